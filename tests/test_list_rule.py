"""Lone ranges on both sides of the rule that chooses bucket lists for them: the
same results by the library's choice, with lists and without, as the oracle has."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

KEYS = ("count", "pi_4_1", "pi_4_3", "pi_3_1", "pi_3_2", "max_gap", "max_gap_start", "num_gaps")


# primes per SM past the split 221184 from 88 000 to 272 000, segments on one SM
# each (5 * 10^7) or shared by two to four
@pytest.mark.parametrize("a,w", [(2 * 10**12, 5 * 10**7), (4 * 10**12, 5 * 10**7), (11 * 10**12, 25 * 10**6 + 1),
                                 (2 * 10**13, 3 * 10**7 - 1), (4 * 10**13 + 7, 25 * 10**6), (7 * 10**13, 16 * 10**6),
                                 (7 * 10**13 + 1, 2 * 10**7), (7 * 10**13, 25 * 10**6), (10**14, 2 * 10**7)])
def test_either_route(vg, oracle_lib, a, w):
    from voss_gb300 import _capi
    from voss_gb300.autotune import TuneEntry, set_table
    lib, n, own = _capi._lib, ctypes.c_uint32(), (TuneEntry * 64)()
    assert lib.voss_gb300_get_tuning(64, own, ctypes.byref(n)) == 0
    own = [tuple(getattr(e, f) for f, _ in TuneEntry._fields_) for e in own[:n.value]]
    orc = oracle_lib.range_stats(a, a + w)
    want = [orc[k] for k in KEYS], [int(x) for x in orc["hist"]]
    try:
        for table in (own, [e[:4] + (0,) for e in own], [(1, 1, 1024, 64, 0)] + own):
            set_table(lib, table)
            st = vg.range_stats(a, a + w, full=True)
            assert ([getattr(st, k) for k in KEYS], st.gap_hist_full) == want
    finally:
        set_table(lib, own)
