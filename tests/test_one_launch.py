"""Lone ranges run in one launch where they fit one wave: every split of the
primes over CTAs and every number of segments, against the oracle, and calls of
all kinds one after another (each run leaves the buffers clean for the next)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEYS = ("count", "pi_4_1", "pi_4_3", "pi_3_1", "pi_3_2", "max_gap", "max_gap_start", "num_gaps")


def _check(vg, oracle_lib, a, b):
    st, orc = vg.range_stats(a, b, full=True), oracle_lib.range_stats(a, b)
    for k in KEYS:
        assert getattr(st, k) == orc[k], (a, b, k, getattr(st, k), orc[k])
    assert (st.first_prime, st.last_prime) == (orc["first"], orc["last"]), (a, b)
    assert np.array_equal(np.array(st.gap_hist_full, dtype=np.uint64), orc["hist"]), (a, b)


@pytest.mark.parametrize("a", [0, 3, 3899, 10**8 + 1, 10**10 - 77, 10**12 + 13, 10**13 - 10**6, 10**14 + 10**9])
def test_widths_vs_oracle(vg, oracle_lib, a):
    # one segment shared by many CTAs .. several segments .. one CTA each; the
    # last one at 10^10 and above is the first that may take lists or waves
    for width in (1, 37, 4096, 122881, 491521, 983041, 3 * 10**6 + 1, 10**7, 3 * 10**7 + 7):
        _check(vg, oracle_lib, a, a + width)


@pytest.mark.parametrize("cfg", [dict(seg_bytes=1024, threads=64), dict(seg_bytes=4096, threads=1024),
                                 dict(seg_bytes=16384, threads=96), dict(seg_bytes=222848, threads=1024),
                                 dict(seg_bytes=16384, threads=1024, ctas_per_sm=2)])
def test_configurations_vs_oracle(vg, oracle_lib, cfg):
    base = vg.primes.get_config()
    try:
        vg.primes.set_config(tier_split=512, bucket_split=0, auto_tune=0, **cfg)
        for a, w in ((0, 10**6), (5, 29), (10**6 - 3, 30 * cfg["seg_bytes"] + 1), (10**12 + 7, 5 * 10**5),
                     (4000, 150 * 30 * min(cfg["seg_bytes"], 16384))):
            _check(vg, oracle_lib, a, a + w)
    finally:
        vg.primes.set_config(**base)


def test_calls_in_turn(vg, oracle_lib):
    P = vg.primes
    rng = np.random.default_rng(3)
    for i in range(200):
        a = int(10 ** rng.uniform(0, 14)) - 1
        b = min(a + int(10 ** rng.uniform(0, 6)), 10**14 + 10**10)
        orc = oracle_lib.range_stats(a, b)
        assert vg.range_stats(a, b).count == orc["count"], (a, b)
        if i % 4 == 0 and orc["count"]:
            assert P.next_prime(max(a - 1, 0)) == orc["first"] and P.prev_prime(max(b, 3)) == (orc["last"]), (a, b)
        if i % 20 == 0:
            assert P.prime_count(10**6 + i) == oracle_lib.range_stats(0, 10**6 + i + 1)["count"]
            assert P.in_range(a, min(a + 1000, b)) == oracle_lib.primes_in_range(a, min(a + 1000, b)).tolist()
    # a gap list from the one-launch form (it is empty below 3 * 10^11) and after it
    with vg.Context(10**9) as ctx:
        assert ctx.large_gaps() == [] and ctx.prime_count() == 50847534
