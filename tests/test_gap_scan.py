"""The gap scan at its edges, against the oracle: windows of a few wheel bytes
(the largest gap may lie inside a byte), word and run ends, gaps beyond the
shared histogram, and requests that follow one another in a CTA (the byte and
gap histograms are flushed between them)."""
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


@pytest.mark.parametrize("a", [0, 7, 30, 89, 113, 1327, 30 * 1024 - 7, 10**6 + 1, 10**9 - 9])
def test_small_windows(vg, oracle_lib, a):
    for width in (1, 2, 6, 14, 29, 30, 31, 59, 60, 61, 119, 120, 121, 240, 599, 3840, 3841, 30 * 4096, 30 * 4097 + 1):
        _check(vg, oracle_lib, a, a + width)


@pytest.mark.parametrize("end", [304599508537, 416608695821, 738832928467, 100000305501563])
def test_gaps_beyond_the_shared_bins(vg, oracle_lib, end):
    # gaps of 514, 532, 540 and 550 that end here
    for a, b in ((end - 10**5, end + 10**5), (end - 700, end + 1), (end - 3 * 10**7, end + 10**6), (end - 700, end)):
        _check(vg, oracle_lib, a, b)


def test_requests_in_turn(vg, oracle_lib):
    rng = np.random.default_rng(5)
    ranges = []
    for _ in range(600):                       # disjoint, so each is a request of its own
        a = int(rng.integers(0, 10**11))
        ranges.append((a, a + int(10 ** rng.uniform(0, 5.5))))
    for (a, b), st in zip(ranges, vg.range_stats_batch(ranges)):
        orc = oracle_lib.range_stats(a, b)
        for k in KEYS:
            assert getattr(st, k) == orc[k], (a, b, k)
        assert st.gap_hist[:201] == [int(x) for x in orc["hist"][:201]], (a, b)
