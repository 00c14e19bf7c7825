"""The first prime of the largest gap where a window has that gap twice: the
earliest counts, also where the earlier one joins two threads' runs and the later
one lies inside the second run."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# windows whose largest gap joins two runs and occurs again inside the next one
TIES = [(114, 230, 199, 12), (206, 410, 293, 14), (39950, 40342, 40039, 24), (15092417, 15092597, 15092513, 20),
        (15415904, 15416196, 15415999, 34), (10764640, 10765818, 10764709, None), (12644079, 12644964, None, 78)]


@pytest.mark.parametrize("a,b,start,gap", TIES)
def test_a_joining_gap_wins_ties(vg, oracle_lib, a, b, start, gap):
    orc = oracle_lib.range_stats(a, b)
    assert start in (None, orc["max_gap_start"]) and gap in (None, orc["max_gap"])
    alone, (batched, _) = vg.range_stats(a, b), vg.range_stats_batch([(a, b), (10**9, 10**9 + 50)])
    for st in (alone, batched):
        assert (st.max_gap, st.max_gap_start) == (orc["max_gap"], orc["max_gap_start"])


def test_random_narrow_windows(vg, oracle_lib):
    rng = np.random.default_rng(11)
    ranges = []
    for _ in range(4000):
        a = int(rng.integers(0, 2 * 10**7))
        ranges.append((a, a + int(rng.integers(60, 1000 if rng.random() < 0.75 else 4000))))
    want = [oracle_lib.range_stats(a, b) for a, b in ranges]
    # one by one, a CTA or a few for each; and in batches, cut where they overlap
    for (a, b), orc in zip(ranges, want):
        st = vg.range_stats(a, b)
        assert (st.max_gap, st.max_gap_start) == (orc["max_gap"], orc["max_gap_start"]), (a, b)
    for i in range(0, len(ranges), 400):
        for (a, b), orc, st in zip(ranges[i:i + 400], want[i:i + 400], vg.range_stats_batch(ranges[i:i + 400])):
            assert (st.max_gap, st.max_gap_start) == (orc["max_gap"], orc["max_gap_start"]), (a, b)
