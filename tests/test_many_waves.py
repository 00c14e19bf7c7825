"""A lone range of more segments than CTAs in one launch: one segment past a
wave, many waves, a last segment of a few bytes, counts alone, gaps of 500 and
more, and runs in turn (each leaves the buffers clean for the next)."""
import pytest

from test_gpu_parity import assert_range_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seg_bytes,threads,segments", [(1024, 1024, 153), (1024, 64, 1025), (4096, 1024, 305),
                                                        (33024, 1024, 200), (222848, 1024, 154)])
def test_waves_vs_oracle(vg, oracle_lib, seg_bytes, threads, segments):
    base = vg.primes.get_config()
    try:
        vg.primes.set_config(seg_bytes=seg_bytes, threads=threads, tier_split=2048, bucket_split=0, auto_tune=0)
        width = 30 * seg_bytes * (segments - 1)
        for a, b in ((0, width + 31), (29, width + 30 * seg_bytes), (10**12 - width, 10**12 + 1)):
            orc = oracle_lib.range_stats(a, b)
            assert_range_equal(vg.range_stats(a, b, full=True), orc, (seg_bytes, a, b))
            if a == 0:
                assert vg.primes.prime_count(b - 1) == orc["count"]
    finally:
        vg.primes.set_config(**base)


def test_large_gaps_and_turns(vg, oracle_lib):
    # 738832927927 + 540 is the first gap of 540, inside; a plan in between
    for a, b in ((738832927927 - 10**9, 738832927927 + 10**9), (0, 3 * 10**9)):
        orc = oracle_lib.range_stats(a, b)
        for _ in range(2):
            assert_range_equal(vg.range_stats(a, b, full=True), orc, (a, b))
            assert [r.count for r in vg.range_stats_batch([(a, b), (5, 100)])] == [orc["count"], 23]
    with vg.Context(4 * 10**9) as ctx:
        assert ctx.large_gaps() == [] and ctx.prime_count() == 189961812
