"""The warp-per-prime tier at the edges of its rotation: streams with no step,
one step, fewer steps than the longest skip, one more than 32, and a last
segment of a few bytes."""
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("seg_bytes", [1024, 1152, 4096, 33024, 222848])
@pytest.mark.parametrize("tier_split", [160, 2048, 4600])
def test_small_tier_vs_oracle(vg, oracle_lib, seg_bytes, tier_split):
    base = vg.primes.get_config()
    try:
        vg.primes.set_config(seg_bytes=seg_bytes, threads=1024, tier_split=tier_split, bucket_split=0, auto_tune=0)
        span = 30 * seg_bytes
        for a, b in ((0, 2 * span + 31), (4600**2 - span, 4600**2 + 3), (10**9 + 7, 10**9 + 3 * span),
                     (10**12 - span - 1, 10**12 + 120)):
            st, orc = vg.range_stats(a, b), oracle_lib.range_stats(a, b)
            for k in ("count", "pi_4_1", "pi_4_3", "pi_3_1", "pi_3_2", "max_gap", "max_gap_start", "num_gaps"):
                assert getattr(st, k) == orc[k], (a, b, k)
    finally:
        vg.primes.set_config(**base)
