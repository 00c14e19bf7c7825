"""Bucket lists where the fill can go wrong: two segments, a last segment of a
few bytes, more segments than one item takes, more hits than an item's bins
hold on average, primes whose square lies inside the range, hits in clusters
(primes near the square root of the range)."""
import pytest

from test_gpu_parity import assert_range_equal


@pytest.mark.gpu
@pytest.mark.parametrize("seg_bytes,segments", [(1024, 2), (1024, 161), (1152, 1000), (4096, 160), (65536, 33), (222848, 3)])
def test_bucket_fill_vs_oracle(vg, oracle_lib, seg_bytes, segments):
    base = vg.primes.get_config()
    try:
        vg.primes.set_config(seg_bytes=seg_bytes, threads=1024, tier_split=512, bucket_split=seg_bytes, auto_tune=0)
        width = 30 * seg_bytes * segments
        first = seg_bytes + 12345
        for a, b in ((first**2 - width // 2, first**2 + width // 2 + 61), (10**12 - width, 10**12 + 1),
                     (10**14 + 10**10 - width + 77, 10**14 + 10**10)):
            assert_range_equal(vg.range_stats(a, b, full=True), oracle_lib.range_stats(a, b), (seg_bytes, a, b))
    finally:
        vg.primes.set_config(**base)
