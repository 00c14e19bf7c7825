"""The synchronous calls that read a wheel bitmap keep their buffers between
calls: results do not depend on what ran before, in sizes up and down, after an
error and after a configuration change."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_kept_buffers_in_any_order(vg, oracle_lib):
    P = vg.primes
    def listed(a, b):
        assert P.in_range(a, b) == oracle_lib.primes_in_range(a, b).tolist(), (a, b)
    def goldbach(N):
        mine, orc = vg.conjectures.goldbach_minp(N), oracle_lib.goldbach_minp(N)
        assert np.array_equal(mine["minp"], orc["minp"]) and np.array_equal(mine["hist"], orc["hist"]), N
        assert vg.conjectures.goldbach_minp(N, want_array=False)["sum"] == orc["sum"], N
    def sophie(N, want):
        with vg.Context(N) as ctx:
            assert ctx.sophie_germain() == want, N
    goldbach(300001)
    listed(0, 10)
    listed(10**9, 10**9 + 4 * 10**6)
    goldbach(10**4)
    sophie(1000, 37)
    listed(7, 7)
    listed(8, 10)
    goldbach(3 * 10**6 + 1)
    with pytest.raises(vg.VossError):
        P.in_range_with_limit(0, 10**6, 1000)         # counted first
    with pytest.raises(vg.VossError):
        P.in_range_with_limit(10**6, 10**6 + 10**5, 7000)     # counted with the bitmap (7216 primes)
    assert len(P.in_range_with_limit(10**6, 10**6 + 10**5, 7216)) == 7216
    listed(2, 6)
    base = P.get_config()
    try:
        P.set_config(seg_bytes=16384, auto_tune=0)
        goldbach(3 * 10**6 + 1)
        listed(10**12, 10**12 + 10**6)
    finally:
        P.set_config(**base)
    sophie(30, 6)
    goldbach(6)


@pytest.mark.parametrize("a,b", [(2, 2), (2, 7), (0, 29), (7, 31), (10**6 - 17, 10**6 + 1), (10**12, 10**12 + 3),
                                 (10**9, 10**9 + 30 * 4 * 4096 - 1), (10**9, 10**9 + 30 * 4 * 4096),
                                 (10**11 + 1, 10**11 + 30 * 4 * 4096 * 3 + 7), (0, 10**6), (10**13 - 5, 10**13 + 10**6)])
def test_lists_at_block_edges(vg, oracle_lib, a, b):
    # one extraction block holds 4096 words of 120 integers
    want = oracle_lib.primes_in_range(a, b).tolist()
    assert vg.primes.in_range(a, b) == want
    if want:
        assert vg.primes.in_range_with_limit(a, b, len(want)) == want
        if len(want) > 1:
            with pytest.raises(vg.VossError):
                vg.primes.in_range_with_limit(a, b, len(want) - 1)
