"""Goldbach min-p at tile and word edges (the bitmap words of a tile stay in
registers and move on by one word per 64 of p), with and without the array,
against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TILE = 2 * 65536


@pytest.mark.parametrize("N", [7, 63, 64, 130, 4100, 5 + TILE, 6 + TILE, 7 + TILE, 2 * TILE + 64, 3 * TILE - 58,
                               20 * TILE + 31, 10**7 - 1])
def test_goldbach_edges(vg, oracle_lib, N):
    orc = oracle_lib.goldbach_minp(N)
    for want in (True, False):
        mine = vg.conjectures.goldbach_minp(N, want_array=want)
        assert (mine["max"], mine["sum"], mine["counterexamples"]) == (orc["max"], orc["sum"], 0)
        assert np.array_equal(mine["hist"], orc["hist"])
        if want:
            assert np.array_equal(mine["minp"], orc["minp"])
