"""The radix sort's look-back at the edges of its tiles (3072 keys) and groups of
16 tiles: Morton permutations against a stable sort of the oracle's codes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GROUP = 16 * 3072


@pytest.mark.parametrize("n", [GROUP - 3072, GROUP, GROUP + 1, 2 * GROUP, 2 * GROUP + 3073,
                               17 * GROUP, 17 * GROUP + 1, 18 * GROUP - 1])
def test_permutation(nbx, oracle, n):
    b = nbx.cold_square(n, 6)
    k = n // 2  # a run of one code longer than several tiles
    b["px"][k:k + 10000], b["py"][k:k + 10000] = b["px"][0], b["py"][0]
    sim = nbx.Simulation(b, collisions=0)
    sim.phase("build")
    codes, perm = sim.morton()
    sim.close()
    want = oracle.morton(b["px"], b["py"], oracle.root_square(b["px"], b["py"]))
    order = np.argsort(want, kind="stable")  # codes stay in the bodies' order
    assert np.array_equal(codes, want) and np.array_equal(perm, order)
