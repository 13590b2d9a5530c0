"""Partner lists at the lengths where the passes that make them change over,
and buckets that cells share: the pairs in resolution order and the resolved
bodies against the CPU oracle, bit for bit."""
import numpy as np
import pytest

from conftest import same_bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ties", [False, True])
@pytest.mark.parametrize("count", [2, 3, 4, 5, 6, 7, 16, 17, 18, 24])
def test_clumps(nbx, oracle, ties, count):
    """Clumps of `count` bodies that all touch (lists of count - 1), some of them
    at one x, among bodies that touch nobody."""
    rng = np.random.default_rng(count)
    b = nbx.cold_square(3000, 9)
    b["px"] *= np.float32(50)
    b["py"] *= np.float32(50)
    for c in range(9):
        k = slice(c * count, (c + 1) * count)
        r = b["radius"][k].min()
        b["px"][k] = b["px"][c * count] + r * rng.uniform(-0.4, 0.4, count).astype(np.float32)
        b["py"][k] = b["py"][c * count] + r * rng.uniform(-0.4, 0.4, count).astype(np.float32)
        if ties:
            b["px"][k][1::2] = b["px"][c * count]
            b["radius"][k] = r
    b["vx"], b["vy"] = rng.normal(0, 1, (2, len(b))).astype(np.float32)
    sim = nbx.Simulation(b)
    sim.phase("collide")
    later, earlier = sim.pairs()
    olater, oearlier = oracle.collision_pairs(b)
    assert len(olater) >= 9 * count * (count - 1) // 2
    assert np.array_equal(later, olater) and np.array_equal(earlier, oearlier)
    ref, _ = oracle.collide(b)
    assert same_bits(sim.download(), ref)
    sim.close()
