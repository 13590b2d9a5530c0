"""The step's sorts of few bodies (one cluster each) at the edges of their
chunks and of the sizes they take: whole steps, permutations and pair orders
against the CPU oracle, bit for bit."""
import numpy as np
import pytest

from conftest import same_bits

pytestmark = pytest.mark.gpu


def system(nbx, name, n):
    b = nbx.cold_square(n, 11)
    rng = np.random.default_rng(n)
    if name == "moving":  # many contacts with every kind of approach
        b["px"] *= np.float32(0.6)
        b["py"] *= np.float32(0.6)
        b["vx"], b["vy"] = rng.normal(0, 3, (2, n)).astype(np.float32)
    if name == "runs":  # runs of equal high code bits and of equal coarse keys
        k = min(n // 3, 60)  # more overlap than the partner lists hold
        b["px"][:k] = b["px"][0]
        b["py"][:k] = b["py"][0] + rng.uniform(0, 1e-3, k).astype(np.float32)
        b["radius"][:k] = np.float32(1e-4)
    return b


@pytest.mark.parametrize("name", ["moving", "runs"])
@pytest.mark.parametrize("n", [1, 2, 31, 33, 255, 257, 1000, 8191, 8192, 8193, 16385])
def test_steps(nbx, oracle, name, n):
    b = system(nbx, name, n)
    sim = nbx.Simulation(b, exact_math=1)
    sim.step(2)
    assert same_bits(sim.download(), oracle.step(b, steps=2))
    sim.close()


@pytest.mark.parametrize("n", [20479, 20480, 20481, 32769, 39999, 40000, 40001, 65536, 65537])
def test_orders(nbx, oracle, n):
    """Around the largest sizes of each variant: the Morton permutation and
    the pairs in resolution order."""
    b = system(nbx, "moving", n)
    sim = nbx.Simulation(b)
    sim.phase("collide")
    later, earlier = sim.pairs()
    olater, oearlier = oracle.collision_pairs(b)
    assert np.array_equal(later, olater) and np.array_equal(earlier, oearlier)
    moved = sim.download()
    sim.phase("build")
    codes, perm = sim.morton()
    _, ocodes, operm, _, _ = oracle.morton_build(moved)
    assert np.array_equal(codes, ocodes) and np.array_equal(perm, operm)
    sim.close()
