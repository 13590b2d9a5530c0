"""The default force walk (one walk per group of up to 32 bodies) at the
sizes where groups, lists and records have edges, against the CPU oracle's
traversal of the same tree."""
import numpy as np
import pytest

from conftest import same_bits

pytestmark = pytest.mark.gpu


def system(nbx, name, n):
    b = nbx.cold_square(n, 7)
    if name == "coincident":  # half the bodies on one point: a chain of 32 nodes
        b["px"][: n // 2], b["py"][: n // 2] = b["px"][0], b["py"][0]
    if name == "clumps":  # tight pairs far apart: long chains above each pair
        k = n // 2
        b["px"][k:2 * k] = np.nextafter(b["px"][:k], np.float32(1e9))
        b["py"][k:2 * k] = b["py"][:k]
    return b


def term_sums(b, eps):
    """Sum over the other bodies of each body's |term| of the force law."""
    x, y, m = (b[k].astype(np.float64) for k in ("px", "py", "mass"))
    d2 = (x[:, None] - x) ** 2 + (y[:, None] - y) ** 2
    return (m / (d2 + eps * eps)).sum(1)


@pytest.mark.parametrize("name", ["square", "coincident", "clumps"])
@pytest.mark.parametrize("n", [1, 2, 16, 17, 31, 32, 33, 64, 65, 97, 1000])
@pytest.mark.parametrize("leaf,theta", [(16, 1.0), (1, 0.5), (64, 0.5), (3, 2.5), (16, 0.0)])
def test_group_walk(nbx, oracle, name, n, leaf, theta):
    b = system(nbx, name, n)
    try:
        _, _, _, sb, tree = oracle.morton_build(b, leaf)
    except RuntimeError:
        pytest.skip("deeper than the reference's node capacity of 8 n + 8")
    ox, oy = oracle.tree_forces(sb["px"], sb["py"], sb["mass"], tree, theta, 1.0)
    sim = nbx.Simulation(b, theta=theta, leaf_capacity=leaf)
    sim.phase("attract")
    g = sim.download()
    sim.close()
    # n terms of a few rounded operations each, summed in another order: at
    # most (n + 16) half-ulps of the sum of the terms' sizes; a cell's term is
    # at most a few times its bodies' (it lies no nearer than they do, to a
    # factor that theta bounds), hence the 4
    tol = 4.0 * (n + 16) * 2.0 ** -24 * term_sums(sb, 1.0)
    err = np.hypot(g["ax"].astype(np.float64) - ox, g["ay"].astype(np.float64) - oy)
    assert (err <= tol).all(), (err / tol).max()


def test_group_walk_instances(nbx):
    """Instances whose sizes leave ragged groups: the same bits as on their own."""
    sizes = [1, 33, 2, 31, 32, 65, 500, 17]
    bodies = np.concatenate([nbx.cold_square(s, 3 + s) for s in sizes])
    ens = nbx.Handle(sizes, theta=0.5)
    ens.upload(bodies)
    ens.phase("attract")
    got = ens.download()
    ens.close()
    start = 0
    for s in sizes:
        one = nbx.Handle([s], theta=0.5)
        one.upload(bodies[start:start + s])
        one.phase("attract")
        assert same_bits(got[start:start + s], one.download()), s
        one.close()
        start += s


@pytest.mark.parametrize("n", [1, 2, 127, 128, 129, 255, 256, 257, 259, 600])
@pytest.mark.parametrize("eps", [1.0, 1e-19, 1e-20, 0.0])
def test_naive_tiles(nbx, oracle, n, eps):
    """The all-pairs law around its block and tile sizes, with a normal (the
    paired kernel), a subnormal and a zero eps^2 (the checked one), alone and
    as an instance that shares blocks with others."""
    b = nbx.cold_square(n, 5)
    x, y, m = (b[k].astype(np.float64) for k in ("px", "py", "mass"))
    dx, dy = x - x[:, None], y - y[:, None]
    s = dx * dx + dy * dy + float(np.float32(eps)) ** 2
    with np.errstate(divide="ignore", invalid="ignore"):
        f = np.where(dx * dx + dy * dy > 0, m / (s * np.sqrt(s)), 0.0)
    ex, ey = (dx * f).sum(1), (dy * f).sum(1)
    # n terms of about ten rounded operations each: (n + 16) half-ulps of the
    # sum of their sizes
    tol = (n + 16) * 2.0 ** -24 * (np.hypot(dx, dy) * f).sum(1) + 1e-30
    others = nbx.cold_square(70, 9)
    for sizes, bodies, at in (([n], b, 0), ([70, n, 70], np.concatenate([others, b, others]), 70)):
        sim = nbx.Handle(sizes, force_law=1, epsilon=eps)
        sim.upload(bodies)
        sim.phase("attract")
        g = sim.download()[at:at + n]
        sim.close()
        err = np.hypot(g["ax"] - ex, g["ay"] - ey)
        assert (err <= tol).all(), (sizes, (err / tol).max())


@pytest.mark.parametrize("nq", [1, 2, 33, 64, 65, 100, 3000, 20001])
@pytest.mark.parametrize("spread", [1.0, 1e-3, 30.0])
@pytest.mark.parametrize("theta", [1.0, 0.5, 0.2])
def test_points(nbx, nq, spread, theta):
    """Accelerations at points in any order, few and many, close together and
    far outside: the default arithmetic against the reference's (exact_math)."""
    b = nbx.cold_square(3000, 1)
    rng = np.random.default_rng(nq)
    half = 3.0 * np.sqrt(3000.0) * spread
    p = rng.uniform(-half, half, (2, nq)).astype(np.float32)
    p[:, : nq // 3] = p[:, :1]  # many at one place
    sim = nbx.Simulation(b, theta=theta)
    sim.phase("build")
    ax, ay = sim.accel_at(p[0], p[1])
    sim.set_params(exact_math=1)
    ex, ey = sim.accel_at(p[0], p[1])
    sim.close()
    x, y = b["px"].astype(np.float64), b["py"].astype(np.float64)
    terms = np.array([(1.0 / ((x - u) ** 2 + (y - v) ** 2 + 1.0)).sum()
                      for u, v in p.T[:500].astype(np.float64)])
    err = np.hypot(ax - ex.astype(np.float64), ay - ey.astype(np.float64))[:500]
    # as in test_group_walk, 3000 terms at most
    assert (err <= 4.0 * 3016 * 2.0 ** -24 * terms).all()
    if nq > 500:  # the rest: the same bits as the same points alone
        again = nbx.Simulation(b, theta=theta)
        again.phase("build")
        k = rng.choice(nq, 300, replace=False)
        sx, sy = again.accel_at(p[0, k], p[1, k])
        again.close()
        assert same_bits(sx, ax[k]) and same_bits(sy, ay[k])


def test_points_beyond_the_clamp_limit(nbx):
    """Points where squared distances overflow take the clamped law, and a
    NaN point stays NaN without touching its neighbours."""
    b = nbx.cold_square(200, 1)
    sim = nbx.Simulation(b)
    sim.phase("build")
    p = np.array([[1e19, -2e19, 3.0, np.nan, 5.0], [0.0, 1e19, 4.0, 1.0, 6.0]], np.float32)
    ax, ay = sim.accel_at(p[0], p[1])
    sim.set_params(exact_math=1)
    ex, ey = sim.accel_at(p[0], p[1])
    sim.close()
    assert np.isnan(ax[3]) and np.isnan(ex[3])
    k = [0, 1, 2, 4]
    assert np.allclose(ax[k], ex[k], rtol=1e-4, atol=0) and np.allclose(ay[k], ey[k], rtol=1e-4, atol=0)


@pytest.mark.parametrize("sizes", [[1], [16], [17], [300], [4000, 1, 70, 3, 2600], [9000] * 3])
@pytest.mark.parametrize("leaf", [1, 16])
def test_tree_sums(nbx, oracle, sizes, leaf):
    """The tree's sums where nodes stay in a block of 256 records, reach beyond
    it, and share blocks with other instances' (also after an earlier build, whose
    counters must have been left empty): the exact traversal's bits."""
    parts = [nbx.cold_square(s, 2 + k) for k, s in enumerate(sizes)]
    h = nbx.Handle(sizes, theta=0.5, exact_math=1, leaf_capacity=leaf)
    h.upload(np.concatenate(parts))
    for _ in range(2):
        h.phase("attract")
    g = h.download()
    h.close()
    at = 0
    for p in parts:
        _, _, _, sb, tree = oracle.morton_build(p, leaf)
        ox, oy = oracle.tree_forces(sb["px"], sb["py"], sb["mass"], tree, 0.5, 1.0)
        assert same_bits(g["ax"][at:at + len(p)], ox) and same_bits(g["ay"][at:at + len(p)], oy)
        at += len(p)


@pytest.mark.parametrize("nq", [600, 601, 1350, 1351, 5000])
def test_points_around_the_handles_own_room(nbx, nq):
    """300 bodies' staging takes 1350 points on the host and 600 on the device;
    more go through buffers of their own, also after smaller calls: the same
    bits as in calls of 100."""
    b = nbx.cold_square(300, 1)
    p = np.random.default_rng(nq).uniform(-60, 60, (2, nq)).astype(np.float32)
    sim = nbx.Simulation(b)
    sim.phase("build")
    few = [sim.accel_at(p[0, k:k + 100], p[1, k:k + 100]) for k in range(0, nq, 100)]
    for _ in range(2):
        ax, ay = sim.accel_at(p[0], p[1])
        assert same_bits(ax, np.concatenate([f[0] for f in few]))
        assert same_bits(ay, np.concatenate([f[1] for f in few]))
        sim.accel_at(p[0, :50], p[1, :50])
    sim.close()
