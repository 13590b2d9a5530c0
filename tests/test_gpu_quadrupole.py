"""The force pass with the analytic quadrupole term at the sizes where it walks in
groups: against a CPU walk of the oracle's tree, and with the bits of the walk
that knows no groups."""
import numpy as np
import pytest

from conftest import same_bits

pytestmark = pytest.mark.gpu

F = np.float32


def system(nbx, name, n):
    b = nbx.cold_square(n, 7)
    if name == "coincident":  # half the bodies on one point: a chain of 32 nodes
        b["px"][: n // 2], b["py"][: n // 2] = b["px"][0], b["py"][0]
    if name == "clumps":  # tight pairs far apart: long chains above each pair
        k = n // 2
        b["px"][k:2 * k] = np.nextafter(b["px"][:k], F(1e9))
        b["py"][k:2 * k] = b["py"][:k]
    if name == "cusp":  # groups that do not fit
        r = np.random.default_rng(n)
        a, rad = r.uniform(0, 2 * np.pi, n), 3 * np.sqrt(n) * r.uniform(0, 1, n) ** 5
        b["px"], b["py"] = rad * np.cos(a), rad * np.sin(a)
    return b


def law(d2, m):
    """m * fastInvSqrt(d2) / (d2 + 1) in FP32."""
    g = (np.uint32(0x5f3759df) - (d2.view(np.uint32) >> np.uint32(1))).view(F)
    return m * (g * (F(1.5) - F(0.5) * d2 * g * g)) / (d2 + F(1))


def quadrupole_forces(sb, tree, theta, band):
    """(force, sum of the terms' sizes, sizes of the terms that another rounding of
    d^2 would accept or correct otherwise): FP64 sums, moments and corrections."""
    x, y, m = sb["px"], sb["py"], sb["mass"]
    n = len(x)
    out, size, doubt = np.zeros((n, 2)), np.zeros(n), np.zeros(n)
    f, i = tree.f, tree.i
    t2, b2 = F(theta) * F(theta), F(band) * F(band)

    def correction(k, dx, dy):
        X, Y = np.float64(f["comX"][k]), np.float64(f["comY"][k])
        s = slice(i["start"][k], i["end"][k])
        ux, uy, w = x[s].astype(np.float64) - X, y[s].astype(np.float64) - Y, m[s].astype(float)
        ixx, iyy, ixy = (w * ux * ux).sum(), (w * uy * uy).sum(), (w * ux * uy).sum()
        d2 = dx * dx + dy * dy
        r, q = np.sqrt(d2), d2 + 1.0
        # g(r) = 1 / (r (r^2 + 1)), derivatives in closed form
        g = 1.0 / (r * q)
        g1 = -g * (3 * d2 + 1.0) / (r * q)
        g2 = g * (-6.0 * d2 / (d2 * q) + (3 * d2 + 1.0) * (2.0 / (d2 * q) + 4.0 / q ** 2))
        idx, idy = ixx * dx + ixy * dy, ixy * dx + iyy * dy
        did, tr = dx * idx + dy * idy, ixx + iyy
        a, b = g1 / r, (g2 - g1 / r) / d2
        qx = 0.5 * (a * (2 * idx + tr * dx) + b * dx * did)
        qy = 0.5 * (a * (2 * idy + tr * dy) + b * dy * did)
        mag = 0.5 * (np.abs(a) * 3 * tr * r + np.abs(b) * r * d2 * tr)
        M = max(float(f["mass"][k]), 1e-30)
        return qx / (M * g), qy / (M * g), mag / (M * g)

    stack = [(0, np.arange(n))]
    while stack:
        k, at = stack.pop()
        dx, dy = f["comX"][k] - x[at], f["comY"][k] - y[at]
        d2 = dx * dx + dy * dy
        s2 = f["size"][k] * f["size"][k]
        near = lambda c: np.abs(s2 - d2 * c) <= F(2.0 ** -21) * s2
        accept = s2 < d2 * t2
        if f["mass"][k] > 0 and accept.any():
            j, ex, ey = at[accept], dx[accept].astype(np.float64), dy[accept].astype(np.float64)
            fac = np.abs(law(d2[accept], f["mass"][k]).astype(np.float64))
            qx, qy, mag = correction(k, ex, ey)
            on = (s2 >= d2 * b2)[accept]
            out[j, 0] += fac * np.where(on, ex + qx, ex)
            out[j, 1] += fac * np.where(on, ey + qy, ey)
            whole = fac * (np.hypot(ex, ey) + mag)
            size[j] += whole
            doubt[j] += np.where((near(t2) | near(b2))[accept], 2.0 * whole, 0.0)
        at = at[~accept]
        if len(at) == 0:
            continue
        if i["children"][k] == 0:
            for q in range(i["start"][k], i["end"][k]):
                ex, ey = x[q] - x[at], y[q] - y[at]
                fac = law(ex * ex + ey * ey, m[q]).astype(np.float64)
                out[at, 0] += fac * ex
                out[at, 1] += fac * ey
                size[at] += np.abs(fac) * np.hypot(ex, ey)
        else:
            stack.extend((i["children"][k] + q, at) for q in range(4))
    return out, size, doubt


@pytest.mark.parametrize("name", ["square", "coincident", "clumps"])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 97, 1000])
@pytest.mark.parametrize("leaf", [1, 16])
@pytest.mark.parametrize("theta,band", [(0.65, 0.4), (1.0, 0.01), (0.5, 0.49)])
def test_against_the_oracles_tree(nbx, oracle, name, n, leaf, theta, band):
    b = system(nbx, name, n)
    try:
        _, _, _, sb, tree = oracle.morton_build(b, leaf)
    except RuntimeError:
        pytest.skip("deeper than the reference's node capacity of 8 n + 8")
    want, size, doubt = quadrupole_forces(sb, tree, theta, band)
    h = nbx.Handle([n], theta=theta, leaf_capacity=leaf, use_mlp=2, mlp_band=band)
    h.upload(b)
    h.phase("attract")
    g = h.download()
    h.close()
    # sums of at most n terms, whose moments are sums of at most n, each of a
    # few rounded operations: (2 n + 64) half-ulps of the sum of the terms' sizes
    tol = (2 * n + 64) * 2.0 ** -24 * size + doubt + 1e-30
    err = np.hypot(g["ax"] - want[:, 0], g["ay"] - want[:, 1])
    assert (err <= tol).all(), (err / tol).max()


@pytest.mark.parametrize("name", ["square", "coincident", "clumps", "cusp"])
@pytest.mark.parametrize("n", [1, 33, 1000, 20000, 65535, 65536])
@pytest.mark.parametrize("leaf", [1, 16])
def test_same_bits_beside_more_bodies(nbx, name, n, leaf):
    """Alone (in groups) and as the first instance of more than 65,536 bodies (with a
    cursor per lane)."""
    b = system(nbx, name, n)
    got = []
    for parts in ([b], [b, nbx.cold_square(65537, 2)]):
        h = nbx.Handle([len(p) for p in parts], theta=0.7, use_mlp=2, mlp_band=0.4,
                       leaf_capacity=leaf, collisions=0)
        h.upload(np.concatenate(parts))
        try:
            h.phase("attract")
        except nbx.NbxError as e:
            assert e.code == 3
            pytest.skip("deeper than the node capacity")
        got.append(h.download()[:n])
        h.close()
    assert same_bits(got[0]["ax"], got[1]["ax"]) and same_bits(got[0]["ay"], got[1]["ay"])


@pytest.mark.parametrize("n", [1000, 30000])
def test_forces_from_a_tree_without_moments(nbx, n):
    """The term switched on after a step that built no moments: the same bits in
    groups' range and beyond it, whatever moments an earlier tree left."""
    b = nbx.cold_square(n, 3)
    got = []
    for parts in ([b], [b, nbx.cold_square(65537, 2)]):
        h = nbx.Handle([len(p) for p in parts], theta=0.7, collisions=0, leaf_capacity=1)
        h.upload(np.concatenate(parts))
        h.phase("build")  # moments of another, larger tree
        h.set_params(leaf_capacity=16)
        h.step(1)
        h.set_params(use_mlp=2, mlp_band=0.4)
        h.phase("forces")
        got.append(h.download()[:n])
        h.close()
    assert same_bits(got[0]["ax"], got[1]["ax"]) and same_bits(got[0]["ay"], got[1]["ay"])
