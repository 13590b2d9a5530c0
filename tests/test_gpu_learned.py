"""The force pass with the learned correction: which cells it corrects and how
their terms enter the sums, with a network whose outputs are its last biases;
and that a body's sum does not depend on the bodies it shares a warp with."""
import os

import numpy as np
import pytest

from conftest import same_bits

pytestmark = pytest.mark.gpu

F = np.float32
B3 = 1440  # the last layer's biases in the parameter vector
T0, T1 = F(0.25), F(-0.125)


def law(d2, m):
    """m * fastInvSqrt(d2) / (d2 + 1) in FP32."""
    g = (np.uint32(0x5f3759df) - (d2.view(np.uint32) >> np.uint32(1))).view(F)
    return m * (g * (F(1.5) - F(0.5) * d2 * g * g)) / (d2 + F(1))


def constant_forces(sb, tree, theta, band):
    """(force, sum of the terms' sizes, sizes of the terms that another rounding
    of d^2 would accept or correct otherwise), FP64 sums of FP32 terms."""
    x, y, m = sb["px"], sb["py"], sb["mass"]
    n = len(x)
    out, size, doubt = np.zeros((n, 2)), np.zeros(n), np.zeros(n)
    f, i = tree.f, tree.i
    t2, b2 = F(theta) * F(theta), F(band) * F(band)

    def add(at, dx, dy, mass, corrected, margin):
        d2 = dx * dx + dy * dy
        fac = law(d2, mass).astype(np.float64)
        r = np.sqrt(d2.astype(np.float64))
        ux, uy = dx / np.maximum(r, 1e-30), dy / np.maximum(r, 1e-30)
        ex = np.where(corrected, dx * (1.0 + T0) - r * T1 * uy, dx)
        ey = np.where(corrected, dy * (1.0 + T0) + r * T1 * ux, dy)
        out[at, 0] += fac * ex
        out[at, 1] += fac * ey
        size[at] += np.abs(fac) * r * 1.5
        doubt[at] += np.where(margin, np.abs(fac) * r * 3.0, 0.0)

    stack = [(0, np.arange(n))]
    while stack:
        k, at = stack.pop()
        dx, dy = f["comX"][k] - x[at], f["comY"][k] - y[at]
        d2 = dx * dx + dy * dy
        s2 = f["size"][k] * f["size"][k]
        near = lambda c: np.abs(s2 - d2 * c) <= F(2.0 ** -21) * s2
        accept = s2 < d2 * t2
        if f["mass"][k] > 0:
            add(at[accept], dx[accept], dy[accept], f["mass"][k],
                (s2 >= d2 * b2)[accept], (near(t2) | near(b2))[accept])
        at = at[~accept]
        if len(at) == 0:
            continue
        if i["children"][k] == 0:
            for j in range(i["start"][k], i["end"][k]):
                add(at, x[j] - x[at], y[j] - y[at], m[j], False, np.zeros(len(at), bool))
        else:
            stack.extend((i["children"][k] + q, at) for q in range(4))
    return out, size, doubt


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 300, 1000])
@pytest.mark.parametrize("leaf", [1, 16, 64])
@pytest.mark.parametrize("theta,band", [(0.7, 0.5), (0.7, 0.01), (1.0, 0.99)])
def test_corrected_cells(nbx, oracle, n, leaf, theta, band):
    b = nbx.cold_square(n, 3)
    _, _, _, sb, tree = oracle.morton_build(b, leaf)
    want, size, doubt = constant_forces(sb, tree, theta, band)
    w = np.zeros(1442, F)
    w[B3:] = T0, T1
    sim = nbx.Simulation(b, theta=theta, leaf_capacity=leaf, use_mlp=1, mlp_band=band)
    sim.mlp_set_params(w)
    sim.phase("attract")
    g = sim.download()
    sim.close()
    # FP32 sums of at most n terms, each of a few rounded operations, against
    # sums in FP64: (n + 16) half-ulps of the sum of the terms' sizes
    tol = (n + 16) * 2.0 ** -24 * size + doubt + 1e-30
    err = np.hypot(g["ax"] - want[:, 0], g["ay"] - want[:, 1])
    assert (err <= tol).all(), (err / tol).max()


@pytest.mark.parametrize("first", [1, 5, 31, 100])
@pytest.mark.parametrize("n", [33, 700, 3001])
def test_sums_do_not_depend_on_the_warp(nbx, first, n):
    w = np.fromfile(os.path.join(os.path.dirname(nbx.__file__), "weights",
                                 "farfield_mlp.f32"), "<f4")
    a, b = nbx.cold_square(first, 4), nbx.uniform_disc(n, 5)
    got = []
    for parts in ([a, b], [b]):
        h = nbx.Handle([len(p) for p in parts], theta=0.7, use_mlp=1, mlp_band=0.4)
        h.mlp_set_params(w)
        h.upload(np.concatenate(parts))
        h.phase("attract")
        got.append(h.download()[-n:])
        h.close()
    assert same_bits(got[0]["ax"], got[1]["ax"]) and same_bits(got[0]["ay"], got[1]["ay"])


@pytest.mark.parametrize("n", [1, 33, 3001])
@pytest.mark.parametrize("theta,band", [(0.7, 0.7), (0.7, 1.5), (1.0, 1.0)])
def test_a_band_that_no_accepted_cell_reaches(nbx, oracle, n, theta, band):
    b = nbx.cold_square(n, 3)
    _, _, _, sb, tree = oracle.morton_build(b, 16)
    want, size, doubt = constant_forces(sb, tree, theta, band)
    w = np.zeros(1442, F)
    w[B3:] = T0, T1
    sim = nbx.Simulation(b, theta=theta, use_mlp=1, mlp_band=band)
    sim.mlp_set_params(w)
    sim.phase("attract")
    g = sim.download()
    sim.set_params(mlp_band=band * 100)
    sim.phase("attract")
    far = sim.download()
    sim.close()
    # as in test_corrected_cells
    tol = (n + 16) * 2.0 ** -24 * size + doubt + 1e-30
    err = np.hypot(g["ax"] - want[:, 0], g["ay"] - want[:, 1])
    assert (err <= tol).all(), (err / tol).max()
    assert same_bits(far["ax"], g["ax"]) and same_bits(far["ay"], g["ay"])


def test_no_rounds_without_corrections(nbx):
    """With no cell in the band the pass costs no more than a walk (the rounds with
    a few rows took 1.1 times as long as with none)."""
    ms = []
    for band in (0.7, 0.69):
        h = nbx.Handle([1 << 20], theta=0.7, use_mlp=1, mlp_band=band, collisions=0, dt=1e-6)
        h.mlp_set_params(np.zeros(1442, F))
        h.upload(nbx.uniform_disc(1 << 20, 0))
        h.step(2)
        h.sync()
        ms.append(np.median([h.profile_step()["forces"] for _ in range(6)][1:]))
        h.close()
    assert ms[0] < 0.8 * ms[1]
