"""The default force walk where bodies lie unevenly: cusps and concentrated
systems in which groups of 32 bodies do not fit their scratch, and ensembles of
very different instances.  Which route a body takes decides nothing but the
time."""
import numpy as np
import pytest

from conftest import same_bits

pytestmark = pytest.mark.gpu


def system(nbx, name, n):
    b = nbx.cold_square(n, 1)
    r = np.random.default_rng(n)
    a = r.uniform(0, 2 * np.pi, n)
    u = r.uniform(1e-6, 1, n)
    half = 3.0 * np.sqrt(n)
    if name == "cusp":  # density as r^-1.6
        rad = half * u ** 5
    elif name == "plummer":
        rad = np.minimum(0.1 * half / np.sqrt(1.0 / u - 1.0 + 1e-9), 100 * half)
    else:  # two cusps far apart
        rad = half * u ** 5
    b["px"], b["py"] = rad * np.cos(a), rad * np.sin(a)
    if name == "two":
        b["px"][: n // 2] += np.float32(40 * half)
    b["radius"] = 1e-3
    return b


def attract(nbx, parts, **kw):
    h = nbx.Handle([len(p) for p in parts], **kw)
    h.upload(np.concatenate(parts))
    h.phase("attract")
    g = h.download()
    h.phase("forces")  # again from the same tree
    assert same_bits(h.download(), g)
    h.close()
    return g


@pytest.mark.parametrize("name", ["cusp", "plummer", "two"])
@pytest.mark.parametrize("n", [33, 1000, 20000, 32768, 32769, 50000, 100001])
@pytest.mark.parametrize("theta", [0.4, 0.5, 0.7])
def test_sums_do_not_depend_on_the_route(nbx, name, n, theta):
    """The instance alone and behind a larger one that moves it to another
    route, group and warp; and the reference's arithmetic."""
    b = system(nbx, name, n)
    alone = attract(nbx, [b], theta=theta)
    beside = attract(nbx, [nbx.cold_square(40001, 2), b, nbx.cold_square(7, 3)], theta=theta)
    mine = beside[40001:40001 + n]
    assert same_bits(alone["ax"], mine["ax"]) and same_bits(alone["ay"], mine["ay"])
    exact = attract(nbx, [b], theta=theta, exact_math=1)
    k = np.random.default_rng(0).choice(n, min(n, 200), replace=False)
    x, y, m = (exact[f].astype(np.float64) for f in ("px", "py", "mass"))
    terms = np.array([(m / ((x - x[i]) ** 2 + (y - y[i]) ** 2 + 1.0)).sum() for i in k])
    err = np.hypot(alone["ax"].astype(np.float64) - exact["ax"],
                   alone["ay"].astype(np.float64) - exact["ay"])[k]
    # n terms of a few rounded operations each, in two orders
    assert (err <= 4.0 * (n + 16) * 2.0 ** -24 * terms).all()


def force_ms(nbx, parts, **kw):
    h = nbx.Handle([len(p) for p in parts], collisions=0, dt=1e-6, **kw)
    h.upload(np.concatenate(parts))
    h.step(2)
    h.sync()
    ms = [h.profile_step()["forces"] for _ in range(6)]
    h.close()
    return float(np.median(ms[1:]))


@pytest.mark.parametrize("name,n,theta", [("cusp", 10000, 0.5), ("cusp", 100000, 0.75),
                                          ("cusp", 1 << 20, 0.5), ("plummer", 1 << 20, 0.5),
                                          ("plummer", 1 << 22, 0.5)])
def test_groups_that_do_not_fit_cost_little(nbx, name, n, theta):
    """Not much more than the walk that knows no groups (a few per cent in all
    but the smallest; 7 to 34 times as much when each group that did not fit was
    walked piece by piece)."""
    b = [system(nbx, name, n)]
    assert force_ms(nbx, b, theta=theta) < 2.0 * force_ms(nbx, b, theta=theta, leaf_pairs=0)


def test_a_large_instance_among_small_ones(nbx):
    """Whether groups fit is a matter of the instance that holds the bodies."""
    parts = [nbx.uniform_disc(1 << 20, 0)] + [nbx.uniform_disc(1000, k) for k in range(200)]
    assert force_ms(nbx, parts, theta=0.33) < 1.5 * force_ms(nbx, parts, theta=0.33, leaf_pairs=0)


def test_groups_that_do_not_pay(nbx):
    """Short walks of many bodies: a large theta, bodies on a line."""
    n = 1 << 20
    b = nbx.cold_square(n, 1)
    b["px"] = np.random.default_rng(1).uniform(-3e3, 3e3, n)
    b["py"], b["radius"] = 0.0, 1e-3
    assert force_ms(nbx, [b], theta=1.3) < 1.5 * force_ms(nbx, [b], theta=1.3, leaf_pairs=0)


@pytest.mark.parametrize("n,theta", [(40000, 0.5), (300001, 0.5), (300001, 1.0)])
def test_every_kind_of_step(nbx, n, theta):
    """Plain, timed and host-body steps (whose force pass runs in ranges, without the
    step's chain of launches) of a cusp give the same bits."""
    import torch
    b = system(nbx, "cusp", n)
    got = []
    for kind in ("step", "step_timed", "io"):
        h = nbx.Handle([n], theta=theta, collisions=0, dt=1e-4)
        h.upload(b)
        if kind == "io":
            buf = torch.empty((n, 9), dtype=torch.float32, pin_memory=True)
            out = buf.numpy().view(np.uint8).reshape(-1).view(b.dtype)
            out[:] = b
            for _ in range(2):
                h.step_io_ptr(buf.data_ptr(), buf.data_ptr(), n)
            got.append(out.copy())
        else:
            getattr(h, kind)(2)
            got.append(h.download())
        h.close()
    assert same_bits(got[0], got[1]) and same_bits(got[0], got[2])
