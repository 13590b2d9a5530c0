"""After a bounded device wait has given up: what it leaves behind stays in
bounds and spoils no later call."""
import numpy as np
import pytest

from conftest import same_bits

pytestmark = pytest.mark.gpu

TIMEOUT = 5


def expire(nbx, h):
    h._c(nbx.lib().nbx_debug_expire_wait(h.h))
    with pytest.raises(nbx.NbxError) as e:
        h.sync()
    assert e.value.code == TIMEOUT


@pytest.mark.parametrize("sizes", [[20], [300], [5000], [300, 1, 700]])
def test_records_that_lead_nowhere(nbx, sizes):
    """Children that every body opens, with links far beyond the records: the
    group walk gives up within its scratch and the cursor walk, whose records are
    whole, gives every body its sum."""
    b = np.concatenate([nbx.cold_square(n, 1) for n in sizes])
    b["px"] *= np.float32(1e-13)  # the records' children are then far too near
    b["py"] *= np.float32(1e-13)
    h = nbx.Handle(sizes, collisions=0)
    h.upload(b)
    h.phase("attract")
    want = h.download()
    expire(nbx, h)
    h.phase("forces")
    got = h.download()
    h.close()
    assert np.isfinite(got["ax"]).all() and same_bits(got, want)


@pytest.mark.parametrize("sizes", [[3000], [100001], [9000, 1, 20000]])
@pytest.mark.parametrize("form", [{}, {"use_mlp": 2, "mlp_band": 0.4, "theta": 0.7}])
def test_remainders_of_a_tree(nbx, sizes, form):
    """Arrivals that an unsorted build left at nodes it never completed: later builds
    of the same handle start from nothing, with the bodies it has and with others."""
    b = np.concatenate([nbx.cold_square(n, 1) for n in sizes])
    fresh = []
    for bodies in (b, b[::-1].copy()):
        h = nbx.Handle(sizes, collisions=0, **form)
        h.upload(bodies)
        h.step(3)
        fresh.append(h.download())
        h.close()
    h = nbx.Handle(sizes, collisions=0, **form)
    h.upload(b)
    h.step(1)
    h.sync()
    expire(nbx, h)
    h.step(2)
    assert same_bits(h.download(), fresh[0])
    expire(nbx, h)
    h.upload(b[::-1].copy())
    h.step(3)
    assert same_bits(h.download(), fresh[1])
    h.close()


@pytest.mark.parametrize("nq", [1, 64, 65, 600, 601, 5000])
def test_points_after_an_expired_wait(nbx, nq):
    """Accelerations at points that were sorted (more than 64) are not handed out as
    good when a wait gave up; of fewer the status stays for the next call that
    reports it.  All are good again after the next build."""
    b = nbx.cold_square(300, 1)
    p = np.random.default_rng(nq).uniform(-60, 60, (2, nq)).astype(np.float32)
    h = nbx.Handle([300])
    h.upload(b)
    h.phase("build")
    want = h.accel_at(p[0], p[1])
    h._c(nbx.lib().nbx_debug_expire_wait(h.h))
    with pytest.raises(nbx.NbxError) as e:
        h.accel_at(p[0], p[1])
        assert nq <= 64
        h.sync()
    assert e.value.code == TIMEOUT
    h.upload(b)
    h.phase("build")
    assert all(same_bits(a, w) for a, w in zip(h.accel_at(p[0], p[1]), want))
    h.close()
