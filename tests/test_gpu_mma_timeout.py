"""The tensor-core derivatives' bounded waits (finished blocks not signalled, a
test hook): every block gives up, counts itself and stores nothing, the
synchronous calls return EMIX_ERR_TIMEOUT, and the next call is right."""
import numpy as np
import pytest

from emix_gb300 import fields as F
from helpers import assert_close

pytestmark = pytest.mark.gpu

TIMEOUT = 5


@pytest.fixture
def dropped():
    """Blocks go unsignalled while the test is inside `with dropped():`."""
    import contextlib
    import torch
    from emix_gb300 import _lib
    lib = _lib.load()

    @contextlib.contextmanager
    def drop():
        _lib.check(lib.emix_deriv_mma_test_drop(1), "emix_deriv_mma_test_drop")
        try:
            yield
            torch.cuda.synchronize()
        finally:
            _lib.check(lib.emix_deriv_mma_test_drop(0), "emix_deriv_mma_test_drop")
    yield drop


def _raises(call):
    from emix_gb300 import _lib
    with pytest.raises(_lib.EmixError) as e:
        call()
    assert e.value.rc == TIMEOUT


def _fields(n, count):
    return [F.uniform(31, k, (n, n + 1, n + 2)) for k in range(count)]


@pytest.mark.parametrize("scheme", [F.SCHEME_C, F.SCHEME_BPER])
def test_host_calls_report_it(emix, oracle, dropped, scheme):
    f = _fields(48, 6)
    h = tuple(1.0 / n for n in (50, 49, 48))
    jbn = F.Grid(50, 49, 48).jbn()
    vel, temp = np.stack(f[:3]), f[3]
    before = emix.pencil_tma_timeouts()
    with dropped():
        _raises(lambda: emix.cudaDeriv(vel, temp, h, scheme))
        _raises(lambda: emix.cuDivergence(*f, jbn, h, scheme))
    after = emix.pencil_tma_timeouts()
    assert after > before
    dvel, dtemp = emix.cudaDeriv(vel, temp, h, scheme)
    rvel, rtemp = oracle.cudaDeriv(scheme, vel, temp, h)
    assert_close(dvel, rvel, what="dvel")
    assert_close(dtemp, rtemp, what="dtemp")
    rs, rsv = emix.cuDivergence(*f, jbn, h, scheme)
    ref, refv = oracle.cuDivergence(scheme, *f, jbn, h)
    assert_close(rs, ref, what="rs")
    assert_close(rsv, refv, what="rsv")
    assert emix.pencil_tma_timeouts() == after


@pytest.mark.parametrize("axis", [0, 1, 2])
def test_nothing_is_stored(emix, dropped, axis):
    import torch
    from emix_gb300 import _lib
    x = torch.from_numpy(_fields(64, 1)[0]).cuda()
    out = torch.full_like(x, 7.0)
    nz, ny, nx = x.shape
    call = lambda: _lib.check(_lib.load().emix_deriv_dev(F.SCHEME_B, axis, 1, out.data_ptr(), x.data_ptr(), 0.01, nx, ny,
                                                         nz, None), "emix_deriv_dev")
    torch.cuda.synchronize()
    with dropped():
        call()
    assert bool((out == 7.0).all())
    call()
    torch.cuda.synchronize()
    assert torch.equal(out, emix.deriv_dev(x, axis, 0.01, F.SCHEME_B))


def test_the_gradient_and_the_host_step_report_it(emix, dropped):
    w = F.stirred_tank(n=40, nz=20, impeller=True, impeller_omega=1.3)
    r = emix.TankGradient(w, 1, 1, bc_walls=1)
    want = r.run(1.3, 0.1)
    with dropped():
        _raises(lambda: r.run(1.3, 0.1))
    assert r.run(1.3, 0.1) == want
    with dropped():
        _raises(lambda: r.adj.backward())   # recomputes the step
    assert r.run(1.3, 0.1) == want
    r.adj.backward()
    r.close()
    c = emix.Context(w, bc_walls=1)
    um, phi = np.ascontiguousarray(w.um.copy()), np.ascontiguousarray(w.phi.copy())
    with dropped():
        _raises(lambda: c.step_host(um, phi, 1))
    c.close()
