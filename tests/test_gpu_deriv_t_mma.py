"""D^T of the closed schemes on the tensor cores (x pencils of 40 rows and
more): against the sweeps along z of the transposed field (their lengths at the
edges of blocks, end types and tiles; both agree with a dense transpose to a few
1e-15, so to 1e-13), storing and accumulating, with pencils outside the
fixed-point range; and the reverse sweep of a tank whose axes all use it (y and
z too) against a directional difference."""
import numpy as np
import pytest

from emix_gb300 import fields as F
from helpers import assert_close

pytestmark = pytest.mark.gpu

CLOSED = [F.SCHEME_A, F.SCHEME_B, F.SCHEME_C]


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _both(emix, y, scheme, out=None):
    """D^T along x by both kernels (the second along z of the transposed field)."""
    h = 1.0 / (y.shape[-1] - 1)
    t = None if out is None else out.transpose(1, 3).contiguous()
    o = None if out is None else out.clone()
    a = emix.deriv_t_dev(y, 0, h, scheme, out=o)
    b = emix.deriv_t_dev(y.transpose(1, 3).contiguous(), 2, h, scheme, out=t)
    a, b = (a, b) if out is None else (o, t)
    return a.cpu().numpy(), b.transpose(1, 3).contiguous().cpu().numpy()


@pytest.mark.parametrize("scheme", CLOSED)
@pytest.mark.parametrize("n, others", [(40, (13, 10)), (47, (6, 130)), (48, (129, 6)), (96, (8, 16)), (97, (31, 33)),
                                       (112, (9, 7)), (145, (140, 150))])
def test_lengths(emix, scheme, n, others):
    y = _dev(F.uniform(61, n, (2,) + others + (n,)))
    x = _dev(F.uniform(62, n, (2,) + others + (n,)))
    a, b = _both(emix, y, scheme)
    assert_close(a, b, tol=1e-13, what="store")
    a, b = _both(emix, y, scheme, out=x)
    assert_close(a, b, tol=1e-13, what="accumulate")


@pytest.mark.parametrize("scheme", CLOSED)
def test_pencils_outside_the_fixed_point_range(emix, scheme):
    y = F.uniform(63, 1, (1, 9, 20, 56))
    want, _ = _both(emix, _dev(y), scheme)
    y[0, 2, 3, 17] = np.inf
    y[0, 4, 5, 50] = np.nan
    y[0, 6, 7] *= 1e-290
    y[0, 8, 9] = 0.0
    a, b = _both(emix, _dev(y), scheme)
    for k, j in ((2, 3), (4, 5)):
        assert np.array_equal(np.isnan(a[0, k, j]), np.isnan(b[0, k, j]))
    assert_close(a[0, 6, 7] * 1e290, b[0, 6, 7] * 1e290, tol=1e-13, what="tiny")
    assert np.all(a[0, 8, 9] == 0.0)
    plain = np.ones((9, 20), bool)
    for k, j in ((2, 3), (4, 5), (6, 7), (8, 9)):
        plain[k, j] = False
    assert np.array_equal(a[0][plain], want[0][plain])   # the others do not notice


def test_reverse_sweep_of_a_tank(emix):
    """44 rows an axis; steps and tolerance of the same test on 18."""
    w = F.stirred_tank(n=44, impeller=True, impeller_omega=1.3, height=2.0)
    X, Y, Z = w.grid.coords()
    w.phi = np.ascontiguousarray(Z - 1.0 + 0.05 * np.sin(3 * X) * np.cos(2 * Y))
    r = emix.TankGradient(w, 2, 1, bc_walls=1)
    r.run(1.3, 0.1)
    r.adj.backward()
    lum = r.adj.state_gradient()[0].cpu().numpy()
    um0 = w.um.copy()
    du = np.stack([1e-2 * F.uniform(93, m, w.phi.shape) for m in range(5)])
    du *= np.abs(um0).max(axis=(1, 2, 3))[:, None, None, None]
    vals = []
    for eps in (1e-4, -1e-4):
        w.um = np.ascontiguousarray(um0 + eps * du)
        vals.append(r.run(1.3, 0.1))
    pred, fd = float((lum * du).sum()), (vals[0] - vals[1]) / 2e-4
    assert pred != 0.0
    assert abs(pred - fd) <= 1e-6 * abs(fd), (pred, fd)
    w.um = um0
    r.close()
