"""The compact derivative on the tensor cores (axes of 40 rows and more):
every scheme and axis against the oracle at the ends of its blocks of 16
outputs, of its tiles of 128 pencils and of its range of lengths, storing and
accumulating; constants and linear functions; pencils that its fixed-point
form does not cover (infinities, NaN, magnitudes near the ends of the FP64
range), alone and beside ordinary ones; and the same bits however a launch
cuts its tiles."""
import numpy as np
import pytest

from emix_gb300 import fields as F
from helpers import assert_close

pytestmark = pytest.mark.gpu

SCHEMES = [F.SCHEME_A, F.SCHEME_B, F.SCHEME_BPER, F.SCHEME_C]


def _field(shape, seed):
    """Smooth waves along each axis and noise of a tenth."""
    z, y, x = (np.linspace(0.0, 1.0, n) for n in shape)
    f = (np.sin(9.0 * x)[None, None, :] * np.cos(7.0 * y)[None, :, None] + np.cos(8.0 * z)[:, None, None])
    return np.ascontiguousarray(f + 0.1 * F.uniform(seed, 1, shape))


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("scheme", SCHEMES)
@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("n, others", [(40, (13, 10)), (47, (1, 128)), (48, (129, 1)), (49, (8, 16)), (63, (127, 9)),
                                       (97, (31, 33)), (112, (64, 80)), (113, (9, 7)), (144, (20, 13)), (145, (7, 11)),
                                       (520, (9, 15)), (4096, (6, 6))])
def test_lengths_and_remainders(emix, oracle, scheme, axis, n, others):
    dims = [max(6, others[0]), max(6, others[1])]
    dims.insert(2 - axis, n)   # (nz, ny, nx)
    f = np.stack([_field(tuple(dims), 3), _field(tuple(dims), 4)])
    h = 1.0 / n if scheme == F.SCHEME_BPER else 1.0 / (n - 1)
    got = emix.deriv_dev(_dev(f), axis, h, scheme).cpu().numpy()
    for c in range(2):
        assert_close(got[c], oracle.deriv3d(scheme, axis, f[c], h), what=f"scheme {scheme} axis {axis} n {n} field {c}")


@pytest.mark.parametrize("scheme", SCHEMES)
@pytest.mark.parametrize("shape", [(41, 53, 64), (80, 45, 50)])
def test_accumulating(emix, oracle, scheme, shape):
    f = [_field(shape, 10 + k) for k in range(6)]
    jbn = F.Grid(shape[2], shape[1], shape[0], (1.3, 0.9, 1.1)).jbn()
    h = tuple(1.0 / (n if scheme == F.SCHEME_BPER else n - 1) for n in shape[::-1])
    rs, rsv = emix.cuDivergence_dev(*[_dev(q) for q in f], _dev(jbn), h, scheme)
    ref, refv = oracle.cuDivergence(scheme, *f, jbn, h)
    assert_close(rs.cpu().numpy(), ref, what="rs")
    assert_close(rsv.cpu().numpy(), refv, what="rsv")


@pytest.mark.parametrize("scheme", SCHEMES)
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_constants_and_linear_functions(emix, scheme, axis):
    n = 72
    const = _dev(np.full((n, n, n), 1.2345))
    assert float(emix.deriv_dev(const, axis, 0.01, scheme).abs().max()) == 0.0
    signed = np.zeros((n, n, n))
    signed[::2, ::3, 1::2] = -0.0
    assert float(emix.deriv_dev(_dev(signed), axis, 0.01, scheme).abs().max()) == 0.0
    if scheme != F.SCHEME_BPER:
        # integer values: differences are exact, the entries' rows sum to 1/h
        ramp = np.arange(n, dtype=np.float64).reshape([n if 2 - axis == a else 1 for a in range(3)]) + np.zeros((n, n, n))
        d = emix.deriv_dev(_dev(ramp), axis, 1.0, scheme).cpu().numpy()
        assert np.max(np.abs(d - 1.0)) <= 2.3e-16


@pytest.mark.parametrize("scheme", [F.SCHEME_B, F.SCHEME_BPER])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_pencils_outside_the_fixed_point_range(emix, oracle, scheme, axis):
    shape = (48, 50, 52)
    n = shape[2 - axis]
    h = 1.0 / n
    f = _field(shape, 5)
    plain = emix.deriv_dev(_dev(f), axis, h, scheme).cpu().numpy()
    g = np.moveaxis(f.copy(), 2 - axis, -1)   # pencils along the last axis
    g[1, 2] *= 1e250
    g[3, 4] *= 1e-250
    g[5, 6, n // 2] = np.nan
    g[7, 8, 3] = np.inf
    g[9, 10] = 0.0
    bad = np.ascontiguousarray(np.moveaxis(g, -1, 2 - axis))
    got = np.moveaxis(emix.deriv_dev(_dev(bad), axis, h, scheme).cpu().numpy(), 2 - axis, -1)
    want = np.moveaxis(plain, 2 - axis, -1)
    odd = [(1, 2), (3, 4), (5, 6), (7, 8), (9, 10)]
    keep = np.ones(g.shape[:2], dtype=bool)
    for p in odd:
        keep[p] = False
    assert np.array_equal(got[keep], want[keep])
    for p in odd[:2]:
        assert_close(got[p], oracle.deriv_pencil(scheme, np.ascontiguousarray(g[p]), h), what=f"pencil {p}")
    assert np.all(np.isnan(got[5, 6]))
    assert not np.any(np.isfinite(got[7, 8]))
    assert np.all(got[9, 10] == 0.0)


@pytest.mark.parametrize("axis", [0, 1, 2])
def test_the_same_bits_however_tiles_are_cut(emix, axis):
    """One field alone (tiles cut into segments) and among others (whole tiles)."""
    f = np.stack([_field((130, 140, 150), 20 + k) for k in range(5)])
    many = emix.deriv_dev(_dev(f), axis, 0.01, F.SCHEME_C).cpu().numpy()
    for k in (0, 4):
        one = emix.deriv_dev(_dev(f[k]), axis, 0.01, F.SCHEME_C).cpu().numpy()
        assert np.array_equal(many[k], one)


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("n, others", [(48, (170, 130)), (64, (170, 130)), (64, (9, 10)), (80, (90, 130))])
def test_short_cyclic_pencils_of_whole_groups(emix, oracle, axis, n, others):
    """Cyclic pencils of whole groups of 16, held at once up to 64 rows: several
    tiles a CTA (and the cut ones), few pencils, and the length above."""
    dims = list(others)
    dims.insert(2 - axis, n)   # (nz, ny, nx)
    f = np.stack([_field(tuple(dims), 7), _field(tuple(dims), 8)])
    got = emix.deriv_dev(_dev(f), axis, 1.0 / n, F.SCHEME_BPER).cpu().numpy()
    for c in range(2):
        assert_close(got[c], oracle.deriv3d(F.SCHEME_BPER, axis, f[c], 1.0 / n), what=f"axis {axis} n {n} field {c}")
