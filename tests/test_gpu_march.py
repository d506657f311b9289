"""The z-marching kernels (level-set stage, reinitialisation) at the ends of
their 16 x 16 columns and with chunks of one plane up to all of them, and the
small grids' one-launch gradients at the ends of their one-warp blocks,
against the oracle."""
import numpy as np
import pytest

from emix_gb300 import fields as F
from helpers import assert_close

pytestmark = pytest.mark.gpu


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _level_set(shape, seed):
    z, y, x = np.meshgrid(*(np.linspace(0, 1, n) for n in shape), indexing="ij")
    d = np.sqrt((x - 0.5) ** 2 + (y - 0.45) ** 2 + (z - 0.55) ** 2) - 0.25
    phi = d * (1.0 + 0.3 * np.sin(5 * x)) + 1e-3 * F.uniform(seed, 0, shape)
    jbn = np.zeros((11,) + shape)
    for c in (0, 4, 8):
        jbn[c] = 1.0 + 0.05 * F.uniform(seed, 1 + c, shape)
    return np.ascontiguousarray(phi), jbn


SHAPES = [(11, 16, 17), (12, 33, 16), (48, 15, 32), (200, 11, 13), (19, 49, 70)]


# (the reinitialisation mirrors 5 ghost layers of an interior at least as deep)
@pytest.mark.parametrize("shape", [(15, 16, 17), (16, 33, 16), (48, 15, 32), (200, 15, 16), (19, 49, 70)])
@pytest.mark.parametrize("zero_band", [False, True])
def test_reinit_columns_and_chunks(emix, oracle, shape, zero_band):
    phi, jbn = _level_set(shape, 2)
    if zero_band:
        phi[np.abs(phi) < 0.05] = 0.0    # sign 0: the mean of both Godunov forms
    h = tuple(1.0 / (n - 1) for n in shape[::-1])
    dm = np.full(shape, min(h))
    ref = oracle.reinit(phi, jbn, dm, h, 5, min(h), iters=2)
    got = emix.reinit_dev(_dev(phi), _dev(jbn), _dev(dm), h, 5, min(h), iters=2)
    assert_close(got.cpu().numpy(), ref, what=f"reinit {shape}")


@pytest.mark.parametrize("shape", SHAPES)
def test_advection_columns_and_chunks(emix, oracle, shape):
    phi, jbn = _level_set(shape, 3)
    vel = np.stack([F.uniform(4, c, shape) for c in range(3)])
    h = tuple(1.0 / (n - 1) for n in shape[::-1])
    dt = 0.2 * min(h)
    ref = oracle.weno_advect(phi, vel, jbn, h, dt)
    got = emix.weno5_advect_dev(_dev(phi), _dev(vel), _dev(jbn), h, dt)
    assert_close(got.cpu().numpy(), ref, what=f"advection {shape}")


@pytest.mark.parametrize("scheme", [F.SCHEME_A, F.SCHEME_B, F.SCHEME_BPER, F.SCHEME_C])
@pytest.mark.parametrize("shape", [(6, 6, 6), (39, 7, 33), (8, 39, 32), (31, 9, 39)])
def test_small_gradients_in_one_launch(emix, oracle, scheme, shape):
    vel = np.stack([F.uniform(5, c, shape) for c in range(3)])
    temp = F.uniform(5, 3, shape)
    h = tuple(1.0 / (n if scheme == F.SCHEME_BPER else n - 1) for n in shape[::-1])
    dvel, dtemp = emix.cudaDeriv_dev(_dev(vel), _dev(temp), h, scheme)
    rvel, rtemp = oracle.cudaDeriv(scheme, vel, temp, h)
    for c in range(9):
        assert_close(dvel[c].cpu().numpy(), rvel[c], what=f"dvel[{c}]")
    for c in range(3):
        assert_close(dtemp[c].cpu().numpy(), rtemp[c], what=f"dtemp[{c}]")
    alone, none = emix.cudaDeriv_dev(_dev(vel), None, h, scheme)
    assert none is None and np.array_equal(alone.cpu().numpy(), dvel.cpu().numpy())
