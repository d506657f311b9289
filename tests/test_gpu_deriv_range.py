"""Pencils whose differences span many orders of magnitude from one place to
another (a bump over a ripple, an exponential, a spike, a shear layer) or are
small against the values (a ripple on an offset): on axes that go to the tensor
cores, every window of 32 rows against a solve in long double, relative to the
window's own largest derivative.

The tensor cores' form is kept for pencils whose windows' largest differences
are within 2^10 of the pencil's largest, and errs by 2^-55.5 of that one at most
(the operator's cut at 40 rows 2^-55.8, its digit products 2^-57): 2^-45.5 of a
window's, 2.0e-14.  A difference of 1 makes a derivative of at least 0.4 / h there
(the operator's largest row entry less its neighbours'), so 5e-14; other pencils
take the sweeps, a few 1e-15.  The tolerance is 1e-13."""
import numpy as np
import pytest

from emix_gb300 import fields as F

pytestmark = pytest.mark.gpu

TOL = 1e-13
LD = np.longdouble


def exact(scheme, f, h):
    """D f of pencils along the last axis, factored and solved in long double (the
    cyclic scheme on three periods with the ends cut: the solution forgets them by
    0.38 a row)."""
    n = f.shape[-1]
    per = scheme == F.SCHEME_BPER
    f = f.astype(LD)
    if per:
        f = np.concatenate([f, f, f], axis=-1)
    m = f.shape[-1]
    one = LD(1)
    al, a, b = (one / 4, 3 * one / 4, 0 * one) if scheme == F.SCHEME_A else (one / 3, 7 * one / 9, one / 36)
    lo, up = np.full(m, al), np.full(m, al)
    r = np.zeros_like(f)
    r[..., 2:-2] = a * (f[..., 3:-1] - f[..., 1:-3]) + b * (f[..., 4:] - f[..., :-4])
    c = [-5 * one / 2, 2 * one, one / 2, 0 * one] if scheme == F.SCHEME_B else \
        [-17 * one / 6, 3 * one / 2, 3 * one / 2, -one / 6]
    a1 = 2 * one if scheme == F.SCHEME_B else 3 * one
    # (the closures' coefficients sum to zero: on differences)
    e = [f[..., k] - f[..., 0] for k in range(4)]
    g = [f[..., m - 1 - k] - f[..., m - 1] for k in range(4)]
    r[..., 0] = sum(c[k] * e[k] for k in range(1, 4))
    r[..., m - 1] = -sum(c[k] * g[k] for k in range(1, 4))
    r[..., 1] = 3 * one / 4 * (f[..., 2] - f[..., 0])
    r[..., m - 2] = 3 * one / 4 * (f[..., m - 1] - f[..., m - 3])
    lo[0], up[0], lo[1], up[1] = 0, a1, one / 4, one / 4
    lo[m - 2], up[m - 2], lo[m - 1], up[m - 1] = one / 4, one / 4, a1, 0
    gam = np.zeros(m, LD)
    bet = one
    r[..., 0] = r[..., 0] / bet
    for i in range(1, m):
        gam[i] = up[i - 1] / bet
        bet = one - lo[i] * gam[i]
        r[..., i] = (r[..., i] - lo[i] * r[..., i - 1]) / bet
    for i in range(m - 2, -1, -1):
        r[..., i] -= gam[i + 1] * r[..., i + 1]
    if per:
        r = r[..., n:2 * n]
    return r / LD(h)


def pencils(n):
    i = np.arange(n, dtype=np.float64)
    x = i / n
    wave = lambda k: np.sin(2 * np.pi * k * x + 0.3)   # periodic
    bump = np.exp(-((x - 0.25) / 0.03) ** 2)
    spike = wave(2).copy()
    spike[20] = 1e12
    wall = 1.0 + 0.02 * wave(2)
    wall[0] = wall[-1] = 0.0
    step = np.where((x > 0.3) & (x < 0.7), 1.0, -1.0) + 1e-9 * wave(5)
    return {
        "waves": wave(1) + 0.3 * wave(4),
        "bump on a ripple of 1e-6": bump + 1e-6 * wave(3),
        "bump on a ripple of 1e-3": bump + 1e-3 * wave(9),
        "ripple of 1e-8 beside an oscillation": np.where(x < 0.5, np.sin(1.3 * i), 0.0) + 1e-8 * wave(3),
        "decay": np.exp(-35.0 * x),
        "steep decay": np.exp(-100.0 * x),
        "gaussian": np.exp(-((x - 0.5) / 0.08) ** 2 / 2),
        "spike of 1e12": spike,
        "walls": wall,
        "shear layers": step,
        "ripple of 1e-9 on 1": 1.0 + 1e-9 * wave(3),
        "ripple on 1e10": 1e10 + wave(4),
        "noise": F.uniform(5, 0, (n,)),
    }


def worst(scheme, got, ref, f, h):
    """Largest error of a window of 32 rows, relative to its largest derivative; in
    the windows at closed ends of the largest value over h too, whose rounding the
    closures' coefficients carry."""
    n = got.shape[-1]
    out = 0.0
    for k in range(0, n - 31, 32):
        w = slice(k, n if n - k < 64 else k + 32)
        den = float(np.max(np.abs(ref[w])))
        if scheme != F.SCHEME_BPER and (k == 0 or n - k < 64):
            den += float(np.max(np.abs(f[w]))) / h * 0.1
        out = max(out, float(np.max(np.abs(got[w] - ref[w]))) / den)
    return out


@pytest.mark.parametrize("scheme", [F.SCHEME_A, F.SCHEME_B, F.SCHEME_BPER, F.SCHEME_C])
@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("n", [64, 128, 256, 301])
def test_every_window_of_a_pencil(emix, scheme, axis, n):
    import torch
    cases = pencils(n)
    if scheme == F.SCHEME_BPER:
        # a jump where the period closes: the sweeps' cyclic correction, which ends
        # where its weights do, leaves 1e-11 of such a tail
        del cases["decay"], cases["steep decay"]
    h = 1.0 / n
    rows = np.stack([cases[k] for k in cases])
    ref = exact(scheme, rows, h)
    # the pencils of each kind among others of all kinds, 12 x 13 of them
    pick = (np.arange(12)[:, None] * 7 + np.arange(13)[None, :]) % len(cases)
    f = np.moveaxis(rows[pick], -1, 2 - axis)
    got = emix.deriv_dev(torch.from_numpy(np.ascontiguousarray(f)).cuda(), axis, h, scheme).cpu().numpy()
    got = np.moveaxis(got, 2 - axis, -1)
    bad = {}
    for k, name in enumerate(cases):
        for g in got[pick == k]:
            e = worst(scheme, g, ref[k], rows[k], h)
            if not e <= TOL:
                bad[name] = max(bad.get(name, 0.0), e)
    assert not bad, bad


@pytest.mark.parametrize("scheme", [F.SCHEME_A, F.SCHEME_B, F.SCHEME_BPER, F.SCHEME_C])
@pytest.mark.parametrize("size, h", [(1e-200, 1e100), (1e200, 1e-100), (1.0, 1e-200), (1.0, 1e200), (1e230, 1e-70)])
def test_results_near_the_ends_of_the_range(emix, scheme, size, h):
    """Values and spacings far from 1: results within the FP64 range come out, in the
    sweeps' accuracy."""
    import torch
    n = 64
    f = size * (pencils(n)["waves"] + 0.1 * F.uniform(7, 0, (n,)))
    x = torch.from_numpy(np.ascontiguousarray(np.broadcast_to(f, (6, 7, n)))).cuda()
    got = emix.deriv_dev(x, 0, h, scheme).cpu().numpy()
    ref = (exact(scheme, (f / size)[None], 1.0)[0] * (LD(size) / LD(h))).astype(np.float64)
    assert np.all(np.isfinite(ref)) and np.all(np.isfinite(got))
    assert np.max(np.abs(got - ref)) <= 1e-13 * np.max(np.abs(ref))
