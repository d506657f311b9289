"""D^T of the closed schemes on pencils whose values span many orders of
magnitude from one place to another, as the adjoint's fields do away from the
objective: along x against the sweeps along z of the transposed field, every
window of 32 rows relative to the window's own largest value (both are FP64
solves, a few 1e-15 of the rows they couple; 1e-13)."""
import numpy as np
import pytest

from emix_gb300 import fields as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scheme", [F.SCHEME_A, F.SCHEME_B, F.SCHEME_C])
@pytest.mark.parametrize("n", [40, 64, 128, 257])
@pytest.mark.parametrize("accumulate", [False, True])
def test_every_window_of_a_pencil(emix, scheme, n, accumulate):
    import torch
    x = np.arange(n) / n
    rows = np.stack([np.exp(-35.0 * x) * (1.0 + 0.1 * F.uniform(3, 0, (n,))),
                     np.exp(-((x - 0.25) / 0.03) ** 2) + 1e-6 * F.uniform(3, 1, (n,)),
                     np.where(np.arange(n) == 20, 1e12, 1.0) * F.uniform(3, 2, (n,)),
                     F.uniform(3, 3, (n,))])
    y = rows[(np.arange(9)[:, None] + np.arange(10)[None, :]) % 4]           # (9, 10, n)
    y = torch.from_numpy(np.ascontiguousarray(y[None])).cuda()
    h = 1.0 / (n - 1)
    a = b = None
    if accumulate:
        a = 1e-3 * y
        b = a.transpose(1, 3).contiguous()
    got = emix.deriv_t_dev(y, 0, h, scheme, out=a)
    ref = emix.deriv_t_dev(y.transpose(1, 3).contiguous(), 2, h, scheme, out=b)
    got, ref = (a, b) if accumulate else (got, ref)
    got = got.cpu().numpy()[0]
    ref = ref.transpose(1, 3).cpu().numpy()[0]
    for k in range(0, n - 31, 32):
        w = slice(k, n if n - k < 64 else k + 32)
        den = np.abs(ref[..., w]).max(axis=-1)
        assert np.all(np.abs(got[..., w] - ref[..., w]).max(axis=-1) <= 1e-13 * den), (scheme, n, k)
