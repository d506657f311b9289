"""Batched grids whose derivatives go to the tensor cores (axes of 40 rows and
more) next to grids and axes that do not, closed and cyclic in one batch, and
more grids than SMs: one batched step against the per-grid steps, to rounding
(the compiler may contract multiply-adds differently in the batched kernels:
1e-13 as for the other batched kernels)."""
import numpy as np
import pytest

from emix_gb300 import fields as F
from helpers import assert_close

pytestmark = pytest.mark.gpu

# (nx, ny, nz, cyclic): edges of the 40-row rule, of 16-row blocks and of
# 128-pencil tiles; an axis of 33 or 39 keeps the sweeps
SETS = {
    "mixed": [(40, 33, 47, False), (48, 40, 64, True), (39, 38, 36, False), (65, 41, 40, False), (32, 96, 56, True)],
    "one": [(56, 43, 81, True)],
    "sweeps": [(33, 24, 39, False), (32, 36, 28, True)],
    "many": [(40, 41, 42, bool(k & 1)) for k in range(80)],
}


@pytest.mark.parametrize("name", list(SETS))
@pytest.mark.parametrize("use_graph", [False, True])
def test_batched_tensor_core_derivatives(emix, name, use_graph):
    n0 = emix.pencil_tma_timeouts()
    b = emix.Batch([F.random_box(x, y, z, seed=5 + k, periodic=per) for k, (x, y, z, per) in enumerate(SETS[name])])
    count = len(SETS[name])
    b.step_per_grid(2)
    ref = [b.download(g) for g in range(count)]
    for overlap in ((3,) if name == "many" else (0, 3)):
        b.upload()
        b.set_overlap(overlap)
        b.step(2, use_graph=use_graph)
        for g in range(count):
            um, phi = b.download(g)
            assert np.isfinite(um).all()
            assert_close(um, ref[g][0], tol=1e-13, what=f"grid {g} um, overlap {overlap}")
            assert_close(phi, ref[g][1], tol=1e-13, what=f"grid {g} phi, overlap {overlap}")
    b.close()
    assert emix.pencil_tma_timeouts() == n0
