"""The pencil sweeps with rows by TMA on the axes that take them: y and z under
40 rows (longer axes go to the tensor cores), the cyclic ring and the closed
blocks of 32, 64 and 128 pencils, against the same sweeps with loads, bit for bit;
and that they run at all (copies dropped by the test hook: blocks give up)."""
import numpy as np
import pytest

from emix_gb300 import fields as F

pytestmark = pytest.mark.gpu


def _pair(w, **kw):
    from emix_gb300 import ops
    a = ops.Context(w, **kw)
    b = ops.Context(w, **kw)
    a.set_pencil_tma(True)
    b.set_pencil_tma(False)
    return a, b


# cyclic: at least 2^16 pencils in every y and z launch, a partial last chunk of 4
# rows or none; closed: few pencils, and more than 8 blocks an SM
CASES = [((512, 36, 38), True), ((514, 39, 39), True), ((1024, 25, 32), True),
         ((24, 39, 26), False), ((130, 20, 38), False), ((512, 36, 39), False), ((192, 39, 39), False)]


@pytest.mark.parametrize("dims, periodic", CASES)
def test_rows_by_tma_give_the_same_bits(emix, dims, periodic):
    w = F.random_box(*dims, periodic=periodic)
    timeouts = emix.pencil_tma_timeouts()
    a, b = _pair(w, level_set=False)
    assert a.pencil_tma_launches() == 9 and b.pencil_tma_launches() == 0
    for use_graph in (True, False):
        for c in (a, b):
            c.upload(w.um, w.phi)
            c.step(3, use_graph=use_graph)
        assert np.array_equal(a.download()[0], b.download()[0])
    a.close()
    b.close()
    assert emix.pencil_tma_timeouts() == timeouts


@pytest.mark.parametrize("dims, periodic", [((512, 36, 38), True), ((130, 20, 38), False)])
def test_they_run(emix, dims, periodic):
    import torch
    from emix_gb300 import _lib
    lib = _lib.load()
    w = F.random_box(*dims, periodic=periodic)
    a, b = _pair(w, level_set=False)
    before = emix.pencil_tma_timeouts()
    _lib.check(lib.emix_pencil_tma_test_drop(1), "emix_pencil_tma_test_drop")
    try:
        b.step(1)
        torch.cuda.synchronize()
        assert emix.pencil_tma_timeouts() == before      # no copies there to drop
        a.step(1)
        torch.cuda.synchronize()
    finally:
        _lib.check(lib.emix_pencil_tma_test_drop(0), "emix_pencil_tma_test_drop")
    # per substep the divergence's y and z passes and the gradients' pair, in blocks
    # of 128 pencils at most
    least = 3 * (5 * (w.grid.nx * (w.grid.ny + w.grid.nz)) + 3 * w.grid.nx * (w.grid.ny + w.grid.nz)) // 128
    assert emix.pencil_tma_timeouts() - before >= least
    a.close()
    b.close()
