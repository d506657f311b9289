"""Large grids (2^21 cells and more) whose derivatives on the tensor cores are gated:
a sample of a step's pencils decides between them and the sweeps.  The decision
is seen by the tensor cores' test hook (their blocks then give up and are
counted), the values against a batch of the one grid, which is not gated."""
import numpy as np
import pytest

from emix_gb300 import fields as F

pytestmark = pytest.mark.gpu

SIZES = [(128, 128, 128), (161, 96, 137), (2048, 40, 26)]


def _state(dims, periodic, kind):
    """loud: waves and noise.  quiet: a bump of 1 over ripples of 1e-6 in every pencil
    of u, v and w.  half: the same and noise in every other pencil along x, so that
    pencils along y and z have it in every other row."""
    w = F.random_box(*dims, periodic=periodic)
    if kind != "loud":
        x = [np.arange(m) / m for m in dims]
        e = [np.exp(-((c - 0.3) / 0.04) ** 2) + 1e-6 * np.sin(2 * np.pi * 3 * c) for c in x]
        u = e[2][:, None, None] + e[1][None, :, None] + e[0][None, None, :]
        w.um[0] = 1.0
        w.um[1:4] = 0.05 * u
        w.um[4] = 1.0
        if kind == "half":
            odd = (np.arange(dims[2])[:, None] + np.arange(dims[1])[None, :]) % 2
            w.um[1:4] += 0.01 * odd[..., None] * F.uniform(3, 0, (3,) + u.shape)
    return w


def _gave_up(emix, ctx):
    import torch
    from emix_gb300 import _lib
    lib = _lib.load()
    before = emix.pencil_tma_timeouts()
    _lib.check(lib.emix_deriv_mma_test_drop(1), "emix_deriv_mma_test_drop")
    try:
        ctx.step(1)
        torch.cuda.synchronize()
    finally:
        _lib.check(lib.emix_deriv_mma_test_drop(0), "emix_deriv_mma_test_drop")
    return emix.pencil_tma_timeouts() - before


@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("kind", ["loud", "quiet", "half"])
@pytest.mark.parametrize("dims", SIZES)
def test_values_and_forms(emix, dims, periodic, kind):
    w = _state(dims, periodic, kind)
    b = emix.Batch([w], level_set=False)
    b.upload()
    b.step(2)
    ref = b.download(0)[0]
    b.close()
    out = []
    for fused, graph in ((True, True), (True, False), (False, False)):
        c = emix.Context(w, level_set=False)
        c.set_fusion(fused)
        c.step(2, use_graph=graph)
        out.append(c.download()[0])
        c.close()
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])
    # both forms' derivatives are within a few 1e-15 of a field's largest
    for m in range(5):
        assert np.max(np.abs(out[0][m] - ref[m])) <= 1e-12 * np.max(np.abs(ref[m]))


def test_the_sample_decides(emix):
    """Blocks that give up in a step of 18 launches.  Noise everywhere: those of every
    launch.  Half of the pencils along x quiet somewhere: not those of the x gradients,
    three launches that do not start (ungated they would: every tile has the other
    half's pencils)."""
    count = {}
    for kind in ("loud", "half"):
        c = emix.Context(_state((128, 128, 128), False, kind), level_set=False)
        count[kind] = _gave_up(emix, c)
        c.close()
    assert count["loud"] > 0 and count["half"] <= count["loud"] * 15 // 18
