"""A batch of more grids than SMs whose derivatives go to the tensor cores: each
item of a launch is one CTA's work, and the launch has more CTAs than the GPU SMs;
against the per-grid steps (1e-13 as for the other batched kernels)."""
import pytest

from emix_gb300 import fields as F
from helpers import assert_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("periodic", [False, True])
def test_more_items_than_sms(emix, periodic):
    import torch
    count = torch.cuda.get_device_properties(0).multi_processor_count + 8
    # x: one item a grid; y and z: one launch of two
    b = emix.Batch([F.random_box(40 + k % 3, 41, 40, seed=9 + k % 5, periodic=periodic) for k in range(count)])
    b.step_per_grid(1)
    ref = [b.download(g) for g in range(count)]
    b.upload()
    b.step(1, use_graph=False)
    for g in range(count):
        um, phi = b.download(g)
        assert_close(um, ref[g][0], tol=1e-13, what=f"grid {g} um")
        assert_close(phi, ref[g][1], tol=1e-13, what=f"grid {g} phi")
    b.close()
