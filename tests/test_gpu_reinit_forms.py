"""The reinitialisation's stage by cells: on the small grids that take it and on
ones just outside, beyond a marching launch's reach in y, and where the marching
form's scratch does not fit, against the oracle (the tolerance of the other
reinitialisation tests)."""
import subprocess
import sys

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
    phi[np.abs(phi) < 0.02] = 0.0        # sign 0: the mean of both Godunov forms
    jbn = np.zeros((11,) + shape)
    for c in (0, 4, 8):
        jbn[c] = 1.0 + 0.05 * F.uniform(seed, 1 + c, shape)
    return np.ascontiguousarray(phi), jbn


# blocks of 16 x 16 columns by planes: 504, 480 and 160 (by cells); 608 (too many cells),
# 450 and 612 (not)
@pytest.mark.parametrize("shape", [(42, 50, 37), (30, 50, 49), (40, 30, 30), (38, 49, 49), (25, 43, 81), (51, 48, 50)])
@pytest.mark.parametrize("ref_bugs", [0, 1])
def test_small_grids(emix, oracle, shape, ref_bugs):
    phi, jbn = _level_set(shape, 6)
    h = tuple(1.0 / (n - 1) for n in shape[::-1])
    dm = np.full(shape, min(h))
    ref = oracle.reinit(phi, jbn, dm, h, 5, min(h), iters=2, ref_bugs=ref_bugs)
    got = emix.reinit_dev(_dev(phi), _dev(jbn), _dev(dm), h, 5, min(h), iters=2, ref_bugs=ref_bugs)
    assert_close(got.cpu().numpy(), ref, what=f"reinit {shape}")


def test_beyond_a_marching_launch_in_y(emix, oracle):
    shape = (4, 16 * 65535 + 5, 4)
    phi = np.ascontiguousarray(F.uniform(7, 0, shape))
    jbn = np.ones((11,) + shape)
    dm = np.full(shape, 0.5)
    ref = oracle.reinit(phi, jbn, dm, (1.0, 1.0, 1.0), 0, 0.5, iters=1)
    got = emix.reinit_dev(_dev(phi), _dev(jbn), _dev(dm), (1.0, 1.0, 1.0), 0, 0.5, iters=1)
    assert_close(got.cpu().numpy(), ref, what="reinit")


SCRIPT = """
import sys
sys.path[:0] = [{root!r}, {root!r} + "/tests"]
import numpy as np, torch
from emix_gb300 import ops
from test_gpu_reinit_forms import _level_set, _dev
from helpers import assert_close
shape = (150, 150, 150)                                  # a field: 27 MB
phi, jbn = _level_set(shape, 8)
h = tuple(1.0 / (n - 1) for n in shape)
args = [_dev(jbn), _dev(np.full(shape, h[0]))]
small, full = _dev(phi), _dev(phi)
torch.cuda.synchronize()
hog = torch.empty(torch.cuda.mem_get_info()[0] - 160 * 2 ** 20, dtype=torch.uint8, device="cuda")
ops.reinit_dev(small, *args, h, 5, h[0], iters=2)        # 243 MB would be nine fields
torch.cuda.synchronize()
del hog
torch.cuda.empty_cache()
ops.reinit_dev(full, *args, h, 5, h[0], iters=2)
torch.cuda.synchronize()
assert not torch.equal(small, full)                      # the other form, to rounding
assert_close(small.cpu().numpy(), full.cpu().numpy())
print("done")
"""


def test_where_the_scratch_does_not_fit(emix):
    from conftest import ROOT
    p = subprocess.run([sys.executable, "-c", SCRIPT.format(root=str(ROOT))], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0 and "done" in p.stdout, p.stdout + p.stderr
