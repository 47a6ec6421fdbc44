"""The first work of a process's backward thread may be a weight gradient alone (a first layer whose
features need no gradient): its tensor map is encoded by the driver, on a host thread that has made no
runtime call.  In a process of its own, as the thread's state outlives a test."""

import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = """
import torch, fvdb
grid = fvdb.GridBatch.from_ijk(torch.randint(0, 24, (4000, 3), device="cuda", dtype=torch.int32))
pack, _ = grid.sparse_conv_kernel_map(3, 1)
x = torch.randn(grid.total_voxels, 24, device="cuda").{dtype}()
w = torch.randn(24, 24, 3, 3, 3, device="cuda").{dtype}().requires_grad_()
held = [torch.empty(1 << s, dtype=torch.uint8, device="cuda") for s in range(8, 27)]
y = pack.sparse_conv_3d(x, w).jdata
dy = torch.ones_like(y)
del held  # the gradient's buffers come from here, without a call to the driver
torch.cuda.synchronize()
(dw,) = torch.autograd.grad(y, w, dy)
m = pack._impl.kmap()[: grid.total_voxels].long()
want = torch.stack([(x.double()[m[:, k].clamp(min=0)] * (m[:, k] >= 0)[:, None]).sum(0) for k in range(27)])
got = dw.double().permute(4, 3, 2, 1, 0).reshape(27, 24, 24)
err = (got - want[:, :, None]).norm() / (want.norm() * 24 ** 0.5)
assert float(err) <= torch.finfo(dw.dtype).eps / 2 + 2e-5, float(err)
"""


@pytest.mark.parametrize("dtype", ["half", "bfloat16"])
def test_weight_gradient_first(dtype):
    env = dict(os.environ, PYTHONPATH=os.path.join(ROOT, "fvdb-core_gb300"))
    r = subprocess.run([sys.executable, "-c", SCRIPT.format(dtype=dtype)], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
