"""FP32 / FP64 contractions whose tiles stage their map rows: kernel sizes that do and do not divide the
threads, last tiles of every fill, maps with a row stride of their own, and both sides of the rule between
short-row kernel and tiles (rows times channels), against FP64.

Tolerance (relative L2): FP32 accumulation over at most 32 x 32 products (2e-6), 1e-13 in FP64."""

import ctypes

import numpy as np
import pytest
import torch

from oracle import oracle as orc
from tests.helpers import dense_ijk, random_sparse_ijk

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30))


def f64(t):
    return t.detach().double().cpu().numpy()


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 2e-6), (torch.float64, 1e-13)])
@pytest.mark.parametrize("cin,cout,n,ks,dense", [
    (16, 32, 14336, 3, True), (16, 32, 14337, 3, True), (8, 24, 28673, 3, False), (32, 96, 3001, (3, 3, 2), False),
    (1, 16, 900, 3, False), (3, 33, 1000, 2, False), (5, 40, 777, (4, 4, 2), True), (32, 33, 129, (1, 3, 1), False),
    (4, 36, 127, (5, 3, 2), True)])
def test_forward(cuda_device, dtype, tol, cin, cout, n, ks, dense):
    import fvdb
    from fvdb import _lib

    ijk = dense_ijk((32, 32, (n + 1023) // 1024))[:n] if dense else random_sparse_ijk(n, 40, n)
    grid = fvdb.GridBatch.from_ijk(torch.from_numpy(ijk).to(cuda_device))
    pack, _ = grid.sparse_conv_kernel_map(ks, 1)
    kz = (ks,) * 3 if isinstance(ks, int) else ks
    K = int(np.prod(kz))
    g = torch.Generator().manual_seed(cin + cout)
    x = torch.randn(n, cin, generator=g, dtype=dtype).to(cuda_device)
    w = (torch.randn(cout, cin, *kz, generator=g, dtype=dtype) / (K * cin) ** 0.5).to(cuda_device)
    v = grid.ijk.jdata.cpu().numpy()
    want = orc.conv_forward_f64(f64(x), f64(w), orc.kernel_map(v, np.array([0, n]), v, np.array([0, n]), kz, 1))
    first = pack.sparse_conv_3d(x, w).jdata
    assert rel(f64(first), want) <= tol
    # over the row order the same sums in the same order
    assert torch.equal(pack.sparse_conv_3d(x, w).jdata, first)
    # a map with a row stride of its own, entries past the input's rows among the absent ones
    wide = torch.full((n, K + 5), n + 7, dtype=torch.int32, device=cuda_device)
    m = pack._impl.kmap()[:n]
    wide[:, :K] = torch.where(m >= 0, m, n + 3)
    wk = w.permute(4, 3, 2, 1, 0).reshape(K, cin, cout).contiguous()
    y = torch.empty_like(first)
    i64, P = ctypes.c_int64, lambda t: ctypes.c_void_p(t.data_ptr())
    assert _lib.cdll().fvgb_conv_fwd_simt(
        0 if dtype == torch.float32 else 1, P(x), i64(n), cin, i64(cin), P(wide), i64(n), K, i64(K + 5), P(wk), i64(cin * cout),
        i64(cout), i64(1), P(y), cout, i64(cout), 0, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    torch.cuda.synchronize()
    assert rel(f64(y), want) <= tol
