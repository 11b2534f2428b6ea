"""GPU: the exact MTTKRP's runs of one to all steps per lane group, against plain
FP64 sums; the kernel over unsorted nonzeros beside it.

Tolerance: sums of at most a few thousand products of O(1) values in another
order, 1e-12 of the largest entry."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R", [5, 16, 25, 40, 100])
@pytest.mark.parametrize("nnz", [1, 3, 2431, 77823, 77825, 170001, 700003])
def test_exact_mttkrp_run_lengths(nnz, R):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import fast_tensor_leverage_gb300 as ftl
    from fast_tensor_leverage_gb300 import _lib
    rng = np.random.default_rng(nnz + R)
    dims, j = [900, 300, 200], 0
    idx = np.stack([rng.integers(0, d, size=nnz) for d in dims], axis=1).astype(np.uint32)
    vals = rng.normal(size=nnz)
    sp = ftl.SparseTensor(idx, vals, "sort", dims=dims)
    g = torch.Generator(device="cuda")
    g.manual_seed(R)
    U = [torch.randn((d, R), generator=g, device="cuda", dtype=torch.float64) for d in dims]
    st = torch.cuda.current_stream().cuda_stream
    a, b = (torch.full((dims[j], R), np.nan, dtype=torch.float64, device="cuda") for _ in range(2))
    sp._exact_mttkrp_dev(U, j, a.data_ptr(), dims[j], st)
    ptrs = (ctypes.c_void_p * 3)(*[u.data_ptr() for u in U])
    _lib.call("ftl_sparse_exact_mttkrp", sp.idx_dev.data_ptr(), sp.vals_dev.data_ptr(), nnz, 3, j, ptrs, R,
              b.data_ptr(), dims[j], st)
    i = torch.from_numpy(idx.astype(np.int64)).cuda()
    p = torch.from_numpy(vals).cuda().unsqueeze(1) * U[1][i[:, 1]] * U[2][i[:, 2]]
    want = torch.zeros((dims[j], R), dtype=torch.float64, device="cuda").index_add_(0, i[:, 0], p)
    tol = 1e-12 * max(1.0, float(want.abs().max()))
    assert float((a - want).abs().max()) <= tol
    assert float((b - want).abs().max()) <= tol
