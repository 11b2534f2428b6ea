"""GPU: the row-grouped sparse kernels (exact MTTKRP, range finder) at the
edges of their lane groups and runs, against plain FP64 sums.

Tolerance: FP64 sums of at most a few hundred products of O(1) values whose
order differs: 1e-12 of the largest entry; range finder: its FP32 normals
against FP64 ones from the same bits, 1e-5 (as the suite's range-finder test)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ftl():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import fast_tensor_leverage_gb300 as m
    return m


def tensor(dims, nnz, seed):
    rng = np.random.default_rng(seed)
    idx = np.stack([np.minimum((d * rng.random(nnz) ** 3).astype(np.int64), d - 1) for d in dims], axis=1)
    idx = np.unique(idx, axis=0).astype(np.uint32)
    return rng, idx, rng.normal(size=idx.shape[0])


@pytest.mark.parametrize("R", [1, 2, 8, 9, 16, 17, 25, 32, 33, 64, 65, 128])
@pytest.mark.parametrize("dims,nnz,j", [([700, 30, 40], 5000, 0), ([5, 300, 7, 11], 3000, 2), ([60, 80], 257, 1),
                                        ([3, 4, 2, 3, 5, 4], 700, 5), ([1, 1, 1], 1, 0)])
def test_exact_mttkrp_rows(ftl, dims, nnz, j, R):
    rng, idx, vals = tensor(dims, nnz, R + nnz)
    sp = ftl.SparseTensor(idx, vals, "sort", dims=dims)
    U = [rng.normal(size=(d, R)) for d in dims]
    out = torch.full((dims[j] + 3, R), np.nan, dtype=torch.float64, device="cuda")
    sp._exact_mttkrp_dev([torch.from_numpy(u).cuda() for u in U], j, out.data_ptr(), dims[j] + 3,
                         torch.cuda.current_stream().cuda_stream)
    p = vals[:, None].repeat(R, axis=1)
    for k in range(len(dims)):
        if k != j:
            p = p * U[k][idx[:, k]]
    ref = np.zeros((dims[j] + 3, R))
    np.add.at(ref, idx[:, j], p)
    np.testing.assert_allclose(out.cpu().numpy(), ref, rtol=0, atol=1e-12 * max(1.0, np.abs(ref).max()))


@pytest.mark.parametrize("R", [1, 2, 5, 16, 25, 31, 32, 33, 63, 64, 65, 128])
def test_range_finder_rows(ftl, R):
    from fast_tensor_leverage_gb300 import _lib
    from oracle import oracle as O
    dims, seed = [300, 20, 25], 9
    _, idx, vals = tensor(dims, 2000, R)
    sp = ftl.SparseTensor(idx, vals, "sort", dims=dims)
    U = O.rrf(idx, vals, dims, dims, R, seed)
    for j in range(3):
        rrows, rkeys, rvals = sp.rows[j]
        out = torch.full((dims[j], R), np.nan, dtype=torch.float64, device="cuda")
        _lib.call("ftl_sparse_rrf", rrows.data_ptr(), rkeys.data_ptr(), rvals.data_ptr(), sp.nnz, R, seed, j,
                  out.data_ptr(), dims[j], torch.cuda.current_stream().cuda_stream)
        np.testing.assert_allclose(out.cpu().numpy(), U[j], rtol=0, atol=1e-5 * max(1.0, np.abs(U[j]).max()))


@pytest.mark.parametrize("R", [1, 8, 25, 33, 128])
@pytest.mark.parametrize("dims,nnz", [([700, 30, 40], 5000), ([60, 80], 257), ([5, 300, 7, 11], 3000),
                                      ([3, 4, 2, 3, 5, 4], 700), ([2, 3, 2, 3, 2, 3, 4], 500), ([900, 800, 700], 100)])
def test_residual_terms(ftl, dims, nnz, R):
    rng, idx, vals = tensor(dims, nnz, R + nnz)
    sp = ftl.SparseTensor(idx, vals, "sort", dims=dims)
    U = [rng.normal(size=(d, R)) for d in dims]
    s = rng.random(R) + 0.5
    m = np.ones((idx.shape[0], R)) * s
    G = np.outer(s, s)
    for k in range(len(dims)):
        m = m * U[k][idx[:, k]]
        G = G * (U[k].T @ U[k])
    terms = sp.residual_terms_async(torch.from_numpy(s).cuda(), [torch.from_numpy(u).cuda() for u in U]).cpu().numpy()
    first = vals ** 2 - 2.0 * vals * m.sum(axis=1)
    assert abs(terms[0] - first.sum()) <= 1e-12 * max(1.0, (vals ** 2 + 2.0 * np.abs(vals) * np.abs(m).sum(axis=1)).sum())
    assert abs(terms[1] - G.sum()) <= 1e-12 * np.abs(G).sum()
