"""GPU: the weighted Gram and the row solve at the edges of their block
shapes, against plain FP64 products (sums of up to 1,500 products of O(1)
values in another order: 1e-12 of the largest entry)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from fast_tensor_leverage_gb300 import _lib
    return _lib


def close(a, b):
    np.testing.assert_allclose(a, b, rtol=0, atol=1e-12 * max(1.0, np.abs(b).max()))


@pytest.mark.parametrize("R", [1, 2, 4, 5, 8, 16, 25, 31, 32, 40, 63, 64, 65, 100, 125, 128])
@pytest.mark.parametrize("n", [1, 31, 33, 1500])
def test_weighted_gram_and_solve_rows(lib, R, n):
    rng = np.random.default_rng(R * 10000 + n)
    st = torch.cuda.current_stream().cuda_stream
    A = rng.normal(size=(n, R))
    A[rng.random(n) < 0.3] = 0.0
    idx = rng.permutation(n)[: max(1, n // 2)].astype(np.int32)
    w, cnt = rng.random(n) + 0.5, rng.integers(1, 5, size=idx.size).astype(np.int32)
    pinv = rng.normal(size=(R, R))
    pinv = pinv + pinv.T
    d = {k: torch.from_numpy(v).cuda() for k, v in dict(A=A, idx=idx, w=w, cnt=cnt, pinv=pinv).items()}
    nu = torch.tensor([idx.size], dtype=torch.int64, device="cuda")
    nb = lib.ws_bytes("gram", R)
    ws = torch.empty(nb, dtype=torch.uint8, device="cuda")
    g = torch.empty((R, R), dtype=torch.float64, device="cuda")
    lib.call("ftl_weighted_gram", d["A"].data_ptr(), None, None, None, None, n, R, ws.data_ptr(), nb, g.data_ptr(), st)
    close(g.cpu().numpy(), A.T @ A)
    lib.call("ftl_weighted_gram", d["A"].data_ptr(), d["idx"].data_ptr(), d["w"].data_ptr(), d["cnt"].data_ptr(),
             nu.data_ptr(), n, R, ws.data_ptr(), nb, g.data_ptr(), st)
    close(g.cpu().numpy(), (A[idx] * (w[idx] * cnt)[:, None]).T @ A[idx])
    u = torch.full((n, R), 7.0, dtype=torch.float64, device="cuda")
    lib.call("ftl_solve_rows", d["A"].data_ptr(), d["pinv"].data_ptr(), n, R, u.data_ptr(), st)
    close(u.cpu().numpy(), A @ pinv)
    assert np.all(u.cpu().numpy()[~A.any(axis=1)] == 0.0)
    u.fill_(7.0)
    lib.call("ftl_solve_rows_at", d["A"].data_ptr(), d["pinv"].data_ptr(), d["idx"].data_ptr(), nu.data_ptr(), n, R,
             u.data_ptr(), st)
    ref = np.full((n, R), 7.0)
    ref[idx] = A[idx] @ pinv
    close(u.cpu().numpy(), ref)


@pytest.mark.parametrize("Rr,R", [(1, 1), (16, 64), (8, 25), (128, 128), (25, 100)])
def test_low_rank_solve_in_the_middle(lib, Rr, R):
    rng = np.random.default_rng(Rr + R)
    st = torch.cuda.current_stream().cuda_stream
    dims, J, j = [70, 50, 60], 300, 1
    V = [rng.normal(size=(n, Rr)) for n in dims]
    S = np.stack([rng.integers(0, n, size=J) for n in dims])
    h, w, s = rng.normal(size=(J, R)), rng.random(J), rng.random(Rr)
    pinv = rng.normal(size=(R, R))
    pinv = pinv + pinv.T
    d = [torch.from_numpy(v).cuda() for v in V]
    t = {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() for k, v in dict(S=S, h=h, w=w, s=s, pinv=pinv).items()}
    import ctypes
    ptrs = (ctypes.c_void_p * 3)(*[v.data_ptr() for v in d])
    nb = lib.ws_bytes("lowrank_mttkrp", Rr, R)
    ws = torch.empty(nb, dtype=torch.uint8, device="cuda")
    out = torch.empty((dims[j] + 2, R), dtype=torch.float64, device="cuda")
    lib.call("ftl_lowrank_sampled_solve", ptrs, t["s"].data_ptr(), 3, Rr, j, t["S"].data_ptr(), J, None, None, None, J,
             t["w"].data_ptr(), t["h"].data_ptr(), R, t["pinv"].data_ptr(), ws.data_ptr(), nb, out.data_ptr(), dims[j],
             dims[j] + 2, st)
    P = s * V[0][S[0]] * V[2][S[2]]
    ref = np.zeros((dims[j] + 2, R))
    ref[: dims[j]] = V[j] @ (P.T @ (h * w[:, None])) @ pinv
    np.testing.assert_allclose(out.cpu().numpy(), ref, rtol=0, atol=1e-11 * np.abs(ref).max())
