"""GPU: FP64 Jacobi eigensolves of matrices D C D whose columns lie 50 or 55
decades apart (D) over a well-conditioned C: the rotations that couple the two
scales are below FP32's range of the largest entry, and leaving one out changes
the small eigenvalue by its correlation with the large one.

Tolerance, e = 2^-53: two-sided Jacobi with a relative stopping rule changes C,
not D C D, by about 6 e |C| a round, 10 sweeps of R rounds: 64 R e |C| (Demmel
and Veselic); the inverse moves by |C^-1| |C| = cond(C) times that of its own
size, the eigenvector products by a small multiple."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu

E = 2.0 ** -53


@pytest.fixture(scope="module")
def ftl():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import fast_tensor_leverage_gb300 as m
    return m


@pytest.mark.parametrize("R", [3, 9, 32, 33, 41])
def test_pseudo_inverse_of_graded_pairs(ftl, R):
    """Pairs [[S^2, cS], [cS, 1]], and a last row of zeros so that the
    eigendecomposition runs (not a Cholesky factor)."""
    from fast_tensor_leverage_gb300 import _lib
    S, c = 1e50, 0.9
    pairs = (R - 1) // 2
    M = np.zeros((R, R))
    inv = np.zeros((R, R))
    d = np.ones(R)
    for i in range(pairs):
        a, b = 2 * i, 2 * i + 1
        M[a, a], M[a, b], M[b, a], M[b, b] = S * S, c * S, c * S, 1.0
        d[a] = S
        inv[a, a] = inv[b, b] = 1.0 / (1.0 - c * c)
        inv[a, b] = inv[b, a] = -c / (1.0 - c * c)
    dev = torch.from_numpy(M).cuda()
    out = torch.empty((R, R), dtype=torch.float64, device="cuda")
    scr = torch.empty((R, R), dtype=torch.float64, device="cuda")
    _lib.call("ftl_pinv_square", dev.data_ptr(), R, R, None, 1e-11, out.data_ptr(), scr.data_ptr(),
              torch.cuda.current_stream().cuda_stream)
    got = out.cpu().numpy() * np.outer(d, d)
    cond = (1.0 + c) / (1.0 - c)
    assert np.abs(got - inv).max() <= 64 * R * E * cond * np.abs(inv).max()


@pytest.mark.parametrize("R", [8, 25, 33, 64, 101])
def test_compute_m_of_balanced_scales(ftl, R):
    """Two factors whose column scales cancel: computeM's middle matrix has
    them squared, and its W^T W, taken back to scale, is that matrix."""
    from fast_tensor_leverage_gb300 import _lib
    rng = np.random.default_rng(R)
    D = np.where(np.arange(R) % 3 == 0, 2.0 ** 183, 1.0)      # about 1e55
    U = [rng.normal(size=(n, R)) + rng.normal(size=(n, 1)) for n in (300, 400)]
    U = [u / np.sqrt((u * u).sum(axis=0)) for u in U]
    G = [u.T @ u for u in U]
    s = ftl.Sampler([U[0] * D, U[1] / D], 16, R, "efficient", precision="fp64", seed=1, overlap_computem=False)
    _lib.call("ftl_krp_compute_m", ctypes.byref(s._plan), 3, torch.cuda.current_stream().cuda_stream)
    M = s.M.cpu().numpy()[: 3 * R * R].reshape(3, R, R)
    C = G[1] * np.linalg.inv(G[0] * G[1])                     # times 1 / (D_a D_b): the middle matrix
    W = M[1] * D
    tol = (4 * 64 * R + 2 * (R + 16) * R) * E * np.linalg.norm(C, 2) * np.linalg.cond(G[0] * G[1])
    assert np.abs(W.T @ W - C).max() <= tol
