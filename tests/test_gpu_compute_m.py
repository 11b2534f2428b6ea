"""GPU: computeM above R = 32 in FP64 (eigensolves by clusters) against plain
numpy, at odd and even ranks and where the last blocks of a cluster hold few or
no rows of the eigenvectors; the same bits on every repetition.

Tolerances, e = 2^-53.  A root Gram: sums of R products per leaf and of at most
16 levels, so an entry of the Hadamard product S of n of them is off by
n (R + 16) e of its diagonals (at most 1: unit columns, graded ones times powers
of two).  A Jacobi round
moves the matrix by about 6 e of its norm, and 10 sweeps of R rounds make
d(A) = 64 R e |A|.  Eigenvalues and W^T W are within d(A) plus the matrix's own
error, the (pseudo-)inverse within 4 |A^+|^2 times that (Wedin's constant 1.62
for two matrices of equal rank, twice the error when one is cut to it)."""
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


def factors(dims, R, kind, rng):
    U = []
    for n in dims:
        u = rng.normal(size=(n, R)) + rng.normal(size=(n, 1))
        u /= np.sqrt((u * u).sum(axis=0))
        if kind == "rank deficient":    # columns that coincide in every factor
            u[:, 1::4] = u[:, 0:1]
        U.append(u)
    if kind == "graded":                # 2^0 .. 2^-4 per factor and column: no eigenvalue falls below the cut of 1e-8
        d = 2.0 ** -np.round(np.linspace(0.0, 4.0, R))
        U = [u * d for u in U]
        return U, d
    return U, np.ones(R)


@pytest.mark.parametrize("R", [33, 34, 64, 65, 100, 127, 128])
@pytest.mark.parametrize("j", [0, 1, 4])
@pytest.mark.parametrize("kind", ["plain", "rank deficient", "graded"])
def test_compute_m_clusters(ftl, R, j, kind):
    from fast_tensor_leverage_gb300 import _lib
    rng = np.random.default_rng(R + 1000 * j)
    dims = [300, 257, 400]
    U, d = factors(dims, R, kind, rng)
    N = len(U)
    s = ftl.Sampler(U, 16, R, "efficient", precision="fp64", seed=1, overlap_computem=False)
    st = torch.cuda.current_stream().cuda_stream
    bufs = (s.M, s.lam, s.eig_G, s.pinv32)
    first = None
    for _ in range(20):
        _lib.call("ftl_krp_compute_m", ctypes.byref(s._plan), j, st)
        torch.cuda.synchronize()
        now = [b.clone() for b in (s.lam, s.eig_G, s.pinv32)] + [s.M[: (N + 1) * R * R].clone()]
        if first is None:
            first = now
        assert all(torch.equal(a.view(torch.uint8), b.view(torch.uint8)) for a, b in zip(first, now))
    M = s.M.cpu().numpy()[: (N + 1) * R * R].reshape(N + 1, R, R)
    lam = s.lam.cpu().numpy().reshape(N + 1, R)
    eig = s.eig_G.cpu().numpy().reshape(N, 2 * R - 1, -1)

    modes = [k for k in range(N) if k != j]
    roots = {k: O.packed_to_upper(O.tree_build(U[k], min(R, dims[k]))[0], R) for k in modes}
    roots = {k: np.triu(g) + np.triu(g, 1).T for k, g in roots.items()}
    suffix, S = {}, np.ones((R, R))
    for k in reversed(modes):
        S = S * roots[k]
        suffix[k] = S.copy()
    root_err = len(modes) * (R + 16) * E

    def off(A):
        return (root_err * R + 64 * R * E) * np.linalg.norm(A, 2)

    top = suffix[modes[0]]
    dd = d ** len(modes)
    C = top / np.outer(dd, dd)          # exact: powers of two
    assert np.abs(lam[0] - np.linalg.eigvalsh(top)).max() <= off(top)
    if kind == "rank deficient":
        l, Q = np.linalg.eigh(C)
        keep = l > 1e-8
        assert 0 < keep.sum() < R
        inv = (Q[:, keep] / l[keep]) @ Q[:, keep].T
    else:
        inv = np.linalg.inv(C)
    inv = inv / np.outer(dd, dd)
    pinv = M[0]
    assert np.abs(pinv - inv).max() <= 4.0 * np.linalg.norm(inv, 2) ** 2 * off(top)
    for at, k in enumerate(modes):
        last = at + 1 == len(modes)
        o = N if last else modes[at + 1]
        W = M[o]
        if last:
            A = pinv
        else:
            A = suffix[modes[at + 1]] * pinv
            assert np.all(np.diff(lam[o]) >= 0.0)
            assert np.abs(lam[o] - np.linalg.eigvalsh(A)).max() <= off(A)
        # negative rounding noise of the eigenvalues is clamped: once more the error
        assert np.abs(W.T @ W - A).max() <= 2.0 * off(A)
        # the eigen tree over W's rows: sums of up to R products, and the root's own error
        root = O.upper_to_packed(roots[k], R)
        want = O.tree_scale(O.tree_build(np.ascontiguousarray(W), 1), R, root)
        size = O.tree_build(np.ascontiguousarray(np.abs(W)), 1)
        P = want.shape[1]
        assert np.all(np.abs(eig[k][:, :P] - want) <= size * (2.0 * R * E * np.abs(root) + root_err))
        assert np.all(eig[k][:, P:] == 0.0)
