"""GPU: FP64 draws decided by certified fixed-point forms against the FP64
descent (the packed multi-request entry point, which evaluates every form in
FP64): the same samples, rows and weights bit for bit, whatever the shape,
the scale of the factors, zero rows or coinciding columns."""
import ctypes

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


def packed_fp64(s, j, draws):
    from fast_tensor_leverage_gb300 import _lib
    N, J, R = s.N, s.J, s.R
    smp = torch.zeros((N, J), dtype=torch.int64, device="cuda")
    h = torch.empty((J, R), dtype=torch.float64, device="cuda")
    w = torch.empty(J, dtype=torch.float64, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    _lib.call("ftl_krp_compute_m", ctypes.byref(s._plan), j, st)

    def ptrs(*v):
        return (ctypes.c_void_p * len(v))(*v)

    plans = ptrs(ctypes.addressof(s._plan))
    _lib.call("ftl_krp_sample_packed", plans, 1, (ctypes.c_uint32 * 1)(j), ptrs(smp.data_ptr()), ptrs(h.data_ptr()),
              ptrs(w.data_ptr()), ptrs(draws.data_ptr()), (ctypes.c_uint64 * 1)(0), (ctypes.c_uint64 * 1)(0), st)
    torch.cuda.synchronize()
    return smp, h, w


def factors(dims, R, kind, g):
    U = [torch.randn((n, R), generator=g, device="cuda", dtype=torch.float64) for n in dims]
    for u in U:
        u *= torch.where(torch.rand((u.shape[0], 1), generator=g, device="cuda") < 0.01, 100.0, 1.0)
        if kind == "zero rows":
            u[torch.rand(u.shape[0], generator=g, device="cuda") < 0.9] = 0.0
            u[0] = 1.0
        elif kind == "tiny":
            u *= 1e-9
        elif kind == "huge":
            u *= 1e30
        elif kind == "spread columns":
            u *= torch.logspace(-12, 12, R, device="cuda", dtype=torch.float64)
        elif kind == "coinciding columns":
            u[:, 1:] = u[:, :1] * (1.0 + 1e-7 * u[:, 1:])
    return U


@pytest.mark.parametrize("dims,R,J,j", [
    ([1000, 1000, 1000, 1000], 8, 3000, 5),
    ([5, 7, 3], 4, 500, 4),              # single-leaf trees
    ([40000, 33, 2049], 32, 2000, 0),    # full and partial last leaves
    ([300007, 1025], 25, 2000, 3),       # R not a multiple of the vector width
    ([2000, 999], 1, 500, 3),            # one column: one-leaf eigen trees
    ([700, 1500], 33, 1000, 3),
    ([3000, 64, 65], 64, 1000, 1),
    ([1300, 2100], 65, 500, 3),          # four warps per sample
    ([900, 2100], 100, 500, 3),
    ([129, 4000], 128, 400, 3),
])
@pytest.mark.parametrize("kind", ["plain", "zero rows", "tiny", "huge", "spread columns", "coinciding columns"])
def test_fixed_point_draw_equals_fp64_descent(ftl, dims, R, J, j, kind):
    if kind == "huge" and len(dims) * 60 > 300:
        pytest.skip("the product of the Grams overflows FP64")
    g = torch.Generator(device="cuda")
    g.manual_seed(R * 1000 + len(dims))
    U = factors(dims, R, kind, g)
    s = ftl.Sampler(U, J, R, "efficient", precision="fp64", seed=3, overlap_computem=False)
    draws = torch.rand(2 * s.N * J, generator=g, device="cuda", dtype=torch.float64)
    draws[:3] = torch.tensor([0.0, 1.0 - 2.0 ** -53, 2.0 ** -60], device="cuda", dtype=torch.float64)
    smp, h, w = (t.clone() for t in s.draw(j, draws))
    ref, rh, rw = packed_fp64(s, j, draws)
    keep = [k for k in range(s.N) if k != j]
    assert torch.equal(smp[keep], ref[keep])
    assert torch.equal(h.view(torch.int64), rh.view(torch.int64))
    assert torch.equal(w.view(torch.int64), rw.view(torch.int64))
