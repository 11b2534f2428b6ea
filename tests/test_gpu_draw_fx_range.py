"""GPU: FP64 draws on trees and queries near the ends of FP64's range, where the
fixed-point forms leave the decisions to the FP64 descent (an exact zero or a
subnormal value is not small against 2^-(exponent) there, and products that
underflow or overflow in FP64 have no exact form to match): the same samples,
rows and weights as the FP64 descent, bit for bit.

Half of a tree's rows are zero but for one small column, and the uniforms lie
between 2^-32 and 2^-20, where that half's share ends."""
import numpy as np
import pytest
import torch

from tests.test_gpu_draw_fx import packed_fp64

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ftl():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import fast_tensor_leverage_gb300 as m
    return m


@pytest.mark.parametrize("R", [8, 25, 32, 40, 100])
@pytest.mark.parametrize("scales", [(1e-152, 1e151), (1e151, 1e-152), (1e-150, 1e150), (1e-145, 1e145), (1e-140, 1e140),
                                    (1e-120, 1e120), (1e-75, 1e75), (1e75, 1e-75), (1e75, 1e60), (1e-70, 1e-70)])
def test_extreme_scales_equal_fp64_descent(ftl, R, scales):
    g = torch.Generator(device="cuda")
    g.manual_seed(R)
    J = 2000
    U = []
    for n, sc in zip((2048, 1500), scales):
        u = torch.randn((n, R), generator=g, device="cuda", dtype=torch.float64)
        u[: n // 2, 1:] = 0.0
        u[: n // 2, 0] *= 1e-5
        U.append(u * sc)
    s = ftl.Sampler(U, J, R, "efficient", precision="fp64", seed=3, overlap_computem=False)
    draws = torch.rand((4, J), generator=g, device="cuda", dtype=torch.float64)
    draws[2:] = 2.0 ** (-32.0 + 12.0 * torch.rand((2, J), generator=g, device="cuda", dtype=torch.float64))
    draws[2:, ::4] = torch.rand((2, J // 4), generator=g, device="cuda", dtype=torch.float64)
    draws = draws.reshape(-1)
    smp, h, w = (t.clone() for t in s.draw(3, draws))
    ref, rh, rw = packed_fp64(s, 3, draws)
    assert torch.equal(smp, ref)
    assert torch.equal(h.view(torch.int64), rh.view(torch.int64))
    assert torch.equal(w.view(torch.int64), rw.view(torch.int64))
