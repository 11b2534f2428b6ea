"""GPU: FP32 draws at 32 < R <= 64 on either side of one wave of resident warps,
with and without FP32 factor copies, against the packed draw, which runs one
kernel at every J: the same samples, rows and weights bit for bit."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ftl():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import fast_tensor_leverage_gb300 as m
    return m


@pytest.mark.parametrize("R", [33, 48, 49, 64])
@pytest.mark.parametrize("waves,more", [(0, 3), (1, 0), (1, 1), (2, -3), (3, 5), (8, 1)])
@pytest.mark.parametrize("copies", [True, False])
@pytest.mark.parametrize("j", [0, 4])
def test_draw_equals_packed(ftl, R, waves, more, copies, j):
    from fast_tensor_leverage_gb300 import _lib
    J = 16 * torch.cuda.get_device_properties(0).multi_processor_count * waves + more
    g = torch.Generator(device="cuda")
    g.manual_seed(R + J)
    U = [torch.randn((n, R), generator=g, device="cuda", dtype=torch.float64) for n in (5000, 63, 2049)]
    U[0][100:900] = 0.0
    U[2][::7] *= 1e-42          # FP32-subnormal values
    s = ftl.Sampler(U, J, R, "efficient", precision="fp32", seed=7, overlap_computem=False, factor_shadows=copies)
    smp, h, w = (t.clone() for t in s.draw(j))
    N = 3
    ref = (torch.zeros((N, J), dtype=torch.int64, device="cuda"),
           torch.empty((J, R), dtype=torch.float64, device="cuda"), torch.empty(J, dtype=torch.float64, device="cuda"))

    def ptrs(*v):
        return (ctypes.c_void_p * len(v))(*v)

    _lib.call("ftl_krp_sample_packed", ptrs(ctypes.addressof(s._plan)), 1, (ctypes.c_uint32 * 1)(j),
              *(ptrs(t.data_ptr()) for t in ref), ptrs(None), (ctypes.c_uint64 * 1)(7), (ctypes.c_uint64 * 1)(0),
              torch.cuda.current_stream().cuda_stream)
    keep = [k for k in range(N) if k != j]
    assert torch.equal(smp[keep], ref[0][keep])
    assert torch.equal(h.view(torch.int64), ref[1].view(torch.int64))
    assert torch.equal(w.view(torch.int64), ref[2].view(torch.int64))
