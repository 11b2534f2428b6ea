"""GPU: what a CP-ALS request holds on the device while it runs stays within
the bytes it was admitted with."""
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


@pytest.mark.parametrize("R,J", [(128, 1024), (100, 65536), (8, 512), (25, 131072)])
def test_als_request_within_its_estimate(ftl, R, J):
    from fast_tensor_leverage_gb300 import serving as S
    rng = np.random.default_rng(R)
    dims, nnz = [300, 200, 150], 4000
    flat = rng.choice(int(np.prod(dims)), size=nnz, replace=False)
    idx = np.stack(np.unravel_index(flat, dims), axis=1).astype(np.uint32)
    req = S.ALSRequest(idx, rng.random(nnz) + 0.5, dims, R, J, sweeps=2, precision="fp64")
    eng = S.ServingEngine(1 << 32, max_active=1)
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    done = eng.run([(0.0, req)])
    torch.cuda.synchronize()
    assert done[0].status == "ok"
    assert torch.cuda.max_memory_allocated() - before <= S.estimate_bytes(req)
