"""GPU: FP32 draws at R = 32 over trees of one leaf and of more, every variant of
the draw the same samples, rows and weights bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(20, 20, 20), (32, 5, 1), (20, 33, 20), (33, 20, 64)])
@pytest.mark.parametrize("copies", [True, False])
@pytest.mark.parametrize("j", [0, 1, 4])
def test_variants_agree(dims, copies, j):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import fast_tensor_leverage_gb300 as ftl
    from fast_tensor_leverage_gb300 import _lib
    g = torch.Generator(device="cuda")
    g.manual_seed(sum(dims))
    U = [torch.randn((n, 32), generator=g, device="cuda", dtype=torch.float64) for n in dims]
    keep = [k for k in range(3) if k != j]
    out = []
    try:
        for v in (-1, 0, 1, 2, 3):
            _lib.call("ftl_tune_set", 0, 32, 1, v)
            s = ftl.Sampler(U, 3001, 32, "efficient", precision="fp32", seed=9, factor_shadows=copies)
            smp, h, w = s.draw(j)
            out.append((smp[keep].clone(), h.clone().view(torch.int64), w.clone().view(torch.int64)))
    finally:
        _lib.call("ftl_tune_set", 0, 32, 1, -1)
    assert all(torch.equal(a, b) for o in out[1:] for a, b in zip(out[0], o))
