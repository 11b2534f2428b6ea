"""GPU: FP32 draws whose leaf scans round FP64 factor rows themselves against
draws from the FP32 copies of the same factors (rounded when the trees are
built): the same samples, rows and weights bit for bit, with values on both
sides of the range that the branch-free rounding covers."""
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


@pytest.mark.parametrize("R", [1, 5, 16, 17, 25, 31, 32, 33, 48, 64, 65, 100, 128])
@pytest.mark.parametrize("odd", [False, True])
def test_rows_rounded_in_the_scan_equal_the_copies(ftl, R, odd):
    rng = np.random.default_rng(R)
    dims = [3 * R + 1, 2011, 777]
    U = [rng.normal(size=(n, R)) for n in dims]
    for u in U:
        u[rng.random(u.shape[0]) < 0.02] = 0.0
        if odd:  # FP32-subnormal, below it, FP64-subnormal, halfway cases, large
            vals = np.array([1e-40, -3e-45, 1e-60, 5e-324, 1.0 + 2.0 ** -24, 1.0 + 3 * 2.0 ** -24, 1e4, -0.0])
            at = rng.random(u.shape) < 0.02
            u[at] = rng.choice(vals, size=int(at.sum()))
    J = 3000
    a = ftl.Sampler(U, J, R, "efficient", precision="fp32", seed=5, factor_shadows=True)
    b = ftl.Sampler(U, J, R, "efficient", precision="fp32", seed=5, factor_shadows=False)
    for j in (0, 3):
        sa, ha, wa = (t.clone() for t in a.draw(j))
        sb, hb, wb = (t.clone() for t in b.draw(j))
        keep = [k for k in range(3) if k != j]
        assert torch.equal(sa[keep], sb[keep])
        assert torch.equal(ha.view(torch.int64), hb.view(torch.int64))
        assert torch.equal(wa.view(torch.int64), wb.view(torch.int64))
