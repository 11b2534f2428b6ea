"""GPU: draws whose first sampled mode reads its upper forms from the mass
table against draws that evaluate every form (the packed entry point, which
has no table): the same samples, rows and weights bit for bit."""
import numpy as np
import pytest
import torch

from tests.test_gpu_draw_fx import factors, ftl, packed_fp64 as packed  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,R,J,j", [
    ([4096, 900], 4, 30000, 3),            # J = 7,500 R: every level
    ([70000, 1000, 500], 8, 16384, 4),     # the fewest samples with a table
    ([70000, 1000, 500], 8, 16383, 4),     # none
    ([70000, 1000, 500], 8, 20000, 0),     # first sampled mode is 1
    ([65, 3000], 16, 17000, 3),            # 5 leaves: too few levels, no table
    ([40000, 2000], 20, 17000, 3),
    ([100003, 5000], 25, 17000, 2),
    ([300000, 1025, 64], 32, 17000, 4),
    ([50000, 3000], 33, 17000, 3),
    ([70001, 65], 64, 17000, 3),
    ([30000, 500], 100, 17000, 3),
    ([40000, 129], 128, 17000, 3),
])
@pytest.mark.parametrize("precision", ["fp64", "fp32", "tf32x3"])
def test_table_draw_equals_untabled_draw(ftl, dims, R, J, j, precision):  # noqa: F811
    g = torch.Generator(device="cuda")
    g.manual_seed(R + J)
    U = factors(dims, R, "zero rows" if R % 3 == 0 else "plain", g)
    s = ftl.Sampler(U, J, R, "efficient", precision=precision, seed=3, overlap_computem=False)
    draws = torch.rand(2 * s.N * J, generator=g, device="cuda", dtype=torch.float64)
    smp, h, w = (t.clone() for t in s.draw(j, draws))
    ref, rh, rw = packed(s, j, draws)
    keep = [k for k in range(s.N) if k != j]
    assert torch.equal(smp[keep], ref[keep])
    assert torch.equal(h.view(torch.int64), rh.view(torch.int64))
    assert torch.equal(w.view(torch.int64), rw.view(torch.int64))
    assert np.all(smp[keep].cpu().numpy() < np.array(dims)[keep][:, None])
