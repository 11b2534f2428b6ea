"""GPU: the exact MTTKRP of a mode with more than 2^31 rows (indices are uint32)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_rows_past_2_31():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import fast_tensor_leverage_gb300 as ftl
    if torch.cuda.mem_get_info()[0] < 24 << 30:
        pytest.skip("needs 17 GB for the result")
    dims = [(1 << 31) + 8, 4, 3]
    idx = np.array([[5, 0, 1], [(1 << 31) - 1, 3, 2], [1 << 31, 1, 0], [(1 << 31) + 7, 2, 2], [(1 << 31) + 7, 1, 1]],
                   dtype=np.uint32)
    vals = np.array([1.5, -2.0, 3.0, 0.5, 4.0])
    sp = ftl.SparseTensor(idx, vals, "sort", dims=dims)
    rng = np.random.default_rng(0)
    U = [np.zeros((1, 1)), rng.normal(size=(4, 1)), rng.normal(size=(3, 1))]
    out = torch.empty((dims[0], 1), dtype=torch.float64, device="cuda")
    sp._exact_mttkrp_dev([torch.from_numpy(u).cuda() for u in U], 0, out.data_ptr(), dims[0],
                         torch.cuda.current_stream().cuda_stream)
    rows = sorted({int(i) for i in idx[:, 0]})
    want = {r: sum(v * U[1][i[1], 0] * U[2][i[2], 0] for i, v in zip(idx, vals) if i[0] == r) for r in rows}
    got = out[torch.tensor(rows, device="cuda")].cpu().numpy()[:, 0]
    np.testing.assert_allclose(got, [want[r] for r in rows], rtol=1e-14)
