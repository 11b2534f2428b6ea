"""GPU: the weighted Gram takes any workspace of at least one block per SM (the
size ftl_gram_workspace_bytes gave before blocks shared an SM), with the same
result up to the order of its sums, and refuses a smaller one."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R", [1, 8, 25, 64, 100, 128])
def test_smaller_workspaces(R):
    from fast_tensor_leverage_gb300 import _lib
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    st = torch.cuda.current_stream().cuda_stream
    rng = np.random.default_rng(R)
    n = 20000
    A = rng.normal(size=(n, R))
    want = A.T @ A
    d = torch.from_numpy(A).cuda()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    P = R * (R + 1) // 2
    guard = 64
    for blocks in (sms, sms + 1, 2 * sms + 7, 4 * sms):
        nb = blocks * P * 8
        ws = torch.full((nb // 8 + guard,), 7.0, dtype=torch.float64, device="cuda")
        g = torch.empty((R, R), dtype=torch.float64, device="cuda")
        _lib.call("ftl_weighted_gram", d.data_ptr(), None, None, None, None, n, R, ws.data_ptr(), nb, g.data_ptr(), st)
        # 20,000 products of O(1) values: n e of the diagonals at most
        assert np.abs(g.cpu().numpy() - want).max() <= n * 2.0 ** -53 * want.max()
        assert torch.all(ws[nb // 8:] == 7.0)
    nb = sms * P * 8 - 1
    with pytest.raises(Exception, match="workspace"):
        _lib.call("ftl_weighted_gram", d.data_ptr(), None, None, None, None, n, R, ws.data_ptr(), nb, g.data_ptr(), st)
