"""Workspace sizes of a draw plan: the documented sizes, which callers may have
used to size their buffers, and the table scratch beside them."""
import pytest

from fast_tensor_leverage_gb300 import _lib


@pytest.mark.parametrize("R", [1, 2, 16, 17, 32, 33, 100, 128])
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_plan_sizes_stay_as_documented(R, prec):
    for N in (1, 3, 16):
        M = _lib.plan_sizes(N, R, _lib.PREC[prec])[1]
        # (2N + 3) R x R matrices, the packed pseudo-inverse (even length) and a status word
        assert M <= 8 * ((2 * N + 3) * R * R + R * (R + 1) // 2 + 4)


@pytest.mark.parametrize("R", [1, 16, 17, 32, 33, 128])
def test_table_scratch(R):
    for prec, size in (("fp64", 8), ("fp32", 4)):
        p = _lib.PREC[prec]
        assert _lib.table_bytes(R, 16383, p) == 0
        want = 0 if prec == "fp32" and 16 < R <= 32 else (256 + 4096 * R) * size
        assert _lib.table_bytes(R, 16384, p) == want
        assert _lib.table_bytes(R, 1 << 40, p) == want
