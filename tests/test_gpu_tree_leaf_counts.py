"""GPU: leaf Grams where the kernel and its shape depend on the number of leaves
and on their length, around the lines of the rules, against the CPU oracle's
tree (tolerances of test_gpu_tree_leaf)."""
import math

import numpy as np
import pytest
import torch

from oracle import oracle as O
from tests.test_gpu_tree_tc import build, check_close

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ftl():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import fast_tensor_leverage_gb300 as m
    return m


@pytest.mark.parametrize("R,F,leaves", [
    # one leaf per SM and one more (152), 32 per SM and one more (4,864)
    (25, 25, 152), (25, 25, 153), (25, 25, 4864), (25, 25, 4865), (30, 30, 700), (65, 65, 151), (65, 65, 154),
    (40, 40, 1216), (8, 8, 4864), (8, 8, 4865), (16, 16, 304), (56, 56, 13), (80, 80, 9), (5, 5, 40000),
    # leaves much shorter than R
    (16, 1, 500), (15, 1, 500), (17, 1, 500), (17, 2, 400), (20, 2, 400), (20, 3, 400), (25, 2, 300), (25, 3, 300),
    (31, 1, 300), (33, 1, 300), (40, 4, 200), (40, 5, 200), (80, 8, 150), (80, 9, 150), (100, 10, 100), (100, 11, 100),
    (125, 12, 80), (48, 3, 200), (48, 4, 200), (64, 4, 150),
    (64, 5, 150), (128, 8, 80), (128, 9, 80), (33, 6, 300), (33, 7, 300), (64, 12, 150),
    (64, 13, 150), (128, 25, 60), (128, 26, 60),
    # packed FP32 nodes on either side of the wrapped-diagonal ones
    (9, 9, 4900), (12, 12, 300), (13, 13, 4864), (15, 15, 20), (16, 16, 4865), (34, 34, 700), (63, 63, 310), (64, 64, 160),
    (96, 96, 20), (127, 127, 9), (128, 128, 40), (57, 57, 608), (57, 57, 609), (64, 64, 608), (64, 64, 609), (56, 56, 100),
    (9, 2, 300), (9, 3, 300), (16, 2, 700), (16, 3, 700),
])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_leaf_grams_match_oracle(ftl, R, F, leaves, precision):
    n = leaves * F - (F > 1)
    rng = np.random.default_rng(n + R)
    U = rng.normal(size=(n, R))
    U[rng.random(n) < 0.02] *= 100.0
    U[rng.random(n) < 0.05] = 0.0
    G, U32 = build(ftl, U, R, F, precision, with_copy=precision == "fp32")
    levels = math.ceil(math.log2(max(2, leaves))) + 1
    tol = 2 * (F + levels) * 2.0 ** -53 if precision == "fp64" else (F + levels + 3) * 2.0 ** -24
    check_close(G, O.tree_build(U, F), R, tol)
    if precision == "fp32":
        assert np.array_equal(U32, U.astype(np.float32))
