"""GPU: leaf Grams on the CUDA cores, both kernels and every tile shape, against
the CPU oracle's tree.

Tolerances (entrywise, relative to sqrt(G_aa G_bb) of the oracle's node): each
entry sums at most F products and `levels` node sums in the working precision,
one rounding u each on either side; an FP32 tree also rounds the two factors.
  * fp64: 2 (F + levels) 2^-53;
  * fp32: (F + levels + 3) 2^-24.
The FP32 copy is the factor rounded to nearest FP32 exactly."""
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


@pytest.mark.parametrize("n,R,F", [
    (1, 1, 1),            # one row, one column
    (1000, 1, 1),         # one value per row: 64 leaves per CTA
    (5, 3, 3),            # fewer rows than a CTA stages; partial last leaf
    (4097, 4, 4),         # one tile per leaf, no off-diagonal tiles
    (6400, 8, 8),         # whole batches
    (6401, 8, 8),         # last batch of one row
    (3000, 9, 9),         # one column past a tile
    (3001, 16, 16),
    (2500, 20, 20),       # wrapped-diagonal FP32 nodes below 32 columns
    (2511, 25, 25),       # 5 x 5 tiles (FP64)
    (2000, 31, 31),
    (2000, 32, 32),       # rows kernel in both precisions
    (1500, 33, 33),       # one column past eight tiles
    (1500, 35, 35),       # 5 x 5 tiles above 32 columns
    (700, 100, 100),
    (700, 125, 125),
    (1029, 128, 128),     # more tiles than threads
    (64, 128, 64),        # n = F < R
    (1000, 24, 7),        # leaves shorter than R
    (3000, 12, 60),       # leaves longer than R
    (4000, 25, 128),      # the longest leaf
])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_leaf_grams_match_oracle(ftl, n, R, F, precision):
    rng = np.random.default_rng(n + R)
    U = rng.normal(size=(n, R))
    U[rng.random(n) < 0.02] *= 100.0
    U[rng.random(n) < 0.05] = 0.0
    G, U32 = build(ftl, U, R, F, precision, with_copy=precision == "fp32")
    levels = math.ceil(math.log2(max(2, -(-n // F)))) + 1
    tol = 2 * (F + levels) * 2.0 ** -53 if precision == "fp64" else (F + levels + 3) * 2.0 ** -24
    check_close(G, O.tree_build(U, F), R, tol)
    if precision == "fp32":
        assert np.array_equal(U32, U.astype(np.float32))
