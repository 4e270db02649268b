"""The adjoint of left multiplication against the C oracle where its layouts change: rows
of fewer words than a warp, a warp's and a block's rows on either side of 1024 words, rows
too long for shared memory, batches on either side of the row-per-warp and row-per-block
rules, and truncated degrees.

Tolerance: an output word is a sum of up to T terms; T eps <= 2^16 * 1.1e-16 < 1e-11 of the
sum of absolute values, which for these inputs (random signs, level k scaled by 1/k!)
exceeds a level's largest word by less than 1e2: 1e-9.  Float32 rows: float64 sums of exact
products, rounded once, 6e-8 of the level's largest word and below 1e-6 with the margin.
"""
import numpy as np
import pytest
import torch

import oracle
from roughpy_b200 import _internals as I
from roughpy_b200 import compute as rpc
from tests._util import level_rel_err, level_scaled

pytestmark = pytest.mark.gpu

SHAPES = [(2, 1, 3), (2, 2, 5), (2, 4, 149), (2, 9, 2), (2, 10, 3), (2, 13, 1), (2, 15, 1),
          (3, 2, 4), (3, 3, 1200), (3, 5, 33), (3, 8, 2), (4, 2, 7), (4, 5, 64), (4, 7, 65),
          (5, 3, 150), (5, 4, 70), (6, 4, 63), (7, 4, 3), (8, 3, 1184), (8, 5, 1), (9, 3, 2),
          (16, 2, 3), (20, 2, 2)]


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("w,d,batch", SHAPES)
def test_adjoint_left_mul_against_oracle(w, d, batch, dtype):
    basis = rpc.TensorBasis(w, d)
    tol = 1e-9 if dtype == np.float64 else 1e-6
    op = level_scaled(np.random.default_rng(3), w, d, batch, True, dtype)
    arg = level_scaled(np.random.default_rng(4), w, d, batch, True, dtype)
    opd, argd = torch.from_numpy(op).cuda(), torch.from_numpy(arg).cuda()
    for depths in sorted({(-1, -1, -1), (max(0, d - 1), -1, -1), (-1, 1, -1), (-1, 0, max(0, d - 1))}):
        got = torch.zeros_like(argd)
        I.dense_ft_adjoint_left_mul(got, opd, argd, basis, *depths)
        want = oracle.adjoint_left_mul(w, d, op, arg, *depths)
        assert level_rel_err(got.cpu().numpy(), want, w, d) <= tol
