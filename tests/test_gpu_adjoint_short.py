"""The adjoint of left multiplication of short rows, on either side of the batch and the row
length from which a thread has a whole word's sum, against the C oracle.

Tolerance: a sum of at most 85 terms in float64, 85 * 1.1e-16 < 1e-14 of their absolute sum,
which for these inputs exceeds a level's largest word by less than 1e2: 1e-12.  Float32 rows:
the same sums of exact products rounded once, 6e-8, below 1e-6 with the margin."""
import numpy as np
import pytest
import torch

import oracle
from roughpy_b200 import _internals as I
from roughpy_b200 import compute as rpc
from tests._strict import strict_level_rel_err
from tests._util import level_scaled

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("w,d", [(2, 0), (2, 1), (2, 2), (2, 4), (2, 5), (3, 1), (3, 2), (3, 3),
                                 (4, 2), (4, 3), (6, 2), (7, 1), (8, 1), (8, 2), (63, 1), (64, 1)])
def test_short_rows(w, d, dtype):
    basis = rpc.TensorBasis(w, d)
    few, tol = 7, 1e-12 if dtype == np.float64 else 1e-6
    op = level_scaled(np.random.default_rng(8), w, d, few, True, dtype)
    arg = level_scaled(np.random.default_rng(9), w, d, few, True, dtype)
    for depths in sorted({(-1, -1, -1), (max(0, d - 1), -1, -1), (-1, 0, -1), (-1, -1, max(0, d - 1))}):
        want = oracle.adjoint_left_mul(w, d, op, arg, *depths)
        for n in (1, 3, 1183, 1184, 5000):
            rows = np.arange(n) % few
            opd, argd = (torch.from_numpy(x[rows]).cuda() for x in (op, arg))
            got = torch.zeros_like(argd)
            I.dense_ft_adjoint_left_mul(got, opd, argd, basis, *depths)
            assert strict_level_rel_err(got.cpu().numpy(), want[rows], w, d) <= tol
    got = rpc.ft_adjoint_left_mul(rpc.FreeTensor(opd, basis), rpc.ShuffleTensor(argd, basis)).data
    want = oracle.adjoint_left_mul(w, d, op, arg)
    assert strict_level_rel_err(got.cpu().numpy(), want[rows], w, d) <= tol
