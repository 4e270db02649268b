"""exp, fmexp and log of a few of the longest rows that run with a runtime width, which take a
launch a step, against the C oracle.

Tolerance: a word of level k <= 4 is a sum of at most 5 terms in each of 4 steps, 20 eps =
2.2e-15 of the terms' absolute sum, which for these inputs (level k scaled by 1/k!) is below
1e2 times a level's largest word: 1e-12.  Float32 log is the same series in float64, rounded
once: 6e-8 of a level's largest word, 1e-6 with the margin."""
import numpy as np
import pytest
import torch

import oracle
from roughpy_b200 import _internals as I
from roughpy_b200 import compute as rpc
from tests._strict import strict_level_rel_err
from tests._util import level_scaled

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 32, 63, 64])
@pytest.mark.parametrize("w", [13, 16])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_few_long_rows(w, n, dtype):
    d, basis = 4, rpc.TensorBasis(w, 4)
    x = level_scaled(np.random.default_rng(w), w, d, n, False, dtype)
    x[:, 0] = 0.0
    y = level_scaled(np.random.default_rng(n), w, d, n, True, dtype)
    xd, yd = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
    tol = 1e-12 if dtype == np.float64 else 1e-6

    def err(got, want):
        return strict_level_rel_err(got.cpu().numpy(), want, w, d)

    assert err(rpc.ft_log(rpc.FreeTensor(yd, basis)).data, oracle.ft_log(w, d, y)) <= tol
    out = torch.full_like(yd, float("nan"))
    out[:, 0] = 0.0                       # dense_ft_log reads its out's scalar
    I.dense_ft_log(out, yd, basis)
    assert err(out, oracle.ft_log(w, d, y)) <= tol
    if dtype == np.float64:
        assert err(rpc.ft_exp(rpc.FreeTensor(xd, basis)).data, oracle.ft_exp(w, d, x)) <= tol
        assert err(rpc.ft_fmexp(rpc.FreeTensor(yd, basis), rpc.FreeTensor(xd, basis)).data,
                   oracle.ft_fmexp(w, d, y, x)) <= tol
