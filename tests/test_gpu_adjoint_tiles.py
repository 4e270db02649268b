"""The adjoint of left multiplication at 64 rows of long outputs with few terms: bounded
degrees make the staged words of a row few although its result is long, so that the
row-per-block form runs at the batch where unstaged rows change their tile width.

Tolerance: a word is a sum of at most T <= 2^16 terms added in float64, T eps <= 1e-11 of
their absolute sum, which for these inputs exceeds a level's largest word by less than 1e2:
1e-9.  Float32 rows: the same sums of exact products rounded once, 6e-8 of the level's
largest word, below 1e-6 with the margin.
"""
import ctypes

import numpy as np
import pytest
import torch

import oracle
from roughpy_b200 import _internals as I
from roughpy_b200 import _lib
from roughpy_b200 import compute as rpc
from tests._strict import strict_level_rel_err
from tests._util import level_scaled

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [63, 64, 65])
@pytest.mark.parametrize("w,d,dtype,depths", [
    (4, 7, np.float32, (-1, 1, -1)), (4, 7, np.float64, (-1, -1, 6)),
    (7, 5, np.float32, (-1, 1, -1)), (7, 5, np.float64, (-1, -1, 4)),
    (8, 5, np.float64, (-1, -1, 4)), (2, 14, np.float32, (-1, 2, -1)),
    (4, 7, np.float32, (-1, -1, -1))])
def test_bounded_adjoint_around_64_rows(w, d, dtype, depths, batch):
    basis = rpc.TensorBasis(w, d)
    tol = 1e-9 if dtype == np.float64 else 1e-6
    op = level_scaled(np.random.default_rng(5), w, d, batch, True, dtype)
    arg = level_scaled(np.random.default_rng(6), w, d, batch, True, dtype)
    opd, argd = torch.from_numpy(op).cuda(), torch.from_numpy(arg).cuda()
    want = oracle.adjoint_left_mul(w, d, op, arg, *depths)
    got = torch.zeros_like(argd)
    I.dense_ft_adjoint_left_mul(got, opd, argd, basis, *depths)
    assert strict_level_rel_err(got.cpu().numpy(), want, w, d) <= tol
    # the fresh entry writes every word
    got = torch.full_like(argd, float("nan"))
    T = basis.size()
    code = _lib.F64 if dtype == np.float64 else _lib.F32
    _lib.check(_lib.lib.rpyb_ft_adjoint_left_mul_fresh(
        code, w, d, batch, got.data_ptr(), opd.data_ptr(), argd.data_ptr(), T, T, T,
        (ctypes.c_int32 * 3)(*depths), torch.cuda.current_stream().cuda_stream))
    assert strict_level_rel_err(got.cpu().numpy(), want, w, d) <= tol
