"""Results into memory full of NaN against the C oracle: every word that a fresh result has to
hold is written, by every kernel that the shapes and batches reach (row-resident, slabs,
blocked, launch a step, packed map and CSR).

Tolerances: a product's word is a sum of at most 17 terms in float64, a series has at most 16
such steps: 16 * 17 * 1.1e-16 = 3e-14 of the terms' absolute sum, which for these inputs
(level k scaled by 1/k!) exceeds a level's largest word by less than 1e2: 1e-11; adjoints as
in test_gpu_adjoint_left_mul, 1e-9.  Float32 rows: products, logs, adjoints and maps round
float64 sums once, 6e-8 of a level's largest word, 1e-6 with the margin; exp and fmexp by a
launch a step round every step, 16 * 6e-8 = 1e-6 of the absolute sum: 1e-4."""
import ctypes

import numpy as np
import pytest
import torch

import oracle
from roughpy_b200 import _internals as I
from roughpy_b200 import _lib
from roughpy_b200 import compute as rpc
from tests._strict import strict_level_rel_err
from tests._util import degree_begin, level_scaled

pytestmark = pytest.mark.gpu

SHAPES = [(1, 3, 4), (2, 0, 3), (2, 3, 5), (2, 8, 150), (2, 14, 2), (3, 4, 1200), (3, 9, 3), (4, 7, 2),
          (4, 8, 64), (5, 5, 149), (6, 6, 2), (6, 6, 64), (7, 3, 40), (8, 4, 150), (9, 3, 5),
          (9, 4, 150), (12, 3, 700), (16, 4, 2)]


def _inputs(w, d, n, dtype):
    few = min(n, 6)
    rows = np.arange(n) % few
    b, c = (level_scaled(np.random.default_rng(s), w, d, few, True, dtype) for s in (1, 2))
    x = c.copy()
    x[:, 0] = 0.0
    dev = [torch.from_numpy(v[rows]).cuda() for v in (b, c, x)]
    return rows, (b, c, x), dev


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("w,d,n", SHAPES)
def test_every_word_is_written(w, d, n, dtype):
    basis = rpc.TensorBasis(w, d)
    rows, (b, c, x), (bd, cd, xd) = _inputs(w, d, n, dtype)
    f64 = dtype == np.float64

    def check(call, want, tol):
        out = torch.full_like(bd, float("nan"))
        call(out)
        assert strict_level_rel_err(out.cpu().numpy(), want[rows], w, d) <= tol

    tol = 1e-11 if f64 else 1e-6
    check(lambda o: I.ft_mul_into(o, bd, cd, basis), oracle.ft_mul(w, d, b, c), tol)
    check(lambda o: I.ft_log_into(o, bd, basis), oracle.ft_log(w, d, b), tol)
    check(lambda o: I.ft_adjoint_left_mul_into(o, bd, cd, basis),
          oracle.adjoint_left_mul(w, d, b, c), 1e-9 if f64 else tol)
    check(lambda o: I.dense_ft_antipode(o, bd, basis), oracle.antipode(w, d, b), 0.0)
    tol = 1e-11 if f64 else 1e-4
    check(lambda o: I.dense_ft_exp(o, xd, basis), oracle.ft_exp(w, d, x), tol)
    check(lambda o: I.dense_ft_fmexp(o, bd, xd, basis), oracle.ft_fmexp(w, d, b, x), tol)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("bounds", [(0, 3, 0, 5, 0, 5), (0, 5, 1, 4, 2, 5), (2, 4, 0, 1, 0, 2),
                                    (1, 5, 3, 5, 3, 5), (0, 5, 0, 0, 0, 5)])
@pytest.mark.parametrize("w", [2, 4, 6])
def test_bounded_products_write_their_levels(w, bounds, dtype):
    d, n = 5, 7
    db = degree_begin(w, d)
    rows, (b, c, _), (bd, cd, _) = _inputs(w, d, n, dtype)
    T = bd.shape[1]
    out = torch.full_like(bd, float("nan"))
    code = _lib.F64 if dtype == np.float64 else _lib.F32
    _lib.check(_lib.lib.rpyb_ft_mul(code, w, d, n, out.data_ptr(), bd.data_ptr(), cd.data_ptr(), T, T,
                                    T, (ctypes.c_int32 * 6)(*bounds),
                                    torch.cuda.current_stream().cuda_stream))
    want = oracle.ft_fma(w, d, np.zeros_like(b), b, c, bounds)[rows]
    got = out.cpu().numpy()
    c0, c1 = db[bounds[0]], db[bounds[1] + 1]
    assert np.all(np.isnan(got[:, :c0])) and np.all(np.isnan(got[:, c1:]))
    got[:, :c0] = 0.0
    got[:, c1:] = 0.0
    assert strict_level_rel_err(got, want, w, d) <= (1e-11 if dtype == np.float64 else 1e-6)


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("w,d,n", [(2, 3, 1), (2, 6, 40), (3, 4, 700), (5, 4, 9), (6, 3, 2500)])
def test_maps_write_every_word(w, d, n, dtype):
    """Against the dense matrix in float64: sums of at most 2^8 entries, 3e-14 of their absolute
    sum, or float32's 6e-8 of it; bounds 1e-12 and 1e-6 of the largest absolute sum."""
    lb, tb = rpc.LieBasis(w, d), rpc.TensorBasis(w, d)
    g = torch.Generator(device="cuda").manual_seed(4)
    tol = 1e-12 if dtype == torch.float64 else 1e-6
    for m in (lb.get_l2t_matrix(np.float64), lb.get_t2l_matrix(np.float64)):
        dense = torch.from_numpy(m.todense()).cuda()
        x = torch.randn(n, m.shape[1], device="cuda", dtype=dtype, generator=g)
        want = x.double() @ dense.T
        size = float((x.double().abs() @ dense.abs().T).max())
        for _ in range(3):            # the CSR form, then the packed one
            out = torch.full((n, m.shape[0]), float("nan"), device="cuda", dtype=dtype)
            I.lie_map_into(out, x, m)
            assert bool(torch.isfinite(out).all())
            assert float((out.double() - want).abs().max()) <= tol * size
    assert tb.size() == dense.shape[1]
