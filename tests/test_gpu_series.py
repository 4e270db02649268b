"""exp, fmexp and log in the row-resident series kernel against the C oracle at the sizes
where its layout changes: levels shorter than the owned first letters, rows of fewer words than a warp, the largest rows
that stay in shared memory, and a batch on either side of the block-per-row split.

Tolerances: a result word is a sum of at most n = depth + 1 products of terms bounded by
the row's level norms, evaluated in float64 on both sides; the per-level normwise error
of either is below n^2 eps plus the series' own n steps, under 1e-13 for n <= 17 (log's
alternating terms: 1e-12).  Float32 rows add one rounding of the result, 2^-24 = 6e-8,
of the level's largest word: 1e-7.
"""
import numpy as np
import pytest
import torch

import oracle
from roughpy_b200 import _internals as I
from roughpy_b200 import compute as rpc
from tests._util import degree_begin, level_rel_err, level_scaled

pytestmark = pytest.mark.gpu

SHAPES = [(2, 1, 3), (2, 2, 5), (2, 3, 1), (2, 4, 149), (2, 9, 2), (2, 13, 1), (3, 1, 2), (3, 2, 4),
          (3, 5, 33), (3, 8, 2), (4, 2, 7), (4, 5, 3), (5, 3, 150), (5, 5, 2), (6, 4, 3), (6, 6, 1),
          (7, 2, 2), (7, 4, 3), (8, 3, 2), (8, 5, 1), (9, 3, 2), (16, 2, 3), (3, 9, 1)]


def _rows(w, d, batch, dtype, seed, unit):
    x = level_scaled(np.random.default_rng(seed), w, d, batch, unit, dtype)
    return x, torch.from_numpy(x).cuda()


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("w,d,batch", SHAPES)
def test_series_against_oracle(w, d, batch, dtype):
    basis = rpc.TensorBasis(w, d)
    tol = 1e-13 if dtype == np.float64 else 1e-7
    if (w, d) == (3, 9):
        # past the shared-memory limit: one product launch a step, each rounding float32
        # rows (the tolerance of those launches' own tests)
        tol = 1e-13 if dtype == np.float64 else 2e-6
    log_tol = 1e-12 if dtype == np.float64 else 1e-7
    x, xd = _rows(w, d, batch, dtype, 1, True)
    m, md = _rows(w, d, batch, dtype, 2, True)
    for out_depth in sorted({-1, d - 1, 1}):
        if out_depth == 0:
            continue
        top = d if out_depth < 0 else out_depth
        keep = degree_begin(w, d)[top + 1]
        got = torch.full_like(xd, 7.0)
        I.dense_ft_exp(got, xd, basis, out_depth)
        g = got.cpu().numpy()
        want = oracle.ft_exp(w, d, x, out_depth)
        assert level_rel_err(g[:, :keep], want[:, :keep], w, top) <= tol
        assert np.all(g[:, keep:] == 7.0)      # levels above the requested one are untouched
        got.fill_(7.0)
        I.dense_ft_fmexp(got, md, xd, basis, out_depth)
        g = got.cpu().numpy()
        want = oracle.ft_fmexp(w, d, m, x, out_depth)
        assert level_rel_err(g[:, :keep], want[:, :keep], w, top) <= tol
        assert np.all(g[:, keep:] == 7.0)
        for arg_depth in sorted({-1, max(1, d - 1)}):
            got.fill_(0.0)
            got[:, 0] = 0.25                    # the incoming scalar joins the first coefficient
            init = got.cpu().numpy()
            I.dense_ft_log(got, xd, basis, out_depth, arg_depth)
            want = oracle.ft_log(w, d, x, out_depth, arg_depth, init)
            g = got.cpu().numpy()
            assert level_rel_err(g[:, :keep], want[:, :keep], w, top) <= log_tol
            assert np.all(g[:, keep:] == 0.0)
