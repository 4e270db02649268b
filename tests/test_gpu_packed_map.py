"""The packed sparse map against the CSR map at the sizes where its layout changes: one
row and just over a warp's, the sort window, rows staged eight, four, two and one a block
and not staged, and batches with a remainder; with empty rows, columns outside the
matrix, and infinities and NaN beside them.

Both sum a row's terms in the CSR order in float64 and round once, so the results are
equal bit for bit; `scale` multiplies the sum in both.
"""
import ctypes

import numpy as np
import pytest
import torch

from roughpy_b200 import _internals as I
from roughpy_b200 import _lib

pytestmark = pytest.mark.gpu


def _matrix(rows, cols, seed):
    rng = np.random.default_rng(seed)
    counts = rng.integers(0, 9, rows)
    counts[rng.integers(0, rows)] = 40
    ptr = np.concatenate([[0], np.cumsum(counts)])
    idx = rng.integers(0, cols, int(ptr[-1]))
    idx[::17] = cols + 3          # outside the matrix: left out by both maps
    val = rng.choice([-2.0, -1.0, 0.5, 1.0 / 3.0, 1.0], int(ptr[-1]))
    return I.SparseMatrix(ptr, idx, val, (rows, cols))


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("rows,cols,batch", [
    (1, 1, 1), (33, 5, 3), (512, 40, 1), (513, 1500, 2400), (100, 3000, 1200), (70, 6000, 600),
    (1000, 20000, 5), (65, 30000, 4), (2000, 17, 9001)])
def test_packed_map_equals_csr_map(rows, cols, batch, dtype):
    m = _matrix(rows, cols, rows)
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn(batch, cols + 2, dtype=dtype, device="cuda", generator=g)
    x[0, 0] = float("inf")        # reaches the rows that name it, and no padded entry's row
    x[-1, cols - 1] = float("nan")
    y = torch.randn(batch, rows + 3, dtype=dtype, device="cuda", generator=g)
    code = _lib.F64 if dtype == torch.float64 else _lib.F32
    ptr, idx, val = m.device_arrays(x.device)
    block, layout = m.device_packed(x.device)
    s = torch.cuda.current_stream().cuda_stream
    for accumulate in (1, 0):
        want = y.clone()
        if not accumulate:
            want[:, :rows] = 0
        _lib.check(_lib.lib.rpyb_sparse_map(code, rows, cols, batch, ptr.data_ptr(), idx.data_ptr(),
                                            val.data_ptr(), want.data_ptr(), x.data_ptr(),
                                            rows + 3, cols + 2, 0.75, s))
        got = y.clone()
        _lib.check(_lib.lib.rpyb_sparse_map_packed(code, rows, cols, batch, block.data_ptr(),
                                                   layout, got.data_ptr(), x.data_ptr(), rows + 3,
                                                   cols + 2, 0.75, accumulate, s))
        assert torch.equal(torch.nan_to_num(got, 7.0), torch.nan_to_num(want, 7.0))
        assert torch.equal(got.isnan(), want.isnan())


def test_pack_refuses_what_does_not_fit():
    layout = (ctypes.c_int64 * 3)()
    many = I.SparseMatrix([0, 5000], np.arange(5000), np.arange(5000) + 0.5, (1, 5000))
    wide = I.SparseMatrix([0, 1], [0], [1.0], (1, (1 << 20) + 1))
    room = np.empty(1 << 20, dtype=np.uint8)
    for m in (many, wide):
        assert m.device_packed("cuda") is None
        assert _lib.lib.rpyb_sparse_pack(*m.shape, m.indptr.ctypes.data, m.indices.ctypes.data,
                                         m.data.ctypes.data, room.ctypes.data, room.size,
                                         layout) == _lib.E_UNSUPPORTED
