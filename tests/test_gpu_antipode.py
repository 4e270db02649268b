"""The antipode against a plain transposition of each level's letters (a permutation with a
sign: equal bit for bit), at depths on either side of the tiled levels for every width, odd
batches, row strides above the tensor's size, and twice over, which is the identity."""
import numpy as np
import pytest
import torch

from roughpy_b200 import _lib
from roughpy_b200 import compute as rpc
from tests._util import degree_begin

pytestmark = pytest.mark.gpu


def _reference(x, w, d):
    db, out = degree_begin(w, d), np.empty_like(x)
    for k in range(d + 1):
        t = x[:, db[k]:db[k + 1]].reshape([x.shape[0]] + [w] * k)
        t = t.transpose([0] + list(range(k, 0, -1))).reshape(x.shape[0], -1)
        out[:, db[k]:db[k + 1]] = -t if k % 2 else t
    return out


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("w,d,batch", [
    (2, 0, 3), (2, 9, 3), (2, 10, 2), (2, 13, 1), (3, 5, 7), (3, 6, 3), (3, 8, 2), (4, 5, 3),
    (4, 6, 2), (4, 7, 1), (5, 3, 5), (5, 4, 3), (5, 6, 1), (6, 4, 2), (6, 5, 1), (7, 4, 2),
    (7, 5, 1), (8, 3, 3), (8, 4, 2), (8, 5, 1), (9, 3, 2), (12, 4, 1)])
def test_antipode_is_the_signed_reversal(w, d, batch, dtype):
    basis = rpc.TensorBasis(w, d)
    T = basis.size()
    x = np.random.default_rng(w + d).standard_normal((batch, T)).astype(dtype)
    xd = torch.from_numpy(x).cuda()
    got = rpc.antipode(rpc.FreeTensor(xd, basis))
    assert np.array_equal(got.data.cpu().numpy(), _reference(x, w, d))
    assert torch.equal(rpc.antipode(got).data, xd)
    wide_in = torch.zeros(batch, T + 3, dtype=xd.dtype, device="cuda")
    wide_in[:, :T] = xd
    wide_out = torch.full((batch, T + 1), 7.0, dtype=xd.dtype, device="cuda")
    code = _lib.F64 if dtype == np.float64 else _lib.F32
    _lib.check(_lib.lib.rpyb_ft_antipode(code, w, d, batch, wide_out.data_ptr(), wide_in.data_ptr(),
                                         T + 1, T + 3, torch.cuda.current_stream().cuda_stream))
    assert torch.equal(wide_out[:, :T], got.data)
    assert (wide_out[:, T] == 7.0).all()
