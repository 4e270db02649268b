"""The forms that wholly write their result against the accumulating forms on zeroed
results: equal bit for bit whatever the result held before (here NaN), at depths 0 and 1,
on every product kernel, with a truncated right factor, and on both sides of the
row-resident log."""
import numpy as np
import pytest
import torch

from roughpy_b200 import _internals as I
from roughpy_b200 import compute as rpc
from tests._util import level_scaled

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("w,d,batch", [(3, 0, 2), (2, 1, 3), (2, 6, 5), (2, 11, 2), (3, 4, 1),
                                       (5, 3, 9), (7, 3, 2), (8, 4, 2), (9, 2, 4), (2, 14, 1)])
def test_fresh_forms(w, d, batch, dtype):
    basis = rpc.TensorBasis(w, d)
    x, y = (torch.from_numpy(level_scaled(np.random.default_rng(s), w, d, batch, True, dtype)).cuda()
            for s in (1, 2))
    nan = lambda: torch.full_like(x, float("nan"))
    for rd in sorted({-1, d // 2}):
        want, got = torch.zeros_like(x), nan()
        I.dense_ft_fma(want, x, y, basis, rhs_depth=rd)
        I.ft_mul_into(got, x, y, basis, rd)
        assert torch.equal(got, want)
    want, got = torch.zeros_like(x), nan()
    I.dense_ft_log(want, x, basis)
    I.ft_log_into(got, x, basis)
    assert torch.equal(got, want)
    want, got = torch.zeros_like(x), nan()
    I.dense_ft_adjoint_left_mul(want, x, y, basis)
    I.ft_adjoint_left_mul_into(got, x, y, basis)
    assert torch.equal(got, want)


def test_rows_longer_than_the_tensor_keep_zeros_beyond_it():
    basis = rpc.TensorBasis(2, 2)
    data = torch.ones(3, basis.size() + 2, dtype=torch.float64, device="cuda")
    x = rpc.FreeTensor(data, basis)
    for r in (rpc.ft_mul(x, x), rpc.antipode(x), rpc.ft_adjoint_left_mul(x, x)):
        assert r.data.shape == data.shape
        assert not r.data[:, basis.size():].any()
