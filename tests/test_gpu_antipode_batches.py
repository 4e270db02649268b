"""The antipode of batches on either side of the number of words from which the upper levels
go through tiles: the signed reversal, exactly."""
import numpy as np
import pytest
import torch

from roughpy_b200 import compute as rpc
from tests.test_gpu_antipode import _reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("w,d", [(2, 10), (2, 13), (3, 6), (3, 8), (4, 6), (4, 7), (5, 4), (5, 6),
                                 (6, 4), (6, 5), (7, 4), (7, 5), (8, 4), (8, 5), (9, 4)])
def test_antipode_on_both_sides_of_the_rule(w, d, dtype):
    basis = rpc.TensorBasis(w, d)
    T = basis.size()
    x = np.random.default_rng(w + d).standard_normal((5, T)).astype(dtype)
    want = torch.from_numpy(_reference(x, w, d)).cuda()
    xd = torch.from_numpy(x).cuda()
    edge = -(-(1 << 19) // T)   # the first batch of 2^19 words or more
    for n in (1, 2, edge - 1, edge, edge + 1):
        rows = torch.arange(n, device="cuda") % 5
        got = rpc.antipode(rpc.FreeTensor(xd[rows].contiguous(), basis)).data
        assert torch.equal(got, want[rows]), n
