"""The adjoint of left multiplication on the longest rows a tensor may have, just under 2^31
words, where an index of level 0's sum passes the largest 32-bit integer.  Whole numbers in
float32: the comparison is exact."""
import pytest
import torch

from roughpy_b200 import _internals as I
from roughpy_b200 import compute as rpc

pytestmark = pytest.mark.gpu


def test_adjoint_of_a_row_of_nearly_2_31_words():
    width = 2 ** 31 - 3
    T = width + 1
    if torch.cuda.mem_get_info()[0] < 3.5 * 4 * T:
        pytest.skip("needs 30 GB of device memory")
    op = torch.zeros(T, device="cuda", dtype=torch.float32)
    arg = torch.zeros(T, device="cuda", dtype=torch.float32)
    # words on either side of the last full step of 1024 slices of eight terms
    places = torch.tensor([0, 1, 1023, 8192, T // 2, T - 9000, T - 8192, T - 7168, T - 1025,
                           T - 1024, T - 2, T - 1], device="cuda")
    value = torch.arange(1, places.numel() + 1, device="cuda", dtype=torch.float32)
    op[places] = value
    arg[places] = value
    out = torch.zeros_like(arg)
    I.dense_ft_adjoint_left_mul(out, op, arg, rpc.TensorBasis(width, 1))
    assert out[0].item() == (value * value).sum().item()   # every pair of words
    assert torch.equal(out[1:], arg[1:])                   # op's scalar, 1, times the letters
