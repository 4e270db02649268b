"""A row's result does not depend on the batch it is in: batches on either side of the rules
that set the threads of a row's block, the blocks that share a row and the kernel of a
product give the same bits as a batch that fills the GPU."""
import numpy as np
import pytest
import torch

from roughpy_b200 import _internals as I
from roughpy_b200 import compute as rpc
from tests._util import level_scaled

pytestmark = pytest.mark.gpu

BATCHES = (1, 2, 31, 32, 63, 64, 65, 147, 148, 149, 297, 443, 444, 592, 1185, 1777)
SHAPES = [(2, 3), (2, 8), (2, 11), (3, 2), (3, 5), (3, 7), (4, 4), (4, 6), (5, 3), (5, 5), (6, 4),
          (6, 5), (7, 4), (8, 3), (8, 4), (9, 2), (9, 3), (10, 3), (12, 3), (16, 2)]
LONG = [(2, 13), (3, 9), (4, 7), (5, 6), (6, 6), (7, 5), (8, 5), (9, 4), (12, 4)]
LONGEST = [(4, 8), (5, 7), (7, 6), (8, 6), (16, 4)]


def products(b, c, basis):
    got = {}
    out = b.clone()
    I.dense_ft_fma(out, b, c, basis)
    got["fma"] = out
    got["mul"] = rpc.ft_mul(rpc.FreeTensor(b, basis), rpc.FreeTensor(c, basis)).data
    out = b.clone()
    I.dense_ft_inplace_mul(out, c, basis)
    got["inplace"] = out
    return got


def series(b, c, basis):
    x = c.clone()
    x[:, 0] = 0.0
    return {"exp": rpc.ft_exp(rpc.FreeTensor(x, basis)).data,
            "fmexp": rpc.ft_fmexp(rpc.FreeTensor(b, basis), rpc.FreeTensor(x, basis)).data,
            "log": rpc.ft_log(rpc.FreeTensor(b, basis)).data}


def check(w, d, dtype, batches, calls):
    basis = rpc.TensorBasis(w, d)
    few = 5   # distinct rows
    b, c = (torch.from_numpy(level_scaled(np.random.default_rng(s), w, d, few, True, dtype)).cuda()
            for s in (w, d))
    n = max(batches)
    rows = torch.arange(n, device="cuda") % few
    b, c = b[rows].contiguous(), c[rows].contiguous()
    want = {k: v[:few] for k, v in calls(b, c, basis).items()}
    for m in batches:
        for k, v in calls(b[:m], c[:m], basis).items():
            assert torch.equal(v, want[k][rows[:m]]), (k, m)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("w,d", SHAPES)
def test_short_rows(w, d, dtype):
    check(w, d, dtype, BATCHES + (2500,), products)
    check(w, d, dtype, BATCHES + (2500,), series)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("w,d", LONG)
def test_long_rows(w, d, dtype):
    check(w, d, dtype, BATCHES[:13] + (600,), products)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("w,d", LONGEST)
def test_longest_rows(w, d, dtype):
    check(w, d, dtype, (1, 31, 32, 63, 64, 147, 148, 150), products)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("w,d", [(2, 3), (2, 8), (3, 2), (3, 5), (4, 4), (5, 5), (6, 3), (8, 3)])
def test_queries(w, d, dtype):
    """Batches on either side of the rules of the chain kernel; from some size on the queries
    are also dissected on the device."""
    from roughpy_b200 import streams
    rng = np.random.default_rng(w * d)
    times = np.sort(rng.uniform(0.0, 1.0, 200))
    inc = (0.1 * rng.standard_normal((200, w))).astype(dtype)
    st = streams.LieIncrementStream.from_increments(inc, times, w, d, resolution=7, dtype=dtype)
    a = rng.uniform(0.0, 0.9, 1500)
    b = np.minimum(1.0, a + rng.uniform(0.0, 0.5, 1500))
    want = st.log_signature_batch(a, b)
    for m in (1, 2, 100, 148, 149, 255, 256, 300, 383, 384, 600, 1000):
        assert torch.equal(st.log_signature_batch(a[:m], b[:m]), want[:m]), m
