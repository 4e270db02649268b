"""Queries on either side of the batch sizes from which they are dissected on the device, with
and without the range table: the edge cases of test_gpu_device_dissection, equal bit for bit
to the same queries asked a few at a time."""
import numpy as np
import pytest
import torch

from tests.test_gpu_device_dissection import _queries, _stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["f64", "f32c"])
@pytest.mark.parametrize("table", [False, True])
@pytest.mark.parametrize("res,lo,hi", [(9, 0.0, 8.0), (6, -3.0, 5.5), (3, -700.25, 900.0)])
def test_batches_around_the_device_rule(res, lo, hi, table, mode):
    st = _stream(res, lo, hi, mode)
    st.auto_range_table = False
    if table:
        st.build_range_table()
    a, b = (np.tile(x, 2) for x in _queries(res, lo, hi))
    for q in (None, res, res - 2, res + 3):
        want = torch.cat([st.log_signature_batch(a[i:i + 100], b[i:i + 100], resolution=q)
                          for i in range(0, len(a), 100)])
        for n in (399, 400, 599, 600, 800):
            assert torch.equal(st.log_signature_batch(a[:n], b[:n], resolution=q), want[:n])
