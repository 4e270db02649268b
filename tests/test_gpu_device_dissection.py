"""Queries dissected on the device against the same queries one by one, which the host
dissects: equal bit for bit, with and without the range table, over supports on both sides
of 0, explicit resolutions coarser and finer than the stream's, lengths from one leaf to
the support, empty and outside queries, and ends at every kind of alignment."""
import numpy as np
import pytest
import torch

from roughpy_b200.streams import LieIncrementStream, RealInterval

pytestmark = pytest.mark.gpu


def _stream(res, lo, hi, mode):
    rng = np.random.default_rng(5)
    n = 700
    times = np.sort(rng.uniform(lo, hi, n))
    return LieIncrementStream.from_increments(
        rng.standard_normal((n, 2)) * 0.1, indices=times, width=2, depth=3, resolution=res,
        support=RealInterval(lo, hi), mode=mode)


def _queries(res, lo, hi):
    rng = np.random.default_rng(6)
    step = 2.0 ** -res
    a = rng.uniform(lo - 0.2, hi + 0.2, 400)
    b = rng.uniform(lo - 0.2, hi + 0.2, 400)
    a[100:] = np.round(a[100:] / step) * step            # leaf ends
    b[100:] = np.round(b[100:] / step) * step
    b[200:240] = a[200:240] + step                       # one leaf
    b[240:280] = a[240:280] + step / 4                   # a quarter of one
    b[280:300] = a[280:300]                              # nothing
    a[300:310], b[300:310] = lo, hi
    return np.minimum(a, b), np.maximum(a, b)


@pytest.mark.parametrize("mode", ["f64", "f32c"])
@pytest.mark.parametrize("table", [False, True])
@pytest.mark.parametrize("res,lo,hi", [(9, 0.0, 8.0), (6, -3.0, 5.5), (3, -700.25, 900.0), (12, 0.125, 0.75)])
def test_device_dissection_equals_host(res, lo, hi, table, mode):
    st = _stream(res, lo, hi, mode)
    st.auto_range_table = False
    if table:
        st.build_range_table()
    a, b = _queries(res, lo, hi)
    for q in (None, res, res - 2, res + 3):
        got = st.log_signature_batch(a, b, resolution=q)
        want = torch.cat([st.log_signature_batch(a[i:i + 100], b[i:i + 100], resolution=q)
                          for i in range(0, len(a), 100)])
        assert torch.equal(got, want)
        got = st.signature_batch(a, b, resolution=q)
        want = torch.cat([st.signature_batch(a[i:i + 100], b[i:i + 100], resolution=q)
                          for i in range(0, len(a), 100)])
        assert torch.equal(got, want)


def test_invalid_queries_are_refused_in_large_batches():
    st = _stream(4, 0.0, 1.0, "f64")
    a, b = np.zeros(400), np.ones(400)
    a[399] = 2.0
    with pytest.raises(ValueError):
        st.log_signature_batch(a, b)
    a[399] = np.nan
    with pytest.raises(ValueError):
        st.log_signature_batch(a, b)
    with pytest.raises(ValueError):
        st.log_signature_batch(np.zeros(400), np.ones(400), resolution=70)
