"""Interval batches with fewer ends than starts are refused on the host: the library takes one
of each a query."""
import numpy as np
import pytest

from roughpy_b200 import streams


class Recorder(streams._StreamQueries):
    """A stream whose queries are only counted."""
    device = "cpu"

    def __init__(self):
        from roughpy_b200 import compute as rpc
        self.lie_basis, self.tensor_basis = rpc.LieBasis(2, 2), rpc.TensorBasis(2, 2)
        self.asked = []

    def _query(self, infs, sups, resolution, logsig=True, sig=False, out=None):
        self.asked.append((len(infs), len(sups)))


@pytest.mark.parametrize("call", ["log_signature_batch", "signature_batch"])
@pytest.mark.parametrize("n_sup", [0, 1, 4])
def test_fewer_ends_than_starts(call, n_sup):
    st = Recorder()
    with pytest.raises(ValueError):
        getattr(st, call)(np.zeros(5), np.ones(n_sup), chunk=2)
    assert st.asked == []


@pytest.mark.parametrize("cls", [streams.LieIncrementStream, streams.PiecewiseAbelianStream])
def test_query_checks_before_anything_else(cls):
    with pytest.raises(ValueError):
        cls._query(object.__new__(cls), np.zeros(5), np.ones(3), None)


@pytest.mark.parametrize("call", ["log_signature_batch", "signature_batch"])
def test_ends_for_every_start(call):
    st = Recorder()
    assert getattr(st, call)(np.zeros(5), np.ones(5), chunk=2).shape[0] == 5
    assert st.asked == [(2, 2), (2, 2), (1, 1)]
