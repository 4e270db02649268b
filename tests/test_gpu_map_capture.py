"""Lie <-> tensor maps recorded in a CUDA graph after a single call outside it: the map's
arrays that the first call left on the device are what the recorded call uses."""
import pytest
import torch

from roughpy_b200 import compute as rpc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [3, 65536])   # few entries, and enough to pack at once
@pytest.mark.parametrize("warm", [1, 2])
@pytest.mark.parametrize("which", ["lie_to_tensor", "tensor_to_lie"])
def test_capture_after_few_calls(which, warm, rows):
    lb, tb = rpc.LieBasis(4, 4), rpc.TensorBasis(4, 4)
    n = lb.size() if which == "lie_to_tensor" else tb.size()
    x = torch.randn(rows, n, device="cuda", dtype=torch.float64)

    def call(x):
        if which == "lie_to_tensor":
            return rpc.lie_to_tensor(rpc.Lie(x, lb), tb).data
        return rpc.tensor_to_lie(rpc.FreeTensor(x, tb), lb).data

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(warm):
            call(x)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = call(x)
    x.copy_(torch.randn_like(x))
    graph.replay()
    want = call(x.clone())
    assert torch.allclose(got, want, rtol=1e-13, atol=1e-13)   # the two maps' terms are the same
