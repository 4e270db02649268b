"""Calls of one width and several depths from several host threads, each on its own stream:
the kernels they share take different amounts of shared memory, above the 48 KB that need
leave, and no call may take that leave back from another.  Every call must succeed and give
the result that it gives alone, bit for bit."""
import threading

import pytest
import torch

from roughpy_b200 import _lib
from roughpy_b200 import compute as rpc

pytestmark = pytest.mark.gpu

CALLS = 4000


def _fma(w, d, n, o, a, b, ws, s):
    T = o.shape[1]
    return _lib.lib.rpyb_ft_fma(_lib.F64, w, d, n, o.data_ptr(), a.data_ptr(), b.data_ptr(), T, T,
                                T, None, s)


def _exp(w, d, n, o, a, b, ws, s):
    T = o.shape[1]
    return _lib.lib.rpyb_ft_exp(_lib.F64, w, d, n, o.data_ptr(), a.data_ptr(), T, T, -1,
                                ws.data_ptr(), ws.numel(), s)


def _adjoint(w, d, n, o, a, b, ws, s):
    T = o.shape[1]
    return _lib.lib.rpyb_ft_adjoint_left_mul_fresh(_lib.F64, w, d, n, o.data_ptr(), a.data_ptr(),
                                                   b.data_ptr(), T, T, T, None, s)


def _project(w, d, n, o, a, b, ws, s):
    T = o.shape[1]
    return _lib.lib.rpyb_tensor_to_lie(_lib.F64, w, d, n, o.data_ptr(), T, a.data_ptr(), T, s)


@pytest.mark.parametrize("call,depths,w,n", [
    (_fma, (12, 13), 2, 150), (_exp, (12, 13), 2, 150), (_adjoint, (10, 11), 2, 64),
    (_project, (12, 13), 2, 1)])
def test_depths_of_one_width_from_several_threads(call, depths, w, n):
    failed, done = [], []

    def work(d, seed):
        g = torch.Generator(device="cuda")
        g.manual_seed(seed)
        T = rpc.TensorBasis(w, d).size()
        a, b = (torch.randn(n, T, device="cuda", dtype=torch.float64, generator=g) for _ in "ab")
        o = torch.zeros_like(a)
        ws = torch.empty(n * T * 8, device="cuda", dtype=torch.uint8)
        st = torch.cuda.Stream()
        st.wait_stream(torch.cuda.current_stream())
        for _ in range(CALLS):
            rc = call(w, d, n, o, a, b, ws, st.cuda_stream)
            if rc:
                failed.append((d, rc, _lib.lib.rpyb_last_error()))
                break
        st.synchronize()
        if call is _fma:      # accumulates: one call from zero is compared
            o.zero_()
            torch.cuda.synchronize()
            failed.extend([(d, "again")] if call(w, d, n, o, a, b, ws, st.cuda_stream) else [])
            st.synchronize()
        done.append((d, a, b, o))

    threads = [threading.Thread(target=work, args=(depths[i % len(depths)], i)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
    s = torch.cuda.current_stream().cuda_stream
    for d, a, b, o in done:
        want = torch.zeros_like(o)
        ws = torch.empty(o.numel() * 8, device="cuda", dtype=torch.uint8)
        assert call(w, d, n, want, a, b, ws, s) == 0
        assert torch.equal(o, want)
