"""The row-resident product kernel: the same bits as the suffix kernel (which adds the same
terms in the same order; RPYB_PRODUCT_BLOCKED=0 is read once per process, so its results
come from a child process), at depths below the owned first letters, the deepest tops whose
lower levels fit in shared memory for every width, and batches on either side of a block a
row; float32, float64, mixed and gathered rows; and in place, with the rows of the factors
apart, the same, or reaching into one another."""
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SHAPES = [(2, 1, 3), (2, 2, 4), (2, 3, 2), (2, 7, 150), (2, 13, 1), (3, 1, 2), (3, 2, 5), (3, 6, 3),
          (3, 9, 1), (4, 1, 3), (4, 5, 149), (4, 7, 2), (5, 2, 3), (5, 6, 1), (6, 3, 4), (6, 6, 2),
          (7, 5, 1), (7, 2, 9), (8, 5, 2), (8, 3, 150), (9, 4, 2), (10, 5, 1), (16, 2, 3),
          (4, 8, 64), (5, 7, 64), (5, 7, 2), (7, 6, 65), (8, 6, 64)]   # 64 rows on: slabs


def compute_all():
    from roughpy_b200 import _internals as I
    from roughpy_b200 import _lib
    from roughpy_b200 import compute as rpc
    from tests._util import level_scaled
    res = {}
    for w, d, n in SHAPES:
        basis = rpc.TensorBasis(w, d)
        for dt in (np.float64, np.float32):
            rng = np.random.default_rng(7 + d)
            a, b, c = (torch.from_numpy(level_scaled(rng, w, d, n, True, dt)).cuda()
                       for _ in range(3))
            # rows one word apart from their size: every alignment of a row's start
            pad = torch.zeros(n, basis.size() + 1, dtype=a.dtype, device="cuda")
            pad[:, :-1] = b
            t = f"w{w}d{d}_{np.dtype(dt).name}"
            got = a.clone()
            I.dense_ft_fma(got, b, c, basis)
            res[t + "_fma"] = got
            res[t + "_mul"] = rpc.ft_mul(rpc.FreeTensor(b, basis), rpc.FreeTensor(c, basis)).data
            got = b.clone()
            I.dense_ft_inplace_mul(got, c, basis)
            res[t + "_inplace"] = got
            if d > 1:
                got = b.clone()
                I.dense_ft_inplace_mul(got, c, basis, d - 1)
                res[t + "_inplace_short"] = got
            code = _lib.F64 if dt == np.float64 else _lib.F32
            s = torch.cuda.current_stream().cuda_stream
            idx = torch.arange(n - 1, -1, -1, device="cuda")
            out = torch.zeros_like(pad)
            T1 = basis.size() + 1
            _lib.check(_lib.lib.rpyb_ft_mul_gather(code, w, d, n, out.data_ptr(), pad.data_ptr(),
                                                   pad.data_ptr(), T1, idx.data_ptr(), None,
                                                   idx.data_ptr(), 0, s))
            res[t + "_gather"] = out
            if dt == np.float64:
                out = pad.clone()
                pad32 = pad.float()
                _lib.check(_lib.lib.rpyb_ft_mul_gather_mixed(
                    w, d, n, out.data_ptr(), pad.data_ptr(), pad32.data_ptr(), T1, None,
                    idx.data_ptr(), None, 1, s))
                res[t + "_mixed"] = out
    return {k: v.cpu().numpy() for k, v in res.items()}


def test_row_kernel_equals_suffix_kernel_bitwise(tmp_path):
    out = tmp_path / "suffix.npz"
    code = (f"import sys; sys.path.insert(0, {ROOT!r}); import numpy as np; "
            f"from tests.test_gpu_product_rows import compute_all; "
            f"np.savez({str(out)!r}, **compute_all())")
    env = dict(os.environ, RPYB_PRODUCT_BLOCKED="0")
    subprocess.run([sys.executable, "-c", code], cwd=ROOT, env=env, check=True, timeout=600)
    want, got = np.load(out), compute_all()
    assert set(want.files) == set(got)
    for k in got:
        assert np.array_equal(got[k], want[k]), k


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_in_place_with_related_rows(dtype):
    from roughpy_b200 import _internals as I
    from roughpy_b200 import _lib
    from roughpy_b200 import compute as rpc
    w, d, n = 3, 5, 40
    basis = rpc.TensorBasis(w, d)
    T = basis.size()
    code = _lib.F64 if dtype == torch.float64 else _lib.F32
    x = torch.randn(n, T, dtype=dtype, device="cuda", generator=torch.Generator("cuda").manual_seed(3))

    def fresh(a, b):
        out = torch.zeros_like(a)
        I.dense_ft_fma(out, a.contiguous(), b.contiguous(), basis)
        return out

    got = x.clone()                       # the same rows: x <- x (x) x
    I.dense_ft_inplace_mul(got, got, basis)
    assert torch.equal(got, fresh(x, x))
    # rows reaching into one another: every row times the old row before it
    got = x.clone()
    ws = torch.empty(n * T * 8, dtype=torch.uint8, device="cuda")
    _lib.check(_lib.lib.rpyb_ft_inplace_mul(
        code, w, d, n - 1, got[1:].data_ptr(), got.data_ptr(), T, T, None, ws.data_ptr(),
        ws.numel(), torch.cuda.current_stream().cuda_stream))
    assert torch.equal(got[1:], fresh(x[1:], x[:-1]))
    assert torch.equal(got[0], x[0])
