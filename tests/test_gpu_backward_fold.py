"""The backward lane kernel's two folding stages at their edges: every number
of fold warps, streams of one to three steps (the hand-over buffers' first
uses), chunk remainders, and fewer blocks than fit.

Bound against float64 autograd: 1e-10 of the largest gradient, that of the
other float64 checks of this kernel (a gradient is a sum of at most 1e5 terms,
each with an error of a few units in the last place: 1e5 * 4 * 1.1e-16 = 5e-11).
How many blocks run changes no sum, so those results are equal bit for bit."""
import numpy as np
import pytest
import torch

from roughpy_b200 import _lib
from roughpy_b200 import signatures as S

pytestmark = pytest.mark.gpu


def reference(inc, w, d):
    sig = [torch.ones(1, dtype=inc.dtype, device=inc.device)]
    sig += [torch.zeros(w ** k, dtype=inc.dtype, device=inc.device) for k in range(1, d + 1)]
    for x in inc:
        ex = [torch.ones(1, dtype=inc.dtype, device=inc.device)]
        for k in range(1, d + 1):
            ex.append(torch.outer(ex[-1], x).reshape(-1) / k)
        sig = [sum(torch.outer(sig[k - j], ex[j]).reshape(-1) for j in range(k + 1))
               for k in range(d + 1)]
    return torch.cat(sig)


# one fold warp with no, one and more levels to fold; three; one stage
@pytest.mark.parametrize("w,d", [(3, 2), (4, 3), (5, 4), (3, 6), (4, 6), (2, 9), (5, 6), (3, 8)])
def test_fold_stages_against_autograd(w, d):
    lens = [1, 2, 3, 0, 33, 5]
    off = S.offsets_from_lengths(lens)
    rng = np.random.default_rng(w + 10 * d)
    inc = torch.from_numpy(rng.normal(0, 0.3, size=(int(off[-1]), w))).cuda()
    G = torch.from_numpy(rng.normal(size=(len(lens), S.tensor_size(w, d)))).cuda()
    plan = S.SignaturePlan(off, w, d, "f64")
    x = inc.clone().requires_grad_(True)
    (S.signature_with_grad(x, plan, checkpoint_every=16) * G).sum().backward()
    y = inc.clone().requires_grad_(True)
    for s in range(len(lens)):
        if lens[s]:
            (reference(y[off[s]:off[s + 1]], w, d) * G[s]).sum().backward()
    assert float((x.grad - y.grad).abs().max()) <= 1e-10 * max(float(y.grad.abs().max()), 1.0)


@pytest.mark.parametrize("w,d,mode", [(3, 4, "f64"), (8, 3, "f32c"), (5, 5, "f32c")])
def test_fewer_blocks_give_the_same_bits(w, d, mode):
    n, K = 1600, 8
    rng = np.random.default_rng(5)
    off = S.offsets_from_lengths([int(v) for v in rng.integers(0, 40, size=n)])
    dt = torch.float64 if mode == "f64" else torch.float32
    inc = torch.from_numpy(rng.normal(0, 0.3, size=(int(off[-1]), w))).to("cuda", dt)
    G = torch.from_numpy(rng.normal(size=(n, S.tensor_size(w, d)))).to("cuda", dt)
    plan = S.SignaturePlan(off, w, d, mode)
    full = int(_lib.lib.rpyb_signature_backward_workspace_size(
        plan.code, w, d, n, plan.max_len, K))
    ws = torch.empty(full, dtype=torch.uint8, device="cuda")

    def run(n_bytes):
        out = torch.full_like(inc, 7.0)
        rc = _lib.lib.rpyb_signature_backward(
            plan.code, w, d, n, plan.offsets.data_ptr(), plan.max_len, inc.data_ptr(),
            G.data_ptr(), G.stride(0), out.data_ptr(), K, ws.data_ptr(), n_bytes,
            torch.cuda.current_stream().cuda_stream)
        return rc, out

    rc, want = run(full)
    assert rc == 0
    accepted = 0
    for part in (0.95, 0.8, 0.6, 0.1):
        rc, got = run(int(full * part))
        if rc == 0:
            accepted += 1
            assert torch.equal(got, want)
        else:
            assert "workspace too small" in _lib.last_error()
            torch.cuda.synchronize()
            assert bool((got == 7.0).all())
    assert 1 <= accepted < 4
