"""How many blocks the gradient's workspace is for: all that fit while their checkpoints take
little memory; for long streams those of the usual block, never fewer than the least count
that a caller has to provide.  Fewer blocks give the same bits."""
import pytest
import torch

from roughpy_b200 import _lib
from roughpy_b200 import signatures as S

pytestmark = pytest.mark.gpu


def need(w, d, n, max_len, every, mode):
    size = _lib.lib.rpyb_signature_backward_workspace_size
    return int(size(S.MODES[mode], w, d, n, max_len, every))


@pytest.mark.parametrize("mode", ["f64", "f32c"])
@pytest.mark.parametrize("w,d", [(2, 3), (3, 4), (4, 4), (6, 3), (8, 2), (8, 3)])
def test_slots_of_long_streams(w, d, mode):
    n, every = 100000, 32
    short, long_ = 320, 3200000
    slot_short = need(w, d, 1, short, every, mode) - 256
    slot_long = need(w, d, 1, long_, every, mode) - 256
    few = (need(w, d, n, long_, every, mode) - 256) // slot_long
    all_ = (need(w, d, n, short, every, mode) - 256) // slot_short
    assert 148 <= few <= all_


@pytest.mark.parametrize("w,d,mode", [(4, 4, "f32c"), (3, 3, "f64")])
def test_long_streams_give_the_same_bits(w, d, mode):
    n, steps, every = 640, 12000, 4
    dt = torch.float64 if mode == "f64" else torch.float32
    off = S.offsets_from_lengths([steps] * n)
    g = torch.Generator(device="cuda").manual_seed(2)
    x = 0.02 * torch.randn(n * steps, w, device="cuda", dtype=dt, generator=g)
    x.requires_grad_(True)
    plan = S.SignaturePlan(off, w, d, mode)
    G = torch.randn(n, S.tensor_size(w, d), device="cuda", dtype=dt, generator=g)
    (S.signature_with_grad(x, plan, checkpoint_every=every) * G).sum().backward()
    # the same streams, a few at a time
    for s in (0, 17, n - 3):
        part = x.detach()[s * steps:(s + 3) * steps].clone().requires_grad_(True)
        few = S.SignaturePlan(S.offsets_from_lengths([steps] * 3), w, d, mode)
        sig = S.signature_with_grad(part, few, checkpoint_every=every)
        (sig * G[s:s + 3]).sum().backward()
        assert torch.equal(part.grad, x.grad[s * steps:(s + 3) * steps])
