"""Gradients at the shapes whose fold warps are two in one stage, two, or four without shared
levels, in both types, against float64 autograd.

Float64: 1e-10 of the largest gradient, as in test_gpu_backward_fold.  Float32: increments and
the lanes' words are float32, so each of a step's at most 2^7 products of a stream of at most 33
steps carries a few 6e-8: 33 * 8 * 6e-8 = 2e-5 of the largest gradient; 1e-4 with the margin."""
import numpy as np
import pytest
import torch

from roughpy_b200 import signatures as S
from tests.test_gpu_backward_fold import reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["f64", "f32c"])
@pytest.mark.parametrize("w,d", [(2, 2), (2, 3), (2, 4), (2, 5), (2, 6), (3, 2), (3, 3), (3, 4), (3, 5),
                                 (4, 2), (4, 3), (4, 4), (5, 3), (5, 4), (6, 4), (7, 4), (8, 4)])
def test_few_fold_warps_against_autograd(w, d, mode):
    lens = [1, 2, 3, 0, 33, 5, 17]
    off = S.offsets_from_lengths(lens)
    rng = np.random.default_rng(w + 10 * d)
    dt = torch.float64 if mode == "f64" else torch.float32
    inc = torch.from_numpy(rng.normal(0, 0.3, size=(int(off[-1]), w))).to("cuda", dt)
    G = torch.from_numpy(rng.normal(size=(len(lens), S.tensor_size(w, d)))).to("cuda", dt)
    plan = S.SignaturePlan(off, w, d, mode)
    x = inc.clone().requires_grad_(True)
    (S.signature_with_grad(x, plan, checkpoint_every=16) * G).sum().backward()
    y = inc.double().requires_grad_(True)
    for s in range(len(lens)):
        if lens[s]:
            (reference(y[off[s]:off[s + 1]], w, d) * G[s].double()).sum().backward()
    tol = 1e-10 if mode == "f64" else 1e-4
    assert float((x.grad.double() - y.grad).abs().max()) <= tol * max(float(y.grad.abs().max()), 1.0)
