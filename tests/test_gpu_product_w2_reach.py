"""The lane-letter kernel of width 2 at the products it still serves, those of float64 rows too
deep for the row-resident kernel or with bounded degrees that reach level 10: the same bits as
the blocked kernel (RPYB_W2_KERNEL=0 is read once per process, so those come from a child
process), and the C oracle's values.

Tolerance: a word is a sum of at most 15 terms in float64, 1.7e-15 of their absolute sum,
which for these inputs exceeds a level's largest word by less than 1e2: 1e-12."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
# depth, rows, (out, lhs, rhs) highest degrees
CASES = [(14, 3, (-1, -1, -1)), (14, 70, (-1, -1, -1)), (12, 3, (-1, -1, 11)), (12, 5, (-1, 9, -1)),
         (10, 4, (-1, -1, 4)), (13, 2, (11, -1, 10)), (16, 1, (-1, -1, -1))]


def inputs(d, n):
    from tests._util import level_scaled
    rng = np.random.default_rng(70 + d)
    return [level_scaled(rng, 2, d, n) for _ in range(3)]


def compute_all():
    from roughpy_b200 import _internals as I
    from roughpy_b200 import compute as rpc
    res = {}
    for i, (d, n, depths) in enumerate(CASES):
        a, b, c = inputs(d, n)
        I.dense_ft_fma(a, b, c, rpc.TensorBasis(2, d), *depths)
        res[str(i)] = a
    return res


def test_same_bits_as_the_blocked_kernel_and_the_oracle(tmp_path):
    import oracle
    from tests._strict import strict_level_rel_err
    out = tmp_path / "blocked.npz"
    code = (f"import sys; sys.path.insert(0, {ROOT!r}); import numpy as np; "
            f"from tests.test_gpu_product_w2_reach import compute_all; "
            f"np.savez({str(out)!r}, **compute_all())")
    env = dict(os.environ, RPYB_W2_KERNEL="0")
    subprocess.run([sys.executable, "-c", code], cwd=ROOT, env=env, check=True, timeout=600)
    blocked, lane = np.load(out), compute_all()
    for i, (d, n, depths) in enumerate(CASES):
        assert np.array_equal(lane[str(i)], blocked[str(i)]), CASES[i]
        a, b, c = inputs(d, n)
        o, lh, rh = (x if x >= 0 else d for x in depths)
        want = oracle.ft_fma(2, d, a, b, c, (0, o, 0, lh, 0, rh))
        assert strict_level_rel_err(lane[str(i)], want, 2, d) <= 1e-12, CASES[i]
