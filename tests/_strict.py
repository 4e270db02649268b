"""A comparison that words left unwritten cannot pass."""
import numpy as np

from tests._util import level_rel_err


def strict_level_rel_err(got, want, width, depth):
    """``level_rel_err``, infinite where a word of ``got`` is not finite but ``want``'s is (a
    NaN there would be lost in the maximum over levels)."""
    got = np.asarray(got, dtype=np.float64)
    want = np.asarray(want, dtype=np.float64)
    assert got.shape == want.shape
    if np.any(~np.isfinite(got) & np.isfinite(want)):
        return float("inf")
    return level_rel_err(got, want, width, depth)
