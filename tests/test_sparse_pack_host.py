"""Packing of sparse matrices (host code): whatever memory layout a matrix's arrays have, the
packed block holds the same entries as its dense form."""
import numpy as np
import pytest

from roughpy_b200._internals import SparseMatrix


def unpack(matrix):
    """The dense matrix that ``rpyb_sparse_pack``'s block stands for."""
    block, layout = matrix.device_packed("cpu")
    raw = block.numpy()
    groups, slots, ntab = (int(v) for v in layout)
    tab = raw[:8 * ntab].view(np.float64)
    words = raw[8 * ntab:].view(np.uint32)
    goff, words = words[:groups + 1], words[groups + 1:]
    perm, length, ent = words[:32 * groups], words[32 * groups:64 * groups], words[64 * groups:]
    assert ent.shape[0] == slots
    out = np.zeros(matrix.shape)
    for g in range(groups):
        for lane in range(32):
            row = int(perm[32 * g + lane])
            for j in range(int(length[32 * g + lane])):
                e = int(ent[int(goff[g]) + 32 * j + lane])
                out[row, e & 0xfffff] += tab[e >> 20]
    return out


def random_matrix(rng, rows, cols, per_row):
    count = rng.integers(0, per_row + 1, rows)
    indptr = np.concatenate([[0], np.cumsum(count)]).astype(np.int64)
    indices = np.concatenate([rng.permutation(cols)[:c] for c in count]).astype(np.int64)
    data = rng.choice([-2.0, -0.5, 0.25, 1.0, 3.0], indices.shape[0])
    return indptr, indices, data


def strided(a):
    """The same values as every second element of a larger array."""
    big = np.full(2 * a.shape[0], 7, dtype=a.dtype)
    big[::2] = a
    return big[::2]


@pytest.mark.parametrize("rows,cols,per_row", [(1, 1, 1), (31, 40, 6), (33, 50, 20), (200, 64, 12)])
@pytest.mark.parametrize("layout", [np.asarray, strided, lambda a: a[::-1].copy()[::-1]])
def test_packed_entries(rows, cols, per_row, layout):
    indptr, indices, data = random_matrix(np.random.default_rng(rows), rows, cols, per_row)
    want = SparseMatrix(indptr, indices, data, (rows, cols)).todense()
    got = unpack(SparseMatrix(layout(indptr), layout(indices), layout(data), (rows, cols)))
    assert np.array_equal(got, want)


def test_rows_that_end_before_they_begin_are_empty():
    """As the CSR kernel has it, which serves a matrix's first small call."""
    indptr = np.array([0, 3, 1, 4, 4], dtype=np.int64)
    indices = np.array([0, 2, 4, 1], dtype=np.int64)
    data = np.array([1.0, -2.0, 0.5, 3.0])
    want = np.zeros((4, 5))
    want[0, [0, 2, 4]] = data[:3]
    want[2, [2, 4, 1]] = data[1:]
    assert np.array_equal(unpack(SparseMatrix(indptr, indices, data, (4, 5))), want)
