"""GPU: the rows of B = A^T at the edges of the device transpose's cases.

A row of B (a column of A) is sorted by a warp up to 256 entries, in four
sizes; ranked in a bitmap of A's rows above that; and sorted by a block where
a (row, column) pair occurs twice or A has more than 2^19 rows.  The scatter
follows A's rows in steps of 32 and looks further where many are empty.
Every result equals the host's stable counting sort entry for entry.
"""
import numpy as np
import pytest

import casgemm
from matrices import from_coo

pytestmark = pytest.mark.gpu

LENGTHS = [1, 2, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 512, 513, 2049, 0, 1500]


def _columns(n_rows, gaps, twice, dtype):
    """A matrix whose column j has LENGTHS[j] entries, in rows drawn at random
    (`gaps`: from a few stretches, with all rows between them empty)."""
    rng = np.random.default_rng(len(LENGTHS) + n_rows + gaps)
    pool = np.arange(n_rows)
    if gaps:
        pool = np.concatenate([np.arange(3, 1100), np.arange(n_rows // 2, n_rows // 2 + 1000),
                               np.arange(n_rows - 700, n_rows - 500, 2), [n_rows - 33, n_rows - 1]])
    r, c = [], []
    for j, n in enumerate(LENGTHS):
        rows = rng.choice(pool, n, replace=False)
        if twice and n > 600:
            rows[:3] = rows[5:8]
        r.append(rows)
        c.append(np.full(n, j))
    r, c = np.concatenate(r), np.concatenate(c)
    o = rng.permutation(len(r))
    r, c = r[o], c[o]
    o = np.argsort(r, kind="stable")
    v = np.arange(1, len(r) + 1)
    return from_coo(n_rows, len(LENGTHS) + 3, r[o], c[o], v, dtype)


@pytest.mark.parametrize("dtype", [np.int32, np.float64])
@pytest.mark.parametrize("twice", [False, True])
@pytest.mark.parametrize("n_rows,gaps", [(2111, False), (6000, True), (1 << 19, True), ((1 << 19) + 1, True),
                                         (2000003, True), (70000, False)])
def test_rows_of_every_length(n_rows, gaps, twice, dtype):
    A = _columns(n_rows, gaps, twice, dtype)
    want = casgemm.transpose(A)
    with casgemm.Context() as ctx:
        got = ctx.transpose(A)
    np.testing.assert_array_equal(got.row_ptrs, want.row_ptrs)
    np.testing.assert_array_equal(got.cols, want.cols)
    np.testing.assert_array_equal(got.vals, want.vals)
