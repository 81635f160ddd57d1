"""GPU: the walk over the inputs' rows that checks them and sums the row products.

4, 16 or 32 lanes a row by the mean length, and a block for long rows: rows at and over 64 times the lanes, more long
rows than a block lists, empty rows; faults in short and long rows are found, wherever B is A or not.
"""
import numpy as np
import pytest

import casgemm
import oracle
from casgemm import Csr
from matrices import from_coo

pytestmark = pytest.mark.gpu


def square(n, lens, seed=1):
    rng = np.random.default_rng(seed)
    lens = np.resize(lens, n)
    cols = np.concatenate([np.sort(rng.choice(n, k, replace=False)) for k in lens])
    return from_coo(n, n, np.repeat(np.arange(n), lens), cols, rng.integers(1, 4, len(cols)))


SHAPES = {"lanes_4": (1500, [0, 1, 3, 5, 12]), "lanes_16": (1500, [7, 16, 17, 24, 0]), "lanes_32": (900, [31, 32, 90]),
          "long": (2600, [0] * 300 + [255, 256, 257, 1025, 2049]), "many_long": (1200, [1100] + [0] * 3)}


@pytest.mark.parametrize("shape", sorted(SHAPES))
@pytest.mark.parametrize("same", [True, False])
def test_products_and_sorting(ctx, shape, same):
    A = square(*SHAPES[shape])
    for unsorted in (False, True):
        cols, vals = A.cols.copy(), A.vals.copy()
        if unsorted:  # the last entries of the longest row swapped
            e = int(A.row_ptrs[np.argmax(np.diff(A.row_ptrs)) + 1])
            cols[[e - 2, e - 1]], vals[[e - 2, e - 1]] = cols[[e - 1, e - 2]], vals[[e - 1, e - 2]]
        M = Csr(A.num_row, A.num_col, A.row_ptrs, cols, vals)
        dA = casgemm.DeviceCsr.upload(M)
        dB = dA if same else casgemm.DeviceCsr.upload(M)
        C, _ = ctx.spgemm_device(dA, dB, "hsersc")
        try:
            rp, c, v, flop = oracle.oracle_spgemm(A, A, "hsersc")
            assert ctx.stats()["flop"] == flop
            assert ctx.digest(C) == oracle.csr_digest(rp, c, v)[0]
        finally:
            ctx.free(C)


@pytest.mark.parametrize("shape", sorted(SHAPES))
@pytest.mark.parametrize("fault", ["column", "negative", "pointer"])
@pytest.mark.parametrize("where", ["A", "B", "both"])
def test_faults_are_found(ctx, shape, fault, where):
    A = square(*SHAPES[shape])
    rp, cols = A.row_ptrs.copy(), A.cols.copy()
    row = int(np.argmax(np.diff(rp)))
    if fault == "pointer":
        rp[row + 1] = rp[row] - 1 if rp[row] else A.nnz + 1
    else:
        cols[rp[row + 1] - 1] = A.num_col if fault == "column" else -1
    bad = casgemm.DeviceCsr.upload(Csr(A.num_row, A.num_col, rp, cols, A.vals))
    bad.c.num_nnz = A.nnz
    good = casgemm.DeviceCsr.upload(A)
    with pytest.raises(casgemm.CasError) as err:
        ctx.spgemm_device(good if where == "B" else bad, good if where == "A" else bad, "hybacc")
    assert err.value.status == 1  # CAS_ERR_BAD_INPUT
    C, _ = ctx.spgemm_device(good, good, "hybacc")  # the context goes on
    ctx.free(C)
