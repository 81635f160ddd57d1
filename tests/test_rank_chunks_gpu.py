"""GPU: rows whose second chunk of A entries starts among a thread's last products.

A row of 6145 to 8192 products is held 32 products a thread; one of more than 128 A entries is staged in chunks, and a
chunk that starts past product 7936 begins behind the 32nd product of the first threads.  Few and many repeats (they
are listed up to 256), whole-number values: bit for bit.
"""
import numpy as np
import pytest

import oracle
from matrices import from_coo

pytestmark = pytest.mark.gpu

ROWS = 160


@pytest.mark.parametrize("first", [7935, 7936, 7937, 7950, 8064, 8191])  # products of the first 128 entries
@pytest.mark.parametrize("rest", [1, 9, 128])                            # entries of one product behind them
@pytest.mark.parametrize("ncol", [9000, 1900000])
@pytest.mark.parametrize("dtype", [np.float64, np.int32])
def test_second_chunk_at_the_end(ctx, first, rest, ncol, dtype):
    rest = min(rest, 8192 - first)
    rng = np.random.default_rng(first + rest)
    lens = np.append(np.full(128, first // 128), np.ones(rest, np.int64))
    lens[:first % 128] += 1
    mid = 128 + rest
    A = from_coo(ROWS, mid, np.repeat(np.arange(ROWS), mid), np.tile(np.arange(mid), ROWS),
                 rng.integers(1, 8, ROWS * mid), dtype)
    cols = np.concatenate([np.sort(rng.choice(ncol, n, replace=False)) for n in lens])
    B = from_coo(mid, ncol, np.repeat(np.arange(mid), lens), cols, rng.integers(1, 8, len(cols)), dtype)
    out = ctx.spgemm(A, B, "hsersc")
    assert out.stats["numc_bins"]["esc8k"] == ROWS
    rp, c, v, _ = oracle.oracle_spgemm(A, B, "hsersc")
    assert (len(np.unique(cols)) + 256 >= len(cols)) == (ncol > 9000)  # listed or not
    np.testing.assert_array_equal(out.csr.row_ptrs, rp)
    np.testing.assert_array_equal(out.csr.cols.astype(np.int64), c)
    np.testing.assert_array_equal(out.csr.vals.astype(np.float64), v)
