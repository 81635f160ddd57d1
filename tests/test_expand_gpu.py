"""GPU: the block-wide walk over a row's products (hash and dense rows, both phases).

B row lengths at the edges of the walk's groups of 32 products (empty rows, one entry, 31 to 33, 64, thousands), one
to several staged chunks of 256 A entries, rows ending on a group and off it.  Whole-number values: bit for bit.
"""
import numpy as np
import pytest

import oracle
from matrices import from_coo

pytestmark = pytest.mark.gpu

LENGTHS = {"ones": [1], "with_empty": [0, 1, 0, 0, 33], "group_edges": [31, 32, 33, 64], "mixed": [0, 5, 2000, 1, 96],
           "long": [3000, 0, 31]}


def product(lengths, entries, ncol, dtype, seed):
    rng = np.random.default_rng(seed)
    mid, rows = 700, 6
    lens = np.resize(lengths, mid)
    A = from_coo(rows, mid, np.repeat(np.arange(rows), entries),
                 np.concatenate([rng.choice(mid, entries, replace=False) for _ in range(rows)]),
                 rng.integers(1, 8, rows * entries), dtype)
    cols = np.concatenate([np.sort(rng.choice(ncol, n, replace=False)) for n in lens])
    B = from_coo(mid, ncol, np.repeat(np.arange(mid), lens), cols, rng.integers(1, 8, len(cols)), dtype)
    return A, B


@pytest.mark.parametrize("lengths", sorted(LENGTHS))
@pytest.mark.parametrize("entries", [1, 31, 255, 256, 257, 600])
@pytest.mark.parametrize("algo,ncol,dtype", [("hash", 4000, np.float64), ("hash", 4000, np.int32),
                                             ("hsersc", 700001, np.float64)])
def test_walk(ctx, lengths, entries, algo, ncol, dtype):
    A, B = product(LENGTHS[lengths], entries, ncol, dtype, entries)
    out = ctx.spgemm(A, B, algo)
    rp, cols, vals, flop = oracle.oracle_spgemm(A, B, algo)
    assert out.stats["flop"] == flop
    np.testing.assert_array_equal(out.csr.row_ptrs, rp)
    np.testing.assert_array_equal(out.csr.cols.astype(np.int64), cols)
    np.testing.assert_array_equal(out.csr.vals.astype(np.float64), vals)


@pytest.mark.parametrize("per", [40, 700])  # products of a row on either side of 2^17, where rows are split
@pytest.mark.parametrize("entries", [255, 256, 257, 600])
def test_slices_follow_each_other(ctx, per, entries):
    """Rows over four column slices, in one staged chunk and in several: B rows that reach all slices, one of them,
    only the last, and none."""
    rng = np.random.default_rng(entries)
    ncol, mid, rows = 4 * 524288 - 3, 601, 5
    spans = [(0, ncol), (524288, 2 * 524288), (ncol - 9000, ncol), (524280, 524300)]
    cols = [np.zeros(0, np.int64) if k % 5 == 4 else
            np.sort(rng.choice(np.arange(*spans[k % 5]), min(per, spans[k % 5][1] - spans[k % 5][0]), replace=False))
            for k in range(mid)]
    B = from_coo(mid, ncol, np.repeat(np.arange(mid), [len(c) for c in cols]), np.concatenate(cols),
                 rng.integers(1, 8, sum(map(len, cols))))
    A = from_coo(rows, mid, np.repeat(np.arange(rows), entries),
                 np.concatenate([rng.choice(mid, entries, replace=False) for _ in range(rows)]),
                 rng.integers(1, 8, rows * entries))
    out = ctx.spgemm(A, B, "hash")
    rp, want, vals, _ = oracle.oracle_spgemm(A, B, "hash")
    np.testing.assert_array_equal(out.csr.row_ptrs, rp)
    np.testing.assert_array_equal(out.csr.cols.astype(np.int64), want)
    np.testing.assert_array_equal(out.csr.vals.astype(np.float64), vals)


@pytest.mark.parametrize("ncol", [16385, 131072, 524288, 524289, 1100000])
@pytest.mark.parametrize("nnz", [4097, 8192, 20000])
def test_dense_row_columns_leave_in_tiles(ctx, ncol, nnz):
    """Dense rows whose columns fill one tile of 4096 on their way out, end on one, or take several, over one, two
    and three column slices; one row crowds its columns into full bitmap words."""
    rng = np.random.default_rng(nnz)
    per, n_b = 500, max(20, 3 * nnz // 500)
    picks = [np.sort(rng.choice(ncol, min(nnz, ncol), replace=False)), np.arange(min(nnz, ncol)) + (ncol - min(nnz, ncol))]
    cols = [np.sort(rng.choice(picks[k % 2], min(per, len(picks[k % 2])), replace=False)) for k in range(2 * n_b)]
    B = from_coo(2 * n_b, ncol, np.repeat(np.arange(2 * n_b), [len(c) for c in cols]), np.concatenate(cols),
                 rng.integers(1, 8, sum(map(len, cols))))
    A = from_coo(2, 2 * n_b, np.repeat([0, 1], n_b), np.concatenate([np.arange(0, 2 * n_b, 2), np.arange(1, 2 * n_b, 2)]),
                 rng.integers(1, 8, 2 * n_b))
    out = ctx.spgemm(A, B, "hash")
    rp, cols, vals, _ = oracle.oracle_spgemm(A, B, "hash")
    np.testing.assert_array_equal(out.csr.row_ptrs, rp)
    np.testing.assert_array_equal(out.csr.cols.astype(np.int64), cols)
    np.testing.assert_array_equal(out.csr.vals.astype(np.float64), vals)


@pytest.mark.parametrize("ncol", [40, 4096, 32768, 32769, 131072, 131073, 524288, 524289])
@pytest.mark.parametrize("products", [700, 1500, 3000, 6000, 12000, 17000])
def test_symbolic_counts_by_bitmap_and_hash(ctx, ncol, products):
    """Every symbolic bin at the widths where its rows go by bitmap and by hash."""
    rng = np.random.default_rng(ncol + products)
    rows, per = 40, min(ncol, 97)
    entries = -(-products // per)
    A = from_coo(rows, entries + 5, np.repeat(np.arange(rows), entries),
                 np.concatenate([rng.choice(entries + 5, entries, replace=False) for _ in range(rows)]))
    cols = np.concatenate([np.sort(rng.choice(ncol, per, replace=False)) for _ in range(entries + 5)])
    B = from_coo(entries + 5, ncol, np.repeat(np.arange(entries + 5), per), cols)
    for algo in ("hash", "hybacc"):
        out = ctx.spgemm(A, B, algo)
        rp, c, v, _ = oracle.oracle_spgemm(A, B, algo)
        np.testing.assert_array_equal(out.csr.row_ptrs, rp)
        np.testing.assert_array_equal(out.csr.cols.astype(np.int64), c)
        np.testing.assert_array_equal(out.csr.vals.astype(np.float64), v)
