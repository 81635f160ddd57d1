"""GPU: the ranked-bitmap ESC kernel (no sort: a column's place is its rank in a two-level bitmap).

Whole-number values, so every sum is exact in any order: C equals the oracle's bit for bit.  The rows sit at the
kernel's edges: the fused and bin bounds in products, the widths at which the second level starts and ends, one and
several staged chunks of A entries, few and many products per column, unsorted B rows.
"""
import numpy as np
import pytest

import oracle
from casgemm import Csr
from matrices import from_coo

pytestmark = pytest.mark.gpu

ROWS = 160  # at least one per SM


def make(entries, per_b, ncol, span=None, seed=1, hot=0, dtype=np.float64, last=None):
    """ROWS rows of `entries` A entries, B rows of per_b columns in the last `span` of ncol columns; `hot` of them the
    same in every B row; the last B row that every row gathers has `last` columns."""
    rng = np.random.default_rng(seed)
    mid, span = 3 * entries, span or ncol
    r = np.repeat(np.arange(ROWS), entries)
    c = np.concatenate([np.append(rng.choice(mid - 1, entries - 1, replace=False), mid - 1) for _ in range(ROWS)])
    A = from_coo(ROWS, mid, r, c, rng.integers(1, 8, len(r)), dtype)
    cols, lens = [], []
    for k in range(mid):
        n = last if last is not None and k == mid - 1 else per_b
        pick = rng.choice(span - hot, n - min(hot, n), replace=False) + hot if span < 1 << 16 else \
            np.unique(rng.integers(hot, span, 2 * n + 8))[:n - min(hot, n)]
        x = np.concatenate([np.arange(min(hot, n)), np.sort(pick)]) + (ncol - span)
        if k % 7 == 0 and n > 1:
            x[-1] = ncol - 1  # the widest range
            x = np.unique(x)
        cols.append(x)
        lens.append(len(x))
    B = from_coo(mid, ncol, np.repeat(np.arange(mid), lens), np.concatenate(cols),
                 rng.integers(1, 8, int(np.sum(lens))), dtype)
    return A, B


def check(ctx, A, B, algo="hsersc", **tuning):
    saved = ctx.get_tuning()
    try:
        ctx.set_tuning(**tuning)
        out = ctx.spgemm(A, B, algo)
    finally:
        ctx.set_tuning(**saved)
    rp, cols, vals, _ = oracle.oracle_spgemm(A, B, algo)
    np.testing.assert_array_equal(out.csr.row_ptrs, rp)
    np.testing.assert_array_equal(out.csr.cols.astype(np.int64), cols)
    np.testing.assert_array_equal(out.csr.vals.astype(np.float64), vals)
    return out


@pytest.mark.parametrize("ncol", [6000, (1 << 17) - 1, 1 << 17, (1 << 17) + 1, (1 << 18) + 1, 1 << 21, (1 << 21) + 1])
@pytest.mark.parametrize("fuse", [1, 0])
def test_widths(ctx, ncol, fuse):
    """One column per cell up to 2^17, 2 to 16 up to 2^21, and the sorting form beyond."""
    A, B = make(60, 70, ncol)
    out = check(ctx, A, B, fusion=fuse)
    assert out.stats["esc_overflow_rows"] == 0
    if fuse:
        assert out.stats["fused_rows"] == ROWS


@pytest.mark.parametrize("products", [2049, 5119, 5120, 5121, 6144, 6145, 8191, 8192])
@pytest.mark.parametrize("ncol", [100000, 1000003])
def test_product_bounds(ctx, products, ncol):
    """Rows at the bounds of the fused range and of the bins."""
    entries = 40
    per = products // entries
    A, B = make(entries, per, ncol, last=products - per * (entries - 1))
    check(ctx, A, B)


@pytest.mark.parametrize("products", [33, 127, 128, 129, 511, 1023, 1024, 1025, 1535, 2047, 2048])
@pytest.mark.parametrize("ncol", [300, 1 << 15, (1 << 15) + 1, 1 << 16, (1 << 16) + 1, 600001, 1 << 21])
def test_small_bins(ctx, products, ncol):
    """Rows of the 1024 and 2048 bins, at the widths where each starts its second level (2^15 and 2^16 columns)."""
    entries = 3 if products < 100 else 11
    per = products // entries
    A, B = make(entries, per, ncol, last=products - per * (entries - 1), seed=products)
    check(ctx, A, B)


@pytest.mark.parametrize("products", [33, 64, 127, 128, 129, 384, 511, 512, 513])
@pytest.mark.parametrize("entries", [1, 31, 32, 33, 128, 129])
@pytest.mark.parametrize("algo", ["hash", "hsersc"])
def test_warp_rows(ctx, products, entries, algo):
    """Rows at the bounds of what a warp takes: products, A entries (empty B rows among them), widths of one and two
    levels, few and many repeats, both value types (1300 rows: enough for a warp each)."""
    rng = np.random.default_rng(products + entries)
    rows, ncol = 1300, [300, 14000, 16385, 262144, 262145, 2000000][(products + entries) % 6]
    live = max(1, min(entries, products, int(rng.integers(1, entries + 1))) if products > 33 else min(entries, products))
    live = max(live, -(-products // min(ncol, 300)))
    entries = max(entries, live)
    per = np.full(live, products // live)
    per[:products % live] += 1
    lens = np.zeros(entries, np.int64)
    lens[rng.choice(entries, live, replace=False)] = per
    A = from_coo(rows, entries, np.repeat(np.arange(rows), entries), np.tile(np.arange(entries), rows),
                 rng.integers(1, 8, rows * entries), np.int32 if products % 2 else np.float64)
    cols = np.concatenate([np.sort(rng.choice(min(ncol, 20000), n, replace=False)) for n in lens]) if products else []
    if ncol > 20000:
        cols = cols * (ncol // 20000)
    B = from_coo(entries, ncol, np.repeat(np.arange(entries), lens), cols, rng.integers(1, 8, products),
                 np.int32 if products % 2 else np.float64)
    check(ctx, A, B, algo)


@pytest.mark.parametrize("span", [300, 5000])
@pytest.mark.parametrize("dtype", [np.float64, np.int32])
def test_crowded_columns(ctx, span, dtype):
    """Most products repeat a column (hundreds of repeats per row), in the last columns of a wide matrix and with two
    columns that every B row holds."""
    A, B = make(60, 60, 1500001, span=span, hot=2, dtype=dtype)
    check(ctx, A, B)
    check(ctx, A, B, fusion=0)


@pytest.mark.parametrize("entries,per_b", [(128, 30), (129, 30), (257, 17), (1200, 3), (3, 1500)])
def test_staged_chunks(ctx, entries, per_b):
    """Rows of one to ten staged chunks of A entries, with few and with many repeats."""
    for span in (None, 2000 if per_b < 2000 else 4000):
        A, B = make(entries, per_b, 700001, span=span)
        check(ctx, A, B)


def test_unsorted_b_rows(ctx):
    """B's rows in any order: the range is the whole matrix."""
    rng = np.random.default_rng(4)
    A, B = make(60, 60, 500000)
    cols, vals = B.cols.copy(), B.vals.copy()
    for k in range(B.num_row):
        s, e = B.row_ptrs[k], B.row_ptrs[k + 1]
        o = rng.permutation(e - s)
        cols[s:e], vals[s:e] = cols[s:e][o], vals[s:e][o]
    check(ctx, A, Csr(B.num_row, B.num_col, B.row_ptrs, cols, vals))
