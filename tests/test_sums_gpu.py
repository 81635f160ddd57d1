"""GPU: the rounding of the sums in rows of up to 2048 products.

Every row of A gathers k products for one column (as the diagonal of A*A^T gathers one per A entry), in the rows that
a warp takes and in the ranked-bitmap bins, with few and with many repeats beside it.  The error of that column over
5000 rows is compared with that of a pairwise sum of the same products in fp64.  Rounding errors are independent from
row to row, so the ratio of two such errors varies by about 1/sqrt(5000) = 1.4%; partial sums of 32 products that are
added one after another cost up to 7% at k = 100.  Sums that add one product at a time would have sqrt(k / 6) times
the error: 1.6 at k = 16, 2.3 at k = 32.  Values that are not finite come out as they do in a plain sum.
"""
import numpy as np
import pytest

from casgemm import Csr

pytestmark = pytest.mark.gpu

ROWS = 5000
TOLERANCE = 1.2


def pairwise(p):
    while p.shape[1] > 1:
        half = p.shape[1] // 2
        p = np.concatenate([p[:, :half] + p[:, half:2 * half], p[:, 2 * half:]], axis=1)
    return p[:, 0]


# products for the column, products of a B row, columns: warps (first line), then a block a row
@pytest.mark.parametrize("k,per_b,ncol", [(16, 16, 9000), (16, 16, 200), (31, 16, 60000), (65, 7, 150000), (65, 7, 60),
                                          (32, 30, 100000), (40, 25, 100000), (32, 30, 500), (64, 31, 300000),
                                          (64, 31, 700), (100, 20, 90000), (200, 10, 50000)])
@pytest.mark.parametrize("algo", ["hsersc", "hybacc"])
def test_column_of_many_products(ctx, k, per_b, ncol, algo):
    rng = np.random.default_rng(k + ncol)
    mid, hot = 2 * k + 100, ncol // 3
    a_cols = np.sort(np.argsort(rng.random((ROWS, mid)), axis=1)[:, :k], axis=1)
    a_vals = rng.uniform(0.5, 1.5, (ROWS, k))
    b_cols = np.empty((mid, per_b), np.int32)
    for i in range(mid):
        others = rng.choice(ncol - 1, per_b - 1, replace=False)
        b_cols[i] = np.sort(np.append(others + (others >= hot), hot))
    b_vals = rng.uniform(0.5, 1.5, (mid, per_b))
    A = Csr(ROWS, mid, np.arange(ROWS + 1, dtype=np.int64) * k, a_cols.astype(np.int32).ravel(), a_vals.ravel())
    B = Csr(mid, ncol, np.arange(mid + 1, dtype=np.int64) * per_b, b_cols.ravel(), b_vals.ravel())
    out = ctx.spgemm(A, B, algo)
    bins = out.stats["numc_bins"]
    if any(bins[b] for b in ("hash256", "hash1k", "hash4k", "dense")):
        pytest.skip("the hybrid accumulator hashes these rows, whose sums go one product at a time")
    C = out.csr
    at = C.cols == hot
    assert at.sum() == ROWS
    got = C.vals[at]
    b_hot = b_vals[b_cols == hot][a_cols]
    exact = (a_vals.astype(np.longdouble) * b_hot).sum(axis=1)

    def error(x):
        return float(np.sqrt((((x - exact) / exact) ** 2).mean()))

    assert error(got) <= TOLERANCE * error(pairwise(a_vals * b_hot))


@pytest.mark.parametrize("k,per_b,ncol", [(16, 16, 200), (65, 7, 60), (32, 30, 500), (64, 31, 700), (64, 31, 300000),
                                          (64, 70, 20000), (90, 80, 200000)])
@pytest.mark.parametrize("algo", ["hash", "hsersc"])
@pytest.mark.parametrize("special", ["inf", "nan", "cancel", "negative zero", "tiny", "huge"])
def test_special_values(ctx, k, per_b, ncol, algo, special):
    """Infinities and NaN stay in their columns; infinities of both signs meet; sums of -0.0 compare equal to zero;
    sums whose rounding errors leave the normal range, or whose terms are near the largest double."""
    rng = np.random.default_rng(k * per_b)
    rows, mid = 1300, 2 * k + 20
    a_cols = np.sort(np.argsort(rng.random((rows, mid)), axis=1)[:, :k], axis=1)
    b_cols = np.sort(np.argsort(rng.random((mid, ncol if ncol < 1000 else 1000)), axis=1)[:, :per_b], axis=1) * (
        1 if ncol < 1000 else ncol // 1000)
    b_cols[:, 0] = 0  # one column that every row holds
    scale = {"tiny": 1e-150, "huge": 1e+150}.get(special, 1.0)
    a_vals = rng.uniform(0.5, 1.5, (rows, k)) * scale
    b_vals = rng.uniform(0.5, 1.5, (mid, per_b)) * scale
    if special in ("inf", "nan"):
        b_vals[::7, 0] = np.inf if special == "inf" else np.nan
        b_vals[3::11, 1] = -np.inf
    elif special == "cancel":
        b_vals[0::5, 0], b_vals[1::5, 0] = np.inf, -np.inf
    elif special == "negative zero":
        b_vals[:] = -0.0
    elif special == "huge":
        b_vals[:, 0] = 1.7e308 / (1e150 * k)
    A = Csr(rows, mid, np.arange(rows + 1, dtype=np.int64) * k, a_cols.astype(np.int32).ravel(), a_vals.ravel())
    B = Csr(mid, ncol, np.arange(mid + 1, dtype=np.int64) * per_b, b_cols.astype(np.int32).ravel(), b_vals.ravel())
    C = ctx.spgemm(A, B, algo).csr
    want = np.zeros((rows, ncol if ncol < 1000 else 1001))
    seen = np.zeros(want.shape, bool)
    step = 1 if ncol < 1000 else ncol // 1000
    with np.errstate(all="ignore"):
        for j in range(k):
            cols = b_cols[a_cols[:, j]] // step
            r = np.arange(rows)[:, None]
            want[r, cols] += a_vals[:, j:j + 1] * b_vals[a_cols[:, j]]
            seen[r, cols] = True
    r = np.repeat(np.arange(rows), np.diff(C.row_ptrs))
    assert len(r) == seen.sum() and seen[r, C.cols // step].all()
    # two sums of at most k terms of one sign, each within k roundings of the exact one
    np.testing.assert_allclose(C.vals, want[r, C.cols // step], rtol=2 * (k + 1) * 2.0 ** -53)
