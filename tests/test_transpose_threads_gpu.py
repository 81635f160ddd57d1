"""GPU: transposes of matrices of different heights on several threads, each with a context of its own."""
import threading

import numpy as np
import pytest

import casgemm
from matrices import from_coo

pytestmark = pytest.mark.gpu


def _long_columns(rows, dtype):
    """Columns of 300 to 2000 entries, which are ranked in a bitmap of the rows."""
    rng = np.random.default_rng(rows)
    lens = [300, 700, 1500, 2000]
    r = np.concatenate([rng.choice(rows, n, replace=False) for n in lens])
    return from_coo(rows, len(lens), r, np.repeat(np.arange(len(lens)), lens), rng.integers(1, 9, len(r)), dtype)


def test_heights_side_by_side():
    cases = [_long_columns(m, d) for m in (2500, 1 << 19) for d in (np.int32, np.float64)]
    bad = []

    def work(A):
        want = casgemm.transpose(A)
        with casgemm.Context(0) as ctx:
            for _ in range(400):
                try:
                    got = ctx.transpose(A)
                except casgemm.CasError as e:
                    bad.append(str(e))
                    return
                if not (np.array_equal(got.row_ptrs, want.row_ptrs) and np.array_equal(got.cols, want.cols)
                        and np.array_equal(got.vals, want.vals)):
                    bad.append("a transpose of %d rows differs" % A.num_row)
                    return

    threads = [threading.Thread(target=work, args=(A,)) for A in cases for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
