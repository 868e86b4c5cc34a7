"""Rows far longer than the average: LSQR's A z hands them to whole warps.  Lengths
around the switch (4 L + min(8 L, 64) entries for L lanes a row), around the warp's
steps of 128, a full row, and several long rows that one warp meets together."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu

import skills_gb300 as skl  # noqa: E402


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("per_row,lanes", [(6, 4), (24, 8), (50, 16), (110, 32)])
def test_long_rows(per_row, lanes, precision):
    """Scaled Gaussian entries, condition number below 100: it_tol 1e-12 leaves x
    ~1e-10 off; 1e-9 asked for."""
    rng = np.random.default_rng(per_row)
    n, d = 9000, 600
    switch = 4 * lanes + min(8 * lanes, 64)
    lengths = [switch - 1, switch, switch + 1, 127, 128, 129, 257, d, d, d]
    cols = [rng.choice(d, per_row, replace=False) for _ in range(n)]
    for q, length in enumerate(lengths):
        cols[100 + q] = rng.choice(d, length, replace=False)      # neighbours
        cols[7 + 883 * q] = rng.choice(d, length, replace=False)  # spread over the CTAs
    rows = np.repeat(np.arange(n), [len(c) for c in cols])
    c = np.concatenate(cols)
    A = sp.csc_matrix((rng.standard_normal(c.size), (rows, c)), shape=(n, d))
    A.sort_indices()
    b = rng.standard_normal(n)
    x = np.linalg.lstsq(A.toarray(), b, rcond=None)[0]
    kw = dict(abs_tol=0.0, it_tol=1e-12, seed=1, precision=precision)
    r = skl.ls_sparse_spqr(A, b, 1.7, 2, **kw)
    assert r.flag == 0 and r.rank == d
    assert np.linalg.norm(r.x - x) <= 1e-9 * np.linalg.norm(x)
    xs, _, _ = skl.batched_sparse_spqr([(A, b)], 1.7, 2, **kw)
    assert np.array_equal(xs[0], r.x)
