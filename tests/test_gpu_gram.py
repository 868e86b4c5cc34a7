"""Sketch factorization through the Gram matrix (well-conditioned sparse
sketches) against exact least squares and the pivoted factorization.

The least-squares solution of a full-rank problem does not depend on the
preconditioner, so both routes' x must be the FP64 solution to
cond(A D) * it_tol-class accuracy: equilibrated condition numbers here are
below 1e2 and it_tol is 1e-12, so 1e-9 holds with a factor ten to spare.
"""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import skills_gb300 as skl  # noqa: E402
import synthetic  # noqa: E402


# d around the tile edges of the sweep (16, 64, 128, 256) and beyond the
# look-ahead's 1,024; gamma 1.1 is the least well-conditioned sketch
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("d,gamma,k", [(1, 4.0, 1), (15, 1.7, 2), (64, 1.4, 2), (65, 1.1, 3),
                                       (128, 1.7, 2), (129, 1.1, 3), (256, 1.7, 2), (257, 1.4, 2),
                                       (449, 1.1, 3), (1025, 1.7, 2), (1291, 1.4, 3)])
def test_full_rank(d, gamma, k, precision):
    if precision == "fp64" and d > 1200:
        pytest.skip("one FP64 size beyond 1,024 is enough")
    n = 12 * d + 40
    A, b = synthetic.sparse_uniform(n, d, min(n, 40), 3, 1e-3)
    r = skl.ls_sparse_spqr(A, b, gamma=gamma, k=k, it_tol=1e-12, seed=5, precision=precision)
    x = np.linalg.lstsq(A.toarray(), b, rcond=None)[0]
    assert r.rank == d and r.info["unresolved_cols"] == 0
    assert np.linalg.norm(r.x - x) <= 1e-9 * np.linalg.norm(x)


@pytest.mark.parametrize("d,n_dep", [(200, 1), (700, 37), (1300, 64)])
def test_dependent_columns(d, n_dep):
    """Dependent columns are carried: rank, residual and the fit agree with the
    exact projection (the fit is unique, x is not)."""
    A, b, dep = synthetic.sparse_illcond(seed=7, n=20 * d, d=d, per_col=40, n_dep=n_dep,
                                         scale_exp=3.0)
    r = skl.ls_sparse_spqr(A, b, gamma=1.7, k=2, it_tol=1e-12, seed=3)
    assert r.rank == d - n_dep and r.info["unresolved_cols"] == n_dep
    # the projection of b on the span of the independent columns
    D = A.toarray()[:, np.setdiff1d(np.arange(d), dep)]
    s = np.linalg.norm(D, axis=0)
    fit = D @ (np.linalg.lstsq(D / s, b, rcond=None)[0] / s)
    res = np.linalg.norm(b - fit)
    # FP64 rounding of x alone moves the residual by about eps * ||A|| ||x||
    slack = 1e-9 * res + 64 * np.finfo(float).eps * np.linalg.norm(np.abs(A) @ np.abs(r.x))
    assert abs(np.linalg.norm(b - A @ r.x) - res) <= slack


CHILD = """
import sys, numpy as np
sys.path[:0] = {paths!r}
import skills_gb300 as skl, synthetic
out = []
# a tiny genuine column (not dependent), a badly conditioned pair, a zero column
A, b = synthetic.sparse_uniform(9000, 300, 60, 11, 1e-3)
A = A.tolil(); rng = np.random.default_rng(1)
A[:, 7] = A[:, 3] + 1e-3 * rng.standard_normal((9000, 1)) * (rng.random((9000, 1)) < 0.01)
A[:, 20] = 0
A = A.tocsc(); A.eliminate_zeros(); A.sort_indices()
r = skl.ls_sparse_spqr(A, b, gamma=1.7, k=2, it_tol=1e-12, seed=3)
out.append((r.rank, r.info["unresolved_cols"], r.info["residual_norm"]))
r = skl.ls_sparse_spqr(A, b, gamma=1.7, k=2, it_tol=1e-12, seed=3, rank_tol=1e-4)
out.append((r.rank, r.info["unresolved_cols"], r.info["residual_norm"]))
r = skl.ls_sparse_spqr(A, b, gamma=1.7, k=2, it_tol=1e-12, seed=3, precision="fp64")
out.append((r.rank, r.info["unresolved_cols"], r.info["residual_norm"]))
print(repr(out))
"""


def test_rank_matches_the_pivoted_factorization():
    """Near-dependent, zero and ordinary columns: rank, carried columns and the
    residual are those of the pivoted route (SKILLS_GRAM=0)."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    code = CHILD.format(paths=[os.path.join(root, "ski-lls_gb300")])
    got = []
    for v in ("1", "0"):
        p = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, SKILLS_GRAM=v),
                           capture_output=True, text=True, timeout=300)
        assert p.returncode == 0, p.stderr[-2000:]
        got.append(eval(p.stdout.strip().splitlines()[-1]))
    for (rg, ug, resg), (rp, up, resp) in zip(*got):
        assert (rg, ug) == (rp, up)
        assert abs(resg - resp) <= 1e-8 * resp
