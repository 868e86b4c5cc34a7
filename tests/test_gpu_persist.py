"""LSQR's persistent kernel: each of its shapes (one cluster, a grid, 1,024-thread
CTAs) against exact least squares, and bit for bit against the phase kernels
that the batched entry point runs.

x must be the FP64 solution to cond * it_tol accuracy: equilibrated condition
numbers here are below 1e2 and it_tol is 1e-12, so 1e-9 has a factor ten to
spare.
"""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu

import skills_gb300 as skl  # noqa: E402
import synthetic  # noqa: E402


def problem(n, d, per_col, kind, seed=1):
    A, _ = synthetic.sparse_uniform(n, d, per_col, seed, 0.0)
    if kind == "long":      # columns far longer than a chunk, a full one, and short ones
        rng = np.random.default_rng(seed)
        cols = [np.arange(n)] + [rng.choice(n, n // 3, replace=False) for _ in range(3)]
        B = sp.lil_matrix((n, len(cols)))
        for c, r in enumerate(cols):
            B[r, c] = rng.standard_normal((len(r), 1))
        A = sp.hstack([A[:, :d - len(cols)], B.tocsc()]).tocsc()
        A.sort_indices()
    return A, np.random.default_rng(seed + 1).standard_normal(n)


# bytes an iteration reads (24 nnz + 16 n + 4 d^2) choose the shape: one
# 16-CTA cluster to 1.6 MB, a grid above, 1,024 threads from 60 MB
SHAPES = [(40, 1, 30, "uniform"), (90, 3, 20, "uniform"), (700, 17, 40, "uniform"),
          (3001, 130, 40, "uniform"), (3000, 100, 200, "long"), (9000, 257, 300, "uniform"),
          (12001, 301, 100, "long"), (26000, 1300, 60, "uniform"), (40000, 3900, 30, "uniform")]


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("n,d,per_col,kind", SHAPES)
def test_solution(n, d, per_col, kind, precision):
    if precision == "fp64" and d > 400:
        pytest.skip("the FP64 path takes the same shapes")
    A, b = problem(n, d, per_col, kind)
    r = skl.ls_sparse_spqr(A, b, gamma=1.7 if d > 4 else 4.0, k=2 if d > 4 else 1, it_tol=1e-12,
                           seed=2, precision=precision)
    s = np.sqrt(np.asarray(A.multiply(A).sum(axis=0))).ravel()
    E = A.toarray() / s
    G = E.T @ E
    x = np.linalg.solve(G, E.T @ b)
    x = (x + np.linalg.solve(G, E.T @ (b - E @ x))) / s
    assert r.rank == d and r.flag == 0
    assert np.linalg.norm(r.x - x) <= 1e-9 * np.linalg.norm(x)


def test_batched_bits():
    probs = [problem(*sh, seed=11 + i) for i, sh in enumerate(SHAPES[1:8])]
    kw = dict(gamma=1.7, k=2, it_tol=1e-12)
    xs, _, status = skl.batched_sparse_spqr(probs, seed=5, **kw)
    assert not any(status)
    for (A, b), x in zip(probs, xs):
        assert np.array_equal(skl.ls_sparse_spqr(A, b, seed=5, **kw).x, x)


def test_iteration_limit_and_relaunch():
    """max_it below, at and above the iterations of one launch of the kernel."""
    A, b = problem(9000, 300, 60, "uniform")
    for max_it in (1, 7, 255, 256, 257, 300):
        r = skl.ls_sparse_spqr(A, b, gamma=1.1, k=3, it_tol=0.0, max_it=max_it, seed=2)
        assert r.it == max_it and r.flag == 1
