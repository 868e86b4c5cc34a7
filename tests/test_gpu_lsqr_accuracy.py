"""How far LSQR's x is from the exact solution when it runs until nothing moves.

The mixed iteration keeps v, the dense u and the norms in FP64.  Over twelve seeds
that leaves an rms error of 4.1e-15 (sparse) and 1.3e-14 (dense) on the problems
below; with float pairs in their place it is 5.0e-15 and 1.7e-14.  The bounds lie
halfway.  Results are bitwise reproducible, so the margin need not cover noise."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import skills_gb300 as skl  # noqa: E402
import synthetic  # noqa: E402

SEEDS = range(12)


def exact(A, b):
    """Least-squares solution by refinement with residuals in extended precision."""
    x = np.linalg.lstsq(A, b, rcond=None)[0].astype(np.longdouble)
    Al, bl = A.astype(np.longdouble), b.astype(np.longdouble)
    R = np.linalg.qr(A, mode="r")
    for _ in range(3):
        g = (Al.T @ (bl - Al @ x)).astype(float)
        x = x + np.linalg.solve(R, np.linalg.solve(R.T, g))
    return x


def rms(errs):
    return float(np.sqrt(np.mean(np.square(errs))))


def test_sparse():
    errs = []
    for s in SEEDS:
        A, b = synthetic.sparse_uniform(4000, 200, 60, s, 1.0)
        x = exact(A.toarray(), b)
        r = skl.ls_sparse_spqr(A, b, 1.7, 2, abs_tol=0, it_tol=1e-16, max_it=150, seed=1)
        errs.append(float(np.linalg.norm(r.x - x) / np.linalg.norm(x)))
    assert rms(errs) <= 4.6e-15


def test_dense():
    errs = []
    for s in SEEDS:
        rng = np.random.default_rng(100 + s)
        for n, d in ((1500, 150), (4000, 200)):   # the second problem drawn is solved
            A = np.asfortranarray(rng.standard_normal((n, d)) * 10.0 ** rng.uniform(-1, 1, d))
            b = rng.standard_normal(n)
        x = exact(A, b)
        r = skl.ls_dense_hashing_blendenpik_noCPQR(A, b, 1.7, 1, it_tol=1e-16, max_it=150, seed=3)
        errs.append(float(np.linalg.norm(r.x - x) / np.linalg.norm(x)))
    assert rms(errs) <= 1.5e-14
