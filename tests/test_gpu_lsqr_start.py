"""How LSQR starts: a right-hand side that leaves it nothing to do, on the phase
kernels (profile = 1, and every problem of a batch) as in the persistent kernel."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import skills_gb300 as skl  # noqa: E402
import synthetic  # noqa: E402


def test_nothing_to_do():
    """b = 0 with the early exit off: alpha beta = 0 ends LSQR before its first
    iteration (src/IterSolver.cpp:200), flag 0."""
    A, _ = synthetic.sparse_uniform(2000, 60, 40, 3, 0.0)
    b = np.zeros(2000)
    for profile in (0, 1):
        r = skl.ls_sparse_spqr(A, b, 1.7, 2, abs_tol=0.0, seed=1, max_it=50, profile=profile)
        assert (r.it, r.flag) == (0, 0) and not r.x.any()
    xs, infos, _ = skl.batched_sparse_spqr([(A, b)] * 3, 1.7, 2, abs_tol=0.0, seed=1, max_it=50)
    assert all((i.it, i.flag) == (0, 0) for i in infos) and not any(x.any() for x in xs)


@pytest.mark.parametrize("scale", [1e-30, 1e-25, 1e-18, 1e20, 1e30])
def test_scale_of_b(scale):
    """x scales with b: every solver, mixed precision.  Both matrices have condition
    numbers below 100, so it_tol 1e-12 leaves x ~1e-10 off; 1e-9 has a factor ten to
    spare."""
    A, b = synthetic.sparse_uniform(2000, 60, 100, 3, 1.0)
    rng = np.random.default_rng(4)
    D = np.asfortranarray(rng.standard_normal((1500, 150)))
    bd = rng.standard_normal(1500)
    xs = np.linalg.lstsq(A.toarray(), b, rcond=None)[0]
    xd = np.linalg.lstsq(D, bd, rcond=None)[0]
    kw = dict(it_tol=1e-12, max_it=300, seed=1)
    runs = [(skl.ls_sparse_spqr(A, b * scale, 1.7, 2, abs_tol=0.0, **kw), xs),
            (skl.ls_sparse_spqr(A, b * scale, 1.7, 2, abs_tol=0.0, profile=1, **kw), xs),
            (skl.ls_dense_hashing_blendenpik(D, bd * scale, 1.7, 1, abs_tol=0.0, **kw), xd),
            (skl.ls_dense_hashing_blendenpik_noCPQR(D, bd * scale, 1.7, 1, **kw), xd),
            (skl.ls_dense_blendenpik(D, bd * scale, 2.2, **kw), xd)]
    for r, x in runs:
        assert r.flag == 0
        assert np.linalg.norm(r.x / scale - x) <= 1e-9 * np.linalg.norm(x)
    x, _, _ = skl.batched_sparse_spqr([(A, b * scale)], 1.7, 2, abs_tol=0.0, **kw)
    assert np.array_equal(x[0], runs[0][0].x)
