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
