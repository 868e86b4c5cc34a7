"""A solve beside another stream's kernel that keeps an SM: LSQR's resident kernels
need every SM (dense and large sparse problems fill one's registers), so the solve
has to go on without them instead of waiting for that kernel's end."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import skills_gb300 as skl  # noqa: E402
import synthetic  # noqa: E402

HOLD = 4_000_000_000   # cycles: about two seconds


def beside(f):
    """f() while a one-block kernel runs on a stream of its own, and whether that kernel
    still ran when f had returned."""
    import torch
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        torch.cuda._sleep(HOLD)
    r = f()
    running = not side.query()
    side.synchronize()
    return r, running


def test_sparse():
    A, b = synthetic.sparse_uniform(100000, 1500, 1600, 3, 1.0)
    f = lambda: skl.ls_sparse_spqr(A, b, 1.7, 2, abs_tol=0.0, it_tol=1e-12, seed=1)  # noqa: E731
    alone = f()
    r, running = beside(f)
    assert running
    assert np.array_equal(r.x, alone.x) and (r.it, r.rank, r.flag) == (alone.it, alone.rank, alone.flag)


@pytest.mark.parametrize("solver", ["ls_dense_hashing_blendenpik", "ls_dense_hashing_blendenpik_noCPQR"])
def test_dense(solver):
    """Other kernels, other rounding: condition number ~6, it_tol 1e-12, so x ~1e-11
    off; 1e-9 asked for."""
    rng = np.random.default_rng(1)
    A = np.asfortranarray(rng.standard_normal((6000, 700)))
    b = rng.standard_normal(6000)
    f = lambda: getattr(skl, solver)(A, b, 1.7, 1, it_tol=1e-12, seed=3, backward_tol=1e-13)  # noqa: E731
    alone = f()
    r, running = beside(f)
    assert running
    assert (r.rank, r.flag) == (alone.rank, alone.flag)
    assert np.linalg.norm(r.x - alone.x) <= 1e-9 * np.linalg.norm(alone.x)
    again = f()   # the GPU to itself: the resident kernel again
    assert np.array_equal(again.x, alone.x)
