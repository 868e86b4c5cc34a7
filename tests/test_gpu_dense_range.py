"""The dense solvers over the magnitudes of A that they admit: x scales with 1 / A,
the backward error does not change, whichever precision takes the call."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import skills_gb300 as skl  # noqa: E402


@pytest.mark.parametrize("e", [-97, -90, -70, -58, 30, 55, 70, 90, 110])
def test_scale_of_a(e):
    """Condition number below 4 and it_tol 1e-12: x ~1e-11 off, 1e-9 asked for.  A
    backward error between 1e-14 and 1e-11 shows that ||A||_F was neither lost nor
    infinite (0 would pass any target)."""
    rng = np.random.default_rng(5)
    n, d = 1500, 150
    # magnitudes in [0.5, 4]: at 2^-97 and 2^90 the mixed path admits every value, but
    # FP32 cannot hold its squares
    A = np.asfortranarray(np.clip(rng.standard_normal((n, d)), -4, 4))
    A = np.where(np.abs(A) < 0.5, 0.0, A)
    b = rng.standard_normal(n)
    x = np.linalg.lstsq(A, b, rcond=None)[0]
    kw = dict(it_tol=1e-12, max_it=300, seed=3)
    B = np.asfortranarray(A * 2.0 ** e)
    runs = [skl.ls_dense_hashing_blendenpik_noCPQR(B, b, 1.7, 1, **kw), skl.ls_dense_blendenpik(B, b, 2.2, **kw)]
    if e > -20:   # smaller matrices fall under the pivoted solver's absolute rank rule
        runs.append(skl.ls_dense_hashing_blendenpik(B, b, 1.7, 1, abs_tol=0.0, **kw))
    for r in runs:
        assert r.flag == 0 and r.rank == d
        assert np.linalg.norm(r.x * 2.0 ** e - x) <= 1e-9 * np.linalg.norm(x)
        assert 1e-14 < r.info["backward_error"] < 1e-11
