"""The autotuner tunes what the solve runs: a class whose sketches are factorized by
their Gram matrix tries no panel widths until one of its solves takes the CPQR."""
import numpy as np
import pytest
import scipy.sparse as sp

import skills_gb300 as skl
import synthetic

pytestmark = pytest.mark.gpu


def test_panel_width_with_the_first_cpqr():
    n, d = 9000, 640
    A, b = synthetic.sparse_uniform(n, d, 90, 5, 1.0)
    kw = dict(it_tol=1e-12, abs_tol=0.0, seed=1, autotune=1)
    skl.finalize()
    gram = skl.ls_sparse_spqr(A, b, 1.7, 2, **kw)
    assert gram.info["tuned"][2] in (4, 8, 16, 32) and gram.info["tuned"][3] in (4, 8, 16, 32)
    # every column the same but for 1e-4 of it: more failed pivots than the Gram route drops
    g = np.random.default_rng(7)
    c = sp.csc_matrix((g.standard_normal(90), (g.choice(n, 90, replace=False), np.zeros(90, int))), shape=(n, 1))
    B = (c @ sp.csc_matrix(np.ones((1, d))) + 1e-4 * A).tocsc()
    B.sort_indices()
    plain = skl.ls_sparse_spqr(B, b, 1.7, 2, it_tol=1e-12, abs_tol=0.0, seed=1)
    first = skl.ls_sparse_spqr(B, b, 1.7, 2, **kw)
    second = skl.ls_sparse_spqr(B, b, 1.7, 2, **kw)
    assert first.rank == plain.rank == second.rank
    assert second.info["tuned"] == first.info["tuned"] and first.info["tuned"][1] in (32, 40, 48, 56, 64)
    assert np.array_equal(first.x, second.x)
    # the fitted values are unique; condition number ~1e4, it_tol 1e-12
    for r in (first, plain):
        assert abs(r.info["residual_norm"] - plain.info["residual_norm"]) <= 1e-9 * plain.info["residual_norm"]
    skl.finalize()
