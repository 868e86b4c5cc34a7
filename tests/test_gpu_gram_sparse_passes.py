"""Sparse sketches beyond the reach of one Gram matrix: later passes on S A M must
find what the pivoted QR finds (the same rank, as many iterations, the same x).
Column pairs (a, a + eps b) give condition numbers of about 2 / eps: with eps above
~0.012 no pivot of the first sweep fails, below they all do."""
import json
import os
import subprocess
import sys

import numpy as np
import pytest
import scipy.sparse as sp

from conftest import ROOT

pytestmark = pytest.mark.gpu

import skills_gb300 as skl  # noqa: E402

# n, d, entries a column, eps, one pair in so many columns
CASES = [(3000, 70, 60, 0.05, 2), (6000, 300, 100, 0.03, 2), (6000, 300, 100, 3e-3, 50), (20000, 1000, 100, 0.02, 5),
         (20000, 1000, 100, 1e-3, 5), (20000, 1100, 100, 1e-3, 20)]


def solve(n, d, per_col, eps, every):
    g = np.random.default_rng(3)
    R = sp.csc_matrix((g.standard_normal(d * per_col), (g.integers(0, n, d * per_col), np.repeat(np.arange(d), per_col))),
                      shape=(n, d))
    M = sp.eye(d, format="lil")
    at = np.arange(every - 1, d, every)
    M[at, at] = eps
    M[at - 1, at] = 1.0
    A = (R @ M.tocsc()).tocsc()
    A.sort_indices()
    b = g.standard_normal(n)
    r = skl.ls_sparse_spqr(A, b, 1.7, 2, abs_tol=0.0, it_tol=1e-12, seed=1)
    return r.x.tolist(), r.it, r.rank, r.flag, r.info["unresolved_cols"], r.info["rcond_r11"]


_CHILD = """
import json, sys
sys.path[:0] = sys.argv[1].split(":")
import test_gpu_gram_sparse_passes as t
print(json.dumps([t.solve(*c) for c in t.CASES]))
"""


def test_as_with_the_qr():
    path = ":".join(os.path.join(ROOT, p) for p in ("tests", "ski-lls_gb300", "oracle"))
    p = subprocess.run([sys.executable, "-c", _CHILD, path], env=dict(os.environ, SKILLS_GRAM="0"),
                       capture_output=True, text=True, timeout=600)
    assert p.returncode == 0, p.stderr[-2000:]
    for case, qr in zip(CASES, json.loads(p.stdout.strip().splitlines()[-1])):
        x, it, rank, flag, unresolved, rcond = solve(*case)
        assert (rank, flag, unresolved) == (qr[2], 0, qr[4]), case
        assert abs(rcond - qr[5]) > 1e-3 * qr[5], case   # the factors are not the QR's
        assert it <= 1.15 * qr[1] + 3, (case, it, qr[1])
        # condition numbers up to ~1e4 and it_tol 1e-12: x ~1e-8 off
        assert np.linalg.norm(np.array(x) - qr[0]) <= 1e-7 * np.linalg.norm(qr[0]), case
