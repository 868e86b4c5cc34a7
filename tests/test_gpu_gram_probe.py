"""The FP64 path's look at the sketch in FP32 before its own Gram matrix (from 1,500
columns on): rank-deficient sketches go to the pivoted QR and its results, bit for
bit those of SKILLS_GRAM=0; others, also beyond the float range, end as without it."""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

import skills_gb300 as skl  # noqa: E402
import synthetic  # noqa: E402


def runs():
    out = {}
    kw = dict(it_tol=1e-12, seed=1, precision="fp64")
    for dep in (0, 1, 30):
        A, b, _ = synthetic.sparse_illcond(n=16000, d=1520, per_col=60, n_dep=dep, scale_exp=4.0)
        out[f"sparse {dep}"] = skl.ls_sparse_spqr(A, b, 1.2, 2, abs_tol=0.0, **kw)
    rng = np.random.default_rng(2)
    D = np.asfortranarray(rng.standard_normal((2900, 1510)))
    b = rng.standard_normal(2900)
    for scale in (1.0, 2.0 ** 200, 2.0 ** -200):
        out[f"dense {scale:.0e}"] = skl.ls_dense_hashing_blendenpik_noCPQR(D * scale, b, 1.3, 1, **kw)
    D[:, 7] = D[:, 1] - D[:, 1500]
    out["dense dependent"] = skl.ls_dense_hashing_blendenpik(D, b, 1.3, 1, abs_tol=0.0, **kw)
    return {k: (r.x.tolist(), r.rank, r.flag) for k, r in out.items()}


_CHILD = """
import json, sys
sys.path[:0] = sys.argv[1].split(":")
import test_gpu_gram_probe as t
print(json.dumps(t.runs()))
"""


def test_probe():
    path = ":".join(os.path.join(ROOT, p) for p in ("tests", "ski-lls_gb300", "oracle"))
    p = subprocess.run([sys.executable, "-c", _CHILD, path], env=dict(os.environ, SKILLS_GRAM="0"),
                       capture_output=True, text=True, timeout=600)
    assert p.returncode == 0, p.stderr[-2000:]
    other = json.loads(p.stdout.strip().splitlines()[-1])
    for k, (x, rank, flag) in runs().items():
        ox, orank, oflag = other[k]
        assert (rank, flag) == (orank, oflag) and flag == 0, k
        if k in ("sparse 1", "sparse 30", "dense dependent"):
            assert rank < len(x) and x == ox, k
        else:   # condition numbers below 100: both x ~1e-10 off
            assert rank == len(x)
            assert np.linalg.norm(np.subtract(x, ox)) <= 1e-9 * np.linalg.norm(ox), k
