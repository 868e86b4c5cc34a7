"""The Gram route's larger workspace is no condition of a solve: where only the QR's
can be had, the solve takes the QR.  The least workspace that a solve gets along
with (SKILLS_WORKSPACE_MB) must be that of SKILLS_GRAM=0."""
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


def solves():
    rng = np.random.default_rng(1)
    A, b = synthetic.sparse_uniform(6000, 1600, 20, 3, 1.0)
    D = np.asfortranarray(rng.standard_normal((2400, 1300)))
    bd = rng.standard_normal(2400)
    kw = dict(it_tol=1e-12, abs_tol=0.0, seed=1)
    return {"sparse": lambda: skl.ls_sparse_spqr(A, b, 1.7, 2, **kw),
            "sparse fp64": lambda: skl.ls_sparse_spqr(A, b, 1.7, 2, precision="fp64", **kw),
            "dense": lambda: skl.ls_dense_hashing_blendenpik(D, bd, 1.7, 1, **kw),
            "dense fp64": lambda: skl.ls_dense_hashing_blendenpik(D, bd, 1.7, 1, precision="fp64", **kw)}


def least_mb(f):
    """Smallest SKILLS_WORKSPACE_MB that f succeeds with, and its result there."""
    def attempt(mb):
        skl.finalize()   # releases the workspace of the call before
        os.environ["SKILLS_WORKSPACE_MB"] = str(mb)
        try:
            return f()
        except skl.SklError as e:
            assert e.status == skl.SKL_ERR_ALLOC, e
            return None
        finally:
            del os.environ["SKILLS_WORKSPACE_MB"]
    lo, hi = 1, 4096
    assert attempt(hi) is not None
    while hi - lo > 1:
        mid = (lo + hi) // 2
        if attempt(mid) is None:
            lo = mid
        else:
            hi = mid
    return hi, attempt(hi)


def measure():
    out = {}
    for k, f in solves().items():
        mb, r = least_mb(f)
        out[k] = (mb, r.x.tolist(), r.rank)
    return out


_CHILD = """
import json, sys
sys.path[:0] = sys.argv[1].split(":")
import test_gpu_workspace as t
print(json.dumps(t.measure()))
"""


def test_least_workspace():
    path = ":".join(os.path.join(ROOT, p) for p in ("tests", "ski-lls_gb300", "oracle"))
    p = subprocess.run([sys.executable, "-c", _CHILD, path], env=dict(os.environ, SKILLS_GRAM="0"),
                       capture_output=True, text=True, timeout=600)
    assert p.returncode == 0, p.stderr[-2000:]
    qr = json.loads(p.stdout.strip().splitlines()[-1])
    for k, (mb, x, rank) in measure().items():
        assert mb == qr[k][0], k
        assert rank == qr[k][2] and x == qr[k][1], k   # the QR, bit for bit
