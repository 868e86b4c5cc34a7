"""Every route LSQR can take: the kernels of their own (sparse problems whose vectors
do not fit shared memory, dense ones beyond 4,096 columns; here by
SKILLS_LSQR_PERSIST=0, read once per process) and each column-chunk count of the
dense one-pass kernel up to its limit and one column beyond."""
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


def problems():
    rng = np.random.default_rng(8)
    out = {}
    for n, d in ((40, 3), (3001, 65), (12000, 700)):
        A, b = synthetic.sparse_uniform(n, d, max(3, n // 50), d, 1.0)
        for precision in ("mixed", "fp64"):
            out[f"sparse {n}x{d} {precision}"] = lambda A=A, b=b, p=precision: skl.ls_sparse_spqr(
                A, b, 1.7, 2, abs_tol=0.0, it_tol=1e-12, seed=1, precision=p)
    A, b = synthetic.sparse_zipf(n=20000, d=900, cap=5000, target_nnz=150000)
    out["sparse power-law"] = lambda A=A, b=b: skl.ls_sparse_spqr(A, b, 1.7, 2, abs_tol=0.0, it_tol=1e-12, seed=1)
    for n, d in ((40, 3), (2600, 513), (3500, 1025)):
        D = np.asfortranarray(rng.standard_normal((n, d)))
        b = rng.standard_normal(n)
        g = 4.0 if d == 3 else 1.7
        out[f"dense {n}x{d}"] = lambda D=D, b=b, g=g: skl.ls_dense_hashing_blendenpik(
            D, b, g, 1, abs_tol=0.0, it_tol=1e-12, seed=3)
        out[f"dense {n}x{d} unpivoted"] = lambda D=D, b=b, g=g: skl.ls_dense_hashing_blendenpik_noCPQR(
            D, b, g, 1, it_tol=1e-12, seed=3)
    return out


def solve_all():
    return {k: f() for k, f in problems().items()}


_CHILD = """
import json, sys
sys.path[:0] = sys.argv[1].split(":")
import test_gpu_lsqr_routes as t
print(json.dumps({k: [r.x.tolist(), r.rank, r.flag] for k, r in t.solve_all().items()}))
"""


def test_kernels_of_their_own():
    """Condition numbers below 100, so it_tol 1e-12 leaves both x ~1e-10 off."""
    path = ":".join(os.path.join(ROOT, p) for p in ("tests", "ski-lls_gb300", "oracle"))
    p = subprocess.run([sys.executable, "-c", _CHILD, path], env=dict(os.environ, SKILLS_LSQR_PERSIST="0"),
                       capture_output=True, text=True, timeout=600)
    assert p.returncode == 0, p.stderr[-2000:]
    other = json.loads(p.stdout.strip().splitlines()[-1])
    for k, r in solve_all().items():
        x, rank, flag = other[k]
        assert (rank, flag) == (r.rank, r.flag), k
        if "power-law" not in k:   # its columns may coincide, x is then not unique
            assert np.linalg.norm(np.array(x) - r.x) <= 1e-9 * np.linalg.norm(r.x), k


@pytest.mark.parametrize("d", [2561, 3073, 3585, 4096, 4097])
def test_dense_chunk_counts(d):
    """Gaussian with 1.8 rows per column: condition number ~7, x ~1e-11 off."""
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(d)
    n = int(1.8 * d)
    At = torch.randn(d, n, generator=g, device="cuda", dtype=torch.float64)
    b = torch.randn(n, generator=g, device="cuda", dtype=torch.float64)
    q, r = torch.linalg.qr(At.t())
    want = torch.linalg.solve_triangular(r, (q.t() @ b)[:, None], upper=True)[:, 0]
    for use_cpqr in (1, 0):
        x = torch.zeros(d, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        info = skl.dense_solve_device(n, d, At.data_ptr(), n, b.data_ptr(), x.data_ptr(), 1.5, 1, seed=3,
                                      it_tol=1e-12, abs_tol=0.0, use_cpqr=use_cpqr)
        assert (info.rank, info.flag) == (d, 0)
        assert float((x - want).norm() / want.norm()) <= 1e-9
