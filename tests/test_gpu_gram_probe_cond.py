"""The FP64 path's look in FP32, by condition number: within the FP64 Gram matrix's
reach its results, beyond it the pivoted QR's, bit for bit those of SKILLS_GRAM=0."""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

import skills_gb300 as skl  # noqa: E402

D = 1504


def solve(kappa_exp):
    """A = G diag(logspace(0, -kappa_exp)) Q with a Gaussian G and an orthogonal Q."""
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(7)
    n = 2 * D
    X = torch.randn(n, D, generator=g, device="cuda", dtype=torch.float64) / n ** 0.5
    X *= torch.logspace(0.0, -float(kappa_exp), D, dtype=torch.float64, device="cuda")
    Q = torch.linalg.qr(torch.randn(D, D, generator=g, device="cuda", dtype=torch.float64))[0]
    At = (X @ Q).t().contiguous()
    b = At.t() @ torch.ones(D, dtype=torch.float64, device="cuda")
    x = torch.zeros(D, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    info = skl.dense_solve_device(n, D, At.data_ptr(), n, b.data_ptr(), x.data_ptr(), 1.3, 1, seed=3, it_tol=1e-10,
                                  abs_tol=0.0, rcond=1e-14, precision="fp64")
    return x.cpu().numpy().tolist(), int(info.rank), float(info.rcond_r11)


_CHILD = """
import json, sys
sys.path[:0] = sys.argv[1].split(":")
import test_gpu_gram_probe_cond as t
print(json.dumps([t.solve(k) for k in t.KAPPAS]))
"""
KAPPAS = [1, 4, 9, 11]


def test_by_condition():
    path = ":".join(os.path.join(ROOT, p) for p in ("tests", "ski-lls_gb300", "oracle"))
    p = subprocess.run([sys.executable, "-c", _CHILD, path], env=dict(os.environ, SKILLS_GRAM="0"),
                       capture_output=True, text=True, timeout=600)
    assert p.returncode == 0, p.stderr[-2000:]
    for k, (ox, orank, orcond) in zip(KAPPAS, json.loads(p.stdout.strip().splitlines()[-1])):
        x, rank, rcond = solve(k)
        assert rank == orank == D, k
        if k >= 9:
            assert x == ox and rcond == orcond, k
        else:   # consistent system: x = 1 up to the condition number times FP64 rounding
            assert rcond != orcond
            assert np.max(np.abs(np.array(x) - 1.0)) <= 1e-10 * 10.0 ** k, k
