"""Dense solves over condition numbers 1 to 1e8: one to three passes of the Gram route, and
the QR beyond it, must find the same rank and x as the QR alone (SKILLS_GRAM=0).

x is compared with the exact solution of a consistent system: its error is that of FP64
data, cond * 2^-53 * sqrt(d), or LSQR's, cond * it_tol; both runs get a factor 64 over
their sum.  A column that repeats another leaves x open; there b's fit is compared.
"""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CODE = """
import sys
sys.path[:0] = %r
import numpy as np, skills_gb300 as skl
n, d, kexp, f, dup = %d, %d, %g, skl.%s, %d
rng = np.random.default_rng(d)
Q = np.linalg.qr(rng.standard_normal((d, d)))[0]
U = np.linalg.qr(rng.standard_normal((n, d)))[0]
A = (U * np.logspace(0, -kexp, d)) @ Q
if dup: A[:, d - 3] = A[:, 2]
A = np.asfortranarray(A)
x = rng.standard_normal(d)
b = A @ x
r = f(A, b, gamma=1.7, k=1, it_tol=1e-13, seed=3)
print(r.rank, r.flag, np.linalg.norm(r.x - x) / np.linalg.norm(x), np.linalg.norm(A @ r.x - b) / np.linalg.norm(b))
"""
PIV, NOPIV = "ls_dense_hashing_blendenpik", "ls_dense_hashing_blendenpik_noCPQR"


@pytest.mark.parametrize("n,d,kexp,f,dup", [(700, 63, 2.6, PIV, 0), (700, 64, 4, NOPIV, 0), (900, 65, 6, PIV, 0),
                                            (2600, 257, 3, NOPIV, 0), (2600, 255, 5, PIV, 0), (3000, 200, 8, PIV, 0),
                                            (4500, 640, 4, PIV, 0), (900, 65, 1, PIV, 1), (900, 65, 3, PIV, 1)])
def test_passes(n, d, kexp, f, dup):
    out = []
    for v in ("1", "0"):
        p = subprocess.run([sys.executable, "-c", CODE % (sys.path, n, d, kexp, f, dup)], env=dict(os.environ, SKILLS_GRAM=v),
                           capture_output=True, text=True, timeout=300)
        assert p.returncode == 0, p.stderr
        rank, flag, err, fit = p.stdout.split()
        out.append((int(rank), int(flag)))
        if dup:
            assert float(fit) <= 64 * 10.0 ** kexp * (2.0 ** -53 * d ** 0.5 + 1e-13)
        elif kexp < 8:
            assert float(err) <= 64 * 10.0 ** kexp * (2.0 ** -53 * d ** 0.5 + 1e-13)
    assert out[0] == out[1]
