"""The comparison switches of the QR with the QR taken: well-conditioned sketches are
factorized by Cholesky of their Gram matrix, so test_gpu_variants reaches the
panels, products and sample QRP that its switches choose only with SKILLS_GRAM=0.
Same problems, same bound (x to 1e-8 relative)."""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT
from test_gpu_variants import VARIANTS, _CHILD

pytestmark = pytest.mark.gpu


def solve(env):
    p = subprocess.run([sys.executable, "-c", _CHILD, os.path.join(ROOT, "ski-lls_gb300")],
                       env=dict(os.environ, SKILLS_GRAM="0", **env), capture_output=True, text=True, timeout=600)
    assert p.returncode == 0, p.stderr[-2000:]
    return {k: np.array(v) for k, v in json.loads(p.stdout.strip().splitlines()[-1]).items()}


def test_variants_reach_the_same_solution():
    default = solve({})
    for name, env in VARIANTS.items():
        if name == "default":
            continue
        for k, x in solve(env).items():
            if name == "no_pdl":
                assert np.array_equal(x, default[k]), (name, k)
            else:
                assert np.linalg.norm(x - default[k]) <= 1e-8 * np.linalg.norm(default[k]), (name, k)
