"""Sizes beyond the device's 32-bit counters are refused before anything is drawn,
copied or looked for on a device."""
import ctypes

import numpy as np
import pytest

import skills_gb300 as skl

LIMIT = 2 ** 31 - 1 - 2 ** 20


def sparse(m, nnz):
    p = np.array([0, nnz], dtype=np.int64)
    one = np.zeros(1)
    csc = skl.SklCsc(m, 1, nnz, p.ctypes.data, one.ctypes.data, one.ctypes.data)
    o = skl.default_opts()
    return skl.lib().skl_sparse_solve(ctypes.byref(csc), one.ctypes.data, one.ctypes.data, ctypes.byref(o), None)


def dense(n, solve):
    one = np.zeros(1)
    o = skl.default_opts()
    return getattr(skl.lib(), solve)(one.ctypes.data, n, n, 1, one.ctypes.data, one.ctypes.data, ctypes.byref(o), None)


@pytest.mark.parametrize("over", [1, 2 ** 19, 2 ** 20, 2 ** 20 + 1, 2 ** 33])
def test_refused(over):
    assert sparse(LIMIT + over, 1) == skl.SKL_ERR_INVALID
    assert "too large" in skl.last_error()
    assert sparse(1000, LIMIT + over) == skl.SKL_ERR_INVALID
    assert "too large" in skl.last_error()
    for solve in ("skl_dense_solve", "skl_dense_blendenpik_solve", "skl_dense_solve_device"):
        assert dense(LIMIT + over, solve) == skl.SKL_ERR_INVALID
        assert "too large" in skl.last_error()
