"""The dense LSQR's one-pass kernel at the edges of its tiles: columns around
multiples of its chunks (512) and of the tile shapes, rows around the tile
heights, a leading dimension larger than n, columns it does not select.

x must be the least-squares solution of a matrix of condition number ~10 to
cond * it_tol accuracy with it_tol 1e-12: 1e-9 has a factor ten to spare.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import skills_gb300 as skl  # noqa: E402


def lstsq(A, b):
    x = np.linalg.lstsq(A, b, rcond=None)[0]
    return x


@pytest.mark.parametrize("n,d", [(9, 1), (40, 3), (301, 31), (1021, 127), (2049, 511), (2050, 512),
                                 (2600, 513), (3001, 1024), (3500, 1025), (4097, 1537),
                                 (4600, 2048), (5000, 2049)])
def test_solution(n, d):
    rng = np.random.default_rng(d)
    A = np.asfortranarray(rng.standard_normal((n, d)) * (1 + 2 * rng.random(d)))
    b = rng.standard_normal(n)
    for f in (skl.ls_dense_hashing_blendenpik, skl.ls_dense_hashing_blendenpik_noCPQR):
        r = f(A, b, gamma=1.7 if d > 3 else 4.0, k=1, it_tol=1e-12, seed=3)
        x = lstsq(A, b)
        assert r.rank == d and r.flag == 0
        assert np.linalg.norm(r.x - x) <= 1e-9 * np.linalg.norm(x)


def test_range_split_and_strides():
    """Magnitudes over [2^-90, 2^90] of the pairs' range, zeros, and lda > n through the
    device entry point (unpivoted: the pivoted solver's absolute rank rule leaves out
    columns this small); outside the range the FP64 path takes over as before."""
    import torch
    rng = np.random.default_rng(4)
    n, d, lda = 1500, 150, 1511
    B = rng.standard_normal((lda, d)) * 2.0 ** rng.integers(-20, 20, d)
    B[rng.random((lda, d)) < 0.3] = 0.0
    B[5, 7] = 2.0 ** -90
    A = B[:n]
    b = rng.standard_normal(n)
    At = torch.from_numpy(np.ascontiguousarray(B.T)).cuda()
    bd = torch.from_numpy(b).cuda()
    xd = torch.zeros(d, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    info = skl.dense_solve_device(n, d, At.data_ptr(), lda, bd.data_ptr(), xd.data_ptr(), 1.7, 1,
                                  it_tol=1e-12, use_cpqr=0)
    s = np.linalg.norm(A, axis=0)
    x = lstsq(A / s, b) / s
    assert info.fp64_fallback == 0
    assert np.linalg.norm((xd.cpu().numpy() - x) * s) <= 1e-9 * np.linalg.norm(x * s)
    At[3, 3] = 2.0 ** 101
    torch.cuda.synchronize()
    info = skl.dense_solve_device(n, d, At.data_ptr(), lda, bd.data_ptr(), xd.data_ptr(), 1.7, 1,
                                  it_tol=1e-12)
    assert info.fp64_fallback == 1


def test_rank_deficient_selection():
    """Columns the rank rule leaves out have x = 0; the residual is the projection's."""
    rng = np.random.default_rng(9)
    n, d = 2000, 160
    A = rng.standard_normal((n, d))
    A[:, 40:60] = 0.0
    A = np.asfortranarray(A)
    b = rng.standard_normal(n)
    r = skl.ls_dense_hashing_blendenpik(A, b, gamma=1.7, k=1, it_tol=1e-12, seed=3)
    keep = np.r_[0:40, 60:d]
    x = lstsq(A[:, keep], b)
    assert r.rank == d - 20
    assert np.all(r.x[40:60] == 0.0)
    assert np.linalg.norm(r.x[keep] - x) <= 1e-9 * np.linalg.norm(x)
