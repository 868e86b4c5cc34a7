"""The FP32 Hartley transform in shared memory and the FP64 one of the right-hand side
against the oracle's, at lengths that take every pair of radices, a length with one pass
per radix, the smallest ones and the last that fits shared memory (and the first that
does not), with rows that leave zeros at the end and leading dimensions of either parity.

Tolerances as at the other lengths that are tested: 2e-6 (FP32) and 1e-12 (FP64) of the
result's norm.
"""
import numpy as np
import pytest

import ski_lls_oracle as orc

pytestmark = pytest.mark.gpu

import skills_gb300 as skl  # noqa: E402


@pytest.mark.parametrize("N", [2, 4, 6, 8, 10, 14, 18, 24, 28, 30, 40, 42, 50, 126, 210, 1024, 4410, 12348, 48020,
                               32768, 40000, 51200, 51450])
@pytest.mark.parametrize("cut", [0, 3])
def test_transform(N, cut):
    rng = np.random.default_rng(N)
    n = N - cut if N > 4 else N
    A = rng.standard_normal((n, 3))
    D = np.where(rng.random(n) < 0.5, -1.0, 1.0)
    ref = orc.unitary_dht(A, D, N)
    for prec, tol in (("mixed", 2e-6), ("fp64", 1e-12)):
        Y = skl.dht(A, D, N, precision=prec)
        assert np.linalg.norm(Y - ref) <= tol * np.linalg.norm(ref), prec


@pytest.mark.parametrize("n,d,m,k", [(7, 1, 4, 1), (98, 5, 20, 2), (2500, 7, 90, 1), (5000, 3, 1000, 3),
                                     (20000, 160, 500, 1), (51450, 2, 64, 2)])
def test_sketch_and_right_hand_side(n, d, m, k):
    rng = np.random.default_rng(n)
    N = skl.dht_length(n)
    A = rng.standard_normal((n, d))
    b = rng.standard_normal(n)
    g = orc.Rng(9)
    D = orc.rand_signs(g, n)
    rows, vals = orc.gen_hashing(g, m, N, k)
    SA_ref = orc.dense_sketch(orc.unitary_dht(A, D, N), m, k, rows, vals)
    Sb_ref = orc.dense_sketch(orc.unitary_dht(b, D, N), m, k, rows, vals)[:, 0]
    SA, Sb = skl.sketch_dense(A, b, D, N, m, k, rows, vals, precision="mixed")
    assert np.linalg.norm(SA - SA_ref) <= 2e-6 * np.linalg.norm(SA_ref)
    assert np.linalg.norm(Sb - Sb_ref) <= 1e-12 * np.linalg.norm(Sb_ref)


def test_transforms_without_scratch_may_overlap():
    """FP32 transforms in shared memory of two lengths, on two streams at once through the
    entry point whose calls share one scratch: the results of the calls alone, bit for bit."""
    import torch
    rng = np.random.default_rng(3)
    jobs = []
    for N, d in ((40000, 304), (30000, 456)):
        A = torch.from_numpy(rng.standard_normal((d, N))).cuda()
        D = torch.from_numpy(np.where(rng.random(N) < 0.5, -1.0, 1.0)).cuda()
        Y = torch.zeros((d, N), dtype=torch.float64, device="cuda")
        skl.dht_device_noalloc(A.data_ptr(), N, N, d, D.data_ptr(), N, Y.data_ptr(), N)
        torch.cuda.synchronize()
        jobs.append((A, D, N, d, Y.clone(), Y, torch.cuda.Stream()))
    torch.cuda.synchronize()
    for _ in range(5):
        for A, D, N, d, _, Y, st in jobs:
            Y.zero_()
        torch.cuda.synchronize()
        for A, D, N, d, _, Y, st in jobs:
            skl.dht_device_noalloc(A.data_ptr(), N, N, d, D.data_ptr(), N, Y.data_ptr(), N, stream=st.cuda_stream)
        torch.cuda.synchronize()
        for A, D, N, d, ref, Y, st in jobs:
            assert torch.equal(ref, Y)
