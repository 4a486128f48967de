"""Operands sliced a row at a time with few columns (contiguous, from 2^21 elements on): 1 to 32 threads per row, chunks
past K, rows that start on 8 bytes only (odd K), a last block with rows missing, rows of zeros and of subnormal
numbers beside ordinary ones in a warp. The bounds are those of the slices, relative to K max|row| max|col|."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
REL = {"mixed": 2.0 ** -19, "mid": 2.0 ** -27, "high": 2.0 ** -32, "exact": 2.0 ** -45}


@pytest.mark.parametrize("mode", list(REL))
@pytest.mark.parametrize("M,K", [(262147, 8), (83887, 25), (65537, 32), (61681, 34), (26215, 80), (13108, 161), (8193, 257), (2731, 769)])
def test_edges(mode, M, K):
    from helios_gb300 import api
    rng = np.random.default_rng(M + K)
    A = rng.normal(size=(M, K)) * 10.0 ** rng.integers(-3, 4, size=(M, 1))
    A[5] = 0.0
    A[8] *= 2.0 ** -1030
    A[M - 1] = 0.0
    A[M - 1, K - 1] = 2.0 ** -1074
    A[7, K - 1] = 50.0 * np.abs(A[7]).max()             # the last element decides the exponent
    B = rng.normal(size=(2, K)) * 2.0 ** 60
    ref = A.astype(np.longdouble) @ B.astype(np.longdouble).T
    bound = REL[mode] * K * np.abs(A).max(1)[:, None].astype(np.longdouble) * np.abs(B).max(1)[None, :]
    C, _ = api.gemm(A, B, mode)
    # (a product below the smallest normal number is rounded to a multiple of 2^-1074)
    assert np.isfinite(C).all() and (np.abs(C - ref) <= bound + 2.0 ** -1074).all()
