"""Operands sliced a row at a time (1024 < K <= 8192, contiguous, from 2^21 elements on) and beside those limits: chunks past K, rows that
start on 8 bytes only (odd K), blocks with rows missing. The bounds are those of the slices, relative to
K max|row| max|col|."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
REL = {"mixed": 2.0 ** -19, "mid": 2.0 ** -27, "high": 2.0 ** -32, "exact": 2.0 ** -45}


@pytest.mark.parametrize("mode", list(REL))
@pytest.mark.parametrize("M,N,K", [(2100, 3, 1024), (2101, 3, 1025), (1031, 5, 2048), (1030, 6, 2050), (517, 3, 4097), (257, 2, 8192),
                                   (257, 2, 8193)])
def test_edges(mode, M, N, K):
    from helios_gb300 import api
    rng = np.random.default_rng(M + N + K)
    A = rng.normal(size=(M, K)) * 10.0 ** rng.integers(-3, 4, size=(M, 1))
    B = rng.normal(size=(N, K)) * 10.0 ** rng.integers(-3, 4, size=(N, 1))
    A[0, K - 1] = 50.0 * np.abs(A).max()                # the last element decides the exponent
    ref = A.astype(np.longdouble) @ B.astype(np.longdouble).T
    bound = REL[mode] * K * np.abs(A).max(1)[:, None] * np.abs(B).max(1)[None, :]
    C, _ = api.gemm(A, B, mode)
    assert np.isfinite(C).all() and (np.abs(C - ref) <= bound).all()
