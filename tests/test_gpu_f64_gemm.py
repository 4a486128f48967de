"""The FP64 CUDA-core GEMM at the edges of its tiles: 8 x 8 tiles (launches below 304 16 x 16 tiles), 16 x 16
tiles, one-row and one-column problems, K below, at and above its 32-deep k-blocks, and K cut into slices
(K >= 512 over few tiles)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (7, 9, 31), (8, 8, 32), (17, 1, 33), (1, 40, 65), (36, 36, 36), (100, 64, 511),
                                   (24, 24, 512), (9, 7, 1300), (275, 289, 64), (280, 281, 95), (1500, 3, 40)])
def test_tiles_against_bounds(M, N, K):
    from helios_gb300 import api
    rng = np.random.default_rng(M * 10007 + N * 101 + K)
    A, B = rng.normal(size=(M, K)), rng.normal(size=(N, K))
    C, _ = api.gemm(A, B, "fp64")
    ref = A.astype(np.longdouble) @ B.astype(np.longdouble).T
    # K fused multiply-adds and at most K / 128 atomic adds, each within half an ulp of a partial sum
    bound = (K + K // 128 + 1) * 2.0 ** -53 * (np.abs(A) @ np.abs(B).T)
    assert (np.abs(C - ref) <= bound * (1 + 1e-10)).all()
