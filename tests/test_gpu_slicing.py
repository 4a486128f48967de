"""The exact-slice GEMM where its operands meet the edges of tiles and k-blocks: rows and columns beside
multiples of the tile, K beside multiples of 8 (the slice pitch), 32, 64 and the one-pass limit 1024, in
every mode, against the product of the same slices in extended precision."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
# bounds relative to K max|row| max|col| (a row's largest entry is 64..128 units of its leading digit):
# truncating both operands after S digits 2^(-8(S-1)-6), the slice pairs left out (QMAX + 1 or fewer) x
# 2^(-8(QMAX+1)+2), FP32 accumulation of the classes from NX on below 2^(-8NX-15): 2^-22, 2^-28, 2^-35, 2^-51,
# with a few bits to spare
REL = {"mixed": 2.0 ** -19, "mid": 2.0 ** -27, "high": 2.0 ** -32, "exact": 2.0 ** -45}


@pytest.mark.parametrize("mode", list(REL))
@pytest.mark.parametrize("M,N,K", [(129, 33, 9), (127, 65, 64), (128, 64, 65), (3, 500, 95), (500, 3, 1023), (140, 49, 1025),
                                   (200, 97, 1032), (260, 17, 2500)])
def test_edges(mode, M, N, K):
    from helios_gb300 import api
    rng = np.random.default_rng(M * 1009 + N * 31 + K)
    A = rng.normal(size=(M, K)) * 10.0 ** rng.integers(-3, 4, size=(M, 1))
    B = rng.normal(size=(N, K)) * 10.0 ** rng.integers(-3, 4, size=(N, 1))
    A[M // 2] = 0.0
    ref = A.astype(np.longdouble) @ B.astype(np.longdouble).T
    bound = REL[mode] * K * np.abs(A).max(1)[:, None] * np.abs(B).max(1)[None, :]
    for variant in range(len(api.tile_variants(["mixed", "mid", "high", "exact"].index(mode)))):
        C, _ = api.gemm(A, B, mode, variant=variant)
        assert np.isfinite(C).all() and (np.abs(C - ref) <= bound).all()
