"""Row exponents of the exact-slice GEMM where a row holds only zeros and subnormal numbers (their high words do not
tell the exponent), beside ordinary rows, for operands sliced in one pass (K <= 1024) and in two."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
REL = {"mixed": 2.0 ** -19, "mid": 2.0 ** -27, "high": 2.0 ** -32, "exact": 2.0 ** -45}   # per K max|row| max|col|


@pytest.mark.parametrize("mode", list(REL))
@pytest.mark.parametrize("K", [8, 70, 1000, 1300])
def test_subnormal_rows(mode, K):
    from helios_gb300 import api
    rng = np.random.default_rng(K)
    A = rng.normal(size=(40, K))
    B = rng.normal(size=(24, K)) * 2.0 ** 700
    A[3] *= 2.0 ** -1030                        # subnormal
    A[4] = 0.0
    A[4, K // 2] = 2.0 ** -1074                 # the smallest one alone
    A[5] = 0.0
    A[6, 1:] = 0.0
    A[7] *= 2.0 ** -1021                        # on both sides of the smallest normal number
    ref = A.astype(np.longdouble) @ B.astype(np.longdouble).T
    C, _ = api.gemm(A, B, mode)
    bound = REL[mode] * K * np.abs(A).max(1)[:, None].astype(np.longdouble) * np.abs(B).max(1)[None, :]
    assert np.isfinite(C).all() and (np.abs(C - ref) <= bound).all()
