"""The 7-slice GEMM at short K and beside the limit (256) up to which the epilogue adds the classes in fixed
point: entries just below a power of two (the largest digits) of one sign and of both, and normal ones, against extended
precision. The bound, per K max|row| max|col| with a row's largest entry at 64 units of its leading digit or more: what the
slices leave of the operands 2 x 2^-55, the slice pairs left out 6 x 2^-54, the FP32 sums of the lower classes over 256
products 6 x 2^-54, the final rounding 2^-53: 2^-50 in all."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("entries", ["largest", "largest of both signs", "normal"])
@pytest.mark.parametrize("K", [1, 2, 3, 128, 129, 255, 256, 257])
def test_exact_products(K, entries):
    from helios_gb300 import api
    rng = np.random.default_rng(K)
    A, B = rng.normal(size=(200, K)), rng.normal(size=(70, K))
    if entries != "normal":
        A, B = 1.0 - 2.0 ** -20 * rng.random(A.shape), 1.0 - 2.0 ** -20 * rng.random(B.shape)
    if entries == "largest of both signs":
        A *= rng.choice([-1.0, 1.0], size=A.shape)
        B *= rng.choice([-1.0, 1.0], size=B.shape)
    ref = A.astype(np.longdouble) @ B.astype(np.longdouble).T
    bound = 2.0 ** -50 * K * np.abs(A).max(1)[:, None] * np.abs(B).max(1)[None, :]
    for variant in range(len(api.tile_variants(3))):
        C, _ = api.gemm(A, B, "exact", variant=variant)
        assert (np.abs(C - ref) <= bound).all()
