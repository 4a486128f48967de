"""The FP32 activation of the learned-guess network, alone: with zero hidden weights and one output weight of 1 the network
returns silu(b3) of one bias. It has to be z divided by 1 + exp(-z) with a correctly rounded division: between 6 and 16 the
FP32 sum 1 + exp(-z) is known but for the exponential's error (below 2^-18 of it), so the quotients of the one or two
sums possible are the only results allowed. -inf / inf is NaN."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _silu(z):
    from helios_gb300 import api
    P = np.zeros(api.mlp_nparam(), dtype=np.float32)
    H, F = 256, 8
    b3, w4 = H * F + H + H * H + H + H * H, H * F + H + H * H + H + H * H + H     # W1 b1 W2 b2 W3 b3 w4 b4 | shift scale y_scale
    P[b3], P[w4] = z, 1.0
    P[-9:-1] = 1.0
    P[-1] = 1.0
    return api.mlp_predict(P, np.zeros((3, F), dtype=np.float32))


def test_rounding():
    z = np.random.default_rng(3).uniform(6.0, 16.0, 400).astype(np.float32)
    got = np.array([_silu(x)[0] for x in z])
    e = np.exp(-z.astype(np.float64))
    allowed = [z / (1.0 + e * (1.0 + d)).astype(np.float32) for d in (-2.0 ** -18, 0.0, 2.0 ** -18)]     # FP32 quotients
    assert all(a.dtype == np.float32 for a in allowed)
    assert ((got == allowed[0]) | (got == allowed[1]) | (got == allowed[2])).all()
    assert got.dtype == np.float32 and _silu(0.0)[2] == 0.0


def test_large_arguments():
    assert np.isnan(_silu(-np.inf)).all() and (_silu(np.inf) == np.inf).all()
    assert (_silu(200.0) == 200.0).all() and (np.abs(_silu(-100.0)) < 1e-37).all()
