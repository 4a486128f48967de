"""Amplitudes cross the C ABI column-major and come back bit for bit, whatever o and v are against the
32 x 32 tiles of the device's layout kernel; the layout itself is checked through one energy evaluation."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nel", [(2, 2), (5, 8), (9, 2), (12, 12), (40, 6), (40, 74), (66, 66), (35, 4)])
def test_round_trip(n, nel):
    from dataclasses import replace
    from helios_gb300 import api, molecules
    m = molecules.polyene(n)
    nels = np.zeros(n, dtype=np.int32)
    nels[: nel // 2] = 2
    if nel == n:
        nels[:] = 1
    cc = api.CoupledCluster(replace(m, nels=nels, alpha=np.linspace(-300.0, 300.0, n)), api.Keywords())
    cc.initCC()
    o, v = nel // 2, n - nel // 2
    rng = np.random.default_rng(n * 100 + nel)
    t1, t2 = rng.normal(size=(o, v)), rng.normal(size=(o, o, v, v))
    t2 = t2 + t2.transpose(1, 0, 3, 2)
    cc.set_guess(0, t1, t2)
    b1, b2 = cc.amplitudes(0)
    assert np.array_equal(b1, t1) and np.array_equal(b2, t2)
    # the doubles energy of these amplitudes from host integrals: the tensor sits where the engine reads it
    s = cc.scf(0)
    C = s["C"]
    from helios_gb300.lrccsd import coulomb_matrix
    B = np.einsum("mi,ma->mia", C[:, :o], C[:, o:])
    g = np.einsum("mia,mn,njb->iajb", B, coulomb_matrix(m), B, optimize=True)
    L = 2 * g - g.transpose(0, 3, 2, 1)
    terms = np.einsum("iajb,ijab->iajb", L, t2 + np.einsum("ia,jb->ijab", t1, t1))
    e = cc.energyCC()
    assert abs(e[3] - terms.sum()) <= 1e-10 * np.abs(terms).sum() + 1e-12
    cc.finalizeCC()
