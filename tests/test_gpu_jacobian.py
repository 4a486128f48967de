"""Jacobian products on the device (hx_ccsd_jacobian) against the same stencil through set_guess, iterationCC and
amplitudes: sizes beside the 32 x 32 tiles, o != v, both array orders, fewer vectors than copies, FP64 and
7-slice contractions."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nel,precision,nvec", [(2, 2, "fp64", 1), (9, 12, "fp64", 2), (24, 24, "exact", 3), (36, 6, "fp64", 1),
                                                  (40, 72, "exact", 1), (66, 66, "exact", 2)])
def test_against_host_stencil(n, nel, precision, nvec):
    from dataclasses import replace
    from helios_gb300 import api, lrccsd, molecules
    m = molecules.polyene(n)
    nels = np.zeros(n, dtype=np.int32)
    nels[: nel // 2] = 2
    if nel == n:
        nels[:] = 1
    m = replace(m, nels=nels, alpha=np.linspace(-40.0, 40.0, n) if nel != n else m.alpha)
    kw = api.Keywords(bond_alternation=0.1, accuracy=8)
    cc = api.CoupledCluster(m, kw)
    cc.initCC()
    t1, t2 = cc.amplitudes(0)
    C = cc.scf(0)["C"]
    cc.finalizeCC()
    rng = np.random.default_rng(n)
    vecs = []
    for k in range(nvec):
        r1, r2 = rng.normal(size=t1.shape), rng.normal(size=t2.shape)
        r2 = lrccsd.pair_symmetric(r2)
        vecs.append((np.asfortranarray(r1), np.asfortranarray(r2)) if k % 2 else (r1, np.ascontiguousarray(r2)))
    sig = lrccsd.DeviceSigma(m, kw, t1, t2, C, nvec=nvec + 1, precision=precision)
    assert sig.on_device
    dev = sig(vecs)
    sig.on_device = False
    host = sig(vecs)
    sig.close()
    # the host's residuals come back through the step: 18/12h differences of values |t + h r| rounded to
    # 2^-53, times denominators of at most a few hundred eV
    for (d1, d2), (h1, h2) in zip(dev, host):
        scale = max(np.abs(h1).max(), np.abs(h2).max())
        assert np.abs(d1 - h1).max() <= 1e-9 + 1e-11 * scale
        assert np.abs(d2 - h2).max() <= 1e-9 + 1e-11 * scale
        assert np.array_equal(d2, d2.transpose(1, 0, 3, 2))
