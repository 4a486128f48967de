"""What hx_ccsd_jacobian leaves behind: the copies' DIIS history is empty, on the device and in the host's mirror, so a
solve that follows starts as it does from the same amplitudes given by set_guess."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_solve_after_jacobian_has_no_stencil_vector(precision):
    from helios_gb300 import api, lrccsd, molecules
    cc = api.CoupledCluster([molecules.polyene(14)] * 4, api.Keywords(bond_alternation=0.1, accuracy=9, precision=precision))
    cc.initCC()
    t1, t2 = cc.amplitudes(0)
    rng = np.random.default_rng(5)
    r1, r2 = rng.normal(size=t1.shape), lrccsd.pair_symmetric(rng.normal(size=t2.shape))
    cc.jacobian(t1, t2, [(0.1 * r1, 0.1 * r2)], 1e-2)
    left = [cc.amplitudes(k) for k in range(4)]
    out, after = cc.solve_batch(), [cc.trace(k) for k in range(4)]
    cc.initCC()
    for k in range(4):
        cc.set_guess(k, *left[k])
    ref, given = cc.solve_batch(), [cc.trace(k) for k in range(4)]
    cc.finalizeCC()
    assert list(out["status"]) == list(ref["status"]) == [1] * 4
    for a, g in zip(after, given):
        # the first iterations, before rounding (K slices added by atomics) is amplified; a stencil vector in the
        # history changes the second residual in its first digits
        assert np.abs(a[:4, :3] - g[:4, :3]).max() <= 1e-9 * np.abs(g[:4, :3]).max()
