"""The SCF where the number of CTAs that share a molecule changes with the size of the batch (16, 8 or 4), at
sites just above the one-CTA limit and beside multiples of the clusters, against the oracle's RHF."""
import numpy as np
import pytest

from helios_gb300 import molecules

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nmol", [9, 10, 76, 77])
def test_batch(nmol):
    from helios_gb300 import api
    from oracle import rhf
    from oracle.ppp import build_model
    rng = np.random.default_rng(nmol)
    sizes = [26, 34, 40][:3] * nmol
    mols = [molecules.polyene(n, alpha=rng.normal(0.0, 0.3, size=n)) for n in sizes[:nmol]]
    cc = api.CoupledCluster(mols, api.Keywords(bond_alternation=0.1, accuracy=10))
    cc.initCC()
    for k in {0, 1, 2, nmol - 2, nmol - 1}:
        ref = rhf.rhf(build_model(mols[k], alternation=0.1))
        got = cc.scf(k)
        # the energy is stationary: rounding alone, n^2 terms of some 10 eV
        assert abs(got["energy"] - ref["energy"]) < 1e-9
        assert np.abs(rhf.density(got["C"], len(got["C"]) // 2) - ref["D"]).max() < 1e-8     # gradient 1e-10 over gaps above 1 eV, x 10
    cc.finalizeCC()
