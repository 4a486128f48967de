"""SCF orbitals after a given number of iterations (scf:max-iterations reached, so not converged) against the same
iterations with numpy's FP64 eigensolver: every iteration diagonalises to FP64. The density and the orbital energies
differ by rounding alone, which a diagonalisation amplifies by ||F|| / gap: n 2^-53 x 60 eV / 3 eV x 6 iterations = 1.2e-12
at n = 90 for the density, x ||F|| for the energies."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,shape", [(12, "polyene"), (26, "polyene"), (38, "ladder"), (90, "polyene")])
@pytest.mark.parametrize("iterations", [1, 3, 6])
def test_stopped_scf(n, shape, iterations):
    from helios_gb300 import api, molecules
    from oracle.ppp import build_model
    mol = getattr(molecules, shape)(n, alpha=np.random.default_rng(n).normal(0.0, 0.3, n))
    md = build_model(mol, alternation=0.1)
    G, core, o = md["G"], md["core"], n // 2

    def fock(D):
        return core - G * D + 2.0 * np.diag(G @ np.diag(D))

    C = np.linalg.eigh(md["huckelCore"])[1]
    D = C[:, :o] @ C[:, :o].T
    for _ in range(iterations):
        F, R = fock(D), 2.0 * D - np.eye(n)
        e, C = np.linalg.eigh(fock(D - 0.05 * (F @ R - R @ F) @ R))
        D = C[:, :o] @ C[:, :o].T
    cc = api.CoupledCluster(mol, api.Keywords(bond_alternation=0.1, scf_max_iterations=iterations))
    with pytest.raises(api.HxError, match="did not|status"):
        cc.initCC()
    s = cc.scf(0)
    cc.finalizeCC()
    assert s["iterations"] == iterations
    Co = s["C"][:, :o]
    assert np.abs(Co @ Co.T - D).max() <= 1.2e-12
    assert np.abs(s["C"].T @ s["C"] - np.eye(n)).max() <= n * 2.0 ** -50
    assert np.abs(s["eps"] - e).max() <= 60 * 1.2e-12
