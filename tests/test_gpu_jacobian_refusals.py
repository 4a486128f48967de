"""What hx_ccsd_jacobian refuses: molecules of equal size that are not copies of one, more vectors than copies, and
settings under which the step leaves no residuals. The handle stays usable."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _call(mols, nvec=1, step=1e-2, **kw):
    from helios_gb300 import api
    cc = api.CoupledCluster(mols, api.Keywords(bond_alternation=0.1, accuracy=9, **kw))
    cc.initCC()
    t1, t2 = cc.amplitudes(0)
    try:
        return cc.jacobian(t1, t2, [(np.ones_like(t1), np.zeros_like(t2))] * nvec, step)
    finally:
        cc.finalizeCC()


@pytest.mark.parametrize("change", ["site energy", "repulsion", "bond", "geometry", "last copy"])
def test_molecules_of_equal_size_that_are_no_copies(change):
    from dataclasses import replace
    from helios_gb300 import api, molecules
    m = molecules.polyene(10)
    other = {"site energy": lambda: molecules.polyene(10, alpha=np.linspace(0.0, 0.3, 10)),
             "repulsion": lambda: replace(m, gamma=m.gamma * 1.001),
             "bond": lambda: replace(m, bonds=[(i, j, 1.01 * b, k) if i == 3 else (i, j, b, k) for i, j, b, k in m.bonds]),
             "geometry": lambda: replace(m, coords=m.coords * 1.001),
             "last copy": lambda: molecules.polyene(10, alpha=np.linspace(0.0, 1e-9, 10))}[change]()
    mols = [m, m, m, other] if change == "last copy" else [m, other, m, m]
    with pytest.raises(api.HxError, match="not a copy"):
        _call(mols)
    assert len(_call([m] * 4)) == 1
    assert len(_call([m] * 4 + [other])) == 1             # a molecule beyond the copies may be any


@pytest.mark.parametrize("kw", [dict(nvec=2), dict(step=0.0), dict(step=float("nan")), dict(diis_enabled=False), dict(projection_type="1")])
def test_bad_arguments(kw):
    from helios_gb300 import api, molecules
    with pytest.raises(api.HxError):
        _call([molecules.polyene(10)] * 4, **kw)
