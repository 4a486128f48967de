"""Handles of different sizes side by side: the kernels' shared-memory limit is the process's, so a handle of
small molecules made later must leave the larger one's solves as they are."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_large_handle_after_a_small_one(precision):
    from helios_gb300 import api, molecules
    kw = api.Keywords(bond_alternation=0.1, accuracy=8, precision=precision, max_iterations=3)
    large = api.CoupledCluster(molecules.polyene(96), kw)
    alone = api.CoupledCluster(molecules.polyene(96), kw)
    alone.initCC()
    ref = alone.iterate()
    small = api.CoupledCluster(molecules.polyene(4), kw)
    for cc in (small, large):
        cc.initCC()
    small.iterate()
    out = large.iterate()
    assert out["status"] == ref["status"] == -1                # three iterations
    assert abs(out["energy"][0] - ref["energy"][0]) < 1e-9
    for cc in (large, alone, small):
        cc.finalizeCC()
