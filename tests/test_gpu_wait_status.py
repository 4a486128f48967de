"""A tensor-core wait that ran out reaches the caller: host-driven iterations, Jacobian products and solves of the handle
report it instead of returning what the unfinished tiles left. The code is put into the handle's error word by the host."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_timed_out_wait_is_reported():
    from helios_gb300 import api, molecules
    mark = api.library().hx_ccsd_test_wait_code
    cc = api.CoupledCluster([molecules.polyene(12)] * 4, api.Keywords(bond_alternation=0.1, precision="exact"))
    cc.initCC()
    t1, t2 = cc.amplitudes(0)
    calls = {"hx_ccsd_iterate": lambda: cc.iterationCC(1, 1e-10),
             "hx_ccsd_jacobian": lambda: cc.jacobian(t1, t2, [(np.ones_like(t1), np.zeros_like(t2))], 1e-2),
             "timed out": cc.solve_batch}
    for text, call in calls.items():
        cc.initCC()
        call()                                           # no wait ran out
        assert mark(cc._h, 7) == 0
        with pytest.raises(api.HxError, match=text) as e:
            call()
        assert e.value.code == -105
        assert mark(cc._h, 0) == 0
    cc.finalizeCC()
