"""Device memory of a plain-FP64 handle, counted in tensors of (o v)^2 doubles: ten of a molecule (integrals, denominators,
amplitudes, residual, ring intermediates; the last level's products share the ladder's), the ladder's three of N/v, N and N^2/v^2
times that, the hole-hole one, two times diis-steps error and amplitude vectors over the pairs i <= j, and less than
3 % for everything smaller."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [66, 96, 160])
def test_bytes_of_a_handle(n):
    from helios_gb300 import api, molecules
    cc = api.CoupledCluster(molecules.polyene(n), api.Keywords(diis_steps=20))
    got = cc.timing()["device_bytes"]
    cc.finalizeCC()
    o = v = n // 2
    large = 10 * (o * v) ** 2 + o * o * v * n + 2 * (o * n) ** 2 + o ** 4 + 2 * 20 * (o * v + o * (o + 1) // 2 * v * v)
    assert 8 * large < got < 1.03 * 8 * large
