"""The orbitals' signs are those of the FP64 cyclic Jacobi (circle ordering, from the Hueckel matrix and then from
basis to basis): amplitudes that a program keeps follow them. The molecules are ones whose signs change
when the first diagonalisation rounds its rotation angles to FP32."""
import numpy as np
import pytest

from helios_gb300 import molecules

pytestmark = pytest.mark.gpu


def _pairs(n):
    m = n + (n & 1)
    k = np.arange(m // 2)
    for r in range(m - 1):
        p = np.where(k == 0, 0, 1 + (k - 1 + r) % (m - 1))
        q = 1 + (m - 2 - k + r) % (m - 1)
        p, q = np.minimum(p, q), np.maximum(p, q)
        yield p[q < n], q[q < n]


def _jacobi(A, V, pairs):
    while True:
        tot = (A * A).sum()
        off = A - np.diag(np.diag(A))
        if (off * off).sum() <= 1e-30 * tot:
            o = np.argsort(np.diag(A), kind="stable")
            return V[:, o]
        for p, q in pairs:
            apq, d = A[p, q], A[q, q] - A[p, p]
            on = np.abs(apq) > 1e-300
            theta = d / np.where(on, 2.0 * apq, 1.0)
            t = np.where(on, np.where(theta >= 0, 1.0, -1.0) / (np.abs(theta) + np.sqrt(theta * theta + 1.0)), 0.0)
            c = 1.0 / np.sqrt(t * t + 1.0)
            s = t * c
            for X in (A, V):
                x, y = X[:, p].copy(), X[:, q].copy()
                X[:, p], X[:, q] = c * x - s * y, s * x + c * y
            x, y = A[p].copy(), A[q].copy()
            A[p], A[q] = c[:, None] * x - s[:, None] * y, s[:, None] * x + c[:, None] * y


@pytest.mark.parametrize("n,seed", [(112, 11), (90, 11), (90, 14), (27, 3), (20, 3)])
def test_signs(n, seed):
    from helios_gb300 import api
    from oracle import rhf
    from oracle.ppp import build_model
    rng = np.random.default_rng([seed, n])
    nels = np.ones(n, dtype=np.int32)
    alpha = rng.normal(0.0, 0.3, size=n)
    if n % 2:
        nels[-1], alpha[-1] = 2, alpha[-1] - 14.0
    mol = molecules.polyene(n, alpha=alpha)
    mol.nels = nels
    model = build_model(mol, alternation=0.1)
    o, pairs = int(nels.sum()) // 2, list(_pairs(n))
    V = _jacobi(model["huckelCore"].copy(), np.eye(n), pairs)
    D = rhf.density(V, o)
    F = rhf.fock(model["core"], model["G"], D)
    for _ in range(300):
        g = rhf.fmin(F, D)
        F = rhf.fock(model["core"], model["G"], D - 0.05 * g)
        V = _jacobi(V.T @ F @ V, V, pairs)
        D = rhf.density(V, o)
        F = rhf.fock(model["core"], model["G"], D)
        if np.abs(g).max() < 1e-12:
            break
    cc = api.CoupledCluster(mol, api.Keywords(bond_alternation=0.1))
    cc.initCC()
    C = cc.scf(0)["C"]
    cc.finalizeCC()
    assert np.abs(C - V).max() < 1e-6
