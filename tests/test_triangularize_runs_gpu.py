"""triangularize of a matrix that is not quasi-triangular: the rotations of neighbouring subdiagonal
entries overlap and are applied in the reference's order (triang.jl:15-38), last block first."""
import numpy as np
import pytest

from common import EPS


def _sequential(T, Z):
    n = T.shape[0]
    Tc, Zc = T.astype(complex), Z.astype(complex)
    for j in range(n - 1, 0, -1):
        if T[j, j - 1] == 0:
            continue
        s, c = np.sqrt(abs(T[j, j - 1])), np.sqrt(abs(T[j - 1, j]))
        r = np.hypot(s, c)
        G = np.array([[c / r, -1j * s / r], [-1j * s / r, c / r]])
        Tc[j - 1:j + 1] = G @ Tc[j - 1:j + 1]
        Tc[:, j - 1:j + 1] = Tc[:, j - 1:j + 1] @ G.conj().T
        Zc[:, j - 1:j + 1] = Zc[:, j - 1:j + 1] @ G.conj().T
    return np.triu(Tc), Zc


@pytest.mark.gpu
@pytest.mark.parametrize("n,run", [(3, 2), (4, 3), (5, 2), (129, 2), (130, 4), (257, 6), (70, 69)])
def test_triangularize_runs(gs, n, run):
    rng = np.random.default_rng(53 + n)
    T = np.triu(rng.standard_normal((n, n)))
    for i in range(n - 1):
        if i % (run + 2) < run:
            T[i + 1, i] = rng.uniform(0.5, 1.5)
    Z = np.linalg.qr(rng.standard_normal((n, n)))[0]
    Tr, Zr = _sequential(T, Z)
    outs = [gs.triangularize(gs.Schur(T, Z, np.zeros(n, dtype=complex))) for _ in range(4)]
    for S in outs:
        np.testing.assert_array_equal(S.T, outs[0].T)
        np.testing.assert_array_equal(S.Z, outs[0].Z)
    # n unitary 2x2 rotations from either side, a few roundings each
    S = outs[0]
    assert np.linalg.norm(S.T - Tr) <= 10 * n * EPS * np.linalg.norm(T)
    assert np.linalg.norm(S.Z - Zr) <= 10 * n * EPS * np.sqrt(n)
    np.testing.assert_array_equal(S.values, np.diag(S.T))
