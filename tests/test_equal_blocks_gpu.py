"""The large mixed refinement where block pairs of its Sylvester equation are equal or nearly so:
repeated decoupled 2x2 blocks, and the precomputed block solutions themselves.
"""
import ctypes
from fractions import Fraction

import numpy as np
import pytest

from common import EPS, assert_schur_real, randn_matrix
import native_build


def _repeated(rng, k, J, m, first):
    """A random block of order k and m copies of J on the diagonal."""
    n = k + 2 * m
    A = np.zeros((n, n))
    o = 0 if first else 2 * m
    A[o:o + k, o:o + k] = randn_matrix(rng, k)
    for i in range(m):
        p = (k if first else 0) + 2 * i
        A[p:p + 2, p:p + 2] = J
    return A


@pytest.mark.gpu
@pytest.mark.parametrize("first", [True, False])
@pytest.mark.parametrize("J", [((0.0, 1.0), (-1.0, 0.0)), ((0.5, 2.0), (-1.0, 0.5)), ((0.1, 2.0), (-1.1, 0.1))])
@pytest.mark.parametrize("k,m", [(100, 30), (140, 3), (64, 100)])
def test_mixed_repeated_blocks(gs, k, m, J, first):
    """Equal 2x2 blocks have no solution of their block equation: the refinement still converges by
    itself (no FP64 recomputation), since the parts are decoupled."""
    A = _repeated(np.random.default_rng(61), k, np.array(J), m, first)
    S, info = gs.gschur_mixed(A, return_info=True, fallback=False)
    assert info["iterations"] >= 0
    assert_schur_real(A, S.T, S.Z, S.values)


def _solve(tp, tq, R, zp, zq):
    """W of T_pp W - W T_qq = R by rational elimination; None where it is singular."""
    m = zp * zq
    M = [[Fraction(0)] * (m + 1) for _ in range(m)]
    for b in range(zq):
        for a in range(zp):
            r = a + b * zp
            for a2 in range(zp):
                M[r][a2 + b * zp] += Fraction(float(tp[a, a2]))
            for b2 in range(zq):
                M[r][a + b2 * zp] -= Fraction(float(tq[b2, b]))
            M[r][m] = Fraction(float(R[a, b]))
    for c in range(m):
        p = max(range(c, m), key=lambda i: abs(M[i][c]))
        if M[p][c] == 0:
            return None
        M[c], M[p] = M[p], M[c]
        for i in range(m):
            if i != c and M[i][c] != 0:
                f = M[i][c] / M[c][c]
                M[i] = [x - f * y for x, y in zip(M[i], M[c])]
    return np.array([[float(M[a + b * zp][m] / M[a + b * zp][a + b * zp]) for b in range(zq)] for a in range(zp)])


def _block(rng, z, like=None, gap=0.0):
    if z == 1:
        t = np.array([[rng.standard_normal()]])
    else:
        a, b, c = rng.standard_normal(3)
        t = np.array([[a, abs(b) + 0.1], [-abs(c) - 0.1, a]])
    if like is not None:
        t = like + gap * np.eye(z)
    return t


@pytest.mark.gpu
@pytest.mark.parametrize("zp", [1, 2])
@pytest.mark.parametrize("zq", [1, 2])
def test_block_weights_device(gs, tmp_path, zp, zq):
    """The kernel's own function: refuses what is singular or nearly so, and what it accepts is as
    close to the exact solution as its derivation says.

    The entries of Q = A^2 + det(B) I carry an error of 3 eps `big` each (products of entries and their
    sum), which reaches its inverse as 12 eps kappa, kappa = |Q| big / |det Q| <= 1e8, relative to
    |Q^-1|; the products with A, B and R add 8 eps; so |W - W*| <= (12 kappa + 8) eps |Q^-1| (|A| + |B|) |R|
    with |.| at most twice the largest entry of each.
    """
    torch = pytest.importorskip("torch")
    lib = native_build.load("block_weights", tmp_path)
    rng = np.random.default_rng(62)
    pairs = []
    for k in range(400):
        tp = _block(rng, zp)
        if zp == zq and k % 2:
            gap = [0.0, 1e-300, 1e-160, 1e-25, 1e-16, 1e-12, 1e-9, 1e-6, 1e-4, 1e-2, 0.1][(k // 2) % 11]
            tq = _block(rng, zq, tp, gap)
        else:
            tq = _block(rng, zq)
        s = [1.0, 1.0, 1e-4, 1e-10, 1e-24, 1e-100, 1e-170][k % 7]
        pairs.append((tp * s, tq * s, rng.standard_normal((zp, zq)) * s))
    n = len(pairs)
    P, Q, R = np.zeros((n, 2, 2)), np.zeros((n, 2, 2)), np.zeros((n, 2, 2))
    for i, (tp, tq, r) in enumerate(pairs):
        P[i, :zp, :zp], Q[i, :zq, :zq] = tp, tq
        R[i, :zq, :zp] = r.T  # rhs[a + 2 b]
    floor = 1e-3 * EPS
    dev = [torch.from_numpy(x).cuda() for x in (P, Q, np.full(n, zp, np.int32), np.full(n, zq, np.int32), R)]
    w = torch.zeros(n, 4, dtype=torch.float64, device="cuda")
    fine = torch.ones(n, dtype=torch.int32, device="cuda")
    p = [ctypes.c_void_p(x.data_ptr()) for x in dev]
    torch.cuda.synchronize()
    native_build.check(lib, lib.weights(n, *p, ctypes.c_double(floor), ctypes.c_void_p(w.data_ptr()),
                                        ctypes.c_void_p(fine.data_ptr())))
    w, fine = w.cpu().numpy(), fine.cpu().numpy()
    taken = 0
    for i, (tp, tq, r) in enumerate(pairs):
        lp, lq = np.linalg.eigvals(tp), np.linalg.eigvals(tq)
        sep = np.min(np.abs(lp[:, None] - lq[None, :]))
        if zp == 1 and zq == 1:  # floored in place
            m = tp[0, 0] - tq[0, 0]
            m = m if abs(m) >= floor else (-floor if m < 0 else floor)
            assert w[i, 0] == 0 or abs(w[i, 0] - r[0, 0] / m) <= 4 * EPS * abs(r[0, 0] / m)
            taken += 1
            continue
        if sep < floor:
            assert not fine[i], (i, tp, tq)
        if not fine[i]:
            continue
        taken += 1
        W = np.array([[w[i, a + 2 * b] for b in range(zq)] for a in range(zp)])
        assert np.all(np.isfinite(W))
        ref = _solve(tp, tq, r, zp, zq)
        c = np.trace(tq) / zq
        A, B = tp - c * np.eye(zp), tq - c * np.eye(zq)
        det = np.linalg.det(B) if zq == 2 else 0.0
        Qm = A @ A + det * np.eye(zp) if zq == 2 else A
        big = np.max(np.abs(A)) ** 2 + abs(det) if zq == 2 else np.max(np.abs(A))
        inv = np.linalg.inv(Qm)
        kappa = np.max(np.abs(inv)) * big  # |Q| / |det Q| is the inverse's largest entry
        rest = 2 * np.max(np.abs(A)) + 2 * np.max(np.abs(B)) if zq == 2 else 1.0
        bound = (12 * kappa + 8) * EPS * 2 * np.max(np.abs(inv)) * rest * 2 * np.max(np.abs(r))
        assert np.max(np.abs(W - ref)) <= bound, (i, W, ref)
    assert taken >= n // 5
    # an ordinary pair, eigenvalues apart by a hundredth, is always taken
    ok = [fine[i] for i, (tp, tq, _) in enumerate(pairs)
          if np.max(np.abs(tp)) > 0.1 and np.min(np.abs(np.linalg.eigvals(tp)[:, None] - np.linalg.eigvals(tq)[None])) > 0.01]
    assert ok and all(ok)
