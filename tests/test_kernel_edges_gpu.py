"""Kernels at the sizes where their splits change: window and chunk edges of the batched
Schur iterations, shared-memory limits of the reductions and of the real QZ, column splits of
the Hermitian tridiagonalization, tile edges of the refinement's Sylvester solve.

Criteria as in the other tests: backward error and orthogonality 10 n eps of the compute
type, standard form, eigenvalues matched to the oracle's within 1e2 n eps ||A||_F / s_i;
for the real QZ 20 n eps; for the Hermitian path 10 n eps and Weyl's bound 10 n eps ||A||_2.
"""
import numpy as np
import pytest

from common import (EPS, assert_schur_cplx, assert_schur_real, checkblocks, eig_tolerances, match_eigenvalues,
                    randn_matrix)
from oracle import pyoracle as po
from test_hermitian_gpu import _check_eigen, _herm
from test_qz_gpu import _real_pencil_check

EPS32 = np.finfo(np.float32).eps


def _eig_tol32(A):
    """The oracle's FP64 eigenvalues of an FP32 matrix and their tolerances in FP32."""
    w, tol = eig_tolerances(A.astype(np.float64), po)
    return w, tol * (EPS32 / EPS)


# orders around the 28-wide real window with its 4- to 16-reflector chunks, the 32-lane
# rows, four columns per pass of the reductions and the shared-memory limits
REAL = [1, 2, 3, 4, 5, 15, 16, 17, 18, 27, 28, 29, 30, 31, 32, 33, 44, 45, 46, 63, 64, 65, 95, 96, 97, 111, 112, 113,
        117, 118, 119, 127, 128]
# around the 13-wide complex window, its 12-reflector chunks and the bin bounds
CPLX = [1, 2, 3, 12, 13, 14, 15, 24, 25, 26, 27, 31, 32, 33, 47, 48, 49, 79, 80, 81, 111, 112, 113, 117, 127, 128]


def _kinds(rng, n, cplx):
    """A random matrix, and one that deflates in the middle and starts its sweeps below the top."""
    A = randn_matrix(rng, n, cplx)
    B = A.copy()
    if n >= 4:
        B[n // 2:, : n // 2] *= 1e-9
    return [A, B]


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["f64", "f32", "c64"])
@pytest.mark.parametrize("alone", [False, True])
def test_schur_orders(gs, dtype, alone):
    rng = np.random.default_rng(41)
    mats = [M for n in (CPLX if dtype == "c64" else REAL) for M in _kinds(rng, n, dtype == "c64")]
    if dtype == "f32":
        mats = [M.astype(np.float32) for M in mats]
    if alone:
        res = [gs.gschur(A) for A in mats]
        res = [(S.T, S.Z, S.values) for S in res]
    else:
        Ts, Zs, ws, status = gs.gschur_batched(mats)
        assert np.all(status == 0)
        res = list(zip(Ts, Zs, ws))
    for idx, (A, (T, Z, w)) in enumerate(zip(mats, res)):
        n = A.shape[0]
        if dtype == "f32":
            A64, T64, Z64 = A.astype(np.float64), T.astype(np.float64), Z.astype(np.float64)
            assert np.all(np.tril(T, -2) == 0) and checkblocks(T)
            assert np.linalg.norm(A64 - Z64 @ T64 @ Z64.T) <= 10 * n * EPS32 * np.linalg.norm(A64)
            assert np.linalg.norm(Z64.T @ Z64 - np.eye(n)) <= 10 * n * EPS32
        elif dtype == "c64":
            assert_schur_cplx(A, T, Z, w)
        else:
            assert_schur_real(A, T, Z, w)
        if idx % 6 == 0:
            w_ref, tol = _eig_tol32(A) if dtype == "f32" else eig_tolerances(A, po)
            ok, worst = match_eigenvalues(w, w_ref, tol)
            assert ok, "n = %d: worst err/tol %.3g" % (n, worst)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,scale", [("f64", 1e-300), ("f64", 1e300), ("f32", 1e-36), ("f32", 1e36),
                                         ("c64", 1e-300), ("c64", 1e300)])
def test_schur_scaled(gs, dtype, scale):
    """Reflectors whose squares under- or overflow take the guarded path of the reductions."""
    rng = np.random.default_rng(42)
    for n in (3, 17, 33, 64, 97, 128):
        A = randn_matrix(rng, n, dtype == "c64")
        A = A.astype(np.float32) if dtype == "f32" else A
        S = gs.gschur((A * A.dtype.type(scale)).astype(A.dtype))
        T, Z = S.T.astype(np.complex128) / scale, S.Z.astype(np.complex128)
        eps = EPS32 if dtype == "f32" else EPS
        assert np.linalg.norm(A - Z @ T @ Z.conj().T) <= 10 * n * eps * np.linalg.norm(A)
        assert np.linalg.norm(Z.conj().T @ Z - np.eye(n)) <= 10 * n * eps


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["f64", "c64"])
@pytest.mark.parametrize("ctas", [1, 2])
def test_schur_ticket_queue(gs, dtype, ctas, tmp_path):
    """A bin whose CTAs are capped takes its matrices from a ticket counter; the same results."""
    rng = np.random.default_rng(43)
    mats = [randn_matrix(rng, int(n), dtype == "c64") for n in rng.integers(2, 129, size=700)]
    ref = gs.gschur_batched(mats)
    kind = "complex_f64" if dtype == "c64" else "real_f64"
    table = tmp_path / "t.tsv"
    # the same thread counts as the table in use, so that only the queue differs
    old = gs.get_context().tuning()
    rows = [r.split() for r in old.splitlines() if r.startswith(kind)]
    table.write_text("".join("%s %s %s %s %s %d\n" % (*r[:5], ctas) for r in rows))
    new = gs.Context()
    try:
        new.set_tuning(str(table))
        out = gs.gschur_batched(mats, ctx=new)
    finally:
        new.close()
    for a, b in zip(ref[:3], out[:3]):
        for x, y in zip(a, b):
            np.testing.assert_array_equal(x, y)
    np.testing.assert_array_equal(ref[3], out[3])


@pytest.mark.gpu
@pytest.mark.parametrize("n", [5, 31, 33, 81, 82, 83, 84, 116, 117, 118, 119, 128])
def test_real_qz_orders(gs, n):
    """All four matrices, two of them, or none in shared memory."""
    rng = np.random.default_rng(44 + n)
    _real_pencil_check(gs, rng.random((n, n)), rng.random((n, n)), oracle_tol=1e-7)


@pytest.mark.gpu
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 31, 32, 33, 36, 37, 255, 257, 607, 608, 609])
def test_hermitian_orders(gs, cplx, n):
    """One CTA, several, one per SM; from both triangles, and with values only."""
    A = _herm(np.random.default_rng(45 + n), n, cplx)
    w_ref = np.linalg.eigvalsh(A)
    for uplo in ("L", "U"):
        E = gs.geigen(gs.Hermitian(A, uplo), alg="DivideAndConquer")
        _check_eigen(A, E.values, E.vectors)
        assert np.max(np.abs(E.values - w_ref)) <= 10 * n * EPS * np.linalg.norm(A, 2)
    w = gs.eigvals(gs.Hermitian(A, "L"))
    assert np.max(np.abs(w - w_ref)) <= 10 * n * EPS * np.linalg.norm(A, 2)


@pytest.mark.gpu
@pytest.mark.parametrize("cplx,n", [(False, 1928), (False, 1929), (True, 1314), (True, 1315), (True, 1809)])
def test_hermitian_limits(gs, cplx, n):
    """The largest order of the one-kernel reduction, the next one, and an order whose columns
    leave a CTA of the Q accumulation with fewer warps."""
    A = _herm(np.random.default_rng(46), n, cplx)
    E = gs.geigen(gs.Hermitian(A, "L"), alg="DivideAndConquer")
    nA = np.sqrt(2 * n) * 0.9  # below ||A||_2 of this ensemble (about sqrt(2 n))
    V, w = E.vectors, E.values
    assert np.linalg.norm(A @ V - V * w[None, :]) / (n * nA * EPS) < 10
    assert np.linalg.norm(V.conj().T @ V - np.eye(n)) / (n * EPS) < 10


@pytest.mark.gpu
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("kind", ["zero", "diagonal", "tridiagonal", "graded", "tiny", "huge", "arrow"])
def test_hermitian_reflector_paths(gs, cplx, kind):
    """Reflectors with a zero tail, with squares out of range (scaled passes), and ordinary ones in one matrix."""
    n = 70
    rng = np.random.default_rng(47)
    A = _herm(rng, n, cplx)
    scale = 1.0
    if kind == "zero":
        A = np.zeros_like(A)
    elif kind == "diagonal":
        A = np.diag(np.diag(A))
    elif kind == "tridiagonal":
        A = np.triu(np.tril(A, 1), -1)
    elif kind == "graded":
        d = np.logspace(0, -150, n)
        A = A * d[:, None] * d[None, :]
    elif kind == "tiny":
        scale = 2.0 ** -960
    elif kind == "huge":
        scale = 2.0 ** 960
    elif kind == "arrow":
        B = np.diag(np.diag(A))
        B[:, 0], B[0, :] = A[:, 0], A[0, :]
        A = B
    E = gs.geigen(gs.Hermitian(A * scale, "L"), alg="DivideAndConquer")
    w, V = E.values / scale, E.vectors
    nA = max(np.linalg.norm(A, 2), np.finfo(float).tiny)
    assert np.linalg.norm(A @ V - V * w[None, :]) <= 10 * n * EPS * nA
    assert np.linalg.norm(V.conj().T @ V - np.eye(n)) <= 10 * n * EPS
    assert np.max(np.abs(w - np.linalg.eigvalsh(A))) <= 10 * n * EPS * nA


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["real", "pairs", "mixed", "close"])
@pytest.mark.parametrize("n", [129, 160, 161, 193])
def test_mixed_tiles(gs, n, kind):
    """Sylvester tiles of 1x1 blocks, of 2x2 blocks (on tile edges), of both, and with eigenvalues
    too close for the precomputed block inverses."""
    rng = np.random.default_rng(48 + n)
    A = randn_matrix(rng, n)
    if kind == "real":
        A = (A + A.T) / 2 + 1e-3 * np.triu(A, 1)
    elif kind == "pairs":
        A = (A - A.T) / 2 + 0.02 * A
    elif kind == "close":
        lam = np.repeat(np.arange(1, n // 2 + 2), 2)[:n] * (1 + 1e-7 * (np.arange(n) % 2))
        X = np.eye(n) + 0.1 * A / np.sqrt(n)
        A = X @ np.diag(lam) @ np.linalg.inv(X)
    S = gs.gschur_mixed(A)
    assert_schur_real(A, S.T, S.Z, S.values)
    w_ref, tol = eig_tolerances(A, po)
    ok, worst = match_eigenvalues(S.values, w_ref, tol)
    assert ok, "worst err/tol %.3g" % worst


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["real", "pairs", "mixed"])
def test_batched_mixed_blocks(gs, kind):
    """The closing standardisation of the 2x2 blocks, all blocks at once: none, all or some are 2x2."""
    rng = np.random.default_rng(49)
    ns = [1, 2, 3, 15, 16, 17, 32, 33, 63, 64, 65, 96, 127, 128]
    mats = []
    for n in ns:
        A = randn_matrix(rng, n)
        if kind == "real":
            A = (A + A.T) / 2 + 1e-3 * np.triu(A, 1)
        elif kind == "pairs":
            A = (A - A.T) / 2 + 0.02 * A
        mats.append(A * 3.0)
    Ts, Zs, ws, status = gs.gschur_batched(mats, mixed=True)
    assert np.all(status == 0)
    for A, T, Z, w in zip(mats, Ts, Zs, ws):
        assert_schur_real(A, T, Z, w)


@pytest.mark.gpu
@pytest.mark.parametrize("first", [0, 1, 3])
@pytest.mark.parametrize("n", [1, 2, 3, 127, 128, 129, 130, 257])
def test_triangularize_orders(gs, n, first):
    """Blocks on and across the launch's row tiles: 1x1 up to `first`, then 2x2 (every third 1x1)."""
    rng = np.random.default_rng(52 + n)
    T = np.triu(rng.standard_normal((n, n)))
    i, pairs = first, []
    while i + 1 < n:
        if i % 3 != 2:
            T[i + 1, i + 1] = T[i, i]
            T[i, i + 1], T[i + 1, i] = 1.5, -0.75
            pairs.append(i)
            i += 2
        else:
            i += 1
    Z = np.linalg.qr(rng.standard_normal((n, n)))[0]
    S = gs.triangularize(gs.Schur(T, Z, np.zeros(n, dtype=complex)))
    assert np.all(np.tril(S.T, -1) == 0)
    assert np.linalg.norm(S.Z @ S.T @ S.Z.conj().T - Z @ T @ Z.T) <= 10 * n * EPS * np.linalg.norm(T)
    assert np.linalg.norm(S.Z.conj().T @ S.Z - np.eye(n)) <= 10 * n * EPS
    w = np.diag(T).astype(complex)
    for k in pairs:  # in either order
        w[k:k + 2] = S.T[k, k].real + 1j * np.sqrt(1.5 * 0.75) * np.sign(S.T[k, k].imag) * np.array([1, -1])
        assert abs(S.T[k, k].real - T[k, k]) <= 10 * EPS * (abs(T[k, k]) + 1.5)
    assert np.max(np.abs(np.diag(S.T) - w)) <= 10 * EPS * (np.max(np.abs(w)) + 1.5)


def _block_weights(tp, tq, floor=1e-30):
    """The four weights per entry of k_sylv_solve's block solution, as the kernel forms them."""
    zp, zq = tp.shape[0], tq.shape[0]
    if zp == 1 and zq == 1:
        return np.array([[[[1.0 / (tp[0, 0] - tq[0, 0])]]]])
    c = np.trace(tq) / zq
    A, B = tp - c * np.eye(zp), tq - c * np.eye(zq)
    if zq == 2:
        q = A @ A + np.linalg.det(B) * np.eye(zp)
        inv = np.linalg.inv(q)
        K, L = inv @ A, inv
        return np.einsum("ac,bd->abcd", K, np.eye(2)) + np.einsum("ac,db->abcd", L, B)
    return np.einsum("ac,bd->abcd", np.linalg.inv(A), np.eye(1))


@pytest.mark.parametrize("zp", [1, 2])
@pytest.mark.parametrize("zq", [1, 2])
def test_block_weights_solve_sylvester(zp, zq):
    """W[a][b] = sum k[a][b][c][d] R[c][d] solves T_pp W - W T_qq = R (the identity behind the
    weights: B^2 = -det(B) I for a traceless 2x2 B)."""
    rng = np.random.default_rng(50)
    for _ in range(50):
        tp, tq, R = rng.standard_normal((zp, zp)) + 4 * np.eye(zp), rng.standard_normal((zq, zq)), rng.standard_normal((zp, zq))
        W = np.einsum("abcd,cd->ab", _block_weights(tp, tq), R)
        M = np.kron(np.eye(zq), tp) - np.kron(tq.T, np.eye(zp))
        ref = np.linalg.solve(M, R.ravel(order="F")).reshape((zp, zq), order="F")
        # two inversions of order 2 against one elimination of order 4, each to its condition
        assert np.linalg.norm(W - ref) <= 1e3 * EPS * np.linalg.cond(M) ** 2 * np.linalg.norm(ref)


def _level_sum(hs, ls, e):
    """refine_tc.cu's level_sum with the kernel's widths; None where it takes the FP64 operations."""
    t, l = hs + (ls >> 28), ls & 0xfffffff
    neg = t < 0
    if neg:
        t, l = -t - (l != 0), -l & 0xfffffff
    if t == 0 and l == 0:
        return 0.0
    sh = max(0, 28 - (64 - t.bit_length()))
    m = (t << (28 - sh)) | (l >> sh)
    assert m < 2 ** 64
    rest = l & ((1 << sh) - 1)
    z = 64 - m.bit_length()
    m <<= z
    q, low = m >> 11, (m & 2047) | (1 if rest else 0)
    q += low > 1024 or (low == 1024 and q & 1)
    be = 1023 + 63 + sh - z + e
    if be < 1 or be > 2045:
        return None
    bits = (be << 52) + (q - (1 << 52)) | (int(neg) << 63)
    return float(np.uint64(bits).view(np.float64))


def test_level_sum_rounds_to_nearest():
    from fractions import Fraction
    import random
    r = random.Random(51)

    def val():
        k = r.randrange(0, 48)
        v = r.getrandbits(k) if k else 0
        return v if r.random() < 0.5 else -v
    for it in range(20000):
        hs, ls, e = val(), val(), r.randrange(-200, 200)
        if it % 5 == 0:  # ties and their neighbours
            hs, ls = (hs >> 20) << 20, r.choice([0, 1, -1, 1 << 27, -(1 << 27), (1 << 27) + 1])
        exact = Fraction(hs * 2 ** 28 + ls) * Fraction(2) ** e
        assert _level_sum(hs, ls, e) == float(exact)
