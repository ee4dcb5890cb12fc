"""Calls whose launches depend on the order or the number of matrices: the small forms give what the general
ones give."""
import numpy as np
import pytest

EPS = np.finfo(float).eps


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 18])
@pytest.mark.parametrize("wantz", [True, False])
def test_triangularize_one_cta_bound(gs, n, wantz):
    # orders on both sides of the one-CTA bound
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n))
    S = gs.gschur(A, wantZ=wantz)
    C = gs.triangularize(S)
    assert np.all(np.tril(C.T, -1) == 0)
    w = np.sort_complex(np.diag(C.T))
    # the rotations are unitary: eigenvalues and norm stay to rounding
    assert np.abs(np.linalg.norm(C.T) - np.linalg.norm(S.T)) <= 50 * n * EPS * np.linalg.norm(S.T)
    assert np.array_equal(w, np.sort_complex(C.values))
    if wantz:
        R = A @ C.Z - C.Z @ C.T
        assert np.linalg.norm(R) <= 100 * n * EPS * max(np.linalg.norm(A), 1.0)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [np.float64, np.complex128])
@pytest.mark.parametrize("n", [1, 2, 3, 31, 32, 33, 34])
def test_hermitian_one_cta_bound(gs, dtype, n):
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n)).astype(dtype)
    if dtype == np.complex128:
        A = A + 1j * rng.standard_normal((n, n))
    A = (A + A.conj().T) / 2
    E = gs.geigen(gs.Hermitian(A, "L"), alg="DivideAndConquer")
    w, V = E.values, E.vectors
    assert np.linalg.norm(A @ V - V * w) <= 100 * n * EPS * np.linalg.norm(A)
    assert np.linalg.norm(V.conj().T @ V - np.eye(n)) <= 100 * n * EPS


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.complex128])
@pytest.mark.parametrize("orders", [[1], [0, 5], [32, 33], [64, 65, 0], [128], [2] * 160 + [128], [40] * 153, [96, 97, 3]])
def test_batches_without_some_bins(gs, dtype, orders):
    # every matrix as in a batch that has matrices in all size bins and more of them than SMs
    rng = np.random.default_rng(len(orders) + orders[0])
    mats = [rng.standard_normal((n, n)).astype(dtype) for n in orders]
    rest = [rng.standard_normal((n, n)).astype(dtype) for n in [5, 40, 70, 100, 128] * 40]
    for wantz in (True, False):
        Ts, Zs, ws, st = gs.gschur_batched(mats, wantZ=wantz)
        Tr, Zr, wr, sr = gs.gschur_batched(mats + rest, wantZ=wantz)
        assert np.all(st == 0) and np.all(sr == 0)
        for k in range(len(mats)):
            assert np.array_equal(Ts[k], Tr[k]) and np.array_equal(ws[k], wr[k])
            if wantz:
                assert np.array_equal(Zs[k], Zr[k])


@pytest.mark.gpu
@pytest.mark.parametrize("count", [2, 151, 152, 153, 304, 305, 608, 609, 912, 913])
def test_complex_rounds(gs, count):
    # rounds of one launch over the SMs: every matrix once, each as by itself
    rng = np.random.default_rng(count)
    orders = rng.integers(0, 13, size=count)
    orders[:2] = [30, 90]
    mats = [rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) for n in orders]
    Ts, Zs, ws, st = gs.gschur_batched(mats)
    assert np.all(st == 0)
    for k in list(range(0, count, 37)) + [1, count - 1]:
        if orders[k] == 0:
            continue
        S = gs.gschur(mats[k])
        assert np.array_equal(Ts[k], S.T) and np.array_equal(Zs[k], S.Z) and np.array_equal(ws[k], S.values)
    for A, T, Z in zip(mats, Ts, Zs):
        n = A.shape[0]
        if n:
            assert np.linalg.norm(A @ Z - Z @ T) <= 100 * n * EPS * np.linalg.norm(A)
