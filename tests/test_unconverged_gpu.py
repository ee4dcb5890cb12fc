"""A batched real Schur call on matrices that do not converge: the status says so, and the places of
eigenvalues that were not found keep what the caller had there."""
import numpy as np
import pytest


def _run(gs, dtype, wantz, mats, wr0, wi0):
    torch = pytest.importorskip("torch")
    from genericschur_gb300 import _capi
    ctx = gs.get_context()
    ns = np.array([m.shape[0] for m in mats], dtype=np.int32)
    n64 = ns.astype(np.int64)
    offs = np.concatenate([[0], np.cumsum(n64 ** 2)])
    woffs = np.concatenate([[0], np.cumsum(n64)])
    A = torch.from_numpy(np.concatenate([np.asarray(m, dtype=dtype).ravel(order="F") for m in mats])).cuda()
    Z = torch.full_like(A, 0.5)
    wr = torch.full((int(woffs[-1]),), wr0, dtype=A.dtype, device="cuda")
    wi = torch.full_like(wr, wi0)
    status = torch.full((len(ns),), -1, dtype=torch.int32, device="cuda")
    meta = [torch.from_numpy(x).cuda() for x in (ns, offs[:-1].copy(), woffs[:-1].copy())]
    torch.cuda.synchronize()
    fn = ctx.lib.gs_schur_batched_f64 if dtype == np.float64 else ctx.lib.gs_schur_batched_f32
    rc = fn(ctx.handle, len(ns), *[x.data_ptr() for x in meta], A.data_ptr(), Z.data_ptr() if wantz else None, wr.data_ptr(),
            wi.data_ptr(), status.data_ptr(), _capi.GS_SCALE | _capi.GS_DEVICE | (_capi.GS_WANTZ if wantz else 0))
    assert rc == 0
    torch.cuda.synchronize()
    cut = [slice(int(a), int(a + n)) for a, n in zip(woffs, ns)]
    return [wr.cpu().numpy()[c] for c in cut], [wi.cpu().numpy()[c] for c in cut], status.cpu().numpy()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("wantz", [True, False])
def test_unconverged_keeps_eigenvalue_places(gs, dtype, wantz):
    rng = np.random.default_rng(63)
    orders = [3, 4, 5, 17, 33, 64, 65, 97, 117, 128]
    mats = [rng.standard_normal((n, n)).astype(dtype) for n in orders for _ in range(2)]
    for m in mats[::2]:
        m[1, 0] = np.nan
    wr, wi, status = _run(gs, dtype, wantz, mats, 7.25, -3.5)
    for k, m in enumerate(mats):
        if k % 2 == 0:  # nothing deflates
            assert status[k] == 1
            assert np.all(wr[k] == 7.25) and np.all(wi[k] == -3.5), m.shape
        else:
            assert status[k] == 0
            tol = 1e3 * np.finfo(dtype).eps * np.linalg.norm(m)
            assert abs(wr[k].astype(float).sum() - np.trace(m.astype(float))) <= len(m) * tol
            assert abs(wi[k].astype(float).sum()) <= tol
