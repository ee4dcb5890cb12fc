"""The one-kernel tridiagonalization where its CTAs cannot all be resident, and where a wait gives up."""
import ctypes

import numpy as np
import pytest
from scipy.linalg import eigvalsh_tridiagonal

from common import EPS
import native_build
from test_hermitian_gpu import _herm


@pytest.mark.gpu
@pytest.mark.parametrize("cplx,n,sms", [(False, 1900, 4096), (True, 1300, 4096), (False, 300, 40), (True, 300, 40)])
def test_refused_cooperative_launch(gs, tmp_path, cplx, n, sms):
    """As many SMs as the device does not have: the launch is refused, and the launches per column take
    the matrix.  (A few SMs: the cooperative kernel with fewer CTAs.)"""
    torch = pytest.importorskip("torch")
    lib = native_build.load("he_tridiag", tmp_path, link=["hermitian.cu"])
    A = _herm(np.random.default_rng(65), n, cplx)
    dt = torch.complex128 if cplx else torch.float64
    dA = torch.from_numpy(np.ascontiguousarray(A.T)).cuda()
    npart = 1024
    B, W, part, tau = (torch.zeros(k, dtype=dt, device="cuda") for k in (n * n, 2 * n, npart, n))
    ctl = torch.zeros(16, dtype=torch.float64, device="cuda")
    d, e = torch.full((n,), np.nan, dtype=torch.float64, device="cuda"), torch.full((n,), np.nan, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    p = [ctypes.c_void_p(x.data_ptr()) for x in (dA, B, W, part, ctl, tau, d, e)]
    f = lib.tridiag_c if cplx else lib.tridiag_r
    native_build.check(lib, f(p[0], n, p[1], p[2], p[3], npart, p[4], p[5], p[6], p[7], sms))
    w = eigvalsh_tridiagonal(d.cpu().numpy(), e.cpu().numpy()[:n - 1])
    w_ref = np.linalg.eigvalsh(A)
    assert np.max(np.abs(w - w_ref)) <= 10 * n * EPS * np.max(np.abs(w_ref))


GIVE_UP = """
import numpy as np
from common import EPS
rng = np.random.default_rng(66)
for cplx in (False, True):
    for n in (20, 33, 200):
        A = rng.standard_normal((n, n)) + (1j * rng.standard_normal((n, n)) if cplx else 0)
        A = (A + A.conj().T) / 2
        for call in (lambda: gs.geigen(gs.Hermitian(A, "L"), alg="DivideAndConquer"), lambda: gs.geigen(gs.Hermitian(A, "L")),
                     lambda: gs.hessenberg_hermitian(gs.Hermitian(A, "U"))):
            try:
                call()
                assert n <= 32, (cplx, n)  # one CTA waits for no other
            except RuntimeError as e:
                assert n > 32 and "gave up" in str(e), (cplx, n, e)
print("done")
"""


@pytest.mark.gpu
def test_tridiagonalization_wait_runs_out(gs, tmp_path):
    lib = native_build.variant(tmp_path, ["hermitian.cu"], ["GS_HE_WAIT_POLLS=0"])
    assert "done" in native_build.run_with(lib, GIVE_UP)
