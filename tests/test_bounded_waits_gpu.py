"""Waits inside kernels that run out: a library built with limits of zero takes the give-up paths, ends
by itself, and says so."""
import pytest

import native_build

MIXED = """
import numpy as np
from common import assert_schur_real
rng = np.random.default_rng(64)
mats = [rng.standard_normal((n, n)) for n in (1, 2, 17, 33, 64, 65, 96, 128) for _ in range(40)]
Ts, Zs, ws, status = gs.gschur_batched(mats, mixed=True)
assert np.all(status == 0)
for A, T, Z, w in zip(mats, Ts, Zs, ws):
    assert_schur_real(A, T, Z, w)
try:
    gs.get_context().mixed_info()
    raise SystemExit("the timeout was not reported")
except RuntimeError as e:
    assert "timed out" in str(e), e
print("done")
"""


@pytest.mark.gpu
def test_refinement_waits_run_out(gs, tmp_path):
    """Every tensor-core wait gives up at once: the FP64 kernel takes the matrices, the call returns, the
    counters' call reports it."""
    lib = native_build.variant(tmp_path, ["refine_tc.cu"], ["GS_TC_WAIT_CYCLES=0"])
    assert "done" in native_build.run_with(lib, MIXED)
