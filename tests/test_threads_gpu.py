"""Several threads, each with a context of its own, whose calls want different amounts of shared memory from
the same kernels."""
import threading

import numpy as np
import pytest


def _hammer(gs, jobs, reps):
    errors = []

    def work(job):
        ctx = gs.Context()
        try:
            for _ in range(reps):
                job(ctx)
        except Exception as e:  # noqa: BLE001 - reported below
            errors.append(repr(e))
        finally:
            ctx.close()

    threads = [threading.Thread(target=work, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[:3]


@pytest.mark.gpu
def test_batched_calls_from_threads(gs):
    rng = np.random.default_rng(67)
    mats = [rng.standard_normal((n, n)) for n in (100, 128, 60, 20, 97, 65)]
    _hammer(gs, [lambda c, A=A: gs.gschur_batched([A], ctx=c) for A in mats], 60)
    cmats = [A + 1j * A.T for A in mats]
    _hammer(gs, [lambda c, A=A: gs.gschur_batched([A], ctx=c) for A in cmats[:4] + cmats[3:5]], 12)


@pytest.mark.gpu
def test_single_calls_from_threads(gs):
    rng = np.random.default_rng(68)
    mats = [rng.standard_normal((n, n)) for n in (6, 30, 70, 110, 140, 170)]
    _hammer(gs, [lambda c, A=A: gs.gschur(A, ctx=c) for A in mats], 25)


@pytest.mark.gpu
def test_pencils_from_threads(gs):
    rng = np.random.default_rng(69)
    mats = [rng.standard_normal((2, n, n)) for n in (60, 3, 4, 80, 5, 117)]
    _hammer(gs, [lambda c, A=A: gs.ggschur(A[0], A[1], ctx=c) for A in mats], 40)
