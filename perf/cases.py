"""The workloads whose speed is tracked: Schur decompositions and eigen-solvers as a program
that uses this framework calls them, from one 8 x 8 matrix to a batch of 20,000 and a single
matrix of order 2048.

A case is a dict of plain values.  `prepare` makes what the program has in hand before the
call (inputs from a seed, output buffers, the library context), `run` is one pass through
the public entry points, `work` the bytes and FLOPs that a pass cannot do without, `exact`
the outputs in 64 bits from numpy where they are unique.  Schur factors are unique only up
to the order and the phases of their columns, so they have no exact value; sorted eigenvalues,
normalised eigenvectors and eigenvalue gradients do.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "genericschur.jl_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import genericschur_gb300 as g  # noqa: E402
from genericschur_gb300 import _capi, autograd  # noqa: E402

DTYPES = {"f64": (np.float64, torch.float64, 8), "f32": (np.float32, torch.float32, 4),
          "c64": (np.complex128, torch.complex128, 16)}
SIZES_SEED = 4  # the orders of a ragged batch are part of the case, the values come from the seed
TAU = 0.1       # temperature of the differentiated loss, sum_b logsumexp(Re(lambda_b) / TAU)


def listed():
    return [
        # one tiny matrix through the host API: call latency
        {"name": "schur-one-8", "kind": "schur", "dtype": "f64", "n": 8},
        # many small systems (per-element Jacobians, small state spaces), all orders in one warp's reach
        {"name": "batch-f64-small", "kind": "batch", "dtype": "f64", "count": 4000, "lo": 3, "hi": 33},
        # the mixed-size batch of the benchmark (orders uniform in 8..128) in each data type
        {"name": "batch-f64", "kind": "batch", "dtype": "f64", "count": 2000, "lo": 8, "hi": 128},
        {"name": "batch-f32", "kind": "batch", "dtype": "f32", "count": 5000, "lo": 8, "hi": 128},
        {"name": "batch-c64", "kind": "batch", "dtype": "c64", "count": 1250, "lo": 8, "hi": 128},
        # the benchmark's batch at full size: FP32 Schur forms refined to FP64
        {"name": "batch-mixed", "kind": "mixed_batch", "dtype": "f64", "count": 20000, "lo": 8, "hi": 128},
        # eigenvalue gradients of a batch (a training step's forward and backward)
        {"name": "adjoint-64", "kind": "adjoint", "dtype": "c64", "count": 1024, "n": 64},
        # one dense matrix, values and vectors, above the small-matrix bound: real and complex
        {"name": "eigen-f64-1024", "kind": "eigen", "dtype": "f64", "n": 1024},
        {"name": "eigen-c64-256", "kind": "eigen", "dtype": "c64", "n": 256},
        # one large real matrix in the mixed-precision form
        {"name": "mixed-2048", "kind": "mixed", "dtype": "f64", "n": 2048},
        # generalized Schur forms of a batch of pencils
        {"name": "pencils-f64", "kind": "pencils", "dtype": "f64", "count": 64, "lo": 9, "hi": 65},
        # Hermitian eigenproblem, divide and conquer
        {"name": "hermitian-f64-1000", "kind": "hermitian", "dtype": "f64", "n": 1000},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["schur", "batch", "batch", "mixed_batch", "adjoint", "eigen", "mixed", "pencils", "hermitian"])
    if kind == "schur":
        return {"kind": kind, "dtype": rng.choice(["f64", "f32", "c64"]), "n": _logint(rng, 5, 128)}
    if kind == "batch":
        hi = _logint(rng, 12, 128)
        dtype = rng.choice(["f64", "f32", "c64"])
        most = {"f64": 8000, "f32": 16000, "c64": 2500}[dtype]
        return {"kind": kind, "dtype": dtype, "count": _logint(rng, 1, most), "lo": rng.randint(2, 8), "hi": hi}
    if kind == "mixed_batch":
        return {"kind": kind, "dtype": "f64", "count": _logint(rng, 16, 20000), "lo": 8, "hi": _logint(rng, 16, 128)}
    if kind == "adjoint":
        return {"kind": kind, "dtype": "c64", "count": _logint(rng, 8, 1024), "n": _logint(rng, 6, 72)}
    if kind == "eigen":
        dtype = rng.choice(["f64", "c64"])
        return {"kind": kind, "dtype": dtype, "n": _logint(rng, 10, 1000 if dtype == "f64" else 400)}
    if kind == "mixed":
        return {"kind": kind, "dtype": "f64", "n": _logint(rng, 140, 2000)}
    if kind == "pencils":
        return {"kind": kind, "dtype": rng.choice(["f64", "c64"]), "count": _logint(rng, 1, 64), "lo": 4,
                "hi": _logint(rng, 8, 65)}
    return {"kind": kind, "dtype": rng.choice(["f64", "c64"]), "n": _logint(rng, 20, 1000)}


def _orders(case):
    return np.random.default_rng(SIZES_SEED).integers(case["lo"], case["hi"] + 1, size=case["count"]).astype(np.int32)


def _offsets(ns):
    n64 = ns.astype(np.int64)
    offs = np.concatenate([[0], np.cumsum(n64 ** 2)])
    woffs = np.concatenate([[0], np.cumsum(n64)])
    return offs, woffs


def _host_normal(case, seed, shape):
    """iid N(0, 1) entries; complex entries have real and imaginary parts N(0, 1/2)."""
    rng = np.random.default_rng(seed)
    a = rng.standard_normal(shape)
    if case["dtype"] == "c64":
        a = (a + 1j * rng.standard_normal(shape)) / math.sqrt(2.0)
    return a.astype(DTYPES[case["dtype"]][0])


def _device_normal(case, seed, count):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    return torch.randn(count, dtype=DTYPES[case["dtype"]][1], device="cuda", generator=gen)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("batch", "mixed_batch"):
        ns = _orders(case)
        offs, woffs = _offsets(ns)
        A = _device_normal(case, seed, int(offs[-1]))
        real = case["dtype"] != "c64"
        wt = A.dtype
        return {"kind": kind, "case": case, "A": A, "T": torch.empty_like(A), "Z": torch.empty_like(A),
                "w": [torch.empty(int(woffs[-1]), dtype=wt, device="cuda") for _ in range(2 if real else 1)],
                "ns": torch.from_numpy(ns).cuda(), "offs": torch.from_numpy(offs[:-1].copy()).cuda(),
                "woffs": torch.from_numpy(woffs[:-1].copy()).cuda(),
                "status": torch.zeros(len(ns), dtype=torch.int32, device="cuda")}
    if kind == "adjoint":
        n, count = case["n"], case["count"]
        A = _device_normal(case, seed, count * n * n).view(count, n, n) / math.sqrt(n)
        return {"kind": kind, "A": A}
    if kind == "pencils":
        ns = _orders(case)
        flat = _host_normal(case, seed, (2, int((ns.astype(np.int64) ** 2).sum())))
        offs, _ = _offsets(ns)
        cut = [[f[o:o + n * n].reshape(n, n) for o, n in zip(offs, ns)] for f in flat]
        return {"kind": kind, "A": cut[0], "B": cut[1]}
    n = case["n"]
    A = _host_normal(case, seed, (n, n))
    if kind == "hermitian":
        A = g.Hermitian((A + A.conj().T) / 2, "L")
    return {"kind": kind, "A": A}


def _direction(z):
    """Sort key of the eigenvalues: their place along one direction of the plane, so that the two
    values of a conjugate pair, whose real parts agree but for rounding, keep a definite order."""
    return z.real + 0.5 * z.imag


def _batch(st):
    ctx = g.get_context()
    ctx.set_stream(torch.cuda.current_stream().cuda_stream or 1)
    st["T"].copy_(st["A"])  # the call overwrites its matrices with T
    flags = _capi.GS_WANTZ | _capi.GS_SCALE | _capi.GS_DEVICE
    if st["kind"] == "mixed_batch":
        flags |= _capi.GS_MIXED
    fn = {"f64": ctx.lib.gs_schur_batched_f64, "f32": ctx.lib.gs_schur_batched_f32,
          "c64": ctx.lib.gs_schur_batched_c64}[st["case"]["dtype"]]
    rc = fn(ctx.handle, st["case"]["count"], st["ns"].data_ptr(), st["offs"].data_ptr(), st["woffs"].data_ptr(),
            st["T"].data_ptr(), st["Z"].data_ptr(), *[w.data_ptr() for w in st["w"]], st["status"].data_ptr(), flags)
    if rc != _capi.GS_OK:
        raise RuntimeError(ctx.last_error())
    return {"T": st["T"], "Z": st["Z"], "w": st["w"], "status": st["status"]}


def run(state):
    kind = state["kind"]
    if kind in ("batch", "mixed_batch"):
        return _batch(state)
    if kind == "adjoint":
        A = state["A"].detach().requires_grad_(True)
        w = autograd.eigvals_batched(A)
        loss = torch.logsumexp(w.real / TAU, dim=1).sum()
        loss.backward()
        return {"w": w.detach(), "loss": loss.detach(), "grad": A.grad}
    if kind == "schur":
        S = g.gschur(state["A"])
        return {"T": S.T, "Z": S.Z, "w": S.values}
    if kind == "mixed":
        S = g.gschur_mixed(state["A"])
        return {"T": S.T, "Z": S.Z, "w": S.values}
    if kind == "eigen":
        E = g.eigen(state["A"], sortby=_direction)
        return {"values": E.values, "vectors": E.vectors}
    if kind == "hermitian":
        E = g.geigen(state["A"], alg="DivideAndConquer")
        return {"values": E.values, "vectors": E.vectors}
    out, status = g.ggschur_batched(state["A"], state["B"])
    # one array of each factor over the batch
    parts = {f: np.concatenate([np.asarray(getattr(p, f)).ravel(order="F") for p in out])
             for f in ("S", "T", "alpha", "beta", "Q", "Z")}
    return dict(parts, status=status)


def work(case):
    kind, es = case["kind"], DTYPES[case["dtype"]][2]
    real = 4.0 if case["dtype"] == "c64" else 1.0  # a complex operation is four real ones
    if kind in ("batch", "mixed_batch", "pencils"):
        n = _orders(case).astype(np.float64)
    elif kind == "adjoint":
        n = np.full(case["count"], float(case["n"]))
    else:
        n = np.array([float(case["n"])])
    n2, n3 = float((n ** 2).sum()), float((n ** 3).sum())
    # input read once; T and Z (or the vectors, or the gradient) written once
    if kind == "pencils":
        return {"bytes": 6 * es * n2, "flops": real * 66.0 * n3}
    if kind == "hermitian":
        return {"bytes": 2 * es * n2, "flops": real * (4.0 / 3 + 2 + 4.0 / 3) * n3}
    if kind == "adjoint":
        # forward Schur; backward two triangular solves, two back-transforms, one product
        return {"bytes": 2 * es * n2, "flops": real * (25.0 + 2.0 / 3 + 6.0) * n3}
    if kind == "eigen":
        return {"bytes": (es + 16) * n2, "flops": real * 25.0 * n3 + 4.0 * (1.0 / 3 + 2.0) * n3}
    return {"bytes": 3 * es * n2, "flops": real * 25.0 * n3}


def exact(case, seed):
    kind = case["kind"]
    if kind == "eigen":
        w, V = np.linalg.eig(prepare(case, seed)["A"])
        w, V = w.astype(np.complex128), V.astype(np.complex128)
        p = np.argsort(_direction(w))
        w, V = w[p], V[:, p]
        top = V[np.argmax(np.abs(V), axis=0), np.arange(V.shape[1])]
        V = V * (np.conj(top) / np.abs(top)) / np.linalg.norm(V, axis=0)
        return {"values": w, "vectors": V}
    if kind == "hermitian":
        return {"values": np.linalg.eigvalsh(prepare(case, seed)["A"].data), "vectors": None}
    if kind == "adjoint":
        A = prepare(case, seed)["A"].cpu().numpy()
        w, X = np.linalg.eig(A)
        x = w.real / TAU
        top = x.max(axis=1, keepdims=True)
        e = np.exp(x - top)
        s = e.sum(axis=1, keepdims=True)
        gbar = e / s / TAU
        # sum_i gbar_i y_i x_i^H / conj(y_i^H x_i), with y_i^H the rows of X^-1 (y_i^H x_i = 1)
        Yh = np.linalg.inv(X)
        grad = np.conj(np.swapaxes(Yh, 1, 2)) @ (gbar[:, :, None] * np.conj(np.swapaxes(X, 1, 2)))
        return {"w": None, "loss": np.asarray((top[:, 0] + np.log(s[:, 0])).sum()), "grad": grad}
    return None
