"""The kernels' own scalar functions against exact arithmetic: the integer level sums of the tensor-core
products and their FP32 form, and the reciprocal of the FP32 reflectors."""
import ctypes
import math
import random

import numpy as np
import pytest

import native_build


@pytest.fixture(scope="module")
def lib(gs, tmp_path_factory):
    pytest.importorskip("torch")
    return native_build.load("scalars", tmp_path_factory.mktemp("native"))


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _ldexp(x, e):
    try:
        return math.ldexp(x, e)
    except OverflowError:
        return math.copysign(math.inf, x)


@pytest.mark.gpu
def test_level_sum_device(lib):
    """ldexp of the sum rounded to nearest even, over normal, subnormal and overflowing results."""
    import torch
    r = random.Random(70)

    def val():
        k = r.randrange(0, 48)
        v = r.getrandbits(k) if k else 0
        return v if r.random() < 0.5 else -v
    hs, ls, es = [], [], []
    for it in range(60000):
        h, l, e = val(), val(), r.choice([r.randrange(-200, 200), r.randrange(-1200, -950), r.randrange(930, 1030)])
        if it % 4 == 0:  # ties and their neighbours
            h, l = (h >> 20) << 20, r.choice([0, 1, -1, 1 << 27, -(1 << 27), (1 << 27) + 1, (1 << 27) - 1])
        hs.append(h), ls.append(l), es.append(e)
    n = len(hs)
    dev = [torch.tensor(x, dtype=t, device="cuda") for x, t in ((hs, torch.int64), (ls, torch.int64), (es, torch.int32))]
    out = torch.empty(n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    native_build.check(lib, lib.level_sums(n, *[_p(x) for x in dev], _p(out)))
    got = out.cpu().numpy()
    want = np.array([_ldexp(float(h * 2 ** 28 + l), e) for h, l, e in zip(hs, ls, es)])
    np.testing.assert_array_equal(got, want)


@pytest.mark.gpu
@pytest.mark.parametrize("h", [0, 1])
def test_f32_of_device(lib, h):
    import torch
    rng = np.random.default_rng(71)
    m = rng.integers(0, 2 ** 52, size=80000, dtype=np.uint64)
    m[::4] = (m[::4] >> np.uint64(29) << np.uint64(29)) | np.uint64(1 << 28)  # ties
    m[1::4] = m[::4] + rng.choice(np.array([-1, 1]), size=20000).astype(np.int64).view(np.uint64)
    be = np.concatenate([rng.integers(1023 - 160, 1023 + 130, size=60000), rng.integers(0, 2047, size=20000)]).astype(np.uint64)
    sign = rng.integers(0, 2, size=80000, dtype=np.uint64)
    x = ((sign << np.uint64(63)) | (be << np.uint64(52)) | (m & np.uint64(2 ** 52 - 1))).view(np.float64)
    out = torch.empty(len(x), dtype=torch.float32, device="cuda")
    d = torch.from_numpy(x).cuda()
    torch.cuda.synchronize()
    native_build.check(lib, lib.f32_ofs(len(x), _p(d), h, _p(out)))
    with np.errstate(over="ignore", under="ignore"):
        want = (x * 0.5 if h else x).astype(np.float32)
    np.testing.assert_array_equal(out.cpu().numpy(), want)


@pytest.mark.gpu
def test_rcp_markstein_is_correctly_rounded(lib):
    """Every significand, at exponents over the range where argument and reciprocal are normal."""
    import torch
    for ex in (1 + 1, 27, 97, 126, 127, 128, 157, 227, 251):
        for neg in (0, 1):
            bad = torch.zeros(1, dtype=torch.int64, device="cuda")
            torch.cuda.synchronize()
            native_build.check(lib, lib.rcp_differences(ex, neg, _p(bad)))
            assert int(bad.item()) == 0, (ex, neg, int(bad.item()))
