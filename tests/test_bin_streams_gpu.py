"""The size bins of a batched call run in the order of their sizes, and no further ahead of a caller's own
streams than that needs."""
import ctypes
import os

import pytest

import build_lib
import native_build


@pytest.mark.gpu
def test_bin_stream_priorities(gs, tmp_path):
    rest = [f for f in os.listdir(build_lib.CSRC) if f.endswith(".cu") and f != "gschur_api.cu"]
    lib = native_build.load("bin_streams", tmp_path, link=rest)
    out, least, greatest = (ctypes.c_int * 4)(), ctypes.c_int(), ctypes.c_int()
    native_build.check(lib, lib.bin_priorities(out, ctypes.byref(least), ctypes.byref(greatest)))
    prio = list(out)  # lower numbers are higher priorities
    assert prio[3] == least.value  # that of a stream that asks for none
    assert prio == sorted(prio) and len(set(prio)) == 4
    assert prio[0] > greatest.value  # a caller can be ahead of every bin
