"""Small CUDA libraries that give tests access to single device functions of the product: a
file under tests/native/ includes the product's source and adds a kernel around the function."""
import ctypes
import os
import subprocess

import build_lib

HERE = os.path.dirname(os.path.abspath(__file__))


def load(name, tmp, link=(), defines=()):
    """Compile tests/native/<name>.cu, link it with the product's objects of the sources `link`, load it."""
    build_lib.build()
    out = os.path.join(str(tmp), name + ".so")
    cmd = [build_lib.NVCC] + build_lib.ARCH + build_lib.FLAGS + ["-I" + build_lib.CSRC] + ["-D" + d for d in defines]
    cmd += ["-shared", os.path.join(HERE, "native", name + ".cu")]
    cmd += [os.path.join(build_lib.OBJ, src + ".o") for src in link] + ["-o", out, "-lcudart"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return ctypes.CDLL(out)


def check(lib, rc):
    assert rc == 0, "CUDA error %d" % rc
