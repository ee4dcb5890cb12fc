"""Small CUDA libraries that give tests access to single device functions of the product: a
file under tests/native/ includes the product's source and adds a kernel around the function."""
import ctypes
import os
import subprocess
import sys

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


def variant(tmp, sources, defines):
    """The whole library with `sources` (names under csrc) compiled with `defines`; its path."""
    build_lib.build()
    objs = []
    for src in sorted(os.listdir(build_lib.CSRC)):
        if not src.endswith(".cu"):
            continue
        obj = os.path.join(build_lib.OBJ, src + ".o")
        if src in sources:
            obj = os.path.join(str(tmp), src + ".o")
            cmd = [build_lib.NVCC] + build_lib.ARCH + build_lib.FLAGS + ["-D" + d for d in defines]
            r = subprocess.run(cmd + ["-c", os.path.join(build_lib.CSRC, src), "-o", obj], capture_output=True, text=True)
            assert r.returncode == 0, r.stderr
        objs.append(obj)
    out = os.path.join(str(tmp), "libgschur_variant.so")
    r = subprocess.run([build_lib.NVCC] + build_lib.ARCH + ["-shared", "-o", out] + objs + ["-lcudart"],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return out


def run_with(library, code):
    """Run Python code in a process of its own whose `gs` is the host package on `library`."""
    head = "import sys\nsys.path[:0] = %r\nfrom genericschur_gb300 import _capi\n_capi.load(%r)\nimport genericschur_gb300 as gs\n" % (
        [p for p in sys.path if p], library)
    r = subprocess.run([sys.executable, "-c", head + code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout
