"""Small kernels of tests/device/*.cu around the library's device functions,
compiled with the library's own flags when a test asks for them."""
import ctypes
import os
import subprocess

from parphom_gb300 import build

HERE = os.path.dirname(os.path.abspath(__file__))


def load(name, folder):
    out = os.path.join(str(folder), name + ".so")
    cmd = [build.nvcc(), *build.ARCH, *build.FLAGS, "-shared", os.path.join(HERE, "device", name + ".cu"), "-o", out]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return ctypes.CDLL(out)


def ptr(t):
    return ctypes.c_void_p(t.data_ptr())
