"""The library's host code on a stand-in CUDA runtime (fake_cudart.cpp): the objects of
the library, linked with it instead of the CUDA runtime.  Kernels do nothing there."""

import ctypes
import glob
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
OBJ = os.path.join(ROOT, "cuda-cvdv_b200", "lib", "obj")
CUDA = "/usr/local/cuda/include"


def load(folder):
    from cvdv_b200 import _lib
    if len(glob.glob(os.path.join(OBJ, "*.o"))) < len(glob.glob(os.path.join(ROOT, "cuda-cvdv_b200", "csrc", "*.cu"))):
        if ROOT not in sys.path:
            sys.path.insert(0, ROOT)
        import __graft_entry__ as g
        g.build()
    out = os.path.join(str(folder), "libcvdv_host.so")
    # (-Bsymbolic: a CUDA runtime that torch has loaded must not take the calls)
    subprocess.run(["g++", "-shared", "-fPIC", "-std=c++17", "-O1", "-I", CUDA, "-Wl,-Bsymbolic", "-o", out,
                    os.path.join(ROOT, "tests", "fake_cudart.cpp"), *sorted(glob.glob(os.path.join(OBJ, "*.o"))),
                    "-lpthread"], check=True)
    L = ctypes.CDLL(out)
    for name, args, res in _lib.SIGNATURES:
        fn = getattr(L, name)
        fn.argtypes, fn.restype = args, res
    L.fake_device_bytes.restype = ctypes.c_size_t
    L.fake_launches.restype = ctypes.c_long
    L.fake_fail_at.argtypes = [ctypes.c_long]
    L.fake_last_kernel.restype = ctypes.c_char_p
    L.fake_copied_to.argtypes, L.fake_copied_to.restype = [ctypes.c_void_p], ctypes.c_size_t
    L.cudaMalloc.argtypes = [ctypes.POINTER(ctypes.c_void_p), ctypes.c_size_t]
    return L
