"""The library's host code on a CUDA runtime without a device (runtime.cpp), for tests of what it
does when memory runs out."""
import ctypes as C
import os
import subprocess

from yune_gb300 import _native as N
from yune_gb300 import build

HERE = os.path.dirname(os.path.abspath(__file__))


def load(out_dir):
    """Links the library's objects with the runtime of this folder; returns the loaded library."""
    lib = os.path.join(str(out_dir), "libyune_fake.so")
    objs = [build._obj(s) for s in build.CU_SOURCES + build.CXX_SOURCES]
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic",
                    "-I" + os.path.join(os.path.dirname(os.path.dirname(build.NVCC)), "include"),
                    os.path.join(HERE, "runtime.cpp")] + objs + ["-o", lib, "-lpthread"], check=True)
    L = C.CDLL(lib)
    for name, (res, args) in N.SIGNATURES.items():
        fn = getattr(L, name)
        fn.restype, fn.argtypes = res, args
    for name, res, args in (("fake_limit", None, [C.c_uint64]), ("fake_bytes", C.c_uint64, []),
                            ("fake_peak", C.c_uint64, []), ("fake_reset_peak", None, []),
                            ("fake_launches", C.c_longlong, []), ("fake_mallocs", C.c_longlong, []), ("fake_allocations", C.c_int, []),
                            ("fake_store", None, [C.c_uint64, C.c_int, C.c_int])):
        fn = getattr(L, name)
        fn.restype, fn.argtypes = res, args
    return L


NO_LIMIT = 2 ** 64 - 1
