"""The library's objects linked with the host-side runtime of fake_cuda_runtime.cc instead of CUDA's:
the host code runs as built, kernels do nothing."""
import ctypes as C
import glob
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def load(where):
    """The library on the fake runtime, built in the folder `where`. Its own definitions win over
    those of a CUDA runtime that another package has loaded (-Bsymbolic)."""
    from faspxx_b200 import build, capi
    try:
        cuda = os.path.dirname(os.path.dirname(build.nvcc()))
    except RuntimeError:
        pytest.skip("no CUDA toolkit")
    build.build()
    lib = os.path.join(str(where), "libfasp_fake.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-Wl,-Bsymbolic", f"-I{cuda}/include",
                    os.path.join(ROOT, "tests", "fake_cuda_runtime.cc"),
                    *sorted(glob.glob(os.path.join(build.BUILD, "*.o"))), "-o", lib], check=True)
    L = C.CDLL(lib, mode=os.RTLD_LOCAL)
    for name, (res, args) in capi.SIGNATURES.items():
        getattr(L, name).restype, getattr(L, name).argtypes = res, args
    L.fake_stream.restype = C.c_void_p
    L.fake_launches.argtypes = [C.c_char_p]
    return L
