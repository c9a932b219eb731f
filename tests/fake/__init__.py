"""The library linked with a CUDA runtime that needs no GPU (cudart.cpp): the host
code runs, kernels do nothing."""
import ctypes as C
import os
import shutil
import subprocess

import pytest

from dbsr_gb300 import _lib, build

HERE = os.path.dirname(os.path.abspath(__file__))


def library(tmp):
    """ctypes handle of the library's objects with the fake runtime."""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    if not os.path.exists(os.path.join(include, "cuda_runtime_api.h")):
        pytest.skip("no CUDA headers")
    build.build()
    objs = [os.path.join(build.OUT, os.path.basename(s)[:-3] + ".o") for s in build.sources()]
    so = os.path.join(str(tmp), "libdbsrgpu_fake.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-I", include,
                    "-Wl,-Bsymbolic", "-Wl,--wrap=dlopen,--wrap=dlsym",
                    os.path.join(HERE, "cudart.cpp"), *objs, "-o", so, "-lpthread"], check=True)
    L = C.CDLL(so)
    for name, res, args in _lib.SIGNATURES:
        f = getattr(L, name)
        f.restype = res
        f.argtypes = args
    L.fake_limit.argtypes = [C.c_size_t]
    L.fake_used.restype = C.c_size_t
    L.fake_fail.argtypes = [C.c_char_p]
    L.fake_log.restype = C.c_char_p
    return L
