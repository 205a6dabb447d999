"""The library's host code linked against fake_cuda.cpp, the logging stand-in
for the CUDA runtime (no GPU needed, kernels do not run)."""
import ctypes as C
import glob
import os
import subprocess

from pyflct_gb300 import _lib, build

HERE = os.path.dirname(os.path.abspath(__file__))


def load(folder):
    """libflctgpu.so's objects with the stand-in, built in `folder`."""
    build.build()
    out = os.path.join(str(folder), "libflctfake.so")
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build.nvcc()))), "include")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I", inc,
                    os.path.join(HERE, "fake_cuda.cpp"), *sorted(glob.glob(os.path.join(build.BUILD, "*.o"))),
                    "-o", out, "-lpthread"], check=True)
    lib = _lib.load(out)
    lib.fake_log.restype = C.c_char_p
    lib.fake_reset.argtypes = [C.c_long]
    return lib


class Host:
    """One context on the stand-in."""

    def __init__(self, lib):
        self.lib = lib
        self.h = C.c_void_p()
        assert lib.flct_gpu_create(0, C.byref(self.h)) == _lib.OK

    def close(self):
        self.lib.flct_gpu_destroy(self.h)

    def call(self, name, *args, fail_at=0):
        """Status and log lines of one entry point; fail_at: the n-th runtime call fails."""
        self.lib.fake_reset(fail_at)
        rc = getattr(self.lib, "flct_gpu_" + name)(self.h, *args)
        return rc, self.lib.fake_log().decode().splitlines()
