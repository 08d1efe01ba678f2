"""Builds tests/cpp/internals.cu, which calls launchers and device functions of the library that
have no C entry of their own, and loads it."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
PKG = os.path.join(ROOT, "openmbir-tem_gb300")


@pytest.fixture(scope="session")
def internals(lib_built, tmp_path_factory):
    import build as pkg_build
    so = str(tmp_path_factory.mktemp("internals") / "libinternals.so")
    cmd = ([pkg_build.nvcc(), "-std=c++17", "-O2", "-shared", "-Xcompiler", "-fPIC"] +
           pkg_build.ARCH + ["--expt-relaxed-constexpr", "-I", os.path.join(PKG, "csrc"), "-I",
                             os.path.join(ROOT, "include"), "-o", so,
                             os.path.join(HERE, "cpp", "internals.cu"), f"-L{PKG}",
                             "-Xlinker", "-l:libmbir_gb300.so", "-Xlinker", f"-rpath={PKG}"])
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    lib_built.lib()
    return C.CDLL(so)


def ptr(a, t=C.c_void_p):
    return a.ctypes.data_as(t)


def f64(*shape):
    return np.zeros(shape, np.float64)
