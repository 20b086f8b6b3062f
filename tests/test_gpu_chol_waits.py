"""A wait of the Cholesky's panel kernel that runs out is an error of its own
and not a pivot: with no polls at all the warps look once, go on and report it
(error 6); with the default limit the same call factors, and a matrix that is
not positive definite is reported by its pivot alone."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
D = C.POINTER(C.c_double)


@pytest.fixture(scope="module")
def potrf(gpu_ctx, tmp_path_factory):
    from madsdp_gpu import _lib
    _lib.load()
    so = str(tmp_path_factory.mktemp("chol") / "chol_wait_check.so")
    libdir = os.path.join(os.path.dirname(HERE), "madsdp.jl_gb300", "lib")
    subprocess.run([os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc"), "-gencode", "arch=compute_103a,code=sm_103a",
                    "-O2", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-cudart", "shared", "-o", so,
                    os.path.join(HERE, "native", "chol_wait_check.cu"),
                    os.path.join(libdir, "libmadsdp_gpu.so"), "-Xlinker", "-rpath=" + libdir], check=True)
    lib = C.CDLL(so)
    lib.check_potrf.argtypes = [C.c_int, D, C.c_int, C.c_int, C.POINTER(C.c_int), C.POINTER(C.c_int)]

    def run(A, mixed, polls):
        F = np.asfortranarray(A)
        info, err = C.c_int(), C.c_int()
        assert lib.check_potrf(A.shape[0], F.ctypes.data_as(D), mixed, polls, C.byref(info), C.byref(err)) == 0
        return F, info.value, err.value

    return run


def _spd(n):
    B = np.random.default_rng(n).standard_normal((n, n + 4))
    return B @ B.T / n + np.eye(n)


@pytest.mark.parametrize("mixed", [0, 1])
@pytest.mark.parametrize("n", [20, 33, 300])
def test_wait_that_runs_out_is_reported(potrf, n, mixed):
    A = _spd(n)
    _, info, err = potrf(A, mixed, 0)
    assert err == 6 and info != 0
    F, info, err = potrf(A, mixed, -1)
    assert info == 0 and err == 0
    L = np.tril(F)
    assert np.abs(L @ L.T - A).max() <= (1e-4 if mixed else 1e-12) * np.abs(A).max()
    A[n - 2, n - 2] = -1.0
    _, info, err = potrf(A, mixed, -1)
    assert info == n - 1 and err == 0
