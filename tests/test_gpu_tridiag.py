"""The FP64 stage of the Ritz values on the GPU (csrc/tridiag.cuh) against
numpy's eigenvalues.  The stage searches 8e-6 of the norm around
the FP32 value and, where the eigenvalue is not in there, the whole interval:
the shifts below make it miss to either side by all or nothing of that width.
Sturm counts are exact for entries off by 4 eps, and the last bracket is 2 eps
wide: 8 eps of the norm."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
EPS = np.finfo(float).eps
D = C.POINTER(C.c_double)


@pytest.fixture(scope="module")
def lib(gpu_ctx, tmp_path_factory):
    so = str(tmp_path_factory.mktemp("tridiag") / "tridiag_device_check.so")
    subprocess.run([os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc"), "-gencode", "arch=compute_103a,code=sm_103a",
                    "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-o", so,
                    os.path.join(HERE, "native", "tridiag_device_check.cu")], check=True)
    lib = C.CDLL(so)
    lib.check_min64.argtypes = [C.c_int, C.c_int, D, D, C.POINTER(C.c_float), D]
    return lib


@pytest.mark.parametrize("k", [1, 2, 5, 8, 9, 33, 100, 256])
def test_min64_finds_a_missed_bracket(lib, k):
    rng = np.random.default_rng(k)
    shifts = np.array([0.0, 6e-6, 9e-6, 2e-5, 1e-3, 0.3, 1.5, -6e-6, -9e-6, -2e-5, -1e-3, -0.3, -1.5], dtype=np.float32)
    count = 40 * len(shifts)
    shift = np.tile(shifts, 40).copy()
    a = rng.standard_normal((count, k))
    b = np.zeros((count, k))
    b[:, 1:] = rng.standard_normal((count, k - 1)) * np.exp(rng.uniform(-6, 0, (count, 1)))
    out = np.zeros(count)
    rc = lib.check_min64(count, k, a.ctypes.data_as(D), b.ctypes.data_as(D),
                         shift.ctypes.data_as(C.POINTER(C.c_float)), out.ctypes.data_as(D))
    assert rc == 0
    for i in range(count):
        T = np.diag(a[i]) + np.diag(b[i, 1:], 1) + np.diag(b[i, 1:], -1)
        want = np.linalg.eigvalsh(T)[0]
        norm = np.abs(T).sum(axis=1).max()
        # eigvalsh itself: k eps of the norm at most
        assert abs(out[i] - want) <= (8 + k) * EPS * norm, (i, shift[i], out[i], want)
