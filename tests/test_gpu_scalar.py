"""Reciprocals and roots of csrc/scalar.cuh against CUDA's correctly rounded
sqrt and division, for every exponent of float64: mantissas at both ends, one
bit and runs of ones, and pseudo-random ones.  Bounds in last places, of the
correctly rounded value: exact_root none; the others by their chains, whose
relative error before the last rounding is e^3 of the FP32 start, below 2^-60,
plus one rounding of a factor of 2^-22 at most: fast_root's reciprocal and
fast_inverse 1, a quotient by the reciprocal 2, and the corrected root 2,
because near 2^-1022 the residual of its correction is subnormal and good to
half a last place of the root only."""
import ctypes as C
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


def test_against_correctly_rounded(gpu_ctx, tmp_path):
    so = str(tmp_path / "scalar_check.so")
    subprocess.run([os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc"), "-gencode", "arch=compute_103a,code=sm_103a",
                    "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-o", so,
                    os.path.join(HERE, "native", "scalar_check.cu")], check=True)
    lib = C.CDLL(so)
    worst = (C.c_uint64 * 8)()
    assert lib.check_scalar(C.c_uint(20000), worst) == 0
    names = ["root", "inverse root", "exact root", "exact inverse root", "inverse", "quotient", "widen", "truncation"]
    bounds = [2, 1, 0, 0, 1, 2, 0, 0]
    got = dict(zip(names, worst))
    assert all(w <= b for w, b in zip(worst, bounds)), got
