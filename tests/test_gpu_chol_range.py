"""Pivots at the ends of the range (msdp_dense_cholesky): the blocks
[[4, 2], [2, 5]] times a power of four, whose factor [[2, 0], [1, 2]] times a
power of two is exact, down to subnormal numbers and up to the largest
exponents of float64 and, in the mixed precision, of FP32."""
import numpy as np
import pytest
from test_gpu_chol import _factor

pytestmark = pytest.mark.gpu

FP64 = [-1048, -1040, -1024, -1022, -1020, -1000, 0, 1000, 1018, 1020]
FP32 = [-144, -140, -130, -128, -126, -124, 0, 120, 122, 124]


@pytest.mark.parametrize("n", [2, 32, 34, 70])
@pytest.mark.parametrize("prec,k", [(0, k) for k in FP64] + [(1, k) for k in FP32])
def test_exact_factor_at_any_magnitude(gpu_ctx, n, prec, k):
    A = np.kron(np.eye(n // 2), np.array([[4.0, 2.0], [2.0, 5.0]]))
    L = np.kron(np.eye(n // 2), np.array([[2.0, 0.0], [1.0, 2.0]]))
    got, info = _factor(prec, np.ldexp(A, k))
    assert info == 0
    assert np.array_equal(np.tril(got), np.ldexp(L, k // 2))
