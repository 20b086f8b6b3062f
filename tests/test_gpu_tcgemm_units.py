"""The fixed-point unit of the float64 product: 2^-(47 - log2 K) of the order-0
integers, at most 2^-46.  For operands with entries in [1, 2) the unit is
2^(2 - 14 - 47 + log2 K), a last bit of the result (2^-52) or less up to
K = 128, and seven slices hold all 53 bits: A times the identity is A, bit for
bit."""
import numpy as np
import pytest
from test_gpu_tcgemm import _colmajor, _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("beta", [0.0, 1.0])
@pytest.mark.parametrize("M,K", [(1, 1), (128, 2), (129, 31), (64, 32), (200, 33), (65, 64), (300, 100), (257, 128)])
def test_times_identity_is_exact(gpu_ctx, M, K, beta):
    import torch

    from madsdp_gpu import _lib
    lib = _lib.load()
    rng = np.random.default_rng(M + K)
    A = np.ldexp(rng.integers(1 << 52, 1 << 53, size=(M, K)).astype(np.float64), -52)

    def dev(a):
        return torch.from_numpy(np.ascontiguousarray(a.T)).cuda()

    C = _run(lib, torch, 0, 0, 0, M, K, K, 1.0, beta, 0, dev(A), dev(np.eye(K)), dev(np.zeros((M, K))))
    assert np.array_equal(C.cpu().numpy().T, A)
