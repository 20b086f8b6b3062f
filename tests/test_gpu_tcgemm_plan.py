"""Tile widths, K splits and chunk loops of the tensor-core product: sizes at
the edges of the 64- and 96-column tiles, one and several K chunks per block,
K split over blocks, and both operands the same matrix, against float64
products.  Each row of an operand is sliced relative to its largest entry:
the bound is that of test_gpu_tcgemm (max_k |a_rk| sum_k |b_kc| and its
mirror), times 1e-13 (7 slices) or 2e-6 (3 slices)."""
import numpy as np
import pytest
from test_gpu_tcgemm import TOL, _colmajor, _run

pytestmark = pytest.mark.gpu

CASES = [
    # M, N, K, transa, transb, alpha, beta, lower, same operand
    (128, 96, 256, 0, 0, 1.0, 0.0, 0, False),
    (129, 97, 257, 0, 1, -1.0, 1.0, 0, False),
    (65, 193, 31, 1, 0, 1.0, 1.0, 0, False),
    (1601, 1300, 520, 0, 0, 1.0, 0.0, 0, False),
    (1601, 1300, 260, 1, 1, 0.25, -0.5, 0, False),
    (300, 290, 4100, 0, 0, 1.0, 0.0, 0, False),
    (1153, 1153, 700, 1, 0, 1.0, 0.0, 1, True),
    (2305, 2305, 33, 0, 1, -1.0, 1.0, 1, True),
]


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("case", CASES)
def test_product_plans(gpu_ctx, prec, case):
    import torch

    from madsdp_gpu import _lib
    lib = _lib.load()
    M, N, K, ta, tb, alpha, beta, lower, same = case
    rng = np.random.default_rng(M + N + K + prec)
    Ad, A = _colmajor(torch, *((K, M) if ta else (M, K)), rng)
    Bd, B = (Ad, A) if same else _colmajor(torch, *((N, K) if tb else (K, N)), rng)
    C0d, C0 = _colmajor(torch, M, N, rng)
    Cd = _run(lib, torch, prec, ta, tb, M, N, K, alpha, beta, lower, Ad, Bd, C0d)
    opA, opB = (A.T if ta else A), (B.T if tb else B)
    aa, bb = np.abs(opA), np.abs(opB)
    slicing = np.maximum(aa.max(axis=1)[:, None] * bb.sum(axis=0)[None, :],
                         aa.sum(axis=1)[:, None] * bb.max(axis=0)[None, :])
    bound = abs(alpha) * slicing + abs(beta) * np.abs(C0)
    got = Cd.cpu().numpy().T
    mask = np.tril(np.ones((M, N), dtype=bool)) if lower else np.ones((M, N), dtype=bool)
    assert np.array_equal(got[~mask], C0[~mask])
    err = (np.abs(got - (alpha * (opA @ opB) + beta * C0)) / bound)[mask].max()
    assert err <= TOL[prec], err
