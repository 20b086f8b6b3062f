"""The smallest eigenvalue behind EigenStep for matrices of any magnitude,
through msdp_solver_step_eig with L = I: Z times a power of two, between
2^-500 and 2^500, whose squares float64 holds.  All operations scale with it;
the error bound of test_gpu_lanczos (1.4e-12 of the larger of 1 and the norm)
is the norm's from 2^0 up and 1.4e-12 below."""
import numpy as np
import pytest

import madsdp_gpu as M
from madsdp_gpu import generators as g
from madsdp_gpu.solver import InstanceSolver

pytestmark = pytest.mark.gpu

SHIFTS = [0, 90, 99, 101, 110, 120, 125, 127, 128, 130, 200, 400, 500, -90, -99, -101, -130, -400, -500]


@pytest.mark.parametrize("n", [1, 3, 8, 32, 33, 100, 128, 129, 256, 257, 300])
def test_step_eig_at_any_magnitude(gpu_ctx, n):
    rng = np.random.default_rng(n)
    s = InstanceSolver(g.maxcut(max(n, 2), 0.5, seed=n) if n > 1 else g.dense_random([1], 0, 1, seed=1))
    Q = np.linalg.qr(rng.standard_normal((n, n)))[0]
    Z = (Q * np.linspace(-3.0, 5.0, n)) @ Q.T
    Z = (Z + Z.T) / 2
    w = np.linalg.eigvalsh(Z)
    for k in SHIFTS:
        got = s.step_eig(0, np.eye(n), np.ldexp(Z, k))
        bound = 1.4e-12 * max(1.0, np.ldexp(np.abs(w).max(), k))
        assert abs(got - np.ldexp(w[0], k)) <= bound, (k, got, np.ldexp(w[0], k))
    s.close()
