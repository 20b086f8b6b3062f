"""The Lanczos iterations behind EigenStep through msdp_solver_step_eig with
L = I, against numpy's symmetric eigenvalues: the cluster kernel (up to 256)
at the orders where the number of blocks of a cluster changes (32/33, 64/65,
128/129) and at the smallest ones, the two-launch steps above.  The iteration stops when the
smallest Ritz value moved by at most 64 eps max(1, |theta|) in four steps;
with a convergence factor of at most 0.99 per four steps the rest is below
64 eps * 99 = 1.4e-12, relative to the larger of 1 and the norm; above 256 it
stops at a Ritz residual of 1e-12 of the norm, which bounds the error."""
import numpy as np
import pytest

import madsdp_gpu as M
from madsdp_gpu import generators as g
from madsdp_gpu.solver import InstanceSolver

pytestmark = pytest.mark.gpu

ORDERS = [2, 3, 4, 5, 8, 31, 32, 33, 64, 65, 100, 128, 129, 255, 256, 257, 300, 320, 321, 517]


@pytest.fixture(scope="module")
def solvers(gpu_ctx):
    made = {}

    def get(n):
        if n not in made:
            made[n] = InstanceSolver(g.maxcut(n, 0.5, seed=n))
        return made[n]

    yield get
    for s in made.values():
        s.close()


def _spectra(n, rng):
    Q = np.linalg.qr(rng.standard_normal((n, n)))[0]
    yield "spread", (Q * np.linspace(-3.0, 5.0, n)) @ Q.T
    yield "graded", (Q * np.concatenate([[-40.0], np.exp(rng.uniform(-8, 3, n - 1))])) @ Q.T
    yield "clustered", (Q * np.where(np.arange(n) < n // 2, -1.0, 1.0 + 1e-9 * np.arange(n))) @ Q.T
    yield "scaled", 1e-9 * (Q * np.linspace(-1.0, 0.5, n)) @ Q.T
    yield "identity", np.eye(n)
    yield "zero", np.zeros((n, n))


@pytest.mark.parametrize("n", ORDERS)
def test_step_eig_matches_numpy(solvers, n):
    rng = np.random.default_rng(n)
    s = solvers(n)
    for name, Z in _spectra(n, rng):
        Z = (Z + Z.T) / 2
        w = np.linalg.eigvalsh(Z)
        got = s.step_eig(0, np.eye(n), Z)
        assert abs(got - w[0]) <= 1.4e-12 * max(1.0, np.abs(w).max()), (name, got, w[0])


def test_blocks_of_different_orders_in_one_launch(gpu_ctx):
    # one launch holds the X and S sides of every block of a step length
    m = g.dense_random([130, 40, 7, 1], 3, 60, seed=3)
    a = InstanceSolver(m, max_iter=2).solve().stats()
    assert a["iter"] == 2 and 0.0 < a["alpha"] <= 1.0 and 0.0 < a["beta"] <= 1.0
