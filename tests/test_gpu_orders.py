"""Solves at the orders where a route changes, against the oracle's.

- NT in one thread block per problem: from order 96 the basis of the scaling is
  orthonormal to float64 and the trajectories agree as with HKM (1e-6 while the
  gap is above 1e-5).  Below, the FP32 basis is used as it is: |V'V - I| is up to
  8e-6 and W, which V enters twice, off by up to 3e-6 of its norm (n = 48); ten
  times that holds the trajectories.
- The NT eigendecomposition on the whole GPU: FP64 eigensolver (400, 449),
  refined from an FP32 basis (450, 599).
- The step lengths of blocks of different orders in one launch: the first two
  iterations' alpha and beta, 1e-6 as in the trajectories.
- The triangular solves above order 8500, where the vectors do not fit a
  cluster: the backward error of a Cholesky solve, as in test_gpu_chol_solve."""
import numpy as np
import pytest

import madsdp_gpu as M
from madsdp_gpu import generators as g
from oracle import madsdp_oracle as o
from problems import compare_trajectories

pytestmark = pytest.mark.gpu


def test_nt_trajectories_in_one_block(gpu_ctx):
    orders = [3, 8, 16, 17, 33, 48, 49, 64, 95, 96, 97, 127, 128]
    models = [g.maxcut(n, min(0.8, 10.0 / n), seed=n) for n in orders]
    b = M.Batch(models)
    b.solve()
    for p, model in enumerate(models):
        ref = o.Solver(model).solve()
        compare_trajectories(b.trajectory(p), ref.trajectory, rtol=1e-6 if orders[p] >= 96 else 3e-5)
    b.close()


@pytest.mark.parametrize("n", [400, 449, 450, 599])
def test_whole_gpu_eigendecomposition(gpu_ctx, n):
    model = g.maxcut(n, 10.0 / n, seed=n)
    s = M.InstanceSolver(model).solve()
    st, c, traj = s.stats(), s.counters(), s.trajectory()
    s.close()
    ref = o.Solver(model).solve()
    scale = max(1.0, abs(ref.primal_objective()) + abs(ref.dual_objective()))
    assert st["status"] == M.Status.SOLVE_SUCCEEDED
    assert abs(st["pobj"] - ref.primal_objective()) <= 1e-7 * scale
    assert abs(st["dobj"] - ref.dual_objective()) <= 1e-7 * scale
    compare_trajectories(traj, ref.trajectory)
    assert (c["eig_refined"] > 0) == (n >= 450), c


def test_step_lengths_of_different_orders(gpu_ctx):
    model = g.dense_random([130, 40, 7, 1], 3, 60, seed=3)
    s = M.InstanceSolver(model, max_iter=2).solve()
    traj = s.trajectory()
    s.close()
    ref = o.Solver(model).solve()
    assert len(traj) >= 3  # the starting point, then one entry an iteration
    for k in (1, 2):
        for key in ("alpha", "beta"):
            a, b = traj[k][key], ref.trajectory[k][key]
            assert abs(a - b) <= 1e-6 * max(abs(b), 1e-3), (k, key, a, b)


def test_solve_above_the_cluster(gpu_ctx):
    m = 8530
    rng = np.random.default_rng(m)
    B = rng.standard_normal((m, 40))
    H = B @ B.T
    H[np.arange(m), np.arange(m)] += np.exp(rng.uniform(0.0, 4.0, m))
    b = rng.standard_normal(m)
    ws = M.SchurWorkspace(m)
    assert ws.factorize(H)
    x = ws.solve(b)
    ws.close()
    bound = 8 * m * np.finfo(float).eps * np.abs(H).sum(axis=1).max() * np.abs(x).max()
    assert np.abs(b - H @ x).max() <= bound
