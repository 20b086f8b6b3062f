"""The NT eigendecomposition at the orders where its route changes: 8 (first
refined one), the column groups of the one-block FP32 start (8 lanes a pair,
8 columns a step: 9, 31, 33, 64, 65, 96, 97, 127, 128), cuSOLVER's FP32
start (129, 257, 384) and the FP64 eigensolver (7, 385).  Objectives and trajectories
against the oracle with the tolerances of the instance tests (1e-7 of the sum
of the objectives; per iteration 1e-6 while the gap is above 1e-5); the
counters show which route ran."""
import pytest

import madsdp_gpu as M
from madsdp_gpu import generators as g
from oracle import madsdp_oracle as o
from problems import compare_trajectories

pytestmark = pytest.mark.gpu

ORDERS = [7, 8, 9, 31, 33, 64, 65, 96, 97, 127, 128, 129, 257, 384, 385]


@pytest.mark.parametrize("n", ORDERS)
def test_routes_match_oracle(gpu_ctx, n):
    model = g.maxcut(n, min(0.8, 10.0 / n), seed=n)
    s = M.InstanceSolver(model).solve()
    st, c, traj = s.stats(), s.counters(), s.trajectory()
    s.close()
    ref = o.Solver(model).solve()
    scale = max(1.0, abs(ref.primal_objective()) + abs(ref.dual_objective()))
    assert st["status"] == M.Status.SOLVE_SUCCEEDED
    assert abs(st["iter"] - ref.iter) <= 1
    assert abs(st["pobj"] - ref.primal_objective()) <= 1e-7 * scale
    assert abs(st["dobj"] - ref.dual_objective()) <= 1e-7 * scale
    compare_trajectories(traj, ref.trajectory)
    assert (c["eig_refined"] > 0) == (8 <= n <= 384), c
