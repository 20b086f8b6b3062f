"""The cluster triangular solve and the panel kernel at their edges: orders
around one block row (32), around the cluster sizes (block rows 1 to 17) and
with several block rows per warp group (above 2048), through the Schur
component.  The solution of H x = b is held to the backward error of a
Cholesky solve: |b - H x| <= 8 n eps (|H| |x|) componentwise maxima, with
n eps the classical bound of factorization and substitution."""
import numpy as np
import pytest

import madsdp_gpu as M

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


def _system(m, seed):
    rng = np.random.default_rng(seed)
    B = rng.standard_normal((m, m + 8)) * np.exp(rng.uniform(-2, 2, m))[:, None]
    return B @ B.T + 1e-3 * np.eye(m), rng.standard_normal(m)


@pytest.mark.parametrize("m", [1, 2, 31, 32, 33, 64, 65, 127, 129, 255, 257, 511, 513, 545, 1000, 2047, 2100, 2300])
def test_schur_solve_backward_error(gpu_ctx, m):
    H, b = _system(m, m)
    ws = M.SchurWorkspace(m)
    assert ws.factorize(H)
    x = ws.solve(b)
    bound = 8 * m * EPS * np.abs(H).sum(axis=1).max() * np.abs(x).max()
    assert np.abs(b - H @ x).max() <= bound
    # a second right-hand side with the same factor
    y = ws.solve(2.0 * b)
    assert np.abs(2.0 * b - H @ y).max() <= 2 * bound
    ws.close()


@pytest.mark.parametrize("m", [33, 257, 700])
def test_mixed_solve_refines_to_float64(gpu_ctx, m):
    H, b = _system(m, m + 1)
    ws = M.SchurWorkspace(m, precision="mixed")
    assert ws.factorize(H)
    x = ws.solve(b)
    # the refinement stops at 1e-11 |b| or below
    assert np.abs(b - H @ x).max() <= 1.1e-11 * np.abs(b).max() + 8 * m * EPS * np.abs(H).sum(axis=1).max() * np.abs(x).max()
    ws.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("m", [1, 2, 31, 32, 33, 65, 257, 517])
def test_factorize_takes_any_layout(gpu_ctx, m, precision):
    # the lower triangle is read whatever the memory order: the same factor,
    # so the same bits of the solution, and nothing of the upper triangle
    H, b = _system(m, m + 2)
    low = np.where(np.tri(m, dtype=bool), H, np.nan)
    wide = np.full((2 * m, 3 * m), np.nan)
    wide[::2, ::3] = low
    ws = M.SchurWorkspace(m, precision=precision)
    got = []
    for A in (np.ascontiguousarray(low), np.asfortranarray(low), wide[::2, ::3], low.tolist()):
        assert ws.factorize(A)
        got.append(ws.solve(b))
    assert all(np.array_equal(got[0], x) for x in got[1:])
    bound = 8 * m * EPS * np.abs(H).sum(axis=1).max() * np.abs(got[0]).max()
    assert np.abs(b - H @ got[0]).max() <= bound + (1.1e-11 * np.abs(b).max() if precision == "mixed" else 0.0)
    ws.close()
