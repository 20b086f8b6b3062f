"""NT scaling of the batch kernel above order 95 at iterates of any magnitude:
X and S times the same power of two have the same W and 1/s times the S^-1, and
every float64 operation on the way scales with them.  The FP32 start's squares
do not fit FP32 from entries of 1e-19 down and 1e19 up; the result must not
show it.  Against W and S^-1 from numpy's eigenvectors the error is n eps
cond(X) = 128 * 2.2e-16 * 3e3 = 1e-10 at most for the points drawn here
(eigenvalues e^-4 to e^4); between scales only the route can differ, and 1e-12
leaves room for another order of the sweeps."""
import numpy as np
import pytest

import madsdp_gpu as M
from madsdp_gpu import generators as g

pytestmark = pytest.mark.gpu

SHIFTS = [0, -60, -64, -66, -68, -70, -71, -72, -73, -74, -75, -76, -80, -120, 60, 62, 64, 66, 120]


def _point(n, rng):
    Q = np.linalg.qr(rng.standard_normal((n, n)))[0]
    d = np.exp(rng.uniform(-2.0, 2.0, n))
    E = rng.standard_normal((n, n)) / np.sqrt(n)
    E = 0.5 * np.eye(n) + E @ E.T
    X, S = (Q * d ** 2) @ Q.T, (Q / d) @ E @ (Q / d).T
    return (X + X.T) / 2, (S + S.T) / 2


@pytest.mark.parametrize("n", [96, 97, 128, 140])
def test_scaling_at_any_magnitude(gpu_ctx, n):
    X, S = _point(n, np.random.default_rng(n))
    L = np.linalg.cholesky(S)
    lam, V = np.linalg.eigh(L.T @ X @ L)
    R = np.linalg.inv(L).T @ V
    W, Si = (R * np.sqrt(lam)) @ R.T, R @ R.T
    model = g.maxcut(n, 0.1, seed=n)
    b = M.Batch([model] * len(SHIFTS))
    for p, k in enumerate(SHIFTS):
        b.set_iterate(p, [np.ldexp(X, k)], [np.ldexp(S, k)], np.zeros(n))
    assert b.prepare().all()
    base = b.block_matrix(0, 0, "W")
    assert np.abs(base - W).max() <= 1e-10 * np.abs(W).max()
    assert np.abs(b.block_matrix(0, 0, "Si") - Si).max() <= 1e-10 * np.abs(Si).max()
    for p, k in enumerate(SHIFTS):
        assert np.abs(b.block_matrix(p, 0, "W") - base).max() <= 1e-12 * np.abs(base).max(), k
        assert np.abs(np.ldexp(b.block_matrix(p, 0, "Si"), k) - Si).max() <= 1e-10 * np.abs(Si).max(), k
    b.close()
