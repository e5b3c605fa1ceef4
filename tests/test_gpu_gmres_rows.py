"""GMRES of large systems: row counts on both sides of the line from which the
restart cycles run as a sequence of launches instead of one cooperative kernel
(20,736 rows per SM, 3.07 M rows at 148 SMs, or fewer for a small restart length),
and above 4.07 M rows, where that kernel's blocks no longer fit the shared memory.

The matrices are seeded, diagonally dominant and non-symmetric, with columns in
other blocks' rows; row sums of |offdiagonal| / diagonal are 0.9, so the error is
at most ten times the scaled residual in the maximum norm."""
import numpy as np
import pytest

from test_gpu_gmres_shapes import matrix, numpy_gmres, solve

pytestmark = pytest.mark.gpu

MOST_ROWS = 20736


def _matrix(n):
    from scipy.sparse import csr_matrix
    rng = np.random.default_rng(n)
    r = np.arange(n)
    cols = np.stack([r, (r + 1) % n, (r - 1) % n, (r + n // 2) % n, (r + n // 3 + 7) % n], axis=1)
    vals = np.empty((n, 5))
    off = rng.uniform(0.2, 1.0, (n, 4)) * np.array([-1.0, -1.0, -1.0, 1.0])
    vals[:, 1:] = off
    vals[:, 0] = np.abs(off).sum(axis=1) / 0.9
    A = csr_matrix((vals.ravel(), cols.ravel(), np.arange(0, 5 * n + 1, 5)), shape=(n, n))
    A.sort_indices()
    return A


# one kernel, then a row too many, then a restart length below its line (and restarts)
@pytest.mark.parametrize("n,kdim", [(148 * MOST_ROWS, 150), (148 * MOST_ROWS + 1, 150), (4_500_001, 30)])
def test_rows_beyond_the_persistent_kernel(gpu, n, kdim):
    A = _matrix(n)
    x0 = np.random.default_rng(1).uniform(-1, 1, n)
    b = A @ x0
    x, i = solve(A, b, kdim=kdim, tol=1e-10, maxit=400)
    assert i.converged and not i.breakdown and 50 < i.iters < 150
    r = b - A @ x
    res = np.linalg.norm(r) / np.linalg.norm(b)
    assert res <= 1.001e-10 and abs(res - i.res_norm) <= 1e-3 * res
    # |x - x0|_inf <= |D^-1 r|_inf / (1 - 0.9)
    assert np.abs(x - x0).max() <= 10.0 * (np.abs(r / A.diagonal()).max() + 1e-14)


@pytest.mark.parametrize("kdim", [4, 14, 15])  # the line, kdim + 25e6 / n < 150 - 0.68 nnz / n: 14.9
def test_small_restart_lengths(gpu, kdim):
    n = 300_000
    A = matrix(n, 80, seed=3)
    b = np.random.default_rng(1).normal(size=n)
    x, i = solve(A, b, kdim=kdim, tol=1e-11, maxit=300)
    assert i.converged and not i.breakdown
    assert np.linalg.norm(b - A @ x) <= 1e-10 * np.linalg.norm(b)
    _, its = numpy_gmres(A, b, kdim, 1e-11, 300)
    assert abs(i.iters - its) <= 1
