"""The persistent GMRES kernel at the sizes where its row blocks, shared-memory
plan and cycle logic change: a single row, fewer rows than a CTA's minimum,
ragged last blocks, basis and matrix in shared or global memory, a restart
length above the matrix size, an iteration cap inside a cycle, b = 0.

Matrices are seeded, sparse and diagonally dominant (condition number below 10),
so a relative residual of 1e-11 bounds the error by 1e-10; the iteration count
equals that of a plain numpy GMRES with two Gram-Schmidt passes up to one."""
import numpy as np
import pytest

import pgfem_gpu as pg

pytestmark = pytest.mark.gpu


def matrix(n, per_row, seed=0):
    from scipy.sparse import csr_matrix, identity
    rng = np.random.default_rng(seed)
    r = np.repeat(np.arange(n), per_row)
    c = (r + rng.integers(-4 * per_row, 4 * per_row + 1, r.size)) % n
    A = csr_matrix((rng.uniform(-1, 1, r.size), (r, c)), shape=(n, n)) * (0.8 / per_row) + 2.0 * identity(n)
    A = csr_matrix(A)
    A.sum_duplicates()
    A.sort_indices()
    return A


def numpy_gmres(A, b, kdim, tol, maxit):
    dinv = 1.0 / A.diagonal()
    x, its, bn = np.zeros_like(b), 0, np.linalg.norm(b)
    while its < maxit:
        r = b - A @ x
        beta = np.linalg.norm(r)
        if beta <= tol * bn:
            break
        m = min(kdim, maxit - its)
        V, H = [r / beta], np.zeros((m + 1, m))
        for j in range(m):
            w = A @ (dinv * V[j])
            for _ in range(2):
                h = np.array([v @ w for v in V])
                w = w - np.array(V).T @ h
                H[:j + 1, j] += h
            H[j + 1, j] = np.linalg.norm(w)
            e = np.zeros(j + 2)
            e[0] = beta
            y = np.linalg.lstsq(H[:j + 2, :j + 1], e, rcond=None)[0]
            res = np.linalg.norm(H[:j + 2, :j + 1] @ y - e)
            its += 1
            if res <= tol * bn or H[j + 1, j] == 0.0:
                break
            V.append(w / H[j + 1, j])
        x = x + dinv * (np.array(V[:len(y)]).T @ y)
        if res <= tol * bn:
            break
    return x, its


def solve(A, b, **kw):
    import torch
    s = pg.Solver(A.indptr, A.indices, A.shape[0], **kw)
    dK, db = torch.from_numpy(A.data.copy()).cuda(), torch.from_numpy(b).cuda()
    dx = torch.zeros(A.shape[0], dtype=torch.float64, device="cuda")
    i = s.solve(dK.data_ptr(), db.data_ptr(), dx.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    return dx.cpu().numpy(), i


@pytest.mark.parametrize("n,per_row,kdim", [(1, 1, 1), (5, 2, 3), (31, 3, 40), (33, 3, 4), (4735, 6, 7),
                                            (4740, 40, 30), (20003, 80, 50), (60001, 9, 60), (9001, 5, 300)])
def test_gmres_shapes(gpu, n, per_row, kdim):
    A = matrix(n, per_row)
    b = np.random.default_rng(1).normal(size=n)
    x, i = solve(A, b, kdim=kdim, tol=1e-11, maxit=2000)
    assert i.converged and not i.breakdown and i.res_norm <= 1e-10
    assert np.linalg.norm(b - A @ x) <= 1e-10 * np.linalg.norm(b)
    if n <= 5000:
        _, its = numpy_gmres(A, b, kdim, 1e-11, 2000)
        assert abs(i.iters - its) <= 1


def test_gmres_cap_and_zero_right_hand_side(gpu):
    A = matrix(1000, 5)
    b = np.random.default_rng(1).normal(size=1000)
    xo, its = numpy_gmres(A, b, 4, 1e-14, 6)  # the cap falls inside the second cycle
    x, i = solve(A, b, kdim=4, tol=1e-14, maxit=6)
    assert i.iters == 6 and not i.converged and not i.breakdown
    assert np.linalg.norm(x - xo) <= 1e-10 * np.linalg.norm(xo)
    x, i = solve(A, np.zeros(1000), kdim=4, tol=1e-14, maxit=6)
    assert i.converged and i.iters == 0 and not x.any()
