"""Many right-hand sides at the sizes where the kernel changes its way: fewer
rows than a block's warps take, more blocks than rows, rows of more blocks than
the lanes of a group load at once, both layouts of right-hand sides (up to 8,
more) and vectors beyond L2 (rows dealt to the blocks in turn).

Each right-hand side reaches its FP64 residual tol (1.01e-8: another order of
the norm's sum)."""
import numpy as np
import pytest

from monolis_b200 import api
from monolis_b200 import problems as P
from helpers import build
from test_gpu_one_kernel import grid_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("problem,kw,n_rhs", [
    ("laplacian", dict(n=2), 3), ("laplacian", dict(n=5), 33), ("laplacian", dict(n=21), 8),
    ("diffusion_kappa", dict(n=9), 2), ("diffusion_kappa", dict(n=14), 17), ("elasticity", dict(n=6), 11),
])
def test_multi_edges(gpu, problem, kw, n_rhs, precision):
    m, b = build(gpu, problem, **kw)
    m.set_method(api.ITER_CG)
    m.set_precond(api.PREC_DIAG)
    m.set_tolerance(1e-8)
    m.set_maxiter(5000)
    m.set_precision(precision)
    B = np.stack([b * (1 + k) + 0.1 * np.abs(b).max() * P.uniform(40 + k, len(b)) for k in range(n_rhs)])
    X, its, res, st = m.solve_multi(B)
    assert np.all(st == 0) and np.all(res < 1e-8)
    for k in range(n_rhs):
        assert np.linalg.norm(B[k] - m.matvec(X[k])) / np.linalg.norm(B[k]) < 1.01e-8, k


@pytest.mark.parametrize("n_rhs", [17, 32])  # 17 are padded to 32: the same bytes
@pytest.mark.parametrize("precision", [0, 1])
def test_multi_beyond_l2(gpu, precision, n_rhs):
    n = 58 if precision else 46  # six vectors of 32 right-hand sides: 150 MB in either precision
    index, item, val, _ = P.fv_diffusion_csr(n, 5)
    m = api.Monolis(gpu)
    m.set_matrix_BCSR(n ** 3, n ** 3, 1, len(item), val, index, item)
    m.quiet()
    m.set_error_abort(False)
    m.set_method(api.ITER_CG)
    m.set_precond(api.PREC_DIAG)
    m.set_tolerance(1e-8)
    m.set_maxiter(5000)
    m.set_precision(precision)
    B = np.stack([P.uniform(70 + k, n ** 3) for k in range(n_rhs)])
    X, its, res, st = m.solve_multi(B)
    assert np.all(st == 0) and np.all(res < 1e-8)
    for k in (0, 13, n_rhs - 1):
        assert np.linalg.norm(B[k] - P.csr_matvec(index, item, val, X[k])) / np.linalg.norm(B[k]) < 1.01e-8, k


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("ndof,n_rhs", [(1, 29), (2, 6), (2, 13), (4, 23), (5, 8), (5, 31), (6, 3), (6, 25)])
def test_multi_block_sizes(gpu, ndof, n_rhs, precision):
    index, item, val, _ = grid_system((13, 9, 8), ndof, 21)
    n = len(index) - 1
    m = api.Monolis(gpu)
    m.set_matrix_BCSR(n, n, ndof, len(item), val.reshape(-1), index, item)
    m.quiet()
    m.set_error_abort(False)
    m.set_method(api.ITER_CG)
    m.set_precond(api.PREC_DIAG)
    m.set_tolerance(1e-8)
    m.set_maxiter(2000)
    m.set_precision(precision)
    B = np.stack([P.uniform(90 + k, n * ndof) for k in range(n_rhs)])
    X, its, res, st = m.solve_multi(B)
    assert np.all(st == 0) and np.all(res < 1e-8)
    for k in range(n_rhs):
        assert np.linalg.norm(B[k] - m.matvec(X[k])) / np.linalg.norm(B[k]) < 1.01e-8, k
