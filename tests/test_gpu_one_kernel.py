"""FP64 CG and BiCGSTAB and refined CG as one cooperative kernel (small and middle systems) against
the same solves with a kernel per phase, which timing mode runs
(MONOLIS_B200_PRM_I_KERNEL_TIMERS).

FP64: both sum their dot products in double-double, so iterations and solution
are the same bits. FP32-refined CG: the plain FP64 sums of the loop differ by
their grouping, so the counts may differ a little (a refresh moved by an
iteration: 2) and each side must reach the tolerance on its FP64 residual
(1.01e-8: the norm is computed here in another order)."""
import numpy as np
import pytest

from monolis_b200 import api
from monolis_b200 import problems as P
from helpers import bits_equal

pytestmark = pytest.mark.gpu


def grid_system(dims, ndof, seed, shuffle=False, skew=0.0, points=7):
    """7- or 27-point stencil on a grid of dims points with ndof x ndof blocks,
    diagonally dominant; skew != 0: nonsymmetric; shuffle: random numbering."""
    nx, ny, nz = dims
    ids = np.arange(nx * ny * nz).reshape(nz, ny, nx)
    pairs = [(ids[:, :, :-1], ids[:, :, 1:]), (ids[:, :-1], ids[:, 1:]), (ids[:-1], ids[1:])]
    if points == 27:
        def part(d, m):
            return slice(max(0, -d), m - max(0, d)), slice(max(0, d), m + min(0, d))
        offsets = [(0, 0, 1), (0, 1, -1), (0, 1, 0), (0, 1, 1)] + [(1, y, x) for y in (-1, 0, 1) for x in (-1, 0, 1)]
        pairs = [[ids[q] for q in zip(*[part(d, m) for d, m in zip(o, (nz, ny, nx))])] for o in offsets]
    return blocks_on(nx * ny * nz, pairs, ndof, seed, shuffle, skew)


def blocks_on(n, pairs, ndof, seed, shuffle=False, skew=0.0, shift=0.05):
    """The matrix of grid_system on n nodes that are coupled in pairs."""
    rng = np.random.default_rng(seed)
    i = np.concatenate([np.arange(n)] + [a.ravel() for a, _ in pairs] + [b.ravel() for _, b in pairs])
    j = np.concatenate([np.arange(n)] + [b.ravel() for _, b in pairs] + [a.ravel() for a, _ in pairs])
    m = (len(i) - n) // 2
    w = -np.exp(0.3 * rng.standard_normal(m))
    val = np.zeros((len(i), ndof, ndof))
    for r in range(ndof):
        val[n:n + m, r, r] = w * (1 + 0.1 * r) * (1 + skew)
        val[n + m:, r, r] = w * (1 + 0.1 * r) * (1 - skew)
    coupling = 0.1 * rng.standard_normal((ndof, ndof))
    val[:n] = coupling + coupling.T
    diag = shift + np.bincount(i[n:], weights=np.abs(val[n:]).sum(axis=2).max(axis=1), minlength=n) + 0.5 * ndof
    val[np.arange(n), :, :] += diag[:, None, None] * np.eye(ndof)
    if shuffle:
        perm = rng.permutation(n)
        i, j = perm[i], perm[j]
    order = np.lexsort((j, i))
    index = np.concatenate([[0], np.cumsum(np.bincount(i, minlength=n))]).astype(np.int32)
    return index, j[order].astype(np.int32), np.ascontiguousarray(val[order]), rng.uniform(0.0, 1.0, n * ndof)


def residual(index, item, val, b, x):
    ndof = val.shape[1]
    ax = np.add.reduceat(np.einsum("krc,kc->kr", val, x.reshape(-1, ndof)[item]), index[:-1], axis=0)
    return np.linalg.norm(b - ax.reshape(-1)) / np.linalg.norm(b)


def device_solve(m, b, timers, offset=0):
    import torch
    m.Iarray[api.B200_PRM_I_KERNEL_TIMERS] = int(timers)
    d_b = torch.from_numpy(b).cuda()
    d_x = torch.full((len(b) + 2,), 7.0, dtype=torch.float64, device="cuda")  # init_x: overwritten
    torch.cuda.synchronize()
    rc = m.device_solve(d_b.data_ptr(), d_x.data_ptr() + 8 * offset)
    torch.cuda.synchronize()
    return rc, d_x.cpu().numpy()[offset:offset + len(b)], m.get_converge_iter()


# edges of slices (32 rows, 64 in FP32), of 16-byte row groups and of the split
# over the blocks; a grid whose window does not fit (random numbering); blocks
# of every size, with more and fewer slices than warps
@pytest.mark.parametrize("dims,ndof,shuffle", [
    ((1, 1, 1), 1, False), ((31, 1, 1), 1, False), ((33, 1, 1), 3, False), ((13, 5, 1), 1, False), ((5, 5, 5), 2, False),
    ((16, 16, 37), 1, False), ((17, 29, 11), 3, False), ((23, 19, 11), 2, False), ((40, 37, 31), 1, False),
    ((40, 37, 31), 1, True), ((25, 21, 19), 3, True), ((11, 12, 13), 4, False), ((9, 11, 12), 5, False),
    ((12, 11, 9), 6, False),
])
@pytest.mark.parametrize("method,precision", [(api.ITER_CG, 0), (api.ITER_CG, 1), (api.ITER_BICGSTAB, 0)])
def test_one_kernel_matches_kernels_per_phase(gpu, dims, ndof, shuffle, method, precision):
    index, item, val, b = grid_system(dims, ndof, 11, shuffle, skew=0.3 if method == api.ITER_BICGSTAB else 0.0)
    n = len(index) - 1
    m = api.Monolis(gpu)
    m.set_matrix_BCSR(n, n, ndof, len(item), val.reshape(-1), index, item)
    m.quiet()
    m.set_error_abort(False)
    m.set_method(method)
    m.set_precision(precision)
    m.set_tolerance(1e-8)
    m.set_maxiter(2000)
    m.Iarray[api.B200_PRM_I_ITER_RR] = 7  # replacement iterations on the way
    m.device_prepare()
    rc0, x0, it0 = device_solve(m, b, True)
    for offset in (0, 1):  # x on a 16-byte boundary, and not
        rc1, x1, it1 = device_solve(m, b, False, offset)
        assert rc1 == rc0 and m.Iarray[api.B200_PRM_I_LAUNCHES] == 1
        if rc0:  # one row: BiCGSTAB divides by the exact zero residual on either path
            assert n == 1
            continue
        if precision == 0:
            assert it1 == it0 and bits_equal(x1, x0)
        else:
            assert abs(it1 - it0) <= 2, (it0, it1)
            assert residual(index, item, val, b, x1) < 1.01e-8


def test_one_kernel_initial_guess_log_and_limits(gpu):
    """Start from a given x, the residual log, max_iter and a zero right-hand
    side behave as with a kernel per phase."""
    import torch
    index, item, val, b = grid_system((14, 13, 12), 1, 3)
    n = len(index) - 1
    m = api.Monolis(gpu)
    m.set_matrix_BCSR(n, n, 1, len(item), val.reshape(-1), index, item)
    m.quiet()
    m.set_error_abort(False)
    m.set_tolerance(1e-10)
    m.device_prepare()
    m.set_init_x(False)
    d_b = torch.from_numpy(b).cuda()
    out = []
    for timers in (1, 0):
        m.Iarray[api.B200_PRM_I_KERNEL_TIMERS] = timers
        d_x = torch.from_numpy(np.linspace(-1.0, 1.0, n)).cuda()
        m.show_iterlog(True)
        assert m.device_solve(d_b.data_ptr(), d_x.data_ptr()) == 0
        m.show_iterlog(False)
        out.append((d_x.cpu().numpy(), m.get_converge_iter(), m.get_converge_residual()))
    assert bits_equal(out[0][0], out[1][0]) and out[0][1:] == out[1][1:]
    m.set_maxiter(3)
    assert m.device_solve(d_b.data_ptr(), d_x.data_ptr()) == 1 and m.get_converge_iter() == 3
    zero = torch.zeros_like(d_b)
    m.set_init_x(True)
    assert m.device_solve(zero.data_ptr(), d_x.data_ptr()) == 0
    assert not d_x.cpu().numpy().any()


@pytest.mark.parametrize("method", [api.ITER_CG, api.ITER_BICGSTAB])
def test_one_kernel_wait_runs_out(gpu, method):
    """Every wait of the grid is bounded: with 2,000 polls and block 0 starting
    20 ms late (a bounded sleep) the solve returns MONOLIS_B200_TIMEOUT (4), and
    the next solve on the same device succeeds."""
    n = 14
    m = api.Monolis(gpu)
    b = P.convection_diffusion(m, n=n, peclet=0.5)
    m.quiet()
    m.set_error_abort(False)
    m.set_method(method)
    m.set_maxiter(500)
    m.set_tolerance(1e-6)
    m.device_prepare()
    m.Iarray[api.B200_PRM_I_WAIT_LIMIT] = 2000
    m.Iarray[api.B200_PRM_I_WAIT_DELAY_US] = 20000
    rc, _, _ = device_solve(m, b, False)
    assert rc == 4
    m.Iarray[api.B200_PRM_I_WAIT_LIMIT] = 0
    m.Iarray[api.B200_PRM_I_WAIT_DELAY_US] = 0
    rc, x, it = device_solve(m, b, False)
    rc0, x0, it0 = device_solve(m, b, True)
    assert rc == rc0 and it == it0 and bits_equal(x, x0)


@pytest.mark.parametrize("ndof,shuffle,method,precision", [
    (1, False, api.ITER_CG, 0), (1, True, api.ITER_CG, 0), (4, False, api.ITER_CG, 0), (1, False, api.ITER_CG, 1),
    (1, False, api.ITER_BICGSTAB, 0),
])
def test_one_kernel_any_wait_runs_out(gpu, ndof, shuffle, method, precision):
    """Block 0 late at each wait of a solve in turn, the last one included
    (where the other blocks have given up and left, and block 0 finds every sum
    complete): always TIMEOUT, never a verdict over an x that some blocks have
    not written. Late at a wait beyond the last, the solve is the plain one."""
    index, item, val, b = grid_system((15, 14, 13), ndof, 5, shuffle, skew=0.3 if method == api.ITER_BICGSTAB else 0.0)
    n = len(index) - 1
    m = api.Monolis(gpu)
    m.set_matrix_BCSR(n, n, ndof, len(item), val.reshape(-1), index, item)
    m.quiet()
    m.set_error_abort(False)
    m.set_method(method)
    m.set_precision(precision)
    m.set_tolerance(1e-12)
    m.set_maxiter(5)
    m.Iarray[api.B200_PRM_I_ITER_RR] = 3
    m.device_prepare()
    plain = device_solve(m, b, False)
    assert plain[0] == 1 and plain[2] == 5
    m.Iarray[api.B200_PRM_I_WAIT_LIMIT] = 2000
    m.Iarray[api.B200_PRM_I_WAIT_DELAY_US] = 20000
    codes = []
    for k in range(64):
        m.Iarray[api.B200_PRM_I_WAIT_DELAY_AT] = k
        rc, x, it = device_solve(m, b, False)
        codes.append(rc)
        if rc != 4:
            break
    assert codes[:-1] == [4] * (len(codes) - 1) and codes[-1] == 1, codes
    assert len(codes) - 1 >= 2 * 5 + 1  # two waits an iteration at the least
    assert it == 5 and bits_equal(x, plain[1])


@pytest.mark.parametrize("dims,ndof,method,precision,one", [
    ((62, 62, 62), 2, api.ITER_CG, 0, True), ((67, 67, 67), 2, api.ITER_CG, 0, False),  # 63 and 80 MB
    ((132, 132, 34), 2, api.ITER_CG, 1, True), ((132, 132, 38), 2, api.ITER_CG, 1, False),  # 82 and 92 MB
    ((57, 57, 57), 2, api.ITER_BICGSTAB, 0, True), ((62, 62, 62), 2, api.ITER_BICGSTAB, 0, False),  # 49 and 63 MB
    ((50, 50, 50), 3, api.ITER_BICGSTAB, 0, True), ((52, 52, 52), 3, api.ITER_BICGSTAB, 0, False),  # 70 and 78 MB
    ((35, 35, 36), 6, api.ITER_BICGSTAB, 0, False),  # 92 MB
])
def test_one_kernel_rule(gpu, dims, ndof, method, precision, one):
    """One kernel up to the matrix stream at which the kernels per phase take over, by method and block size."""
    index, item, val, b = grid_system(dims, ndof, 2)
    n = len(index) - 1
    m = api.Monolis(gpu)
    m.set_matrix_BCSR(n, n, ndof, len(item), val.reshape(-1), index, item)
    m.quiet()
    m.set_error_abort(False)
    m.set_method(method)
    m.set_precision(precision)
    m.set_maxiter(3)
    m.device_prepare()
    rc, x, it = device_solve(m, b, False)
    assert rc == 1 and it == 3 and (m.Iarray[api.B200_PRM_I_LAUNCHES] == 1) == one


@pytest.mark.parametrize("refuse", [1, 2])
@pytest.mark.parametrize("method,precision", [(api.ITER_CG, 0), (api.ITER_CG, 1), (api.ITER_BICGSTAB, 0)])
def test_one_kernel_refused_by_the_device(gpu, method, precision, refuse):
    """A launch or an allocation of the one kernel that the device refuses (a
    fake of the failing call): the same solve with a kernel per phase."""
    index, item, val, b = grid_system((14, 11, 13), 2, 8)
    n = len(index) - 1
    m = api.Monolis(gpu)
    m.set_matrix_BCSR(n, n, 2, len(item), val.reshape(-1), index, item)
    m.quiet()
    m.set_error_abort(False)
    m.set_method(method)
    m.set_precision(precision)
    m.set_tolerance(1e-8)
    m.device_prepare()
    plain = device_solve(m, b, False)
    assert plain[0] == 0 and m.Iarray[api.B200_PRM_I_LAUNCHES] == 1
    m.Iarray[api.B200_PRM_I_REFUSE_LAUNCH] = refuse
    rc, x, it = device_solve(m, b, False)
    assert rc == 0 and m.Iarray[api.B200_PRM_I_LAUNCHES] > 1
    if precision == 0:
        assert it == plain[2] and bits_equal(x, plain[1])
    else:
        assert abs(it - plain[2]) <= 2 and np.linalg.norm(x - plain[1]) <= 1e-6 * np.linalg.norm(x)


def arrow(ndof, seed):
    """9472 nodes in a ring, the first 64 coupled to 1500 nodes each besides:
    two slices with most of the matrix, the rest short."""
    n, hubs = 9472, 64
    ring = np.arange(n)
    far = np.arange(200, 200 + 6 * 1500, 6)
    pairs = [(ring[:-1], ring[1:]), (np.repeat(np.arange(hubs), len(far)), np.tile(far, hubs))]
    return blocks_on(n, pairs, ndof, seed, shift=5.0)


# what the small grids do not reach: own vectors beyond the shared memory
# (spill), matrix slices read from global memory, alone or beside cached ones,
# slices with 32-bit column ids (a slot spans more than 65,535 columns), refined
# CG without a window at ndof 1 to 3, and column bases beyond the room for them
BOTH, ALL = [(api.ITER_CG, 0), (api.ITER_CG, 1)], [(api.ITER_CG, 0), (api.ITER_CG, 1), (api.ITER_BICGSTAB, 0)]


@pytest.mark.parametrize("make,kw,ndof,method,precision", [
    (make, kw, ndof, me, pr) for make, kw, ndof, which in [
        (grid_system, dict(dims=(80, 80, 80)), 1, [(api.ITER_CG, 0)]),  # spill, all slices streamed
        (grid_system, dict(dims=(96, 96, 100)), 1, [(api.ITER_CG, 1)]),
        (grid_system, dict(dims=(61, 60, 59)), 1, ALL),
        (grid_system, dict(dims=(44, 44, 40), shuffle=True), 1, ALL),  # 32-bit column ids, cached
        (grid_system, dict(dims=(70, 70, 70), shuffle=True), 1, BOTH),  # and streamed
        (grid_system, dict(dims=(64, 64, 62), shuffle=True), 1, [(api.ITER_BICGSTAB, 0)]),
        (grid_system, dict(dims=(31, 31, 32), shuffle=True), 2, ALL),
        (grid_system, dict(dims=(27, 27, 28), shuffle=True), 3, BOTH),
        (grid_system, dict(dims=(31, 32, 31), points=27), 3, ALL),  # cached and streamed slices in a block
        (grid_system, dict(dims=(60, 60, 30), points=27), 3, BOTH),  # window, spill, streamed
        (grid_system, dict(dims=(30, 31, 29)), 6, BOTH),
        (arrow, {}, 1, ALL), (arrow, {}, 3, BOTH),
    ] for me, pr in which])
def test_one_kernel_large(gpu, make, kw, ndof, method, precision):
    if method == api.ITER_BICGSTAB and make is grid_system:
        kw = dict(kw, skew=0.3)
    index, item, val, b = make(ndof=ndof, seed=4, **kw)
    n = len(index) - 1
    m = api.Monolis(gpu)
    m.set_matrix_BCSR(n, n, ndof, len(item), val.reshape(-1), index, item)
    m.quiet()
    m.set_error_abort(False)
    m.set_method(method)
    m.set_precision(precision)
    m.set_tolerance(1e-8)
    m.set_maxiter(500)
    m.Iarray[api.B200_PRM_I_ITER_RR] = 7
    m.device_prepare()
    rc0, x0, it0 = device_solve(m, b, True)
    rc1, x1, it1 = device_solve(m, b, False)
    assert m.Iarray[api.B200_PRM_I_LAUNCHES] == 1
    assert rc1 == rc0 == 0
    wide = m.Iarray[api.B200_PRM_I_WIDE_SLICES_FP32 if precision else api.B200_PRM_I_WIDE_SLICES_FP64]
    if ndof == 1 and kw.get("shuffle"):
        assert wide > 0
    if precision == 0:
        assert it1 == it0 and bits_equal(x1, x0)
    else:
        assert abs(it1 - it0) <= 2 and residual(index, item, val, b, x1) < 1.01e-8


@pytest.mark.parametrize("method,precision", ALL)
def test_one_kernel_odd_values(gpu, method, precision):
    """Rows without entries (whole slices of them in either layout), and right-hand
    sides with Inf, NaN, squares that overflow or vanish: the status and the count
    of the kernels per phase."""
    index, item, val, b = grid_system((16, 15, 14), 1, 6, skew=0.3 if method == api.ITER_BICGSTAB else 0.0)
    n = len(index) - 1
    rows = np.repeat(np.arange(n), np.diff(index))
    gone = lambda k: (k >= 64) & (k < 200)
    keep = ~gone(rows) & ~gone(item)
    index2 = np.concatenate([[0], np.cumsum(np.bincount(rows[keep], minlength=n))]).astype(np.int32)
    rhs = [(index2, item[keep], val[keep], b)]
    for k, v in ((3, np.inf), (700, np.nan), (9, 1e200)):
        c = b.copy()
        c[k] = v
        rhs.append((index, item, val, c))
    rhs.append((index, item, val, b * 1e-200))
    for index_, item_, val_, b_ in rhs:
        m = api.Monolis(gpu)
        m.set_matrix_BCSR(n, n, 1, len(item_), val_.reshape(-1), index_, item_)
        m.quiet()
        m.set_error_abort(False)
        m.set_method(method)
        m.set_precision(precision)
        m.set_tolerance(1e-8)
        m.set_maxiter(6)
        m.device_prepare()
        rc0, x0, it0 = device_solve(m, b_, True)
        rc1, x1, it1 = device_solve(m, b_, False)
        assert rc1 == rc0 and it1 == it0
        if precision == 0 and np.isfinite(x0).all():
            assert bits_equal(x1, x0)
