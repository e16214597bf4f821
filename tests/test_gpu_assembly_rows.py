"""Device assembly at the sizes where the warp-per-row kernels change their way:
rows of more than 32 blocks, nodes of more than 32 elements, elements of more
than 32 nodes, a node twice in an element, a column stored twice in a row,
conditions repeated on a dof. Bit-identical to the host calls made in order."""
import numpy as np
import pytest

from monolis_b200 import api
from helpers import bits_equal

pytestmark = pytest.mark.gpu


def meshes():
    rng = np.random.default_rng(3)
    star = np.stack([np.zeros(50, dtype=int), np.arange(1, 51)], axis=1)  # node 0: 51 blocks, 50 elements
    tris = rng.integers(0, 40, (90, 3))  # repeated nodes in some elements, many elements a node
    tris[:5, 2] = tris[:5, 0]
    big = np.stack([rng.permutation(80)[:40] for _ in range(6)])  # 40 nodes an element
    big[0, 39] = big[0, 0]
    chain = np.stack([np.arange(0, 200), np.arange(1, 201)], axis=1)
    return {"star": (51, star), "tris": (40, tris), "big": (80, big), "chain": (201, chain)}


def device_values(m, lib):
    v = np.empty(m.NZ * m.NDOF ** 2)
    assert lib.monolis_b200_device_get_values(m.p, v.ctypes.data_as(api._dp)) == 0
    return v


def setup(gpu, name, ndof):
    n, elem = meshes()[name]
    ms = []
    for _ in range(2):
        m = api.Monolis(gpu)
        m.get_nonzero_pattern_flat(n, elem.shape[1], ndof, elem)
        m.quiet()
        ms.append(m)
    return n, np.ascontiguousarray(elem, dtype=np.int32), ms


@pytest.mark.parametrize("name", ["star", "tris", "big", "chain"])
@pytest.mark.parametrize("ndof,scaled,own", [(1, True, False), (2, False, True), (3, True, True), (6, False, False)])
def test_rows_and_conditions_match_host(gpu, name, ndof, scaled, own):
    import torch
    n, elem, (mh, md) = setup(gpu, name, ndof)
    rng = np.random.default_rng(7)
    ne, nb = elem.shape
    size = (nb * ndof) ** 2
    val = rng.standard_normal(size * (ne if own else 1))
    scale = rng.standard_normal(ne) if scaled else None
    mh.add_elements(elem, nb, val, size if own else 0, scale=scale)
    mh.add_elements(elem, nb, val, size if own else 0, scale=scale)
    d_elem, d_val = torch.from_numpy(elem).cuda(), torch.from_numpy(val).cuda()
    d_scale = torch.from_numpy(scale).cuda() if scaled else None
    torch.cuda.synchronize()
    assert gpu.monolis_b200_device_clear_matrix(md.p) == 0
    for _ in range(2):
        assert gpu.monolis_b200_device_add_elements_R(md.p, ne, nb, d_elem.data_ptr(), d_val.data_ptr(),
                                                      size if own else 0, d_scale.data_ptr() if scaled else None) == 0
    assert bits_equal(device_values(md, gpu), mh.values())
    # conditions on every fifth node, the first one three times
    nodes = np.array(list(range(0, n, 5)) + [0, 0], dtype=np.int32)
    dofs = (np.arange(len(nodes)) % ndof).astype(np.int32)
    dofs[-2:] = 0
    vals = rng.standard_normal(len(nodes))
    b = rng.standard_normal(n * ndof)
    d_b = torch.from_numpy(b).cuda()
    torch.cuda.synchronize()
    for q in range(len(nodes)):
        mh.set_Dirichlet_bc(b, nodes[q], dofs[q], vals[q])
    assert gpu.monolis_b200_device_set_Dirichlet_bc_R(md.p, d_b.data_ptr(), len(nodes), nodes.ctypes.data_as(api._ip),
                                                      dofs.ctypes.data_as(api._ip), vals.ctypes.data_as(api._dp)) == 0
    assert bits_equal(device_values(md, gpu), mh.values())
    assert bits_equal(d_b.cpu().numpy(), b)
    # the layout the products read has the same values, A^T too (before and
    # after a second assembly on an unchanged pattern)
    x = rng.standard_normal(n * ndof)
    for again in (False, True):
        if again:
            mh.add_elements(elem, nb, val, size if own else 0, scale=scale)
            assert gpu.monolis_b200_device_add_elements_R(md.p, ne, nb, d_elem.data_ptr(), d_val.data_ptr(),
                                                          size if own else 0,
                                                          d_scale.data_ptr() if scaled else None) == 0
        d_x, d_y = torch.from_numpy(x).cuda(), torch.zeros(n * ndof, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        md.device_matvec(d_x.data_ptr(), d_y.data_ptr())
        torch.cuda.synchronize()
        assert bits_equal(d_y.cpu().numpy(), mh.matvec(x))
        assert gpu.monolis_b200_device_matvec_transpose_R(md.p, d_x.data_ptr(), d_y.data_ptr()) == 0
        torch.cuda.synchronize()
        assert bits_equal(d_y.cpu().numpy(), mh.matvec_transpose(x))


def test_column_stored_twice(gpu):
    """A nodal graph that lists the node itself stores its column twice; both
    sides add to the block their binary search finds."""
    import torch
    n = 37
    index = np.arange(0, 3 * n + 1, 3, dtype=np.int32)
    item = np.stack([(np.arange(n) - 1) % n, np.arange(n), (np.arange(n) + 1) % n], axis=1).astype(np.int32).reshape(-1)
    elem = np.stack([np.arange(n), (np.arange(n) + 1) % n], axis=1).astype(np.int32)
    val = np.random.default_rng(5).standard_normal(4)
    ms = []
    for _ in range(2):
        m = api.Monolis(gpu)
        m.get_nonzero_pattern_by_nodal_graph(n, 1, index, item)
        m.quiet()
        ms.append(m)
    ms[0].add_elements(elem, 2, val, 0)
    d_elem, d_val = torch.from_numpy(elem).cuda(), torch.from_numpy(val).cuda()
    torch.cuda.synchronize()
    assert gpu.monolis_b200_device_clear_matrix(ms[1].p) == 0
    assert gpu.monolis_b200_device_add_elements_R(ms[1].p, n, 2, d_elem.data_ptr(), d_val.data_ptr(), 0, None) == 0
    assert bits_equal(device_values(ms[1], gpu), ms[0].values())


def test_bad_elements_leave_the_values(gpu):
    """A node out of range is refused and nothing is added."""
    import torch
    n, elem, (_, m) = setup(gpu, "chain", 1)
    bad = elem.copy()
    bad[17, 1] = n
    d_elem, d_val = torch.from_numpy(bad).cuda(), torch.ones(4, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    assert gpu.monolis_b200_device_clear_matrix(m.p) == 0
    assert gpu.monolis_b200_device_add_elements_R(m.p, len(bad), 2, d_elem.data_ptr(), d_val.data_ptr(), 0, None) == 5
    assert not device_values(m, gpu).any()


@pytest.mark.parametrize("ndof", [1, 3, 6])
def test_refused_calls_change_nothing(gpu, ndof):
    """An element entry outside the pattern (with others inside it) and a
    condition on a row without diagonal block (after a good one): status 5, and
    the values, the right-hand side, the FP64, FP32 and transposed products and
    the DIAG factors stay what they were; the calls that follow work on them."""
    import torch
    n, rng = 75, np.random.default_rng(9)
    cols = [[j for j in (i - 1, i, i + 1) if 0 <= j < n and not i == j == 40] for i in range(n)]
    index = np.concatenate([[0], np.cumsum([len(c) for c in cols])]).astype(np.int32)
    item = np.concatenate(cols).astype(np.int32)
    val = rng.standard_normal(len(item) * ndof * ndof)
    mh, m = api.Monolis(gpu), api.Monolis(gpu)
    for q in (mh, m):
        q.set_matrix_BCSR(n, n, ndof, len(item), val, index, item)
        q.quiet()
    m.set_precision(1)
    m.set_matrix_cache(True)
    m.device_prepare()
    x = torch.from_numpy(rng.standard_normal(n * ndof)).cuda()
    b = rng.standard_normal(n * ndof)
    d_b = torch.from_numpy(b).cuda()

    def state():
        y, yt, y32 = torch.zeros_like(x), torch.zeros_like(x), torch.zeros(n * ndof, dtype=torch.float32, device="cuda")
        x32 = x.float()
        diag = np.empty(n * ndof * ndof)
        torch.cuda.synchronize()
        m.device_matvec(x.data_ptr(), y.data_ptr())
        assert gpu.monolis_b200_device_matvec_R32(m.p, x32.data_ptr(), y32.data_ptr()) == 0
        assert gpu.monolis_b200_device_matvec_transpose_R(m.p, x.data_ptr(), yt.data_ptr()) == 0
        assert gpu.monolis_b200_device_get_diag(m.p, diag.ctypes.data_as(api._dp)) == 0
        torch.cuda.synchronize()
        return [a.cpu().numpy() for a in (y, yt, y32, d_b)] + [diag, device_values(m, gpu)]

    def conditions(nodes, v):
        nodes, dofs, v = np.array(nodes, dtype=np.int32), np.zeros(len(nodes), dtype=np.int32), np.array(v)
        return gpu.monolis_b200_device_set_Dirichlet_bc_R(m.p, d_b.data_ptr(), len(nodes), nodes.ctypes.data_as(api._ip),
                                                          dofs.ctypes.data_as(api._ip), v.ctypes.data_as(api._dp))

    before = state()
    elem = np.array([[3, 4], [20, 22], [60, 61]], dtype=np.int32)
    ke = rng.standard_normal((2 * ndof) ** 2)
    d_elem, d_ke = torch.from_numpy(elem).cuda(), torch.from_numpy(ke).cuda()
    torch.cuda.synchronize()
    assert gpu.monolis_b200_device_add_elements_R(m.p, 3, 2, d_elem.data_ptr(), d_ke.data_ptr(), 0, None) == 5
    assert all(bits_equal(p, q) for p, q in zip(before, state()))
    assert conditions([10, 40], [1.5, 2.5]) == 5
    assert all(bits_equal(p, q) for p, q in zip(before, state()))
    assert conditions([10, 74, 11], [1.5, -2.0, 0.5]) == 0
    for node, v in ((10, 1.5), (74, -2.0), (11, 0.5)):
        mh.set_Dirichlet_bc(b, node, 0, v)
    assert bits_equal(device_values(m, gpu), mh.values()) and bits_equal(d_b.cpu().numpy(), b)


@pytest.mark.parametrize("ndof", [1, 3])
def test_conditions_with_ghost_columns(gpu, ndof):
    """One rank's part of a matrix: columns beyond its rows (ghosts) are never fixed by conditions on its own nodes."""
    import torch
    n, npn, rng = 40, 64, np.random.default_rng(13)
    cols = [sorted({i, max(i - 1, 0), min(i + 1, n - 1), n + (7 * i) % (npn - n), npn - 1}) for i in range(n)]
    index = np.concatenate([[0], np.cumsum([len(c) for c in cols])]).astype(np.int32)
    item = np.concatenate(cols).astype(np.int32)
    rows = np.repeat(np.arange(n), np.diff(index))
    val = rng.standard_normal((len(item), ndof, ndof))
    b = rng.standard_normal(n * ndof)
    m = api.Monolis(gpu)
    m.set_matrix_BCSR(n, npn, ndof, len(item), val.reshape(-1), index, item)
    m.quiet()
    nodes, dofs, vals = np.array([3, 39, 4], dtype=np.int32), np.array([0, ndof - 1, 0], dtype=np.int32), rng.standard_normal(3)
    d_b = torch.from_numpy(b).cuda()
    torch.cuda.synchronize()
    assert gpu.monolis_b200_device_set_Dirichlet_bc_R(m.p, d_b.data_ptr(), 3, nodes.ctypes.data_as(api._ip),
                                                      dofs.ctypes.data_as(api._ip), vals.ctypes.data_as(api._dp)) == 0
    want, wb = val.copy(), b.reshape(n, ndof).copy()
    for node, dof, v in zip(nodes, dofs, vals):  # one after the other, as the host call does
        for k in np.flatnonzero(item == node):
            wb[rows[k]] -= v * want[k, :, dof]
            want[k, :, dof] = 0.0
        want[rows == node, dof, :] = 0.0
        want[(rows == node) & (item == node), dof, dof] = 1.0
        wb[node, dof] = v
    got = np.empty(len(item) * ndof * ndof)
    assert gpu.monolis_b200_device_get_values(m.p, got.ctypes.data_as(api._dp)) == 0
    assert bits_equal(got, want.reshape(-1)) and bits_equal(d_b.cpu().numpy(), wb.reshape(-1))
