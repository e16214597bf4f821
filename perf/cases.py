"""The work that programs have this library do, as measurable cases.

A case is a dict of plain values; `listed()` names the standing ones and
`draw(rng)` makes one more of the same ranges. `prepare` builds what a program
holds before the call (matrix, right-hand side, output buffers), `run` is one
pass through the library's public entry points, `work` the bytes and operations
the path cannot do without, `exact` the same outputs from plain 64-bit torch
(matrix-free operators and a tight Krylov solve), `tolerance` the difference
between two correct implementations.

Grids have nx x ny x nz points, id = ix + nx (iy + ny iz), cubic cells.
Problems:
  laplacian   7-point Laplacian, diagonal 6, ndof 1 (symmetric)
  fv          cell-centred diffusion, log-normal conductivity, ndof 1
  convection  7-point upwind convection-diffusion, ndof 1 (nonsymmetric)
  diffusion   Q1 hexahedra, log-normal coefficient per element, ndof 1
  elasticity  Q1 hexahedra, a modulus per element, ndof 3, face x = 0 clamped
"""
import ctypes
import math

import numpy as np
import torch

from monolis_b200 import api

_LIB = None
METHODS = {"cg": api.ITER_CG, "bicgstab": api.ITER_BICGSTAB, "pipecg": api.ITER_PIPECG}


def library():
    global _LIB
    if _LIB is None:
        _LIB = api.load_product()
    return _LIB


def _solve(name, problem, n, method="cg", precision=0, host=False, **kw):
    nx, ny, nz = n if isinstance(n, tuple) else (n, n, n)
    c = {"kind": "solve", "problem": problem, "nx": nx, "ny": ny, "nz": nz, "method": method,
         "precision": precision, "host": host, "tol": 1e-8}
    c.update(kw)
    return dict(c, name=name) if name else c


def listed():
    return [
        # a coupled or time-stepping code's smallest solve, matrix resident: latency and launches
        _solve("cg_elasticity_8", "elasticity", 8),
        # monolis_solve_R as it is called from a program: host arrays, matrix uploaded on every call
        _solve("host_laplacian_32", "laplacian", 32, host=True),
        _solve("host_elasticity_41_mixed", "elasticity", (41, 37, 33), precision=1, host=True),
        # resident solves of ordinary size: one part of a mesh
        _solve("cg_elasticity_33", "elasticity", 33),
        _solve("bicgstab_convection_101", "convection", (101, 67, 53), method="bicgstab", peclet=5.0),
        _solve("cg_elasticity_57_mixed", "elasticity", (57, 49, 61), precision=1),
        # the largest: memory-bound Krylov loops
        _solve("cg_elasticity_80", "elasticity", 80),
        _solve("bicgstab_convection_176_mixed", "convection", 176, method="bicgstab", precision=1, peclet=0.5),
        # many systems of uneven size in one call; many right-hand sides on one matrix
        {"name": "batch_64", "kind": "batch", "systems": 64, "lo": 10, "hi": 44, "tol": 1e-8},
        {"name": "multi_rhs_50x32_mixed", "kind": "multi", "nx": 50, "ny": 50, "nz": 50, "rhs": 32, "precision": 1,
         "tol": 1e-8},
        # Newton step: element matrices of the current state assembled on the device, then a product
        {"name": "assemble_elasticity_45", "kind": "assemble", "nx": 45, "ny": 41, "nz": 38},
        # one step of a coefficient inversion: assemble, solve, solve the transpose, gradient
        {"name": "adjoint_diffusion_56", "kind": "adjoint", "nx": 56, "ny": 56, "nz": 56, "precision": 0, "tol": 1e-10},
    ]


def draw(rng):
    def log_size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def box(lo, hi):
        n = log_size(lo, hi)
        return tuple(max(lo, min(hi, n + rng.randint(-n // 6, n // 6))) for _ in range(3))

    kind = rng.choice(["solve", "solve", "solve", "host", "batch", "multi", "assemble", "adjoint"])
    if kind == "solve":
        problem = rng.choice(["elasticity", "elasticity", "convection", "fv"])
        precision = rng.choice([0, 1])
        if problem == "elasticity":
            return _solve(None, problem, box(6, 60), precision=precision)
        if problem == "fv":
            method = rng.choice(["cg", "pipecg"]) if precision == 0 else "cg"
            return _solve(None, problem, box(12, 120), method=method, precision=precision)
        return _solve(None, problem, box(14, 140), method="bicgstab", precision=precision,
                      peclet=rng.choice([0.5, 5.0, 50.0]))
    if kind == "host":
        problem = rng.choice(["laplacian", "elasticity"])
        return _solve(None, problem, box(8, 60) if problem == "laplacian" else box(6, 40),
                      precision=rng.choice([0, 1]), host=True)
    if kind == "batch":
        lo = rng.randint(6, 14)
        return {"kind": "batch", "systems": log_size(4, 96), "lo": lo, "hi": rng.randint(lo + 4, 40), "tol": 1e-8}
    nx, ny, nz = box(8, 44)
    if kind == "multi":
        return {"kind": "multi", "nx": nx, "ny": ny, "nz": nz, "rhs": rng.randint(2, 40),
                "precision": rng.choice([0, 1]), "tol": 1e-8}
    if kind == "assemble":
        return {"kind": "assemble", "nx": nx, "ny": ny, "nz": nz}
    return {"kind": "adjoint", "nx": nx, "ny": ny, "nz": nz, "precision": rng.choice([0, 1]), "tol": 1e-10}


# ---------------------------------------------------------------------------
# Problems (numpy)
# ---------------------------------------------------------------------------
def hexahedra(nx, ny, nz):
    ex, ey, ez = np.meshgrid(np.arange(nx - 1), np.arange(ny - 1), np.arange(nz - 1), indexing="ij")
    base = (ex + nx * (ey + ny * ez)).transpose(2, 1, 0).reshape(-1, 1)
    s = nx * ny
    return (base + np.array([0, 1, 1 + nx, nx, s, s + 1, s + 1 + nx, s + nx])).astype(np.int32)


def gauss_gradients(h):
    nat = np.array([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1],
                    [-1, -1, 1], [1, -1, 1], [1, 1, 1], [-1, 1, 1]], dtype=float)
    out = []
    for q in nat / math.sqrt(3.0):
        f = 1.0 + nat * q
        g = np.stack([nat[:, d] * f[:, (d + 1) % 3] * f[:, (d + 2) % 3] for d in range(3)], axis=1)
        out.append(g / (4.0 * h))
    return out, (h / 2.0) ** 3


def element_matrix(problem, h):
    grads, weight = gauss_gradients(h)
    if problem == "diffusion":
        return sum(g @ g.T for g in grads) * weight
    lam, mu = 0.3 / (1.3 * 0.4), 1.0 / 2.6
    K = np.zeros((8, 3, 8, 3))
    for g in grads:
        K += lam * np.einsum("ai,bj->aibj", g, g) + mu * np.einsum("aj,bi->aibj", g, g)
        K += mu * np.einsum("ab,ij->aibj", g @ g.T, np.eye(3))
    return np.ascontiguousarray(K.reshape(24, 24) * weight)


def stencil(case, rng):
    """Diagonal and the six neighbour coefficients of a 7-point problem as
    (nz, ny, nx) arrays or numbers, in the order -z -y -x +x +y +z."""
    shape = (case["nz"], case["ny"], case["nx"])
    if case.get("problem") == "laplacian":
        return 6.0, [-1.0] * 6
    if case.get("problem") == "convection":
        v = 2.0 * case["peclet"] * np.array([1.0, 0.5, 0.25]) * rng.uniform(0.9, 1.1, 3)
        return 6.0 + v.sum(), [-1.0 - v[2], -1.0 - v[1], -1.0 - v[0], -1.0, -1.0, -1.0]
    kappa = np.exp(rng.standard_normal(shape))
    diag, off = np.zeros(shape), []
    for axis, side in ((0, 0), (1, 0), (2, 0), (2, 1), (1, 1), (0, 1)):
        other = np.roll(kappa, 1 if side == 0 else -1, axis)
        t = 2.0 * kappa * other / (kappa + other)
        edge = [slice(None)] * 3
        edge[axis] = 0 if side == 0 else -1
        t[tuple(edge)] = 2.0 * kappa[tuple(edge)]
        diag += t
        off.append(-t)
    return diag, off


def stencil_csr(case, rng):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n = nx * ny * nz
    diag, off = stencil(case, rng)
    ids = np.arange(n, dtype=np.int32).reshape(nz, ny, nx)
    cols = np.full((nz, ny, nx, 7), -1, dtype=np.int32)
    vals = np.empty((nz, ny, nx, 7))
    a, b, every = slice(1, None), slice(None, -1), slice(None)
    to = [(a, every, every), (every, a, every), (every, every, a), (every, every, b), (every, b, every), (b, every, every)]
    frm = [to[5], to[4], to[3], to[2], to[1], to[0]]
    for k in range(6):
        q = k if k < 3 else k + 1
        cols[to[k] + (q,)] = ids[frm[k]]
        vals[..., q] = off[k]
    cols[..., 3], vals[..., 3] = ids, diag
    keep = cols.reshape(-1) >= 0
    index = np.zeros(n + 1, dtype=np.int32)
    index[1:] = np.cumsum(keep.reshape(-1, 7).sum(1))
    return index, cols.reshape(-1)[keep], vals.reshape(-1)[keep]


def batch_sides(case):
    u = (np.arange(case["systems"]) + 0.5) / case["systems"]
    return np.rint(case["lo"] * (case["hi"] / case["lo"]) ** u).astype(int)


def ndof_of(case):
    return 3 if case.get("problem", case["kind"]) in ("elasticity", "assemble") else 1


def is_mesh(case):
    return case["kind"] in ("assemble", "adjoint") or case.get("problem") in ("elasticity", "diffusion")


def inputs(case, seed):
    """Everything that depends on the seed, as numpy arrays."""
    rng = np.random.default_rng(seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    nn, nd = nx * ny * nz, ndof_of(case)
    if not is_mesh(case):
        csr = stencil_csr(case, rng)
        rows = case.get("rhs", 1)
        return {"csr": csr, "b": rng.uniform(0.0, 1.0, (rows, nn) if rows > 1 else nn)}
    elem = hexahedra(nx, ny, nz)
    h = 1.0 / (max(nx, ny, nz) - 1)
    d = {"elem": elem, "nodes": np.arange(0, nn, nx, dtype=np.int32)}
    if nd == 3:
        d["ke"] = element_matrix("elasticity", h)
        d["scale"] = np.exp(0.3 * rng.standard_normal(len(elem)))
        f = rng.normal(0.0, 0.01, (nn, 3))
        f[:, 2] -= 1.0
    else:
        d["ke"] = element_matrix("diffusion", h)
        d["scale"] = np.exp(rng.standard_normal(len(elem)))
        f = np.ones((nn, 1))
    d["b"] = (f * (np.bincount(elem.reshape(-1), minlength=nn) * h ** 3 / 8.0)[:, None]).reshape(-1)
    if case["kind"] == "assemble":
        d["x"] = rng.standard_normal(nn * nd)
        d["bc"] = rng.normal(0.0, 1e-3, len(d["nodes"]) * nd)
    if case["kind"] == "adjoint":
        d["target"] = rng.standard_normal(nn) * 1e-2 + 0.05
    return d


def bc_list(d, nd):
    nodes = np.repeat(d["nodes"], nd)
    dofs = np.tile(np.arange(nd, dtype=np.int32), len(d["nodes"]))
    return np.ascontiguousarray(nodes), dofs, np.ascontiguousarray(d.get("bc", np.zeros(len(nodes))))


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------
def _gpu(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _ok(rc):
    if rc:
        raise RuntimeError("status %d" % rc)


def _int_p(a):
    return a.ctypes.data_as(ctypes.POINTER(ctypes.c_int))


def _dbl_p(a):
    return a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))


def _matrix(case):
    m = api.Monolis(library())
    m.quiet()
    m.set_error_abort(False)
    m.set_method(METHODS[case.get("method", "cg")])
    m.set_precond(api.PREC_DIAG)
    m.set_tolerance(case.get("tol", 1e-8))
    m.set_maxiter(20000)
    m.set_precision(case.get("precision", 0))
    return m


def _device_assemble(s):
    """Element matrices and conditions into the device matrix; b is rewritten."""
    m, lib = s["m"], s["m"].lib
    _ok(lib.monolis_b200_device_clear_matrix(m.p))
    _ok(lib.monolis_b200_device_add_elements_R(m.p, s["n_elem"], 8, s["elem"].data_ptr(), s["ke"].data_ptr(),
                                               s["ke_stride"], s["scale"].data_ptr() if s["scale"] is not None else None))
    nodes, dofs, vals = s["bc"]
    _ok(lib.monolis_b200_device_set_Dirichlet_bc_R(m.p, s["b"].data_ptr(), len(nodes), _int_p(nodes), _int_p(dofs),
                                                   _dbl_p(vals)))


def prepare(case, seed):
    if case["kind"] == "batch":
        return _prepare_batch(case, seed)
    d = inputs(case, seed)
    nd, nn = ndof_of(case), case["nx"] * case["ny"] * case["nz"]
    m = _matrix(case)
    s = {"kind": case["kind"], "host": case.get("host", False), "m": m}
    if not is_mesh(case):
        index, item, val = d["csr"]
        m.set_matrix_BCSR(nn, nn, 1, len(item), val, index, item)
    else:
        m.get_nonzero_pattern_flat(nn, 8, nd, d["elem"])
    if s["host"]:
        s["b"], s["x"] = d["b"].copy(), np.zeros(nn * nd)
        if is_mesh(case):
            m.add_elements(d["elem"], 8, d["ke"].reshape(-1), 0, scale=d["scale"])
            for node in d["nodes"]:
                for k in range(nd):
                    m.set_Dirichlet_bc(s["b"], node, k, 0.0)
        return s
    s["b"] = _gpu(d["b"])
    if is_mesh(case):
        s["n_elem"], s["elem"], s["bc"] = len(d["elem"]), _gpu(d["elem"]), bc_list(d, nd)
        s["ke"], s["ke_stride"], s["scale"] = _gpu(d["ke"]), 0, _gpu(d["scale"])
    if case["kind"] == "assemble":  # a matrix of its own for each element, as a nonlinear material has
        s["ke"] = (s["scale"][:, None] * s["ke"].reshape(1, -1)).contiguous()
        s["ke_stride"], s["scale"] = 576, None
        s["b0"], s["x"], s["y"] = s["b"].clone(), _gpu(d["x"]), torch.empty(nn * nd, dtype=torch.float64, device="cuda")
        s["r"] = torch.empty_like(s["y"])
    elif case["kind"] == "adjoint":
        fixed = np.zeros(nn, dtype=np.int32)
        fixed[d["nodes"]] = 1
        s.update(fixed=_gpu(fixed), target=_gpu(d["target"]), b0=s["b"].clone(),
                 stream=torch.cuda.ExternalStream(api.stream_handle(m.lib)))
        s["x"], s["lam"] = torch.zeros_like(s["b"]), torch.zeros_like(s["b"])
        s["grad"] = torch.zeros(s["n_elem"], dtype=torch.float64, device="cuda")
    elif case["kind"] == "multi":
        s["rhs"], s["x"] = case["rhs"], torch.zeros_like(s["b"])
        s["iter"], s["status"] = np.zeros(case["rhs"], np.int32), np.zeros(case["rhs"], np.int32)
        s["resid"] = np.zeros(case["rhs"])
        m.set_matrix_cache(True)
    else:
        s["x"] = torch.zeros_like(s["b"])
    torch.cuda.synchronize()
    if is_mesh(case):
        _device_assemble(s)
    m.device_prepare()
    torch.cuda.synchronize()
    return s


def _prepare_batch(case, seed):
    batch = api.Batch(library())
    sides = batch_sides(case)
    rhs = []
    for k, side in enumerate(sides):
        n = int(side)
        d = inputs({"kind": "multi", "nx": n, "ny": n, "nz": n}, seed * 1000 + k)
        index, item, val = d["csr"]
        batch.add_csr(n ** 3, 1, index, item, val)
        rhs.append(d["b"])
    batch.prepare(precond=api.PREC_DIAG, autotune=False)
    batch.set_config(4, 512, 8192)  # fixed, so that two runs time the same work
    offsets = batch.offsets()
    d_b, d_x = batch.device_vectors()
    size = int(offsets[-1]) + (len(rhs[-1]) + 63) // 64 * 64
    b = np.zeros(size)
    for o, r in zip(offsets, rhs):
        b[o:o + len(r)] = r

    class View:  # the batch's own device vectors, as tensors
        def __init__(self, ptr):
            self.__cuda_array_interface__ = {"shape": (size,), "typestr": "<f8", "data": (ptr, False), "version": 2}

    view = torch.as_tensor(View(d_x), device="cuda")
    torch.as_tensor(View(d_b), device="cuda").copy_(torch.from_numpy(b))
    torch.cuda.synchronize()
    return {"kind": "batch", "batch": batch, "tol": case["tol"], "view": view, "x": torch.zeros_like(view)}


def run(s):
    if s["kind"] == "batch":
        _, _, status = s["batch"].device_solve(tol=s["tol"], max_iter=10000, refine=True)
        if status.any():
            raise RuntimeError("batch status")
        s["x"].copy_(s["view"])  # the solutions out of the batch, whose memory ends with it
        return s["x"]
    m = s["m"]
    if s["kind"] == "solve":
        if s["host"]:
            m.solve(s["b"], s["x"])
            _ok(m.get_error_tag())
        else:
            _ok(m.device_solve(s["b"].data_ptr(), s["x"].data_ptr()))
        return s["x"]
    if s["kind"] == "multi":
        _ok(m.lib.monolis_b200_device_solve_multi_R(m.p, s["rhs"], s["b"].data_ptr(), s["x"].data_ptr(),
                                                    _int_p(s["iter"]), _dbl_p(s["resid"]), _int_p(s["status"])))
        return s["x"]
    if s["kind"] == "assemble":
        s["b"].copy_(s["b0"])
        torch.cuda.current_stream().synchronize()
        _device_assemble(s)
        m.device_matvec(s["x"].data_ptr(), s["y"].data_ptr())
        return {"y": s["y"], "b": s["b"]}
    with torch.cuda.stream(s["stream"]):
        s["b"].copy_(s["b0"])
        _device_assemble(s)
        m.device_prepare()
        _ok(m.device_solve(s["b"].data_ptr(), s["x"].data_ptr()))
        rhs = s["x"] - s["target"]
        rhs *= (1 - s["fixed"])
        _ok(m.lib.monolis_b200_device_solve_transpose_R(m.p, rhs.data_ptr(), s["lam"].data_ptr()))
        _ok(m.lib.monolis_b200_device_element_gradient_R(m.p, s["n_elem"], 8, s["elem"].data_ptr(), s["ke"].data_ptr(), 0,
                                                         s["lam"].data_ptr(), s["x"].data_ptr(), s["fixed"].data_ptr(),
                                                         -1.0, s["grad"].data_ptr()))
    return {"x": s["x"], "lambda": s["lam"], "grad": s["grad"]}


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
# Iterations per grid point of the longest side, as these problems need at
# their tolerances (they set the bytes; a solve is judged by its time).
ITERATIONS = {"laplacian": 3.8, "fv": 4.4, "convection": 1.8, "elasticity": 12.2, "adjoint": 6.0, "batch": 4.4, "multi": 4.4}


def solve_work(blocks, rows, nd, iterations, precision, products=1, vectors=12):
    """A Krylov solve: per iteration the matrix values once per product, the
    block-diagonal factors once per product and the recurrence's vectors."""
    v = 4 if precision else 8
    per = products * (blocks + rows) * nd * nd * v + vectors * rows * nd * v
    return iterations * per, iterations * (2.0 * products * blocks * nd * nd + 2.0 * vectors * rows * nd)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        b = f = 0.0
        for n in batch_sides(case):
            one = solve_work(7 * n ** 3 - 6 * n * n, n ** 3, 1, ITERATIONS["batch"] * n, 1)
            b, f = b + one[0], f + one[1]
        return {"bytes": float(b), "flops": float(f)}
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    rows, nd, longest = nx * ny * nz, ndof_of(case), max(nx, ny, nz)
    if is_mesh(case):
        blocks = (3 * nx - 2) * (3 * ny - 2) * (3 * nz - 2)
    else:
        blocks = 7 * rows - 2 * (nx * ny + ny * nz + nx * nz)
    if kind == "solve":
        bi = case["method"] == "bicgstab"
        b, f = solve_work(blocks, rows, nd, ITERATIONS[case["problem"]] * longest, case["precision"], 2 if bi else 1,
                          20 if bi else 12)
        if case["host"]:
            b += blocks * (8.0 * nd * nd + 4) + rows * (16.0 * nd + 4)
        return {"bytes": float(b), "flops": float(f)}
    if kind == "multi":
        its, v = ITERATIONS["multi"] * longest, 4 if case["precision"] else 8
        return {"bytes": its * v * (blocks + rows + 12.0 * rows * case["rhs"]),
                "flops": its * (2.0 * blocks + 24.0 * rows) * case["rhs"]}
    elements = (nx - 1) * (ny - 1) * (nz - 1)
    if kind == "assemble":  # element matrices and connectivity in, matrix out and in again for the product
        return {"bytes": float(elements * (576 * 8 + 32) + blocks * (2 * 72 + 4) + rows * 3 * 8 * 4),
                "flops": float(elements * 576 + 18 * blocks)}
    b, f = solve_work(blocks, rows, 1, ITERATIONS["adjoint"] * longest, case["precision"])
    return {"bytes": float(2 * b + elements * (32 + 8 + 8 + 32) + 2 * 8 * blocks), "flops": float(2 * f + 300.0 * elements)}


# ---------------------------------------------------------------------------
# exact
# ---------------------------------------------------------------------------
def _krylov(apply, diag, b, symmetric):
    """A x = b in 64 bits: Jacobi CG or BiCGSTAB restarted on the true
    residual until it no longer falls (about 1e-15 of b)."""
    x, best, best_x = torch.zeros_like(b), math.inf, None
    target = float(b.norm()) * 1e-15
    for _ in range(6):
        r = b - apply(x)
        if float(r.norm()) < best:
            best, best_x = float(r.norm()), x.clone()
        if best <= target or (_ and float(r.norm()) > 0.5 * last):
            break
        last = float(r.norm())
        goal = max(target, last * 1e-11)
        if symmetric:
            z = r / diag
            p, rho = z.clone(), r.dot(z)
            for it in range(6000):
                q = apply(p)
                alpha = rho / p.dot(q)
                x += alpha * p
                r -= alpha * q
                if it % 20 == 19 and float(r.norm()) < goal:
                    break
                z = r / diag
                new = r.dot(z)
                p = z + (new / rho) * p
                rho = new
        else:
            shadow, p, v = r.clone(), torch.zeros_like(r), torch.zeros_like(r)
            rho = alpha = omega = torch.ones((), dtype=r.dtype, device=r.device)
            for it in range(3000):
                new = shadow.dot(r)
                p = r + (new / rho) * (alpha / omega) * (p - omega * v)
                rho = new
                ph = p / diag
                v = apply(ph)
                alpha = rho / shadow.dot(v)
                q = r - alpha * v
                qh = q / diag
                t = apply(qh)
                omega = t.dot(q) / t.dot(t)
                x += alpha * ph + omega * qh
                r = q - omega * t
                if it % 10 == 9 and float(r.norm()) < goal:
                    break
    return best_x


def _stencil_operator(case, rng):
    diag, off = stencil(case, rng)
    shape = (case["nz"], case["ny"], case["nx"])
    diag, *off = [torch.as_tensor(np.broadcast_to(c, shape).copy()).cuda() for c in (diag, *off)]

    def apply(x):
        x = x.view(shape)
        y = diag * x
        y[1:] += off[0][1:] * x[:-1]
        y[:, 1:] += off[1][:, 1:] * x[:, :-1]
        y[:, :, 1:] += off[2][:, :, 1:] * x[:, :, :-1]
        y[:, :, :-1] += off[3][:, :, :-1] * x[:, :, 1:]
        y[:, :-1] += off[4][:, :-1] * x[:, 1:]
        y[:-1] += off[5][:-1] * x[1:]
        return y.reshape(-1)

    return apply, diag.reshape(-1)


def _mesh_operator(d, nd, nn):
    """Matrix-free Q1 operator without conditions, its diagonal, and the mask of fixed dofs."""
    elem = _gpu(d["elem"].astype(np.int64))
    dofs = (elem[:, :, None] * nd + torch.arange(nd, device="cuda")).reshape(len(elem), -1)
    ke, scale = _gpu(d["ke"]), _gpu(d["scale"])[:, None]
    fixed = torch.zeros(nn * nd, dtype=torch.bool, device="cuda")
    fixed.view(nn, nd)[_gpu(d["nodes"].astype(np.int64))] = True

    def apply(x):
        return torch.zeros_like(x).index_add_(0, dofs.reshape(-1), (scale * (x[dofs] @ ke.T)).reshape(-1))

    diag = torch.zeros(nn * nd, dtype=torch.float64, device="cuda")
    diag.index_add_(0, dofs.reshape(-1), (scale * ke.diagonal()).reshape(-1))
    diag[fixed] = 1.0

    def constrained(x):
        y = apply(x.masked_fill(fixed, 0.0))
        y[fixed] = x[fixed]
        return y

    return apply, constrained, diag, fixed, dofs, ke, scale


def exact(case, seed):
    if case["kind"] == "batch":
        outs = []
        for k, side in enumerate(batch_sides(case)):
            n = int(side)
            one = {"kind": "multi", "nx": n, "ny": n, "nz": n}
            d = inputs(one, seed * 1000 + k)
            apply, diag = _stencil_operator(one, np.random.default_rng(seed * 1000 + k))
            x = _krylov(apply, diag, _gpu(d["b"]), True)
            outs.append(torch.cat([x, x.new_zeros((64 - n ** 3 % 64) % 64)]))
        return torch.cat(outs)
    d = inputs(case, seed)
    nd, nn = ndof_of(case), case["nx"] * case["ny"] * case["nz"]
    if not is_mesh(case):
        apply, diag = _stencil_operator(case, np.random.default_rng(seed))
        b = _gpu(d["b"])
        if case["kind"] == "multi":
            return torch.stack([_krylov(apply, diag, r, True) for r in b.view(case["rhs"], -1)]).view_as(b)
        return _krylov(apply, diag, b, case["problem"] != "convection")
    apply, constrained, diag, fixed, dofs, ke, scale = _mesh_operator(d, nd, nn)
    b = _gpu(d["b"])
    if case["kind"] == "assemble":
        g = torch.zeros_like(b)
        g[fixed] = _gpu(d["bc"])
        b = b - apply(g)
        b[fixed] = g[fixed]
        return {"y": constrained(_gpu(d["x"])), "b": b}
    b[fixed] = 0.0
    x = _krylov(constrained, diag, b, True)
    if case["kind"] == "solve":
        return x
    lam = _krylov(constrained, diag, (x - _gpu(d["target"])).masked_fill(fixed, 0.0), True)
    grad = -(lam.masked_fill(fixed, 0.0)[dofs] * (x[dofs] @ ke.T)).sum(1)
    return {"x": x, "lambda": lam, "grad": grad}


def tolerance(case):
    """About four times the largest error against `exact` over the ranges: a
    solve stops at its residual, so its error is set by `tol` (measured up to
    1.7e-9 at 1e-8 and 7e-12 at 1e-10, either precision); the assembled
    product by the rounding of 64-bit sums (1.6e-16)."""
    if case["kind"] == "assemble":
        return {"rel": 1e-15}
    return {"rel": 5e-11 if case["tol"] < 1e-9 else 8e-9}
