"""The calls whose time counts, as a program that uses the library makes them.

Five kinds of pass, each on a seeded structured mesh (jittered interior nodes, one of the
four element types, its Gauss rule, FP32 or FP64):

  assemble  K assembled again on a mesh whose pattern is known: the step that every load
            step, Newton step or design step repeats
  mesh      a mesh taken from host arrays to an assembled K: upload, checks, pattern, values
  spmv      y = K x on device vectors
  analysis  assembly, elimination of the supports, a solve, and the displacements on the host
  learned   one application of the learned preconditioner's network to a residual
"""
from __future__ import annotations

import ctypes as C
import functools
import math

import numpy as np
import torch

from gpufem_b200 import _lib
from gpufem_b200.fem import Context

TYPES = {"q4": _lib.GF_Q4, "q8": _lib.GF_Q8, "brick8": _lib.GF_BRICK8, "brick20": _lib.GF_BRICK20}
DIM = {"q4": 2, "q8": 2, "brick8": 3, "brick20": 3}
NEN = {"q4": 4, "q8": 8, "brick8": 8, "brick20": 20}
WIDTH = {"q4": 18, "q8": 42, "brick8": 81, "brick20": 243}     # entries of the longest row
JITTER = {"q4": 0.2, "q8": 0.15, "brick8": 0.1, "brick20": 0.05}
DTYPES = {"f32": (_lib.GF_F32, torch.float32), "f64": (_lib.GF_F64, torch.float64)}
SOLVERS = {"pcg": _lib.GF_SOLVER_PCG, "twolevel": _lib.GF_SOLVER_TWOLEVEL_PCG}
E0 = 210e3
TOL = 1e-12      # of the analyses: the displacements settle to the matrix's own roundoff

# natural coordinates of the element nodes, in the library's order
NAT = {
    "q4": [(-1, -1), (1, -1), (1, 1), (-1, 1)],
    "q8": [(-1, -1), (0, -1), (1, -1), (1, 0), (1, 1), (0, 1), (-1, 1), (-1, 0)],
    "brick8": [(1, -1, -1), (1, 1, -1), (1, 1, 1), (1, -1, 1),
               (-1, -1, -1), (-1, 1, -1), (-1, 1, 1), (-1, -1, 1)],
    "brick20": [(1, -1, -1), (1, 0, -1), (1, 1, -1), (1, 1, 0), (1, 1, 1), (1, 0, 1),
                (1, -1, 1), (1, -1, 0), (0, -1, -1), (0, 1, -1), (0, 1, 1), (0, -1, 1),
                (-1, -1, -1), (-1, 0, -1), (-1, 1, -1), (-1, 1, 0), (-1, 1, 1), (-1, 0, 1),
                (-1, -1, 1), (-1, -1, 0)],
}


def case(name, kind, elem, nx, ny, nz, dtype, ngauss, field, strain=False, solver=""):
    c = {"kind": kind, "elem": elem, "nx": nx, "ny": ny, "nz": nz, "dtype": dtype,
         "ngauss": ngauss, "field": field, "strain": strain, "solver": solver}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest configured mesh, re-assembled: launches and host work count
        case("assemble_q4_64_f64", "assemble", "q4", 64, 64, 0, "f64", 2, False),
        # the headline workload: every element its own modulus
        case("assemble_q8_512_f32", "assemble", "q8", 512, 512, 0, "f32", 3, True),
        # a ragged plane-strain section in FP64, the type that solves start from
        case("assemble_q8_301x173_f64", "assemble", "q8", 301, 173, 0, "f64", 3, True, strain=True),
        # the largest linear-brick solid
        case("assemble_brick8_128_f32", "assemble", "brick8", 128, 128, 128, "f32", 2, False),
        # a ragged linear-brick solid in FP64
        case("assemble_brick8_57x43x61_f64", "assemble", "brick8", 57, 43, 61, "f64", 2, True),
        # the largest matrix of the configured workloads: quadratic bricks, 3x3x3 Gauss
        case("assemble_brick20_64_f32", "assemble", "brick20", 64, 64, 64, "f32", 3, True),
        # a ragged quadratic-brick part in FP64
        case("assemble_brick20_23x31x19_f64", "assemble", "brick20", 23, 31, 19, "f64", 3, True),
        # a mesh that has just been read or generated (adaptive meshing, a sweep of shapes)
        case("mesh_q8_256_f32", "mesh", "q8", 256, 256, 0, "f32", 3, True),
        # the product that iterative methods outside the library are built on
        case("spmv_q8_512_f32", "spmv", "q8", 512, 512, 0, "f32", 3, True),
        # a small whole analysis with the reference's kind of solver
        case("analysis_q4_64_pcg", "analysis", "q4", 64, 64, 0, "f64", 2, False, solver="pcg"),
        # a whole analysis of a solid part with the two-level solver
        case("analysis_brick20_24_twolevel", "analysis", "brick20", 24, 24, 24, "f64", 3, True,
             solver="twolevel"),
        # one application of the network inside a flexible CG iteration
        case("learned_brick8_32", "learned", "brick8", 32, 32, 32, "f32", 2, True),
    ]


def _sizes(rng, elem, low, high):
    """Elements per direction: the geometric mean spread over the logarithm of
    [low, high], each direction within about a third of it, odd or even as it comes."""
    mean = math.exp(rng.uniform(math.log(low), math.log(high)))
    n = [min(high, max(2, round(mean * math.exp(rng.uniform(-0.3, 0.3))))) for _ in range(DIM[elem])]
    return n + [0] * (3 - len(n))


def draw(rng):
    kind = rng.choice(["assemble"] * 7 + ["mesh", "spmv", "analysis", "analysis", "learned"])
    elem = "brick8" if kind == "learned" else rng.choice(list(TYPES))
    high = {"assemble": {"q4": 512, "q8": 512, "brick8": 112, "brick20": 48},
            "mesh": {"q4": 384, "q8": 256, "brick8": 48, "brick20": 20},
            "spmv": {"q4": 512, "q8": 512, "brick8": 96, "brick20": 40},
            "analysis": {"q4": 96, "q8": 64, "brick8": 28, "brick20": 20},
            "learned": {"brick8": 40}}[kind][elem]
    low = {"q4": 16, "q8": 8, "brick8": 6, "brick20": 4}[elem]
    dtype = "f64" if kind == "analysis" else "f32" if kind == "learned" else rng.choice(["f32", "f64"])
    ngauss = 2 if elem in ("q4", "brick8") else rng.choice([2, 3, 3])
    strain = DIM[elem] == 2 and rng.random() < 0.3
    solver = rng.choice(["pcg", "twolevel"]) if kind == "analysis" else ""
    if kind == "analysis" and elem in ("q8", "brick20"):
        ngauss = 3
    return case("", kind, elem, *_sizes(rng, elem, low, high), dtype, ngauss,
                rng.random() < 0.7, strain, solver)


# ---- meshes ------------------------------------------------------------------------------
@functools.lru_cache(maxsize=2)
def _grid(elem, n):
    """Node positions of the regular mesh, 1-based connectivity, the interior corner nodes
    and the two end corners of every mid-side node."""
    dim, quad = DIM[elem], elem in ("q8", "brick20")
    step = 2 if quad else 1
    fine = [step * v + 1 for v in n]
    idx = np.stack([g.ravel(order="F") for g in np.meshgrid(*[np.arange(m) for m in fine], indexing="ij")], 1)
    keep = (idx % 2).sum(1) <= 1 if quad else np.ones(len(idx), bool)
    number = np.cumsum(keep) - 1
    pts = idx[keep]
    mult = np.cumprod([1] + fine[:-1])
    cell = np.stack([g.ravel(order="F") for g in np.meshgrid(*[np.arange(v) for v in n], indexing="ij")], 1)
    nat = np.array(NAT[elem])
    conn = np.stack([number[((2 * cell + 1 + x if quad else cell + (x + 1) // 2) * mult).sum(1)] for x in nat], 1)
    inner = np.nonzero(np.all(pts % step == 0, 1) & np.all((pts > 0) & (pts < np.array(fine) - 1), 1))[0]
    ends = None
    if quad:
        mid = np.nonzero((pts % 2).sum(1) == 1)[0]
        off = (pts[mid] % 2 * mult).sum(1)
        at = (pts[mid] * mult).sum(1)
        ends = mid, number[at - off], number[at + off]
    return pts / (step * np.array(n, float)), (conn + 1).astype(np.int32), inner, ends


def _mesh(c, seed):
    """Coordinates, connectivity, element moduli (or None) and Poisson's ratio."""
    elem, dim = c["elem"], DIM[c["elem"]]
    n = (c["nx"], c["ny"], c["nz"])[:dim]
    x, conn, inner, ends = _grid(elem, n)
    x = x.copy()
    rng = np.random.default_rng(seed)
    x[inner] += rng.uniform(-JITTER[elem], JITTER[elem], (len(inner), dim)) / np.array(n, float)
    if ends is not None:
        x[ends[0]] = 0.5 * (x[ends[1]] + x[ends[2]])
    E = E0 * np.exp(0.5 * rng.standard_normal(len(conn))) if c["field"] else None
    return x, conn, E, float(rng.uniform(0.25, 0.35))


def _loads(c, x, seed):
    """Supports (one side clamped) and the load on the side across from it."""
    axis = 0 if DIM[c["elem"]] == 2 else 2
    fixed = np.nonzero(x[:, axis] < 1e-12)[0]
    sup = np.ones((len(fixed), x.shape[1] + 1), np.int32)
    sup[:, 0] = fixed + 1
    f = np.zeros_like(x)
    side = np.nonzero(x[:, axis] > 1 - 1e-12)[0]
    f[side] = np.random.default_rng(seed + 1).uniform(0.5, 1.0, (len(side), x.shape[1])) / len(side)
    return sup, fixed, f.ravel()


def _weights(dim, seed):
    """Network weights of a trained network's size, in the library's order."""
    rng = np.random.default_rng(seed + 2)
    part = lambda rows, cols, s: (rng.standard_normal(rows * cols) * s).astype(np.float32)  # noqa: E731
    w = [part(64, 4 * dim, (4 * dim) ** -0.5), part(64, 1, 0.05)]
    for _ in range(3):
        w += [part(64, 64, 0.125), part(64, 64, 0.125), part(64, 1, 0.05)]
    return np.concatenate(w + [part(dim, 64, 0.05), part(dim, 1, 0.05)])


class _Array:
    """Device memory of a context, for torch.as_tensor; the tensor keeps the context open."""

    def __init__(self, ctx, ptr, shape, typestr):
        self.ctx = ctx
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 3}


def _matrix(ctx, dtype):
    """The device arrays of the assembled ELL matrix: row lengths, columns, values."""
    n, w, p = C.c_int32(), C.c_int32(), [C.c_void_p() for _ in range(3)]
    _lib.check(_lib.lib.gf_ell_view(ctx.h, DTYPES[dtype][0], C.byref(n), C.byref(w), *map(C.byref, p)), ctx.h)
    shapes = [((n.value,), "<i4"), ((w.value, n.value), "<i4"),
              ((w.value, n.value), "<f8" if dtype == "f64" else "<f4")]
    return [torch.as_tensor(_Array(ctx, q.value, *s), device="cuda") for q, s in zip(p, shapes)]


def prepare(case, seed):
    c, kind = case, case["kind"]
    x, conn, E, nu = _mesh(c, seed)
    ctx = Context(torch.cuda.current_device())
    args = (TYPES[c["elem"]], x, conn, c["ngauss"], E0, E, nu,
            _lib.GF_PLANE_STRAIN if c["strain"] else _lib.GF_PLANE_STRESS)
    s = {"case": c, "ctx": ctx, "args": args}
    if kind == "mesh":
        return s
    ctx.mesh_create(*args)
    ctx.build_pattern()
    d, dt = DTYPES["f64" if kind == "learned" else c["dtype"]]
    if kind == "analysis":
        sup, _, s["f"] = _loads(c, x, seed)
        ctx.set_supports(sup)
        return s
    ctx.assemble(d, _lib.GF_SCATTER_AUTO)
    if kind == "assemble":
        s["K"] = _matrix(ctx, c["dtype"])[2]
        return s
    gen = torch.Generator("cuda").manual_seed(seed)
    s["x"] = torch.randn(x.size, device="cuda", dtype=DTYPES[c["dtype"]][1], generator=gen)
    s["y"] = torch.empty_like(s["x"])
    if kind == "learned":
        ctx.set_supports(_loads(c, x, seed)[0])
        ctx.apply_constraints(_lib.GF_BC_ELIMINATION)
        ctx.lp_init(DIM[c["elem"]], seed)
        ctx.lp_set_weights(_weights(DIM[c["elem"]], seed))
    return s


def run(state):
    c, ctx = state["case"], state["ctx"]
    kind, dtype = c["kind"], DTYPES[c["dtype"]][0]
    if kind == "assemble":
        ctx.assemble(dtype, _lib.GF_SCATTER_AUTO)
        return {"values": state["K"]}
    if kind == "mesh":
        ctx.mesh_create(*state["args"])
        ctx.build_pattern()
        ctx.assemble(dtype, _lib.GF_SCATTER_AUTO)
        return dict(zip(("rownnz", "colidx", "values"), _matrix(ctx, c["dtype"])))
    if kind == "analysis":
        ctx.set_force(state["f"])
        ctx.assemble(dtype, _lib.GF_SCATTER_AUTO)
        ctx.apply_constraints(_lib.GF_BC_ELIMINATION)
        ctx.solve(SOLVERS[c["solver"]], dtype, tol=TOL, max_iter=100000)
        return {"u": ctx.solution()}
    px, py = C.c_void_p(state["x"].data_ptr()), C.c_void_p(state["y"].data_ptr())
    if kind == "spmv":
        _lib.check(_lib.lib.gf_spmv(ctx.h, dtype, px, py), ctx.h)
    else:
        _lib.check(_lib.lib.gf_lp_apply(ctx.h, px, py), ctx.h)
    return {"y": state["y"]}


# ---- what a pass cannot do without -----------------------------------------------------
def _counts(c):
    """Elements, nodes, node pairs that share an element, Gauss points."""
    elem, dim = c["elem"], DIM[c["elem"]]
    n = [c["nx"], c["ny"], c["nz"]][:dim]
    nelem = math.prod(n)
    # classes of nodes along each axis (0: on a grid plane, 1: between two) and their number
    quad = elem in ("q8", "brick20")
    classes = [(0,) * dim] + ([tuple(int(a == k) for a in range(dim)) for k in range(dim)] if quad else [])
    nodes = sum(math.prod(v if t else v + 1 for v, t in zip(n, k)) for k in classes)
    # ordered pairs of nodes with a common element: along an axis, classes (0, 0) pair over at
    # most one cell, (0, 1) over the two sides of a cell, (1, 1) only within one cell
    one = {(0, 0): lambda v: 3 * v + 1, (0, 1): lambda v: 2 * v, (1, 0): lambda v: 2 * v, (1, 1): lambda v: v}
    pairs = sum(math.prod(one[(a, b)](v) for v, a, b in zip(n, k, m)) for k in classes for m in classes)
    return nelem, nodes, pairs, c["ngauss"] ** dim


def work(case):
    c = case
    elem, dim, nen = c["elem"], DIM[c["elem"]], NEN[c["elem"]]
    nelem, nodes, pairs, ngp = _counts(c)
    size = 8 if c["dtype"] == "f64" else 4
    ndof = nodes * dim
    ell = ndof * min(WIDTH[elem], ndof)
    mesh = nodes * dim * 8 + nelem * (nen * 4 + (8 if c["field"] else 0))
    # symmetric half of the node-pair blocks, dim^2 multiply-adds at each Gauss point
    assembly = nelem * ngp * (nen * (nen + 1) // 2 * dim * dim * 2 + 4 * nen * dim * dim)
    spmv = pairs * (dim * dim * size + 4) + 2 * ndof * size
    if c["kind"] == "assemble":
        return {"bytes": mesh + ell * size, "flops": assembly}
    if c["kind"] == "mesh":
        return {"bytes": mesh + ell * (size + 4) + ndof * 4, "flops": assembly}
    if c["kind"] == "spmv":
        return {"bytes": spmv, "flops": 2 * pairs * dim * dim}
    if c["kind"] == "analysis":
        # iterations to TOL: about ten per element of the longest side with Jacobi, a hundred
        # with the coarse space
        its = 10 * max(c["nx"], c["ny"], c["nz"]) if c["solver"] == "pcg" else 100
        return {"bytes": mesh + 2 * ell * size + its * spmv, "flops": assembly + its * 2 * pairs * dim * dim}
    # learned: two products with K (FP32), three neighbour sums, four dense layers and the input
    layer = nodes * 64 * 4
    return {"bytes": 2 * spmv + 8 * layer, "flops": 4 * pairs * dim * dim + 3 * pairs * 64
            + 2 * nodes * 64 * (4 * dim + 6 * 64 + dim)}


# ---- the same results in 64 bits ---------------------------------------------------------
def _shape(elem, p):
    """Derivatives of the shape functions at a natural point, [dim][nen]."""
    dim, nat = len(p), np.array(NAT[elem], float)
    out = np.zeros((dim, len(nat)))
    for i, t in enumerate(nat):
        fac = np.where(t != 0, 1 + t * p, 1 - p * p)
        dfac = np.where(t != 0, t, -2 * p)
        scale = 0.5 ** np.count_nonzero(t)
        prod = lambda skip: np.prod([fac[b] for b in range(dim) if b != skip])  # noqa: E731
        corner = elem in ("q8", "brick20") and np.all(t != 0)
        extra = t @ p - (dim - 1) if corner else 1.0
        for a in range(dim):
            out[a, i] = scale * (dfac[a] * prod(a) * extra + (np.prod(fac) * t[a] if corner else 0.0))
    return out


def _blocks(c, x, conn, E, nu):
    """Node adjacency (offsets, sorted neighbours) and the dim x dim block of each pair."""
    elem, dim, nen = c["elem"], DIM[c["elem"]], NEN[c["elem"]]
    nodes = len(x)
    x, conn = torch.tensor(x, device="cuda"), torch.tensor(conn, device="cuda").long() - 1
    E = torch.full((len(conn),), E0, device="cuda", dtype=torch.float64) if E is None else torch.tensor(E, device="cuda")
    if dim == 2 and not c["strain"]:
        lam, mu = nu / (1 - nu * nu), 1 / (2 * (1 + nu))
    else:
        lam, mu = nu / ((1 + nu) * (1 - 2 * nu)), 1 / (2 * (1 + nu))
    pts, wts = np.polynomial.legendre.leggauss(c["ngauss"])
    tensor = np.stack(np.meshgrid(*[np.arange(c["ngauss"])] * dim, indexing="ij"), -1).reshape(-1, dim)
    dN = torch.tensor(np.stack([_shape(elem, pts[t]) for t in tensor]), device="cuda")
    w = torch.tensor(np.array([np.prod(wts[t]) for t in tensor]), device="cuda")
    keys = (conn[:, :, None] * nodes + conn[:, None, :]).reshape(-1)
    uniq, inv = torch.unique(keys, return_inverse=True)
    del keys
    off = torch.searchsorted(uniq, torch.arange(nodes + 1, device="cuda") * nodes)
    K = torch.zeros((len(uniq), dim, dim), device="cuda", dtype=torch.float64)
    eye = torch.eye(dim, device="cuda", dtype=torch.float64)
    for e in range(0, len(conn), 1 << 15):
        at = slice(e, min(len(conn), e + (1 << 15)))
        X = x[conn[at]]
        J = torch.einsum("gai,eib->egab", dN, X)
        g = torch.einsum("egba,gai->egib", torch.linalg.inv(J), dN)
        wd = torch.linalg.det(J) * w * E[at, None]
        m = g.shape[0]
        G = g.reshape(m, len(w), nen * dim)
        H = torch.bmm((G * wd[:, :, None]).transpose(1, 2), G).reshape(m, nen, dim, nen, dim).permute(0, 1, 3, 2, 4)
        V = lam * H + mu * H.transpose(3, 4) + mu * eye * H.diagonal(dim1=3, dim2=4).sum(-1)[..., None, None]
        K.index_add_(0, inv[at.start * nen * nen:at.stop * nen * nen], V.reshape(-1, dim, dim))
    return off, uniq % nodes, uniq // nodes, K


def _csr(c, x, fixed, off, col, row, K):
    """CSR matrix with the supported dofs eliminated (unit diagonal), and its diagonal."""
    dim, n = x.shape[1], x.size
    hold = torch.zeros(len(x), dtype=torch.bool, device="cuda")
    hold[torch.tensor(fixed, device="cuda")] = True
    K = K.clone()
    K[hold[row] | hold[col]] = 0
    K[(row == col) & hold[row]] = torch.eye(dim, device="cuda", dtype=torch.float64)
    diag = K[row == col].diagonal(dim1=1, dim2=2).reshape(-1)
    deg = off[1:] - off[:-1]
    crow = torch.zeros(n + 1, dtype=torch.long, device="cuda")
    crow[1:] = (deg * dim).repeat_interleave(dim).cumsum(0)
    k = torch.arange(len(row), device="cuda") - off[row]
    at = (crow[:-1].reshape(-1, dim)[row][:, :, None] + (k * dim)[:, None, None]
          + torch.arange(dim, device="cuda")).reshape(-1)
    ccol = torch.empty(len(at), dtype=torch.long, device="cuda")
    ccol[at] = (col[:, None, None] * dim + torch.arange(dim, device="cuda")).expand(-1, dim, -1).reshape(-1)
    val = torch.empty(len(at), dtype=torch.float64, device="cuda")
    val[at] = K.reshape(-1)
    return torch.sparse_csr_tensor(crow, ccol, val, (n, n)), diag


def _cg(A, diag, b):
    """Jacobi-preconditioned CG to a recursive residual of 1e-15, then once more on what is left."""
    u = torch.zeros_like(b)
    for _ in range(3):
        r = b - A @ u
        stop = 1e-13 * float(r.norm())
        d, z = torch.zeros_like(b), r / diag
        p, rz = z.clone(), r @ z
        for k in range(20000):
            q = A @ p
            a = rz / (p @ q)
            d += a * p
            r -= a * q
            if k % 16 == 0 and float(r.norm()) <= stop:
                break
            z = r / diag
            new = r @ z
            p = z + (new / rz) * p
            rz = new
        u = u + d
    return u


def exact(case, seed):
    c = case
    dim = DIM[c["elem"]]
    x, conn, E, nu = _mesh(c, seed)
    if c["kind"] == "analysis" and x.size > 300_000:
        return None
    off, col, row, K = _blocks(c, x, conn, E, nu)
    if c["kind"] in ("assemble", "mesh"):
        k = torch.arange(len(row), device="cuda") - off[row]
        n, w = x.size, int((off[1:] - off[:-1]).max()) * dim
        out = torch.zeros((w // dim, dim, len(x), dim), device="cuda", dtype=torch.float64)
        for b in range(dim):     # block column b: slot k * dim + b, the rows of the node
            out[k, b, row] = K[:, :, b]
        out = out.reshape(w, n)
        return {"values": out} if c["kind"] == "assemble" else {"rownnz": None, "colidx": None, "values": out}
    _, fixed, f = _loads(c, x, seed)
    if c["kind"] == "analysis":
        A, diag = _csr(c, x, fixed, off, col, row, K)
        b = torch.tensor(f, device="cuda")
        b.view(-1, dim)[torch.tensor(fixed, device="cuda")] = 0
        return {"u": _cg(A, diag, b).cpu().numpy()}
    dt = DTYPES[c["dtype"]][1]
    v = torch.randn(x.size, device="cuda", dtype=dt, generator=torch.Generator("cuda").manual_seed(seed)).double()
    none = np.zeros(0, np.int64)
    if c["kind"] == "spmv":
        return {"y": _csr(c, x, none, off, col, row, K)[0] @ v}
    A, d = _csr(c, x, fixed, off, col, row, K)
    W = torch.tensor(_weights(dim, seed), device="cuda").bfloat16().double()
    size = [64 * 4 * dim, 64] + [64 * 64, 64 * 64, 64] * 3 + [dim * 64, dim]
    P = [t.reshape(-1, 64) if len(t) == 64 * 64 or len(t) == dim * 64 else t for t in torch.split(W, size)]
    mean = torch.sparse_csr_tensor(off, col, (1.0 / (off[1:] - off[:-1]).double())[row], (len(x), len(x)))
    rho = v / d
    v1 = (A @ rho) / d
    v2 = (A @ v1) / d
    rms = rho.square().mean().sqrt()
    logd = d.log() - d.log().mean()
    h = torch.cat([t.reshape(-1, dim) for t in (rho / rms, v1 / rms, v2 / rms, logd)], 1)
    h = torch.relu(h @ P[0].reshape(64, 4 * dim).T + P[1].reshape(-1))
    for k in range(3):
        Ws, Wn, bias = P[2 + 3 * k:5 + 3 * k]
        h = torch.relu(h @ Ws.T + (mean @ h) @ Wn.T + bias.reshape(-1))
    return {"y": rho + rms * (h @ P[11].T + P[12].reshape(-1)).reshape(-1)}
