"""The one-kernel (P)CG of small systems, at the sizes where its slices, warps and CTAs end, and
one size past what it takes: iterates against a numpy restatement of the same recurrences."""
import numpy as np
import pytest
import scipy.sparse as sp

from gpufem_b200 import _lib
from gpufem_b200 import meshgen as mg

pytestmark = pytest.mark.gpu


def problem(et, n):
    from gpufem_b200.fem import Context
    m = mg.clamp_and_load(mg.structured(et, n, jitter=0.05, seed=2, ngauss=2 if et in (mg.Q4, mg.BRICK8) else 3))
    m.E = mg.lognormal_iid(m, 0.5, seed=3)
    ctx = Context(0)
    ctx.mesh_create(m.elem_type, m.coords, m.conn, m.ngauss, m.E0, m.E, m.nu)
    ctx.set_supports(m.supports)
    ctx.set_force(m.f)
    ctx.assemble(_lib.GF_F64, _lib.GF_SCATTER_AUTO)
    ctx.apply_constraints(_lib.GF_BC_ELIMINATION)
    ctx.convert_f64_to_f32()
    rn, ci, v = ctx.ell_download(_lib.GF_F64)
    mask = np.arange(ci.shape[0])[:, None] < rn[None, :]
    rows = np.broadcast_to(np.arange(rn.size)[None, :], ci.shape)
    K = sp.csr_matrix((v[mask], (rows[mask], ci[mask])), shape=(rn.size, rn.size))
    return ctx, K, ctx.get_force()


def pcg(K, b, dinv, its):
    x, r = np.zeros_like(b), b.copy()
    z = dinv * r
    p, rz = z.copy(), r @ z
    for _ in range(its):
        q = K @ p
        a = rz / (p @ q)
        x += a * p
        r -= a * q
        z = dinv * r
        rz, old = r @ z, rz
        p = z + rz / old * p
    return x


# 4, 32 and 33 nodes (one slice, full and one over); 3-D rows; several warps per slice and one;
# 8,281 nodes fill the cluster's shared memory, 10,201 do not fit
SIZES = [(mg.Q4, (1, 1)), (mg.Q4, (7, 3)), (mg.Q4, (10, 2)), (mg.Q8, (9, 7)), (mg.BRICK8, (5, 4, 3)),
         (mg.BRICK20, (3, 2, 2)), (mg.Q4, (90, 90)), (mg.Q4, (100, 100))]


@pytest.mark.parametrize("et,n", SIZES)
@pytest.mark.parametrize("solver", [_lib.GF_SOLVER_PCG, _lib.GF_SOLVER_CG])
def test_iterates_match_numpy(et, n, solver):
    """After a few iterations the rounding of two orders of summation has not grown: 1e-10."""
    ctx, K, b = problem(et, n)
    with ctx:
        d = 1.0 / K.diagonal() if solver == _lib.GF_SOLVER_PCG else np.ones_like(b)
        for its in (1, 4):
            info = ctx.solve(solver, _lib.GF_F64, tol=1e-30, max_iter=its, raise_on_error=False)
            assert info.iterations == its and info.status == _lib.GF_ERR_NOT_CONVERGED
            x = pcg(K, b, d, its)
            assert np.linalg.norm(ctx.solution() - x) <= 1e-10 * np.linalg.norm(x)


@pytest.mark.parametrize("et,n", SIZES)
def test_converged_solution(et, n):
    ctx, K, b = problem(et, n)
    with ctx:
        x = sp.linalg.spsolve(K.tocsc(), b)
        for kw in ({}, {"max_seconds": 100.0, "check_every": 7}):   # one launch, or one per 7
            ctx.solve(_lib.GF_SOLVER_PCG, _lib.GF_F64, tol=1e-12, max_iter=20000, **kw)
            assert np.linalg.norm(ctx.solution() - x) <= 1e-8 * np.linalg.norm(x)
        ctx.solve(_lib.GF_SOLVER_PCG, _lib.GF_F32, tol=1e-6, max_iter=20000)
        r = b - K @ ctx.solution()   # the FP32 recursion's own accuracy
        assert np.linalg.norm(r) <= 1e-2 * np.linalg.norm(b)


def test_time_limit_stops_between_chunks():
    ctx, _, _ = problem(mg.Q4, (30, 30))
    with ctx:
        info = ctx.solve(_lib.GF_SOLVER_PCG, _lib.GF_F64, tol=1e-12, max_iter=20000, check_every=16,
                         max_seconds=1e-9, raise_on_error=False)
        assert info.status == _lib.GF_ERR_NOT_CONVERGED and info.iterations == 16


def test_solves_repeat_bit_for_bit():
    ctx, _, _ = problem(mg.Q8, (12, 12))
    with ctx:
        u = []
        for _ in range(2):
            ctx.solve(_lib.GF_SOLVER_PCG, _lib.GF_F64, tol=1e-10, max_iter=20000)
            u.append(ctx.solution())
        assert np.array_equal(*u)


# Copies of the direction in every CTA and directions gathered from their homes, on both sides of
# the sizes where the copies stop fitting (5,041 and 5,776 nodes in 2-D, 1,000 and 1,331 in 3-D);
# shuffled node ids give a node up to 16 CTAs that read it.
@pytest.mark.parametrize("et,n", [(mg.Q4, (70, 70)), (mg.Q4, (75, 75)), (mg.Q8, (20, 17)),
                                  (mg.BRICK8, (9, 9, 9)), (mg.BRICK8, (10, 10, 10)),
                                  (mg.BRICK20, (4, 3, 3))])
@pytest.mark.parametrize("shuffled", [False, True])
def test_copies_and_gathers_match_numpy(et, n, shuffled):
    from gpufem_b200.fem import Context
    m = mg.clamp_and_load(mg.structured(et, n, jitter=0.05, seed=2, ngauss=2))
    m.E = mg.lognormal_iid(m, 0.5, seed=3)
    xy, conn, sup, f = m.coords, m.conn, m.supports, m.f
    if shuffled:
        q = np.random.default_rng(1).permutation(m.nnodes)
        xy, f = np.empty_like(m.coords), np.empty_like(m.f)
        xy[q] = m.coords
        f.reshape(-1, m.dim)[q] = m.f.reshape(-1, m.dim)
        conn = (q[m.conn - 1] + 1).astype(np.int32)
        sup = m.supports.copy()
        sup[:, 0] = q[m.supports[:, 0].astype(int) - 1] + 1
    with Context(0) as ctx:
        ctx.mesh_create(m.elem_type, xy, conn, m.ngauss, m.E0, m.E, m.nu)
        ctx.set_supports(sup)
        ctx.set_force(f)
        ctx.assemble(_lib.GF_F64, _lib.GF_SCATTER_AUTO)
        ctx.apply_constraints(_lib.GF_BC_ELIMINATION)
        rn, ci, v = ctx.ell_download(_lib.GF_F64)
        mask = np.arange(ci.shape[0])[:, None] < rn[None, :]
        rows = np.broadcast_to(np.arange(rn.size)[None, :], ci.shape)
        K = sp.csr_matrix((v[mask], (rows[mask], ci[mask])), shape=(rn.size, rn.size))
        b = ctx.get_force()
        for its in (1, 4):
            ctx.solve(_lib.GF_SOLVER_PCG, _lib.GF_F64, tol=1e-30, max_iter=its, raise_on_error=False)
            want = pcg(K, b, 1.0 / K.diagonal(), its)
            assert np.linalg.norm(ctx.solution() - want) <= 1e-10 * np.linalg.norm(want)
