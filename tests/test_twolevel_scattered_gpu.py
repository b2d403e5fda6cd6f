"""The two-level PCG on randomly numbered nodes, where the update of x and r runs by rows and the
restriction alone: against the numpy oracle, and the time of an iteration."""
import numpy as np
import pytest

from gpufem_b200 import _lib
from gpufem_b200 import meshgen as mg
from oracle import twolevel_oracle as tl

pytestmark = pytest.mark.gpu


def context(et, n, scattered):
    from gpufem_b200.fem import Context
    m = mg.clamp_and_load(mg.structured(et, n, jitter=0.1, seed=3, ngauss=2))
    q = np.random.default_rng(1).permutation(m.nnodes) if scattered else np.arange(m.nnodes)
    x, f, sup = np.empty_like(m.coords), np.empty_like(m.f), m.supports.copy()
    x[q] = m.coords
    f.reshape(-1, m.dim)[q] = m.f.reshape(-1, m.dim)
    sup[:, 0] = q[m.supports[:, 0].astype(int) - 1] + 1
    fixed = np.zeros(m.ndof, np.uint8)
    for row in sup:
        fixed[(row[0] - 1) * m.dim:row[0] * m.dim] |= (row[1:1 + m.dim] == 1).astype(np.uint8)
    ctx = Context(0)
    ctx.mesh_create(m.elem_type, x, (q[m.conn - 1] + 1).astype(np.int32), m.ngauss, m.E0, None, m.nu)
    ctx.set_supports(sup)
    ctx.set_force(f)
    ctx.assemble(_lib.GF_F64, _lib.GF_SCATTER_AUTO)
    ctx.apply_constraints(_lib.GF_BC_ELIMINATION)
    ctx.convert_f64_to_f32()
    return ctx, x, np.where(fixed == 1, 0.0, f), fixed


# 22,801 and 32,768 nodes, of which 32 consecutive ones have neighbours in nearly as many blocks
@pytest.mark.parametrize("et,n", [(mg.Q4, (150, 150)), (mg.BRICK8, (31, 31, 31))])
def test_scattered_nodes_match_oracle(et, n):
    """Bounds as in test_twolevel_update_gpu."""
    ctx, x, f, fixed = context(et, n, True)
    with ctx:
        ctx.twolevel_setup(0)
        agg, side = ctx.twolevel_aggregates()
        rn, ci, v = ctx.ell_download(_lib.GF_F64)
        pc = tl.TwoLevel(x, rn, ci, v, fixed, agg=agg, side=side)
        ustar, it_o = pc.pcg(f, 1e-12)
        ctx.twolevel_apply(np.ones(f.size))  # leaves its own partial sums behind
        info = ctx.solve(_lib.GF_SOLVER_TWOLEVEL_PCG, tol=1e-12, max_iter=200000)
        assert info.status == _lib.GF_OK
        assert abs(info.iterations - it_o) <= max(2, it_o // 20), (info.iterations, it_o)
        assert np.linalg.norm(ctx.solution() - ustar) <= 1e-8 * np.linalg.norm(ustar)
        info32 = ctx.solve(_lib.GF_SOLVER_TWOLEVEL_PCG32, _lib.GF_F32, tol=1e-8, max_iter=200000)
        assert info32.status == _lib.GF_OK and info32.rel_residual <= 1e-8
        assert np.linalg.norm(ctx.solution() - ustar) <= 1e-5 * np.linalg.norm(ustar)


def test_iteration_time_of_scattered_nodes():
    """1.19 of the ordered mesh's time, most of it the product; 1.6 with every vector gathered."""
    t = []
    for scattered in (False, True):
        ctx, _, _, _ = context(mg.Q8, (400, 400), scattered)
        with ctx:
            t.append(min(i.seconds / i.iterations for i in
                         (ctx.solve(_lib.GF_SOLVER_TWOLEVEL_PCG, tol=1e-30, max_iter=60,
                                    raise_on_error=False) for _ in range(4))))
    assert t[1] <= 1.38 * t[0], t
