"""The two-level PCG's fused update and restriction (blocks that share an aggregate's nodes) and
its coarse product's own r.z: iteration counts and solutions against the numpy oracle, for one
aggregate with one and with many blocks, for blocks with a last node over, and for the FP32
recursion.  Bounds as for the solver's other tests."""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spla

from gpufem_b200 import _lib
from gpufem_b200 import meshgen as mg
from oracle import twolevel_oracle as tl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("et,n,target", [
    (mg.Q4, (3, 2), 3), (mg.Q4, (42, 2), 3), (mg.Q4, (31, 23), 48), (mg.Q8, (10, 9), 3),
    (mg.BRICK8, (3, 3, 2), 6), (mg.BRICK8, (7, 3, 3), 6), (mg.BRICK8, (9, 8, 7), 60),
    (mg.BRICK20, (3, 2, 2), 6), (mg.BRICK20, (5, 4, 3), 40)])
def test_update_by_shares_of_aggregates(et, n, target):
    from gpufem_b200.fem import Context
    m = mg.clamp_and_load(mg.structured(et, n, jitter=0.1, seed=3, ngauss=2))
    fixed = np.zeros(m.ndof, np.uint8)
    for row in m.supports:
        for c in range(m.dim):
            if row[1 + c] == 1:
                fixed[(row[0] - 1) * m.dim + c] = 1
    with Context(0) as ctx:
        ctx.mesh_create(m.elem_type, m.coords, m.conn, m.ngauss, m.E0, m.E, m.nu)
        ctx.set_supports(m.supports)
        ctx.set_force(m.f)
        ctx.assemble(_lib.GF_F64, _lib.GF_SCATTER_AUTO)
        ctx.apply_constraints(_lib.GF_BC_ELIMINATION)
        ctx.convert_f64_to_f32()
        ctx.twolevel_setup(target)
        agg, side = ctx.twolevel_aggregates()
        rn, ci, v = ctx.ell_download(_lib.GF_F64)
        live = np.arange(ci.shape[0])[:, None] < rn[None, :]
        rows = np.broadcast_to(np.arange(m.ndof), ci.shape)
        K = sp.csr_matrix((v[live], (rows[live], ci[live])), shape=(m.ndof, m.ndof))
        f = np.where(fixed == 1, 0.0, m.f)
        pc = tl.TwoLevel(m.coords, rn, ci, v, fixed, agg=agg, side=side)
        _, it_o = pc.pcg(f, 1e-12)
        ustar = spla.spsolve(K.tocsc(), f)
        ctx.twolevel_apply(np.ones(m.ndof))  # leaves its own partial sums behind
        info = ctx.solve(_lib.GF_SOLVER_TWOLEVEL_PCG, tol=1e-12, max_iter=200000)
        assert info.status == _lib.GF_OK and info.rel_residual <= 1e-11
        assert abs(info.iterations - it_o) <= max(2, it_o // 20), (info.iterations, it_o)
        u = ctx.solution()
        assert np.linalg.norm(u - ustar) <= 1e-8 * np.linalg.norm(ustar)
        info32 = ctx.solve(_lib.GF_SOLVER_TWOLEVEL_PCG32, _lib.GF_F32, tol=1e-10, max_iter=200000)
        assert info32.status == _lib.GF_OK and info32.rel_residual <= 1e-10
        assert info32.iterations <= 2 * info.iterations + 10
        assert np.linalg.norm(ctx.solution() - ustar) <= 1e-7 * np.linalg.norm(ustar)
