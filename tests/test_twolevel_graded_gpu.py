"""The two-level PCG on graded meshes, where one aggregate holds most nodes: its blocks in the
fused update against the numpy oracle, and the time of an iteration against a uniform mesh's."""
import numpy as np
import pytest

from gpufem_b200 import _lib
from gpufem_b200 import meshgen as mg
from oracle import twolevel_oracle as tl

pytestmark = pytest.mark.gpu


def context(et, n, squeeze):
    """0.9^dim of the mesh squeezed into 0.108 of every axis."""
    from gpufem_b200.fem import Context
    # (no jitter: where elements are 80 times wider it would invert them)
    m = mg.clamp_and_load(mg.structured(et, n, ngauss=2))
    x = m.coords
    if squeeze:
        x = np.where(x <= 0.9, 0.12 * x, 0.108 + 8.92 * (x - 0.9))
    ctx = Context(0)
    ctx.mesh_create(m.elem_type, x, m.conn, m.ngauss, m.E0, None, m.nu)
    ctx.set_supports(m.supports)
    ctx.set_force(m.f)
    ctx.assemble(_lib.GF_F64, _lib.GF_SCATTER_AUTO)
    ctx.apply_constraints(_lib.GF_BC_ELIMINATION)
    ctx.convert_f64_to_f32()
    return ctx, m, x


# the largest aggregate takes 2, 9 and the most (64) blocks, 3 in Q8, 4 and 9 in 3-D
@pytest.mark.parametrize("et,n,target", [
    (mg.Q4, (15, 14), 12), (mg.Q4, (40, 40), 48), (mg.Q4, (110, 100), 192), (mg.Q8, (10, 10), 24),
    (mg.BRICK8, (9, 8, 7), 48), (mg.BRICK8, (11, 10, 10), 96)])
def test_uneven_aggregates_match_oracle(et, n, target):
    """Iteration counts as for even ones (test_twolevel_update_gpu).  The recursion to 1e-12 leaves
    a true residual of up to 1e-10 (rounding of K u; the oracle's own is 9e-11) and an error of up
    to 3e-12 (the oracle's against a direct solve): 1e-9 for the solution, and 1e-8 for the FP32
    recursion, which stops on the true residual."""
    ctx, m, x = context(et, n, True)
    fixed = np.zeros(m.ndof, np.uint8)
    for row in m.supports:
        fixed[(row[0] - 1) * m.dim:row[0] * m.dim] |= (row[1:1 + m.dim] == 1).astype(np.uint8)
    with ctx:
        ctx.twolevel_setup(target)
        agg, side = ctx.twolevel_aggregates()
        rn, ci, v = ctx.ell_download(_lib.GF_F64)
        f = np.where(fixed == 1, 0.0, m.f)
        pc = tl.TwoLevel(x, rn, ci, v, fixed, agg=agg, side=side)
        ustar, it_o = pc.pcg(f, 1e-12)
        ctx.twolevel_apply(np.ones(m.ndof))  # leaves its own partial sums behind
        info = ctx.solve(_lib.GF_SOLVER_TWOLEVEL_PCG, tol=1e-12, max_iter=200000)
        assert info.status == _lib.GF_OK
        assert abs(info.iterations - it_o) <= max(2, it_o // 20), (info.iterations, it_o)
        assert np.linalg.norm(ctx.solution() - ustar) <= 1e-9 * np.linalg.norm(ustar)
        z, z_o = ctx.twolevel_apply(m.f), pc.apply(m.f)   # after a solve: the other way round
        assert np.linalg.norm(z - z_o) <= 1e-9 * np.linalg.norm(z_o)
        info32 = ctx.solve(_lib.GF_SOLVER_TWOLEVEL_PCG32, _lib.GF_F32, tol=1e-8, max_iter=200000)
        assert info32.status == _lib.GF_OK and info32.rel_residual <= 1e-8


def test_iteration_time_of_a_graded_mesh():
    """An iteration reads the same matrix and vectors: with even blocks it takes about a third
    longer than on the uniform mesh, waiting for the largest aggregate four times as long."""
    t = []
    for squeeze in (False, True):
        ctx, _, _ = context(mg.BRICK8, (40, 40, 40), squeeze)
        with ctx:
            best = min((i.seconds / i.iterations for i in
                        (ctx.solve(_lib.GF_SOLVER_TWOLEVEL_PCG, tol=1e-30, max_iter=100,
                                   raise_on_error=False) for _ in range(5))))
        t.append(best)
    assert t[1] <= 2.2 * t[0], t
