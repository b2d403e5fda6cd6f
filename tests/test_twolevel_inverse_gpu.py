"""The coarse inverse by symmetric sweeps of 64 x 64 tiles, through z = M r: coarse sizes below,
at and just over a tile, and over several, against the numpy oracle's solve (bound as for the
solver's other sizes)."""
import numpy as np
import pytest

from gpufem_b200 import _lib
from gpufem_b200 import meshgen as mg
from oracle import twolevel_oracle as tl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("et,n,targets", [
    (mg.Q4, (40, 33), (3, 12, 63, 66, 129, 195, 330)),
    (mg.Q8, (24, 24), (48, 192, 600)),
    (mg.BRICK8, (12, 11, 10), (6, 48, 66, 130, 192, 390, 1000))])
def test_inverse_at_tile_edges(et, n, targets):
    from gpufem_b200.fem import Context
    m = mg.clamp_and_load(mg.structured(et, n, jitter=0.1, seed=3, ngauss=2))
    m.E = mg.lognormal_iid(m, 0.5, seed=4)
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
        rn, ci, v = ctx.ell_download(_lib.GF_F64)
        rng = np.random.default_rng(5)
        for target in targets:
            nc = ctx.twolevel_setup(target)
            agg, side = ctx.twolevel_aggregates()
            pc = tl.TwoLevel(m.coords, rn, ci, v, fixed, agg=agg, side=side)
            assert nc == pc.ncoarse
            r = np.where(fixed == 1, 0.0, rng.standard_normal(m.ndof))
            z, zo = ctx.twolevel_apply(r), pc.apply(r)
            assert np.linalg.norm(z - zo) <= 1e-9 * np.linalg.norm(zo), (target, nc)
