"""Assembly by node owners on scattered numberings, where an element's geometry lies in one piece:
values at the edges of the geometry kernel's blocks, and the time against an ordered numbering."""
import numpy as np
import pytest

from gpufem_b200 import _lib
from gpufem_b200 import meshgen as mg
from test_assembly_node_gpu import TOL

pytestmark = pytest.mark.gpu


def scatter(m):
    r = np.random.default_rng(5)
    p, q = r.permutation(m.nnodes), r.permutation(m.nelem)
    xy = np.empty_like(m.coords)
    xy[p] = m.coords
    return xy, (p[m.conn - 1] + 1).astype(np.int32)[q]


# 127, 128, 129 and 255 to 257 elements: blocks of the geometry kernel full, one under and over
@pytest.mark.parametrize("et,n,ng", [
    (mg.Q4, (127, 1), 2), (mg.Q4, (16, 16), 3), (mg.Q4, (43, 3), 3), (mg.Q8, (16, 8), 3),
    (mg.Q8, (257, 1), 3), (mg.Q8, (17, 15), 2), (mg.BRICK8, (43, 3, 1), 2), (mg.BRICK8, (8, 4, 4), 3),
    (mg.BRICK8, (17, 5, 3), 2)])
@pytest.mark.parametrize("dtype", [_lib.GF_F32, _lib.GF_F64])
def test_scattered_matches_oracle(oracle, et, n, ng, dtype):
    """Tolerance (row-relative) as in test_assembly_node_gpu."""
    from gpufem_b200.fem import Context
    m = mg.structured(et, n, jitter=0.1, seed=3, ngauss=ng)
    E = mg.lognormal_iid(m, 0.5, seed=4)
    xy, conn = scatter(m)
    ro, co, vo = oracle.assemble(et, ng, xy, conn, 210e3, 0.3, E_elem=E)
    with Context(0) as ctx:
        ctx.mesh_create(et, xy, conn, ng, 210e3, E, 0.3, _lib.GF_PLANE_STRESS)
        ctx.assemble(dtype, _lib.GF_SCATTER_OWNER)
        rn, ci, v = ctx.ell_download(dtype)
    assert np.array_equal(rn, ro) and np.array_equal(ci, co)
    assert (np.abs(v - vo).max(0) <= TOL[dtype] * np.abs(vo).max(0)).all()


def test_time_on_a_scattered_numbering():
    """Coordinates, incidences and geometry at random addresses cost nearly the time of K's own
    bytes again; with a line for each 16 bytes of geometry it was 4.5 times the ordered time."""
    from gpufem_b200.fem import Context
    m = mg.structured(mg.BRICK8, (64, 64, 64), jitter=0.1, seed=3, ngauss=2)
    t = []
    for xy, conn in ((m.coords, m.conn), scatter(m)):
        with Context(0) as ctx:
            ctx.mesh_create(m.elem_type, xy, conn, m.ngauss, 210e3, None, 0.3)
            t.append(min(ctx.assemble(_lib.GF_F32, _lib.GF_SCATTER_AUTO) for _ in range(8)))
    assert t[1] <= 3.0 * t[0], t
