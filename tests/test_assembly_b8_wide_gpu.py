"""Brick8 by node owners with rows around the widest that its tiles take (154 slots in FP64, 279 in
FP32), in meshes large enough for that kernel: two layers of hexahedra around an axis beside a
structured block."""
import numpy as np
import pytest

from gpufem_b200 import _lib
from gpufem_b200 import meshgen as mg
from test_assembly_node_gpu import TOL

pytestmark = pytest.mark.gpu


def fan(k):
    """Two layers of k hexahedra around an axis; their quadrilaterals are 1.2 long, 2 sin(pi / k)
    wide.  The middle of the axis has rows of 9 (2 k + 1) slots."""
    th = 2 * np.pi * np.arange(k) / k
    xy = np.array([[0.0, 0.0]] + [[np.cos(t), np.sin(t)] for t in th]
                  + [[1.2 * np.cos(t + np.pi / k), 1.2 * np.sin(t + np.pi / k)] for t in th])
    quad = np.array([[1, 2 + j, 2 + k + j, 2 + (j + 1) % k] for j in range(k)], np.int32)
    nn = len(xy)
    xyz = np.concatenate([np.column_stack([xy, np.full(nn, z)]) for z in (0.0, 0.4, 0.8)])
    # element nodes (r, s, t): r = +1 is the upper layer, (s, t) run around the quadrilateral
    conn = np.concatenate([np.column_stack([quad + (l + 1) * nn, quad + l * nn]) for l in (0, 1)])
    return xyz, conn.astype(np.int32)


# k = 8 and 15 are the last that fit; 3,552 nodes take FP64 to this kernel, 11,248 from AUTO too
@pytest.mark.parametrize("dtype,k,block", [
    (_lib.GF_F64, 7, (16, 15, 14)), (_lib.GF_F64, 8, (23, 22, 22)), (_lib.GF_F64, 9, (23, 22, 22)),
    (_lib.GF_F32, 8, (4, 3, 3)), (_lib.GF_F32, 15, (5, 4, 3)), (_lib.GF_F32, 16, (5, 4, 3))])
@pytest.mark.parametrize("first", [False, True])
def test_wide_rows(oracle, dtype, k, block, first):
    from gpufem_b200.fem import Context
    m = mg.structured(mg.BRICK8, block, jitter=0.1, seed=3, ngauss=2)
    xyz, conn = fan(k)
    if first:   # the wide rows lead, or come last
        x, c = np.concatenate([xyz, m.coords + 5.0]), np.concatenate([conn, m.conn + len(xyz)])
    else:
        x, c = np.concatenate([m.coords + 5.0, xyz]), np.concatenate([m.conn, conn + m.nnodes])
    E = np.random.default_rng(7).uniform(1e5, 3e5, len(c))
    ro, co, vo = oracle.assemble(mg.BRICK8, 2, x, c.astype(np.int32), 210e3, 0.3, E_elem=E)
    assert co.shape[0] == max(81, 9 * (2 * k + 1))
    with Context(0) as ctx:
        ctx.mesh_create(mg.BRICK8, x, c.astype(np.int32), 2, 210e3, E, 0.3, _lib.GF_PLANE_STRESS)
        for scatter in (_lib.GF_SCATTER_OWNER, _lib.GF_SCATTER_AUTO):
            ctx.assemble(dtype, scatter)
            rn, ci, v = ctx.ell_download(dtype)
            assert np.array_equal(rn, ro) and np.array_equal(ci, co)
            assert np.all(v[np.arange(co.shape[0])[:, None] >= ro[None, :]] == 0)
            assert (np.abs(v - vo).max(0) <= TOL[dtype] * np.abs(vo).max(0)).all()
