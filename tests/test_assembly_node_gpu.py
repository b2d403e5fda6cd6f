"""The node kernels of the owner schedule (Q4, Q8, Brick8) against the oracle, at the sizes
where their node blocks, geometry groups and row tiles end.  Tolerances (row-relative) as in
test_assembly_gpu: FP64 1e-12, FP32 1e-6."""
import numpy as np
import pytest

from ellutil import ell_to_dense, row_rel_err
from gpufem_b200 import _lib
from gpufem_b200 import meshgen as mg

pytestmark = pytest.mark.gpu

TOL = {_lib.GF_F64: 1e-12, _lib.GF_F32: 1e-6}


def check(et, ng, xy, conn, E, dtypes, scatters, oracle, analysis=_lib.GF_PLANE_STRESS):
    from gpufem_b200.fem import Context
    with Context(0) as ctx:
        ctx.mesh_create(et, xy, conn, ng, 210e3, E, 0.3, analysis)
        ro, co, vo = oracle.assemble(et, ng, xy, conn, 210e3, 0.3, E_elem=E)
        A = ell_to_dense(ro, co, vo)
        pad = np.arange(co.shape[0])[:, None] >= ro[None, :]
        for dtype in dtypes:
            for scatter in scatters:
                ctx.assemble(dtype, scatter)
                rn, ci, v = ctx.ell_download(dtype)
                assert np.array_equal(rn, ro) and np.array_equal(ci, co)
                assert np.all(v[pad] == 0)
                assert row_rel_err(A, ell_to_dense(rn, ci, v.astype(np.float64))) <= TOL[dtype]


# One element (fewer than the 8 of a geometry group); 27 to 33 nodes around Brick8's 28 and
# 32 per warp and the 2-D kernel's blocks of 32; sizes with one node or element over.
@pytest.mark.parametrize("et,n,ng", [
    (mg.Q4, (1, 1), 2), (mg.Q4, (3, 7), 2), (mg.Q4, (10, 2), 3), (mg.Q4, (17, 9), 3),
    (mg.Q8, (1, 1), 3), (mg.Q8, (2, 4), 2), (mg.Q8, (3, 3), 3), (mg.Q8, (9, 7), 3),
    (mg.BRICK8, (1, 1, 1), 2), (mg.BRICK8, (2, 2, 2), 2), (mg.BRICK8, (6, 1, 1), 3),
    (mg.BRICK8, (7, 1, 1), 2), (mg.BRICK8, (3, 3, 1), 2), (mg.BRICK8, (10, 2, 1), 3),
    (mg.BRICK8, (5, 4, 3), 2)])
@pytest.mark.parametrize("shuffled", [False, True])
def test_block_edges_match_oracle(oracle, et, n, ng, shuffled):
    """Shuffled: node ids, element order and each node's slots in no order."""
    m = mg.structured(et, n, jitter=0.1, seed=3, ngauss=ng)
    E = mg.lognormal_iid(m, 0.5, seed=4)
    xy, conn = m.coords, m.conn
    if shuffled:
        r = np.random.default_rng(1)
        p, q = r.permutation(m.nnodes), r.permutation(m.nelem)
        xy = np.empty_like(m.coords)
        xy[p] = m.coords
        conn, E = (p[m.conn - 1] + 1).astype(np.int32)[q], E[q]
    check(et, ng, xy, conn, E, TOL, [_lib.GF_SCATTER_AUTO, _lib.GF_SCATTER_OWNER], oracle)


def fan(k):
    """k quadrilaterals around one centre node."""
    th = 2 * np.pi * np.arange(k) / k
    xy = np.array([[0.0, 0.0]] + [[np.cos(t), np.sin(t)] for t in th]
                  + [[2.0 * np.cos(t + np.pi / k), 2.0 * np.sin(t + np.pi / k)] for t in th])
    conn = np.array([[1, 2 + j, 2 + k + j, 2 + (j + 1) % k] for j in range(k)], np.int32)
    return xy, conn


# Rows of 2 (2 k + 1) slots: a 2-D tile of 112 KB and less holds k = 48, not k = 56 (FP64);
# FP64 only, since the slivers are beyond the FP32 tolerance.
@pytest.mark.parametrize("k", [20, 48, 56])
def test_wide_rows_2d(oracle, k):
    xy, conn = fan(k)
    check(mg.Q4, 2, xy, conn, None, [_lib.GF_F64], [_lib.GF_SCATTER_AUTO], oracle)


# Rows of 6 (2 k + 1) slots with two layers of hexahedra around an axis (9 (2 k + 1) at the
# middle node): k = 7 fits the FP64 Brick8 tile, k = 9 does not (the atomic schedule).
@pytest.mark.parametrize("k", [7, 9])
def test_wide_rows_3d(oracle, k):
    xy, quad = fan(k)
    nn = len(xy)
    xyz = np.concatenate([np.column_stack([xy, np.full(nn, z)]) for z in (0.0, 1.0, 2.0)])
    # element nodes (r, s, t): r = +1 is the upper layer, (s, t) run around the quadrilateral
    conn = np.concatenate([np.column_stack([quad + (l + 1) * nn, quad + l * nn]) for l in (0, 1)])
    check(mg.BRICK8, 2, xyz, conn.astype(np.int32), None, [_lib.GF_F64],
          [_lib.GF_SCATTER_AUTO, _lib.GF_SCATTER_OWNER], oracle)


def test_distorted_brick8_takes_fp64_geometry(oracle):
    """Elements whose detJ varies more than tenfold over the Gauss points."""
    m = mg.structured(mg.BRICK8, (3, 2, 2), seed=1, ngauss=2)
    xyz = m.coords.copy()
    xyz[:, 0] = np.where(np.abs(xyz[:, 0] - 1 / 3) < 1e-9,
                         0.02 + 0.6 * xyz[:, 1] * xyz[:, 2], xyz[:, 0])
    check(mg.BRICK8, 2, xyz, m.conn, None, TOL, [_lib.GF_SCATTER_AUTO], oracle)


# FP64 Brick8 takes the node kernel from a node per lane of every SM's warp on (3552 nodes on 148
# SMs): the last warp full (4032 = 144 x 28) and ragged, on both sides of the line.
@pytest.mark.parametrize("n,ng", [((17, 15, 13), 2), ((16, 15, 14), 3), ((13, 14, 15), 2)])
@pytest.mark.parametrize("shuffled", [False, True])
def test_brick8_fp64_node_kernel_matches_oracle(oracle, n, ng, shuffled):
    m = mg.structured(mg.BRICK8, n, jitter=0.1, seed=3, ngauss=ng)
    E = mg.lognormal_iid(m, 0.5, seed=4)
    xy, conn = m.coords, m.conn
    if shuffled:
        r = np.random.default_rng(1)
        p, q = r.permutation(m.nnodes), r.permutation(m.nelem)
        xy = np.empty_like(m.coords)
        xy[p] = m.coords
        conn, E = (p[m.conn - 1] + 1).astype(np.int32)[q], E[q]
    # row by row, without dense matrices
    from gpufem_b200.fem import Context
    ro, co, vo = oracle.assemble(mg.BRICK8, ng, xy, conn, 210e3, 0.3, E_elem=E)
    with Context(0) as ctx:
        ctx.mesh_create(mg.BRICK8, xy, conn, ng, 210e3, E, 0.3, _lib.GF_PLANE_STRESS)
        for scatter in (_lib.GF_SCATTER_OWNER, _lib.GF_SCATTER_AUTO):
            ctx.assemble(_lib.GF_F64, scatter)
            rn, ci, v = ctx.ell_download(_lib.GF_F64)
            assert np.array_equal(rn, ro) and np.array_equal(ci, co)
            assert (np.abs(v - vo).max(0) <= TOL[_lib.GF_F64] * np.abs(vo).max(0)).all()
