"""Brick20 by coalesced reductions (the atomic schedule) against the oracle: element counts
around a CTA's group of 8 (FP32) or 4 (FP64), more groups than CTAs, shuffled numbering, and
elements whose FP32 points are redone in FP64.  Tolerances as in test_assembly_gpu."""
import numpy as np
import pytest

from gpufem_b200 import _lib
from gpufem_b200 import meshgen as mg
from test_assembly_node_gpu import TOL, check

pytestmark = pytest.mark.gpu

SCATTERS = [_lib.GF_SCATTER_AUTO, _lib.GF_SCATTER_ATOMIC]


@pytest.mark.parametrize("n,ng", [((1, 1, 1), 2), ((3, 1, 1), 3), ((1, 4, 1), 3), ((5, 1, 1), 2),
                                  ((7, 1, 1), 3), ((2, 2, 2), 3), ((3, 3, 1), 2), ((5, 3, 2), 3)])
@pytest.mark.parametrize("shuffled", [False, True])
def test_group_edges_match_oracle(oracle, n, ng, shuffled):
    m = mg.structured(mg.BRICK20, n, jitter=0.1, seed=3, ngauss=ng)
    E = mg.lognormal_iid(m, 0.5, seed=4)
    xy, conn = m.coords, m.conn
    if shuffled:
        r = np.random.default_rng(1)
        p, q = r.permutation(m.nnodes), r.permutation(m.nelem)
        xy = np.empty_like(m.coords)
        xy[p] = m.coords
        conn, E = (p[m.conn - 1] + 1).astype(np.int32)[q], E[q]
    check(mg.BRICK20, ng, xy, conn, E, TOL, SCATTERS, oracle)


def test_distorted_elements_match_oracle(oracle):
    """max/min |detJ| of the first elements is about 65."""
    m = mg.structured(mg.BRICK20, (3, 2, 2), jitter=0.0, seed=3, ngauss=3)
    xy = m.coords.copy()
    xy[:, 0] = (xy[:, 0] - xy[:, 0].min()) ** 3
    check(mg.BRICK20, 3, xy, m.conn, mg.lognormal_iid(m, 0.5, seed=4), TOL, SCATTERS, oracle)


@pytest.mark.parametrize("dtype", [_lib.GF_F32, _lib.GF_F64])
def test_more_groups_than_ctas(dtype):
    """Every CTA takes several groups (2548 elements); colours write each entry by plain sums."""
    from gpufem_b200.fem import Context
    m = mg.structured(mg.BRICK20, (14, 13, 14), jitter=0.1, seed=3, ngauss=2)
    with Context(0) as ctx:
        ctx.mesh_create(m.elem_type, m.coords, m.conn, m.ngauss, 210e3,
                        mg.lognormal_iid(m, 0.5, seed=4), 0.3)
        ctx.assemble(dtype, _lib.GF_SCATTER_COLOR)
        rn, ci, want = ctx.ell_download(dtype)
        ctx.assemble(dtype, _lib.GF_SCATTER_ATOMIC)
        rn2, ci2, got = ctx.ell_download(dtype)
    assert np.array_equal(rn, rn2) and np.array_equal(ci, ci2)
    scale = np.abs(want.astype(np.float64)).max(0)
    err = np.abs(got.astype(np.float64) - want.astype(np.float64)).max(0)
    assert (err <= TOL[dtype] * scale).all()


def test_lines_fetched_ahead():
    """K of 1.7 GB (from 1.5 GB on a group's lines are fetched ahead): K x as after the colour
    schedule.  A row sums up to 8 element entries and then 243 products in FP32; its entries and x
    are of order max |K x| / 1, so 300 roundings of it bound the difference."""
    import ctypes as C

    import torch
    from gpufem_b200.fem import Context
    m = mg.structured(mg.BRICK20, (52, 52, 52), jitter=0.05, seed=1, ngauss=2)
    with Context(0) as ctx:
        ctx.mesh_create(m.elem_type, m.coords, m.conn, m.ngauss, 210e3, None, 0.3)
        x = torch.randn(m.ndof, generator=torch.Generator().manual_seed(3)).cuda()
        ys = []
        for scatter in (_lib.GF_SCATTER_COLOR, _lib.GF_SCATTER_ATOMIC):
            ctx.assemble(_lib.GF_F32, scatter)
            y = torch.empty_like(x)
            _lib.check(_lib.lib.gf_spmv(ctx.h, _lib.GF_F32, C.c_void_p(x.data_ptr()),
                                        C.c_void_p(y.data_ptr())), ctx.h)
            ys.append(y.double())
    assert float((ys[0] - ys[1]).abs().max()) <= 300 * 2.0**-24 * float(ys[0].abs().max())
