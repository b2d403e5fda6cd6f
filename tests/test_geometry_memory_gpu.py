"""Brick8 assembly by owners keeps a geometry buffer; what it must not cost: room that the calls
after it had without it, and a failing allocation on every assembly where it does not fit.  Device
memory is taken up by a tensor, so that allocations return an error."""
import ctypes as C

import numpy as np
import pytest
import torch

from gpufem_b200 import _lib
from gpufem_b200 import meshgen as mg

pytestmark = pytest.mark.gpu
MB = 1 << 20
N = 64   # FP64: K 534 MB, slices 537 + 30, geometry 168; pattern scratch in the pool about 70


def mesh(ctx):
    m = mg.structured(mg.BRICK8, (N, N, N), jitter=0.05, seed=1, ngauss=2)
    ctx.mesh_create(m.elem_type, m.coords, m.conn, m.ngauss, 210e3, None, 0.3)
    ctx.build_pattern()
    return m


def leave(megabytes):
    """Takes up all but `megabytes` of the device's memory."""
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    return torch.empty(free - megabytes * MB, dtype=torch.uint8, device="cuda")


def split(ctx):
    g, s = C.c_double(), C.c_double()
    _lib.check(_lib.lib.gf_last_assembly_split(ctx.h, C.byref(g), C.byref(s)), ctx.h)
    return g.value, s.value


def test_geometry_gives_way_to_the_slices():
    """430 MB and the pool's 70 hold neither the slices' values beside the geometry, nor ask for
    more than there is without it."""
    from gpufem_b200.fem import Context
    with Context(0) as ctx:
        m = mesh(ctx)
        x = torch.randn(m.ndof, dtype=torch.float64, device="cuda")
        y, want = torch.empty_like(x), torch.empty_like(x)
        ctx.assemble(_lib.GF_F64, _lib.GF_SCATTER_AUTO)
        assert split(ctx)[0] > 0   # by owners
        held = leave(430)
        px, py = C.c_void_p(x.data_ptr()), C.c_void_p(y.data_ptr())
        _lib.check(_lib.lib.gf_spmv(ctx.h, _lib.GF_F64, px, py), ctx.h)
        del held
        torch.cuda.empty_cache()
        ctx.assemble(_lib.GF_F64, _lib.GF_SCATTER_AUTO)   # the buffer is had again
        assert split(ctx)[0] > 0
        _lib.check(_lib.lib.gf_spmv(ctx.h, _lib.GF_F64, px, C.c_void_p(want.data_ptr())), ctx.h)
        assert torch.equal(y, want)


def test_assembly_without_room_for_geometry():
    from gpufem_b200.fem import Context
    with Context(0) as ctx:
        mesh(ctx)
        ctx.assemble(_lib.GF_F64, _lib.GF_SCATTER_AUTO)
        assert split(ctx)[0] > 0
        want = ctx.ell_download(_lib.GF_F64)[2]
    with Context(0) as ctx:
        mesh(ctx)
        held = leave(560)
        ctx.assemble(_lib.GF_F64, _lib.GF_SCATTER_AUTO)
        assert split(ctx)[0] == 0   # atomics
        got = ctx.ell_download(_lib.GF_F64)[2]
        del held
        torch.cuda.empty_cache()
        ctx.assemble(_lib.GF_F64, _lib.GF_SCATTER_AUTO)   # known not to fit: not asked for again
        assert split(ctx)[0] == 0
        mesh(ctx)
        ctx.assemble(_lib.GF_F64, _lib.GF_SCATTER_AUTO)   # a new pattern
        assert split(ctx)[0] > 0
    # row-relative: sums of 8 element entries of 8 points in two orders
    assert (np.abs(got - want).max(0) <= 1e-13 * np.abs(want).max(0)).all()
