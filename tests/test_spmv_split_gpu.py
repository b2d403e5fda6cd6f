"""y = K x on node-block slices walked by one, two or four warps: every split, at slice counts that
leave the last slice and the last block ragged, against the FP64 product of the stored matrix."""
import ctypes as C

import numpy as np
import pytest
import torch

from gpufem_b200 import _lib, meshgen as mg
from gpufem_b200.fem import Context

pytestmark = pytest.mark.gpu

# element type, elements per axis; node counts around multiples of 32 and of a block's slices,
# one node-slice in all, and on both sides of the 2-D line (16 slices per SM)
MESHES = [
    ("q4", (1, 1)), ("q4", (7, 3)), ("q4", (8, 6)), ("q4", (331, 257)),
    ("q8", (1, 1)), ("q8", (23, 17)), ("q8", (181, 163)),
    ("brick8", (1, 1, 1)), ("brick8", (3, 1, 3)), ("brick8", (9, 7, 5)), ("brick8", (21, 20, 22)),
    ("brick20", (1, 1, 1)), ("brick20", (2, 3, 1)), ("brick20", (7, 6, 9)),
]
TYPES = {"q4": mg.Q4, "q8": mg.Q8, "brick8": mg.BRICK8, "brick20": mg.BRICK20}


@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("elem,cells", MESHES)
def test_spmv_split(elem, cells, dtype):
    m = mg.structured(TYPES[elem], cells, jitter=0.1, seed=5, ngauss=2)
    gdt, tdt, eps = {"f32": (_lib.GF_F32, torch.float32, 2.0**-24),
                     "f64": (_lib.GF_F64, torch.float64, 2.0**-53)}[dtype]
    ctx = Context(0)
    try:
        ctx.mesh_create(m.elem_type, m.coords, m.conn, m.ngauss, m.E0, None, m.nu)
        ctx.assemble(gdt, _lib.GF_SCATTER_AUTO)
        nnz, col, val = ctx.ell_download(gdt)
        n = m.ndof
        live = np.arange(val.shape[0])[:, None] < nnz[None, :]
        x = torch.randn(n, dtype=tdt, generator=torch.Generator().manual_seed(3))
        xg = np.where(live, x.numpy().astype(np.longdouble)[np.where(live, col, 0)], 0)
        prod = np.where(live, val, 0).astype(np.longdouble) * xg
        want, size = prod.sum(0), np.abs(prod).sum(0)
        xd, y = x.cuda(), torch.full((n,), float("nan"), dtype=tdt, device="cuda")
        _lib.check(_lib.lib.gf_spmv(ctx.h, gdt, C.c_void_p(xd.data_ptr()),
                                    C.c_void_p(y.data_ptr())), ctx.h)
        got = y.cpu().numpy().astype(np.longdouble)
    finally:
        ctx.close()
    # a row of k products: at most k roundings reach any term (FMAs or sums in any order), and
    # the result is rounded once
    bound = (nnz + 2) * eps * size
    assert (np.abs(got - want) <= bound).all()
