"""Brick20 by reductions on matrices of more than 1.5 GB, where an ordered mesh's lines are fetched
to L2 ahead: values against the colour schedule, ordered and with the nodes shuffled in runs of 16
(which fetch nothing ahead), and the time of the latter."""
import ctypes as C

import numpy as np
import pytest
import torch

from gpufem_b200 import _lib
from gpufem_b200 import meshgen as mg

pytestmark = pytest.mark.gpu

# row-relative: a row's entries are sums of at most 8 element entries of 8 points each
TOL = {_lib.GF_F64: 1e-12, _lib.GF_F32: 1e-6}


class _Array:
    def __init__(self, ptr, shape, typestr):
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 3}


def values(ctx, dtype):
    n, w, p = C.c_int32(), C.c_int32(), [C.c_void_p() for _ in range(3)]
    _lib.check(_lib.lib.gf_ell_view(ctx.h, dtype, C.byref(n), C.byref(w), *map(C.byref, p)), ctx.h)
    return torch.as_tensor(_Array(p[2].value, (w.value, n.value), "<f8" if dtype == _lib.GF_F64 else "<f4"),
                           device="cuda")


def runs(m, length=16):
    k = -(-m.nnodes // length)
    old = (np.random.default_rng(2).permutation(k)[:, None] * length + np.arange(length)).ravel()
    old = old[old < m.nnodes]
    new = np.empty(m.nnodes, np.int64)
    new[old] = np.arange(m.nnodes)
    return m.coords[old], (new[m.conn - 1] + 1).astype(np.int32)


@pytest.mark.parametrize("dtype,n", [(_lib.GF_F32, 52), (_lib.GF_F64, 42)])
@pytest.mark.parametrize("shuffled", [False, True])
def test_values_of_every_row(dtype, n, shuffled):
    check(dtype, n, shuffled, 1.5e9)


def test_a_group_per_cta():
    """Shuffled FP32 meshes from 0.3 GB on; 35,937 elements: the last group has one."""
    check(_lib.GF_F32, 33, True, 0.3e9)


def check(dtype, n, shuffled, size):
    from gpufem_b200.fem import Context
    m = mg.structured(mg.BRICK20, (n, n, n), jitter=0.05, seed=1, ngauss=2)
    xy, conn = runs(m) if shuffled else (m.coords, m.conn)
    with Context(0) as ctx:
        ctx.mesh_create(m.elem_type, xy, conn, m.ngauss, 210e3, None, 0.3)
        ctx.assemble(dtype, _lib.GF_SCATTER_COLOR)
        want = values(ctx, dtype).clone()
        ctx.assemble(dtype, _lib.GF_SCATTER_ATOMIC)
        got = values(ctx, dtype)
        assert want.numel() * want.element_size() > size
        worst = 0.0
        for k in range(0, want.shape[1], 1 << 17):   # columns of the array: rows of K
            a, b = got[:, k:k + (1 << 17)].double(), want[:, k:k + (1 << 17)].double()
            worst = max(worst, float(((a - b).abs().amax(0) / b.abs().amax(0)).max()))
    assert worst <= TOL[dtype], worst


def test_time_with_shuffled_runs_of_nodes():
    """1.6 times the ordered mesh's time; 4.0 with lines fetched that nothing else will use."""
    from gpufem_b200.fem import Context
    m = mg.structured(mg.BRICK20, (52, 52, 52), jitter=0.05, seed=1, ngauss=2)
    t = []
    for xy, conn in ((m.coords, m.conn), runs(m)):
        with Context(0) as ctx:
            ctx.mesh_create(m.elem_type, xy, conn, m.ngauss, 210e3, None, 0.3)
            t.append(min(ctx.assemble(_lib.GF_F32, _lib.GF_SCATTER_AUTO) for _ in range(4)))
    assert t[1] <= 3.0 * t[0], t
