"""gf_last_device_seconds and gf_last_assembly_split hold the last call that succeeded."""
import ctypes as C

import pytest
import torch

from gpufem_b200 import _lib
from test_geometry_memory_gpu import leave, mesh, split

pytestmark = pytest.mark.gpu


def test_a_failed_assembly_leaves_the_times():
    """The owner schedule finds no room for its geometry (168 MB) after its timer has started."""
    from gpufem_b200.fem import Context
    with Context(0) as ctx:
        mesh(ctx)
        ctx.assemble(_lib.GF_F64, _lib.GF_SCATTER_ATOMIC)
        before = _lib.lib.gf_last_device_seconds(ctx.h), split(ctx)
        assert before[0] > 0 and before[1] == (0.0, before[0])
        held = leave(40)
        with pytest.raises(_lib.GpufemError) as e:
            ctx.assemble(_lib.GF_F64, _lib.GF_SCATTER_OWNER)
        assert e.value.status == _lib.GF_ERR_OOM
        assert (_lib.lib.gf_last_device_seconds(ctx.h), split(ctx)) == before
        del held
        torch.cuda.empty_cache()
        ctx.assemble(_lib.GF_F64, _lib.GF_SCATTER_OWNER)
        g, s = split(ctx)
        total = _lib.lib.gf_last_device_seconds(ctx.h)
        assert g > 0 and s > 0 and abs(g + s - total) <= 2e-6   # event times in steps of 0.5 us
        # a product between two assemblies has its own
        x = torch.ones(ctx.n, dtype=torch.float64, device="cuda")
        y = torch.empty_like(x)
        _lib.check(_lib.lib.gf_spmv(ctx.h, _lib.GF_F64, C.c_void_p(x.data_ptr()), C.c_void_p(y.data_ptr())),
                   ctx.h)
        assert _lib.lib.gf_last_device_seconds(ctx.h) not in (0.0, total)
        assert split(ctx) == (g, s)
