"""The one-kernel PCG when a CTA's wait for another runs out: limits of a few hundred clocks make
some do, at any point of an iteration, the last one included."""
import ctypes as C

import numpy as np
import pytest

from gpufem_b200 import _lib
from gpufem_b200 import meshgen as mg
from test_pcg_cluster_gpu import pcg, problem

pytestmark = pytest.mark.gpu


def limit(ctx, clocks):
    f = _lib.lib.gftest_pcg_wait
    f.argtypes, f.restype = [C.c_void_p, C.c_longlong], None
    f(ctx.h, clocks)


@pytest.mark.parametrize("et,n", [(mg.Q4, (30, 30)), (mg.BRICK8, (7, 6, 6))])
def test_a_solve_without_error_has_the_iterates(et, n):
    """1e-10 as in test_iterates_match_numpy; in several launches too, which go on from what the
    last one left."""
    ctx, K, b = problem(et, n)
    with ctx:
        for its in (1, 2, 5):
            want = pcg(K, b, 1.0 / K.diagonal(), its)
            for clocks in (0, 150, 400, 800, 1500, 3000) * 4:
                limit(ctx, clocks)
                for kw in ({}, {"max_seconds": 100.0, "check_every": 1}):
                    with pytest.raises(_lib.GpufemError) as e:
                        ctx.solve(_lib.GF_SOLVER_PCG, _lib.GF_F64, tol=1e-30, max_iter=its, **kw)
                    assert e.value.status in (_lib.GF_ERR_NOT_CONVERGED, _lib.GF_ERR_CUDA)
                    if e.value.status == _lib.GF_ERR_NOT_CONVERGED:
                        assert np.linalg.norm(ctx.solution() - want) <= 1e-10 * np.linalg.norm(want)
