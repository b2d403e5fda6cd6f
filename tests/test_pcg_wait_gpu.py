"""The one-kernel PCG when a CTA's wait for another runs out: the first or a later one of an
iteration, in CTA 0 or another, in the last iteration of a launch too.  The solve starts again as a
graph of kernels, from the beginning."""
import ctypes as C

import numpy as np
import pytest

from gpufem_b200 import _lib
from gpufem_b200 import meshgen as mg
from test_pcg_cluster_gpu import pcg, problem

pytestmark = pytest.mark.gpu


def lose(ctx, cta, wait):
    f = _lib.lib.gftest_pcg_late
    f.argtypes, f.restype = [C.c_void_p, C.c_int, C.c_int], None
    f(ctx.h, cta, wait)


# waits of an iteration: the directions, p.q, then r.z and r.r; the launch ends after four
# iterations (waits 0 to 11), or after each
@pytest.mark.parametrize("kw", [{}, {"max_seconds": 100.0, "check_every": 1}])
@pytest.mark.parametrize("cta", [0, 1, 15])
@pytest.mark.parametrize("wait", [0, 1, 2, 7, 9, 10, 11])
def test_iterates_after_a_lost_wait(cta, wait, kw):
    """1e-10 as in test_iterates_match_numpy."""
    ctx, K, b = problem(mg.Q4, (30, 30))
    with ctx:
        want = pcg(K, b, 1.0 / K.diagonal(), 4)
        runs = []
        for c in (-1, cta):
            lose(ctx, c, wait)
            before = ctx.launches()
            info = ctx.solve(_lib.GF_SOLVER_PCG, _lib.GF_F64, tol=1e-30, max_iter=4, raise_on_error=False, **kw)
            runs.append(ctx.launches() - before)
            assert info.iterations == 4 and info.status == _lib.GF_ERR_NOT_CONVERGED
            assert np.linalg.norm(ctx.solution() - want) <= 1e-10 * np.linalg.norm(want)
        # where a launch ends after each iteration, its waits are 0, 1 and 2
        lost = wait < 3 if kw else True
        assert (runs[1] > runs[0]) == lost, runs   # the graph ran


def test_a_solve_after_a_lost_wait():
    import scipy.sparse.linalg as spla
    ctx, K, b = problem(mg.Q8, (9, 7))
    with ctx:
        want = spla.spsolve(K.tocsc(), b)
        for cta in (3, -1):   # without the cluster, and with it again
            lose(ctx, cta, 50)
            for solver in (_lib.GF_SOLVER_PCG, _lib.GF_SOLVER_CG):
                info = ctx.solve(solver, _lib.GF_F64, tol=1e-12, max_iter=20000)
                assert info.status == _lib.GF_OK and info.rel_residual <= 1e-10
                assert np.linalg.norm(ctx.solution() - want) <= 1e-8 * np.linalg.norm(want)
