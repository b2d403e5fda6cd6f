"""FP32 iterates of the one-kernel (P)CG, with copies of the direction and without, and solves that
repeat bit for bit in both types."""
import numpy as np
import pytest

from gpufem_b200 import _lib
from gpufem_b200 import meshgen as mg
from test_pcg_cluster_gpu import pcg, problem

pytestmark = pytest.mark.gpu

# copies: Q4 30^2, Q8, Brick8 9^3, Brick20; gathers (FP32): Q4 110^2, Brick8 13^3
SIZES = [(mg.Q4, (30, 30)), (mg.Q8, (9, 7)), (mg.BRICK8, (9, 9, 9)), (mg.BRICK20, (4, 3, 3)),
         (mg.Q4, (110, 110)), (mg.BRICK8, (13, 13, 13))]


@pytest.mark.parametrize("et,n", SIZES)
@pytest.mark.parametrize("solver", [_lib.GF_SOLVER_PCG, _lib.GF_SOLVER_CG])
def test_fp32_iterates_match_numpy(et, n, solver):
    """A row is at most 243 products, 1.5e-5 of its absolute sum with FP32 roundings in the worst
    case; four iterations: 1e-4."""
    ctx, K, b = problem(et, n)
    with ctx:
        d = 1.0 / K.diagonal() if solver == _lib.GF_SOLVER_PCG else np.ones_like(b)
        for its in (1, 4):
            before = ctx.launches()
            info = ctx.solve(solver, _lib.GF_F32, tol=1e-30, max_iter=its, raise_on_error=False)
            assert ctx.launches() - before < 3 * 16   # no chunk of 16 iterations of three kernels
            assert info.iterations == its and info.status == _lib.GF_ERR_NOT_CONVERGED
            x = pcg(K, b, d, its)
            assert np.linalg.norm(ctx.solution() - x) <= 1e-4 * np.linalg.norm(x)


# FP64 gathers: Q4 75^2, Brick8 10^3
@pytest.mark.parametrize("et,n", SIZES + [(mg.Q4, (75, 75)), (mg.BRICK8, (10, 10, 10))])
@pytest.mark.parametrize("dtype", [_lib.GF_F32, _lib.GF_F64])
def test_solves_repeat(et, n, dtype):
    if dtype == _lib.GF_F64 and n in ((110, 110), (13, 13, 13)):
        pytest.skip("more than the cluster holds in FP64: the graph's sums are atomic")
    ctx, _, _ = problem(et, n)
    with ctx:
        u = []
        for _ in range(3):
            ctx.solve(_lib.GF_SOLVER_PCG, dtype, tol=1e-30, max_iter=40, raise_on_error=False)
            u.append(ctx.solution())
        assert np.array_equal(u[0], u[1]) and np.array_equal(u[0], u[2])
