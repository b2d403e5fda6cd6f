"""The one-kernel PCG without copies of the direction, by the order of the nodes: the cluster while
its gathers are in pieces of some length, the graph of kernels on random numberings."""
import numpy as np
import pytest
import scipy.sparse as sp

from gpufem_b200 import _lib
from gpufem_b200 import meshgen as mg
from test_pcg_cluster_gpu import pcg

pytestmark = pytest.mark.gpu


def problem(et, n, run):
    """Nodes shuffled in runs of `run` (0: in order)."""
    from gpufem_b200.fem import Context
    m = mg.clamp_and_load(mg.structured(et, n, jitter=0.05, seed=2, ngauss=2))
    old = np.arange(m.nnodes)
    if run:
        k = -(-m.nnodes // run)
        old = (np.random.default_rng(1).permutation(k)[:, None] * run + np.arange(run)).ravel()
        old = old[old < m.nnodes]
    new = np.empty(m.nnodes, np.int64)
    new[old] = np.arange(m.nnodes)
    sup = m.supports.copy()
    sup[:, 0] = new[m.supports[:, 0].astype(int) - 1] + 1
    ctx = Context(0)
    ctx.mesh_create(m.elem_type, m.coords[old], (new[m.conn - 1] + 1).astype(np.int32), m.ngauss, m.E0, None, m.nu)
    ctx.set_supports(sup)
    ctx.set_force(m.f.reshape(-1, m.dim)[old].ravel())
    ctx.assemble(_lib.GF_F64, _lib.GF_SCATTER_AUTO)
    ctx.apply_constraints(_lib.GF_BC_ELIMINATION)
    ctx.convert_f64_to_f32()
    return ctx


# FP64 gathers from Q4 75^2 and Brick8 10^3 on, FP32 from Q4 110^2 and Brick8 13^3
@pytest.mark.parametrize("et,n,dtype,run,cluster", [
    (mg.Q4, (80, 80), _lib.GF_F64, 4, True), (mg.Q4, (90, 90), _lib.GF_F64, 1, False),
    (mg.BRICK8, (10, 10, 10), _lib.GF_F64, 32, True), (mg.BRICK8, (10, 10, 10), _lib.GF_F64, 1, False),
    (mg.Q4, (124, 124), _lib.GF_F32, 16, True), (mg.Q4, (124, 124), _lib.GF_F32, 2, False),
    (mg.BRICK8, (13, 13, 13), _lib.GF_F32, 0, True), (mg.BRICK8, (13, 13, 13), _lib.GF_F32, 4, False)])
def test_iterates_by_order(et, n, dtype, run, cluster):
    """FP64 1e-10, FP32 1e-4 as in the other tests of the iterates."""
    with problem(et, n, run) as ctx:
        rn, ci, v = ctx.ell_download(_lib.GF_F64)
        mask = np.arange(ci.shape[0])[:, None] < rn[None, :]
        rows = np.broadcast_to(np.arange(rn.size)[None, :], ci.shape)
        K = sp.csr_matrix((v[mask], (rows[mask], ci[mask])), shape=(rn.size, rn.size))
        b = ctx.get_force()
        ctx.solve(_lib.GF_SOLVER_PCG, dtype, tol=1e-30, max_iter=1, raise_on_error=False)   # the slices
        before = ctx.launches()
        ctx.solve(_lib.GF_SOLVER_PCG, dtype, tol=1e-30, max_iter=4, raise_on_error=False)
        assert (ctx.launches() - before < 3 * 16) == cluster   # else a chunk of 16 iterations
        want = pcg(K, b, 1.0 / K.diagonal(), 4)
        assert np.linalg.norm(ctx.solution() - want) <= (1e-10 if dtype == _lib.GF_F64 else 1e-4) * np.linalg.norm(want)


def test_iteration_time_on_a_random_numbering():
    """11 us against 10 in order; 39 with gathers node by node."""
    t = []
    for run in (0, 1):
        with problem(mg.BRICK8, (13, 13, 13), run) as ctx:
            t.append(min(i.seconds / i.iterations for i in
                         (ctx.solve(_lib.GF_SOLVER_PCG, _lib.GF_F32, tol=1e-30, max_iter=320,
                                    raise_on_error=False) for _ in range(4))))
    assert t[1] <= 2.0 * t[0], t
