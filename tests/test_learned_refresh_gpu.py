"""The learned preconditioner's set-up (diagonal, log means) is kept for one version of the
matrix: every change of its values has to reach the next application."""
import numpy as np
import pytest

from gpufem_b200 import _lib
from gpufem_b200 import meshgen as mg

pytestmark = pytest.mark.gpu


def context(E, dtypes):
    from gpufem_b200.fem import Context
    m = mg.clamp_and_load(mg.structured(mg.BRICK8, (5, 4, 3), jitter=0.1, seed=5))
    ctx = Context(0)
    ctx.mesh_create(m.elem_type, m.coords, m.conn, m.ngauss, m.E0, E * np.linspace(1.0, 2.0, m.nelem), m.nu)
    ctx.set_supports(m.supports)
    for d in dtypes:
        ctx.assemble(d, _lib.GF_SCATTER_AUTO)
    ctx.lp_init(3, seed=1)
    w = np.random.default_rng(2).normal(scale=0.2, size=ctx.lp_num_params(3)).astype(np.float32)
    ctx.lp_set_weights(w)
    return m, ctx


@pytest.mark.parametrize("dtypes", [(_lib.GF_F64,), (_lib.GF_F32,), (_lib.GF_F32, _lib.GF_F64)])
def test_matrix_changes_reach_the_next_application(dtypes):
    """Reassembly with other moduli, then constraints: as a context that never applied before
    (sums of FP32 activations in another order: 1e-5)."""
    m, ctx = context(1.0, dtypes)
    r = np.random.default_rng(0).normal(size=m.ndof).astype(np.float32)
    ctx.lp_apply(r)
    E = np.geomspace(5.0, 0.5, m.nelem)
    ctx.set_modulus(m.E0, E)
    for d in dtypes:
        ctx.assemble(d, _lib.GF_SCATTER_AUTO)
    again = [ctx.lp_apply(r)]
    ctx.apply_constraints(_lib.GF_BC_ELIMINATION)
    again.append(ctx.lp_apply(r))
    _, fresh = context(1.0, ())
    fresh.set_modulus(m.E0, E)
    for d in dtypes:
        fresh.assemble(d, _lib.GF_SCATTER_AUTO)
    want = [fresh.lp_apply(r)]
    _, fresh = context(1.0, ())
    fresh.set_modulus(m.E0, E)
    for d in dtypes:
        fresh.assemble(d, _lib.GF_SCATTER_AUTO)
    fresh.apply_constraints(_lib.GF_BC_ELIMINATION)
    want.append(fresh.lp_apply(r))
    for a, b in zip(again, want):
        assert np.linalg.norm(a - b) <= 1e-5 * np.linalg.norm(b)
    assert np.linalg.norm(want[0] - want[1]) > 1e-3 * np.linalg.norm(want[0])


def test_set_weights_reach_the_next_application():
    """New weights, and the first ones again, many times over."""
    m, ctx = context(1.0, (_lib.GF_F64,))
    r = np.random.default_rng(0).normal(size=m.ndof).astype(np.float32)
    P = ctx.lp_num_params(3)
    ws = [np.random.default_rng(k).normal(scale=0.2, size=P).astype(np.float32) for k in (5, 6)]
    want = []
    for w in ws:
        for _ in range(3):
            ctx.lp_set_weights(w)
        want.append(ctx.lp_apply(r))
    assert np.linalg.norm(want[0] - want[1]) > 1e-3 * np.linalg.norm(want[0])
    for k in range(100):
        ctx.lp_set_weights(ws[k % 2])
        z = ctx.lp_apply(r)
        assert np.linalg.norm(z - want[k % 2]) <= 1e-5 * np.linalg.norm(want[k % 2]), k
