"""Operator calls whose output is one of their inputs (needs a B200): bit for
bit the result of the same call with an output of its own.  Meshes of several
blocks and tiles per direction, so that a node's neighbours belong to others.
"""
import ctypes

import pytest

from helpers import particle_state, random_state

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

CASES = [(2, (46, 37), 2, True, 0.0), (2, (46, 37), 8, False, 0.0), (2, (46, 37), 11, True, 0.0),
         (2, (46, 37), 4, True, 1e-3), (2, (8, 8), 12, False, 0.0), (2, (1, 1), 3, False, 0.0),
         (3, (13, 9, 7), 4, True, 0.0), (3, (13, 9, 7), 7, False, 0.0), (3, (13, 9, 7), 4, True, 1e-3)]


@pytest.mark.parametrize("dim,cells,G,tens,cut", CASES)
def test_output_may_be_an_input(dim, cells, G, tens, cut):
    import hpsint_b200 as hb
    from hpsint_b200 import _lib as L
    mesh, params = hb.Mesh(dim, cells), hb.Params(G, tensorial=tens)
    op = hb.SinteringOperatorGeneric(mesh, params)
    w = [1.5e3, -2e3, 5e2]
    op.set_time_weights(w[0], w[1:], 1.0)
    state = lambda seed: op.to_device((particle_state if cut else random_state)(dim, cells, G, seed=seed))
    lin, old, old2 = state(1), state(2), state(3)
    op.fill_quadrature_point_values(lin)
    if cut:
        op.set_component_mask(lin, cut)
    for dtype in (torch.float64, torch.float32):
        v = state(4).to(dtype)
        want = op.initialize_dof_vector(dtype)
        op.vmult(want, v)
        for _ in range(5):
            x = v.clone()
            op.vmult(x, x)
            assert torch.equal(x, want)
    want = op.initialize_dof_vector()
    op.evaluate_nonlinear_residual(want, lin, 2, [old, old2])
    for which in range(3):
        x = [t.clone() for t in (lin, old, old2)]
        op.evaluate_nonlinear_residual(x[which], x[0], 2, x[1:])
        assert torch.equal(x[which], want)
    if not cut:
        v, s = state(4), torch.cuda.current_stream().cuda_stream
        for which in range(3):  # an output of its own, the direction, the linearisation point
            a, b = lin.clone(), v.clone()
            dst = [op.initialize_dof_vector(), b, a][which]
            L.check(L.lib().sint_jvp_f64_noalloc(ctypes.byref(mesh.to_c()), ctypes.byref(params.to_c()), w[0], 1.0,
                                                 a.data_ptr(), b.data_ptr(), dst.data_ptr(), s), "noalloc")
            if which == 0:
                want = dst
            assert torch.equal(dst, want)
