"""3D kernels of more than five grains against the oracle (needs a B200): the
residual with streamed pair sums and in-place point results (6 to 10 grains
tensorial, 6 to 12 scalar), the scalar-mobility products in place, the FP32
products that run without packed pairs (5 grains and more), with and without
the grain cut-off; partial tiles and every block size of the pair loop with
and without a remainder.

Tolerances per block: 1e-12 (FP64); FP32 against the oracle at the
FP32-rounded inputs, 2e-5 plus twice what rounding the inputs moves the
oracle's own product by (as in test_gpu_fused2d.py).
"""
import numpy as np
import pytest

from helpers import block_rel_err, oracle_mesh, particle_state, random_state
from oracle import oracle as O

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cut", [False, True])
@pytest.mark.parametrize("tens", [True, False])
@pytest.mark.parametrize("G", [5, 6, 7, 8, 9, 10, 11, 12])
def test_many_grains_match_oracle(G, tens, cut):
    import hpsint_b200 as hb
    cells = (9, 6, 5) if G % 2 else (5, 10, 3)
    op = hb.SinteringOperatorGeneric(hb.Mesh(3, cells), hb.Params(G, tensorial=tens))
    u = particle_state(3, cells, G, seed=1) if cut else random_state(3, cells, G, seed=1)
    old, old2 = (random_state(3, cells, G, seed=s) for s in (2, 3))
    src = random_state(3, cells, G, seed=4, smooth=False) - 0.5
    w = [11.0, -7.5, 3.5]
    om, opar, T = oracle_mesh(3, cells), O.make_params(G, tensorial=tens), O.make_time(w[0], 1.0, w[1:])
    op.set_time_weights(w[0], w[1:], 1.0)
    ud = op.to_device(u)
    kw = {}
    if cut:
        op.set_component_mask(ud, 1e-3)
        kw["mask"] = O.grain_mask(om, opar, u, 1e-3)
    r = op.initialize_dof_vector()
    for wtd in (0, 1, 2):
        hist = [op.to_device(old), op.to_device(old2)] if wtd == 2 else []
        op.evaluate_nonlinear_residual(r, ud, wtd, hist)
        ref = O.residual(om, opar, T, u, [old, old2] if wtd == 2 else [], wtd, **kw)
        assert block_rel_err(op.to_host(r), ref) < 1e-12
    op.fill_quadrature_point_values(ud)
    f32 = lambda x: x.astype(np.float32).astype(np.float64)
    exact, rounded = O.jvp(om, opar, T, u, src, **kw), O.jvp(om, opar, T, f32(u), f32(src), **kw)
    for dtype, ref, tol in ((torch.float64, exact, 1e-12),
                            (torch.float32, rounded, 2e-5 + 2 * block_rel_err(rounded, exact))):
        dst = op.initialize_dof_vector(dtype)
        op.vmult(dst, op.to_device(src, dtype))
        assert block_rel_err(op.to_host(dst), ref) < tol
