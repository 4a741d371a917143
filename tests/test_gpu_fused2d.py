"""The one-kernel 2D cell loop against the CPU oracle at its edges (needs a B200).

A block of 16 x 8 threads owns 15 x 7 nodes, so the sizes are one node below,
at and above multiples of those, single rows and columns of cells, and meshes
of several blocks per direction; grain counts on both sides of the rule that
keeps the tiled kernels (FP64 tensorial, more than 10 grains).  Tolerances per
block: 1e-12 (FP64); FP32 against the oracle at the FP32-rounded inputs, 2e-5
plus twice what rounding those inputs moves the oracle's own product by (the
pair terms' 1/|grad eta_i - grad eta_j|^2 amplifies a rounding error where two
gradients nearly agree; FP32 gradients carry errors of that size themselves).
"""
import numpy as np
import pytest

from helpers import block_rel_err, oracle_mesh, random_state
from oracle import oracle as O

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

CASES = [
    # cells, G, tensorial, periodic directions
    ((1, 1), 1, True, ()),
    ((13, 5), 2, True, ()),
    ((14, 6), 2, False, ()),
    ((15, 7), 3, True, ()),
    ((16, 8), 4, True, (0,)),
    ((29, 13), 8, False, ()),
    ((30, 14), 8, True, (0, 1)),
    ((1, 64), 5, True, ()),
    ((97, 1), 6, False, (0,)),
    ((46, 22), 10, True, ()),
    ((31, 15), 11, True, ()),
    ((31, 15), 12, False, ()),
]


@pytest.mark.parametrize("cells,G,tens,periodic", CASES)
def test_fused_2d_matches_oracle(cells, G, tens, periodic):
    import hpsint_b200 as hb
    h = (0.8, 1.1, 1.0)
    op = hb.SinteringOperatorGeneric(hb.Mesh(2, cells, h), hb.Params(G, tensorial=tens))
    op.set_periodicity(periodic)
    u, old, old2 = (random_state(2, cells, G, seed=s) for s in (1, 2, 3))
    src = random_state(2, cells, G, seed=4, smooth=False) - 0.5
    w = [11.0, -7.5, 3.5]
    om, opar, T = oracle_mesh(2, cells, h), O.make_params(G, tensorial=tens), O.make_time(w[0], 1.0, w[1:])
    op.set_time_weights(w[0], w[1:], 1.0)
    ud = op.to_device(u)
    r = op.initialize_dof_vector()
    for wtd in (0, 1, 2):
        hist = [op.to_device(old), op.to_device(old2)] if wtd == 2 else []
        op.evaluate_nonlinear_residual(r, ud, wtd, hist)
        ho = [old, old2] if wtd == 2 else []
        ref = (O.periodic_residual(om, opar, T, u, ho, wtd, periodic) if periodic else
               O.residual(om, opar, T, u, ho, wtd))
        assert block_rel_err(op.to_host(r), ref) < 1e-12
    op.fill_quadrature_point_values(ud)
    jv = lambda a, b: (O.periodic_jvp(om, opar, T, a, b, periodic) if periodic else O.jvp(om, opar, T, a, b))
    f32 = lambda x: x.astype(np.float32).astype(np.float64)
    exact, rounded = jv(u, src), jv(f32(u), f32(src))
    for dtype, ref, tol in ((torch.float64, exact, 1e-12),
                            (torch.float32, rounded, 2e-5 + 2 * block_rel_err(rounded, exact))):
        dst = op.initialize_dof_vector(dtype)
        op.vmult(dst, op.to_device(src, dtype))
        assert block_rel_err(op.to_host(dst), ref) < tol
        assert float(dst[:, op.N:].abs().sum()) == 0.0  # padding untouched
