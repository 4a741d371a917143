"""The warp-per-tile kernels of the cut-off's class without grains against the
oracle at their edges (needs a B200).

Tiles are 4 x 4 x 2 cells: single cells, exact tiles, one cell beyond, partial
tiles in every direction, periodic meshes; no grain relevant anywhere (every
tile is of that class) or on a few cells (tiles of both kinds share nodes).
Tolerances as in test_gpu_cutoff.py: 1e-12 (FP64), and for FP32 2e-5 against
the oracle at the FP32-rounded inputs (scalar mobility: no ill-conditioned
pair terms).
"""
import numpy as np
import pytest

from helpers import block_rel_err, oracle_mesh, random_state
from oracle import oracle as O

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

CASES = [
    # cells, tensorial, grains on some cells, periodic
    ((1, 1, 1), True, False, ()),
    ((4, 4, 2), True, False, ()),
    ((5, 5, 3), False, False, ()),
    ((3, 9, 5), True, True, ()),
    ((13, 8, 7), True, True, ()),
    ((13, 8, 7), False, True, (0, 2)),
    ((33, 6, 2), True, True, (1,)),
]


@pytest.mark.parametrize("cells,tens,grains,periodic", CASES)
def test_light_tiles_match_oracle(cells, tens, grains, periodic):
    import hpsint_b200 as hb
    G, tol, h = 3, 1e-2, (0.9, 1.2, 0.7)
    op = hb.SinteringOperatorGeneric(hb.Mesh(3, cells, h), hb.Params(G, tensorial=tens))
    op.set_periodicity(periodic)
    u, old, old2 = (random_state(3, cells, G, seed=s) for s in (1, 2, 3))
    u[2:] *= 1e-3  # below the cut-off everywhere
    if grains:
        u[2:, : op.N // 3] *= 1e3
    for d in periodic:  # slaves carry their masters' values, as a solver's states do
        a = u.reshape((G + 2,) + tuple(n + 1 for n in reversed(cells)))
        ax = 3 - d
        a[(slice(None),) * ax + (-1,)] = a[(slice(None),) * ax + (0,)]
    src = random_state(3, cells, G, seed=4, smooth=False) - 0.5
    w = [11.0, -7.5, 3.5]
    om, opar, T = oracle_mesh(3, cells, h), O.make_params(G, tensorial=tens), O.make_time(w[0], 1.0, w[1:])
    op.set_time_weights(w[0], w[1:], 1.0)
    ud = op.to_device(u)
    op.set_component_mask(ud, tol)
    mask = O.grain_mask(om, opar, u, tol)
    kw = {"mask": mask}
    r = op.initialize_dof_vector()
    for wtd in (0, 1, 2):
        hist = [op.to_device(old), op.to_device(old2)] if wtd == 2 else []
        op.evaluate_nonlinear_residual(r, ud, wtd, hist)
        ho = [old, old2] if wtd == 2 else []
        ref = (O.periodic_residual(om, opar, T, u, ho, wtd, periodic, **kw) if periodic else
               O.residual(om, opar, T, u, ho, wtd, **kw))
        assert block_rel_err(op.to_host(r), ref) < 1e-12
    op.fill_quadrature_point_values(ud)
    jv = lambda a, b: (O.periodic_jvp(om, opar, T, a, b, periodic, **kw) if periodic else
                       O.jvp(om, opar, T, a, b, **kw))
    f32 = lambda x: x.astype(np.float32).astype(np.float64)
    dst = op.initialize_dof_vector()
    op.vmult(dst, op.to_device(src))
    assert block_rel_err(op.to_host(dst), jv(u, src)) < 1e-12
    if not tens:
        dst = op.initialize_dof_vector(torch.float32)
        op.vmult(dst, op.to_device(src, torch.float32))
        assert block_rel_err(op.to_host(dst), jv(f32(u), f32(src))) < 2e-5
