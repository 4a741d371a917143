"""The Cahn-Hilliard assembly over several slabs and the sweeps of colours
larger than one wave of blocks (needs a B200).

404 x 382 x 3 cells with 12 grains: one cell layer's element rows take more
than half of the assembly's scratch, so every layer is a slab of its own, and
a colour holds 77,000 nodes, more than the sweeps that preload all of their
rows serve.  Against the oracle at the tolerances of
test_gpu_ch_gauss_seidel.py: 1e-12 (matrix and diagonal, FP64 apply), 1e-4
(FP32 apply).
"""
import numpy as np
import pytest

from helpers import block_rel_err, oracle_mesh, random_state
from oracle import oracle as O

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def test_slabs_and_large_colours_match_oracle():
    import hpsint_b200 as hb
    cells, G = (404, 382, 3), 12
    op = hb.SinteringOperatorGeneric(hb.Mesh(3, cells), hb.Params(G, tensorial=False))
    u = random_state(3, cells, G, seed=51)
    op.set_time_weights(1e3, [-1e3], 1.0)
    op.fill_quadrature_point_values(op.to_device(u))
    pc = hb.BlockPreconditioner2(op, block_0="ch_gauss_seidel")
    pc.do_update()
    om, p, T = oracle_mesh(3, cells), O.make_params(G, tensorial=False), O.make_time(1e3, 1.0, [-1e3])
    A = O.ch_matrix(om, p, T, u)
    ours = pc.ch_matrix()[:, :, :op.N].cpu().numpy()
    assert block_rel_err(ours.reshape(27 * 4, -1), A.reshape(27 * 4, -1)) <= 1e-12
    assert block_rel_err(pc.ch_blocks()[:, :op.N].cpu().numpy(), A[13]) <= 1e-12
    d = O.inverse_diagonal(O.ac_diagonal(om, p, T, u))
    assert block_rel_err(pc.inverse_diagonal()[:, :op.N].cpu().numpy(), d) <= 1e-12
    r = random_state(3, cells, G, seed=52, smooth=False) - 0.5
    ref = np.vstack([O.ch_sgs(om, A, r[:2].copy()), d * r[2:]])
    for dtype, tol in ((torch.float64, 1e-12), (torch.float32, 1e-4)):
        z = op.initialize_dof_vector(dtype)
        pc.vmult(z, op.to_device(r, dtype))
        assert block_rel_err(op.to_host(z), ref) <= tol
