"""The Cahn-Hilliard assembly where the device has no room for its scratch
(needs a B200): it works in the slabs that the tile-face partials hold, or of
one cell layer.  The rest of the device memory is held by one allocation
meanwhile.

Meshes whose slabs are then several layers, with the ring of node layers
wrapping at 3, 4, 5, 6, 12 and 13, a last slab that is full or not, odd and even
node counts in x, and (15 layers, one grain) partials too small for two layers.
The order of the sums does not depend on the slabs: bit for bit the matrix,
diagonal and applies of a context with all of its scratch, and 1e-12 per block
against the oracle as in test_gpu_ch_gauss_seidel.py.
"""
import numpy as np
import pytest

from helpers import block_rel_err, oracle_mesh, random_state
from oracle import oracle as O

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,cells,G,tens", [(3, (24, 20, 44), 4, True), (3, (24, 21, 52), 4, False),
                                              (3, (27, 26, 41), 12, True), (3, (26, 23, 47), 12, False),
                                              (3, (40, 29, 15), 1, True), (2, (1000, 60), 8, True),
                                              (2, (1001, 83), 3, False)])
def test_set_up_without_room_for_its_scratch(dim, cells, G, tens):
    import hpsint_b200 as hb
    N, nk = int(np.prod([c + 1 for c in cells])), 3**dim
    u = random_state(dim, cells, G, seed=61)
    r = random_state(dim, cells, G, seed=62, smooth=False) - 0.5

    def results(room):
        op = hb.SinteringOperatorGeneric(hb.Mesh(dim, cells), hb.Params(G, tensorial=tens))
        op.set_time_weights(1e3, [-1e3], 1.0)
        op.fill_quadrature_point_values(op.to_device(u))
        pc = hb.BlockPreconditioner2(op, block_0="ch_gauss_seidel")
        held = None
        if room is not None:
            torch.cuda.synchronize()
            torch.cuda.empty_cache()
            held = torch.empty(torch.cuda.mem_get_info()[0] - room, dtype=torch.uint8, device="cuda")
        pc.do_update()
        torch.cuda.synchronize()
        del held
        torch.cuda.empty_cache()
        out = [pc.ch_matrix(), pc.inverse_diagonal()]
        for dtype in (torch.float64, torch.float32):
            z, v = op.initialize_dof_vector(dtype), op.to_device(r, dtype)
            pc.vmult(z, v)
            out.append(z)
            w = op.initialize_dof_vector(dtype)
            op.vmult(w, v)
            out.append(w)
        return op, out

    op, want = results(None)
    # the matrix (FP64 rows of 3^dim + 1 blocks, FP32 of 3^dim) and 14 MiB, less than any scratch here (30 MiB and more)
    _, got = results(N * ((nk + 1) * 32 + nk * 16) + (14 << 20))
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    A = O.ch_matrix(oracle_mesh(dim, cells), O.make_params(G, tensorial=tens), O.make_time(1e3, 1.0, [-1e3]), u)
    ours = got[0][:, :, :op.N].cpu().numpy()
    assert block_rel_err(ours.reshape(nk * 4, -1), A.reshape(nk * 4, -1)) <= 1e-12
