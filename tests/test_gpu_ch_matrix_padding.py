"""The exported Cahn-Hilliard matrix fills the caller's whole array: zeros in
the entries behind the last node of every block (needs a B200)."""
import pytest

from helpers import random_state

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,cells", [(2, (9, 6)), (3, (4, 5, 3)), (2, (7, 7)), (2, (1, 1))])
def test_padding_of_the_exported_matrix_is_zero(dim, cells):
    import hpsint_b200 as hb
    from hpsint_b200 import _lib as L
    op = hb.SinteringOperatorGeneric(hb.Mesh(dim, cells), hb.Params(2))
    op.set_time_weights(1e3, [-1e3], 1.0)
    op.fill_quadrature_point_values(op.to_device(random_state(dim, cells, 2, seed=1)))
    pc = hb.BlockPreconditioner2(op, block_0="ch_gauss_seidel")
    pc.do_update()
    A = torch.full((3**dim, 4, op.ld), float("nan"), dtype=torch.float64, device="cuda")
    L.check(L.lib().sint_ch_matrix_f64(op._h, A.data_ptr(), torch.cuda.current_stream().cuda_stream), "ch_matrix")
    assert bool(torch.isfinite(A[:, :, :op.N]).all())
    assert bool((A[:, :, op.N:] == 0.0).all())
