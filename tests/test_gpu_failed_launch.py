"""What a call whose kernel launch fails leaves behind (needs a B200).

The launch is made to fail on the host: a stream whose capture was broken by a
call that captures do not allow takes no work, and every launch into it returns
cudaErrorStreamCaptureInvalidated.  Nothing runs on the GPU.
"""
import contextlib
import ctypes

import pytest

from helpers import random_state

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def refusing_stream():
    """A stream that refuses every launch."""
    from cuda.bindings import runtime as rt
    err, stream = rt.cudaStreamCreateWithFlags(rt.cudaStreamNonBlocking)
    assert err == rt.cudaError_t.cudaSuccess
    assert rt.cudaStreamBeginCapture(stream, rt.cudaStreamCaptureMode.cudaStreamCaptureModeThreadLocal)[0] == err
    assert rt.cudaStreamSynchronize(stream)[0] != err  # not allowed under capture: breaks it
    try:
        yield ctypes.c_void_p(int(stream))
    finally:
        rt.cudaStreamEndCapture(stream)
        rt.cudaGetLastError()
        assert rt.cudaStreamDestroy(stream)[0] == err


@pytest.mark.parametrize("block_0", ["block_jacobi", "ch_gauss_seidel"])
def test_a_failed_set_up_leaves_no_preconditioner(block_0):
    import hpsint_b200 as hb
    from hpsint_b200 import _lib as L
    cells, G = (9, 7), 2
    op = hb.SinteringOperatorGeneric(hb.Mesh(2, cells), hb.Params(G))
    op.set_time_weights(1e3, [-1e3], 1.0)
    op.fill_quadrature_point_values(op.to_device(random_state(2, cells, G, seed=1)))
    pc = hb.BlockPreconditioner2(op, block_0=block_0)
    pc.do_update()
    r = op.to_device(random_state(2, cells, G, seed=2))
    want, z = op.initialize_dof_vector(), op.initialize_dof_vector()
    pc.vmult(want, r)
    with refusing_stream() as s:
        assert L.STATUS_NAMES[L.lib().sint_precond_setup(op._h, s)] == "SINT_ERR_CUDA"
    # neither the earlier set-up's data nor another block's stands in for it
    with pytest.raises(L.SintError) as e:
        pc.vmult(z, r)
    assert e.value.status_name == "SINT_ERR_NOT_READY"
    pc.do_update()
    pc.vmult(z, r)
    assert torch.equal(z, want)
