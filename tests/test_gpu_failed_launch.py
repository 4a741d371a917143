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


@pytest.mark.parametrize("call", ["jvp_2d", "jvp_3d", "dot", "precond_block_jacobi", "precond_ch_gauss_seidel"])
def test_a_failed_launch_fails_its_own_call_only(call):
    import hpsint_b200 as hb
    from hpsint_b200 import _lib as L
    dim, cells, G = (3, (6, 5, 4), 2) if call == "jvp_3d" else (2, (9, 7), 2)
    op = hb.SinteringOperatorGeneric(hb.Mesh(dim, cells), hb.Params(G))
    op.set_time_weights(1e3, [-1e3], 1.0)
    u = op.to_device(random_state(dim, cells, G, seed=3))
    op.fill_quadrature_point_values(u)
    z, h, lib = op.initialize_dof_vector(), op._h, L.lib()
    if call.startswith("precond"):
        pc = hb.BlockPreconditioner2(op, block_0=call[len("precond_"):])
        pc.do_update()
    with refusing_stream() as s:
        if call == "dot":
            rc = lib.sint_vec_dot_f64(h, u.numel(), u.data_ptr(), u.data_ptr(), z.data_ptr(), s)
        else:
            f = lib.sint_jvp_f64 if call.startswith("jvp") else lib.sint_precond_apply_f64
            rc = f(h, z.data_ptr(), u.data_ptr(), s)
        assert L.STATUS_NAMES[rc] == "SINT_ERR_CUDA"
    # the next call's launches succeed, and it must say so
    op.fill_quadrature_point_values(u)
    op.evaluate_nonlinear_residual(z, u, 1)
