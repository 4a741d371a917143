"""The Krylov kernels at the edges of their block counts and instances (needs
a B200).

Dot products and norms of lengths below, at and above one block, one pack per
thread and the fixed grid, against numpy in FP64: relative to sum |x_i y_i|,
1e-14 for FP64 (sqrt-like growth of 2^-53 over 3e5 terms stays below it) and
for FP32 vectors too (products and sums are FP64).  Newton with restart
lengths that run every instance of the fused multi-vector kernels (4, 8, 16
vectors, several passes): all reach residual 1e-11 |R_0|, so the solutions
agree to 1e-8 of the largest entry (a step's increment is O(1) and the
Newton system's condition is far below 1e3 after preconditioning).
"""
import ctypes

import numpy as np
import pytest

from helpers import particle_state

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def make(cells=(45, 38), G=3):
    import hpsint_b200 as hb
    op = hb.SinteringOperatorGeneric(hb.Mesh(2, cells), hb.Params(G, tensorial=False))
    op.set_time_weights(1e3, [-1e3], 1.0)
    return op


@pytest.mark.parametrize("n", [1, 3, 255, 512, 513, 131072, 592 * 512, 592 * 512 + 2, 592 * 1024 + 7])
def test_dot_and_norm_lengths(n):
    from hpsint_b200 import _lib as L
    op = make()
    rng = np.random.default_rng(n)
    x, y = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    out = torch.zeros(1, dtype=torch.float64, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    for dt, dot, norm in ((torch.float64, L.lib().sint_vec_dot_f64, L.lib().sint_vec_norm2_f64),
                          (torch.float32, L.lib().sint_vec_dot_f32, L.lib().sint_vec_norm2_f32)):
        a, b = torch.as_tensor(x, dtype=dt).cuda(), torch.as_tensor(y, dtype=dt).cuda()
        ah, bh = a.double().cpu().numpy(), b.double().cpu().numpy()
        L.check(dot(op._h, n, p(a), p(b), p(out), s), "dot")
        assert abs(float(out.item()) - float(np.dot(ah, bh))) <= 1e-14 * float(np.dot(abs(ah), abs(bh)))
        L.check(norm(op._h, n, p(a), p(out), s), "norm")
        assert abs(float(out.item()) - float(np.linalg.norm(ah))) <= 1e-14 * float(np.linalg.norm(ah))


def test_restart_lengths_give_one_solution():
    import hpsint_b200 as hb
    cells, G = (45, 38), 3
    u0 = particle_state(2, cells, G, seed=5)
    sols = []
    for restart, right in ((40, False), (3, False), (6, False), (12, False), (20, True)):
        op = make(cells, G)
        old = op.to_device(u0)
        u = old.clone()
        st = hb.DampedNewtonSolver(op, hb.NonLinearData(nl_rel_tol=1e-11, nl_max_iter=30, l_rel_tol=1e-3,
                                                        gmres_restart=restart,
                                                        right_preconditioning=right)).solve(u, [old])
        assert st.final_residual <= 1e-11 * st.initial_residual
        sols.append(op.to_host(u))
    assert max(float(np.abs(s - sols[0]).max()) for s in sols[1:]) <= 1e-8 * float(np.abs(sols[0]).max())
