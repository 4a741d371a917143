"""Measured work of the sintering operator: what a solver that uses this
framework asks of it, through the public Python interface.

Kinds of case
  jvp       one Jacobian-vector product J(u) v (SinteringOperatorGeneric.vmult),
            the call a Krylov solver makes most; FP64 or FP32, with or without
            the grain cut-off
  residual  one nonlinear residual evaluation with BDF history
  precond   the block preconditioner: set-up and one apply, or an apply alone
  steps     whole time steps (TimeIntegrator: Newton-GMRES, damping, cut-off)
  guess     one whole-mesh inference of the 3D learned initial guess

The states are seeded packings of overlapping spheres (circles in 2D) with
tanh profiles, coloured to the given number of order parameters, as the
repository's workloads are; lengths are in mesh units.  `exact` restates the
operator in plain FP64 torch, point by point.
"""
import math
import os

import numpy as np
import torch

import hpsint_b200 as hb
from hpsint_b200.time_integration import TimeIntegrationData, TimeIntegrator

A, B, KAPPA_C, KAPPA_P = 16.0, 1.0, 1.0, 0.5
MVOL, MVAP, MSURF, MGB, L = 1e-2, 1e-10, 4.0, 0.4, 1.0
WEIGHTS = os.path.join(os.path.dirname(os.path.abspath(hb.__file__)), "weights", "learned_guess_c5_3d_w8.npz")


def _case(name, kind, cells, grains, **more):
    nx, ny, nz = cells if len(cells) == 3 else (*cells, 0)
    c = {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "h": 1.0, "grains": grains, "tensorial": True, "radius": 10.0}
    c |= more
    return c | {"name": name} if name else c


def listed():
    return [
        # a mesh of a few hundred cells, as unit tests and coarse start-ups use: launches and latency only
        _case("residual_2d_small", "residual", (41, 23), 2, order=1, radius=6.0),
        # the two-particle solve's product: a small 2D problem, one product per Krylov iteration
        _case("jvp64_2d_two", "jvp", (256, 128), 2, precision=64, h=0.3125),
        # the FP32 inner product of the many-grain 2D solve
        _case("jvp32_2d_packing", "jvp", (512, 512), 8, precision=32, tensorial=False, radius=9.0),
        # the 3D operator workload: noisy state, FP64 and tensorial mobility
        _case("jvp64_3d_operator", "jvp", (128, 128, 128), 4, precision=64, radius=15.0, noise=1e-3),
        # the FP32 inner product of the mixed-precision 3D solve
        _case("jvp32_3d_packing", "jvp", (192, 192, 192), 9, precision=32),
        # the same product with the grain cut-off at the largest mesh
        _case("cutoff_jvp32_3d", "jvp", (256, 256, 256), 10, precision=32, cut_off=1e-7, radius=8.0),
        # the FP64 residual of the outer Newton loop, BDF2 history, ragged sizes
        _case("residual_3d_packing", "residual", (189, 175, 162), 9, order=2),
        # a preconditioner rebuild at a new linearisation point and its first FP64 apply
        _case("precond_setup_3d", "precond", (131, 118, 97), 6, precision=64, block_0="ch_gauss_seidel", setup=True),
        # the preconditioner apply of every FP32 Krylov iteration
        _case("precond_apply32_3d", "precond", (192, 192, 192), 9, precision=32, block_0="ch_gauss_seidel",
              setup=False),
        # time steps of the two-particle solve, plain FP64 Newton-GMRES
        _case("steps_2d_two", "steps", (256, 128), 2, precision=64, block_0="block_jacobi", h=0.3125, dt=1e-3,
              steps=2),
        # time steps of a 3D packing with FP32 Krylov vectors, cut-off and the matrix-based preconditioner
        _case("steps_3d_mixed", "steps", (96, 96, 96), 6, precision=32, cut_off=1e-7, block_0="ch_gauss_seidel",
              dt=1e-4, steps=2, radius=8.0),
        # the learned initial guess of one time step over a whole mesh
        _case("guess_3d", "guess", (96, 96, 96), 6, radius=8.0),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def cells2(lo, hi):
        s = log_int(lo, hi)
        return s, max(8, int(s * rng.uniform(0.5, 1.0)))

    def cells3(lo, hi):
        s = log_int(lo, hi)
        return s, max(6, int(s * rng.uniform(0.7, 1.0))), max(6, int(s * rng.uniform(0.6, 1.0)))

    radius = rng.uniform(6.0, 14.0)
    kind = rng.choice(["jvp", "jvp", "jvp", "jvp", "residual", "residual", "precond", "precond", "steps", "guess"])
    three = rng.random() < 0.6
    tens = rng.random() < 0.7
    if kind == "jvp":
        prec = rng.choice([32, 64])
        cut = 10.0 ** rng.uniform(-8, -4) if rng.random() < 0.35 else 0.0
        cells = cells3(16, 224 if cut else 176) if three else cells2(24, 512)
        grains = rng.randint(2, 10) if three else rng.randint(2, 8)
        return _case(None, kind, cells, grains, precision=prec, tensorial=tens, cut_off=cut, radius=radius,
                     noise=0.0 if cut else rng.choice([0.0, 1e-3]))
    if kind == "residual":
        cells = cells3(16, 176) if three else cells2(24, 512)
        return _case(None, kind, cells, rng.randint(2, 9), order=rng.randint(1, 2), tensorial=tens, radius=radius)
    if kind == "precond":
        cells = cells3(16, 176) if three else cells2(24, 512)
        return _case(None, kind, cells, rng.randint(2, 9), precision=rng.choice([32, 64]), tensorial=tens,
                     block_0=rng.choice(["ch_gauss_seidel", "ch_gauss_seidel", "block_jacobi"]),
                     setup=rng.random() < 0.4, radius=radius)
    if kind == "steps":
        cells = cells3(32, 80) if three else cells2(64, 256)
        mixed = rng.random() < 0.5
        return _case(None, kind, cells, rng.randint(2, 6), precision=32 if mixed else 64,
                     cut_off=1e-7 if mixed else 0.0, block_0="ch_gauss_seidel" if mixed else "block_jacobi",
                     dt=1e-4 if three else 1e-3, steps=2, radius=rng.uniform(6.0, 10.0),
                     h=1.0 if three else rng.uniform(0.3, 1.0))
    return _case(None, "guess", cells3(24, 96), rng.randint(2, 6), radius=radius)


# --- inputs -------------------------------------------------------------------

def _cells_of(case):
    return [case["nx"], case["ny"]] + ([case["nz"]] if case["nz"] else [])


def _particles(case, rng):
    """Random sequential packing: every particle touches an earlier one with a
    small overlap; each takes the order parameter whose particles are farthest."""
    cells, h = _cells_of(case), case["h"]
    dim, ext = len(cells), np.array(cells) * case["h"]
    r0 = min(case["radius"], 0.2 * float(ext.min()))
    vol = math.pi * r0 ** 2 if dim == 2 else 4.0 / 3.0 * math.pi * r0 ** 3
    want = int(min(200, max(case["grains"], round(0.05 * float(ext.prod()) / vol))))
    overlap = min(2.0 * h, 0.3 * r0)
    centers, radii = [ext / 2 + rng.uniform(-0.1, 0.1, dim) * ext], [r0 * math.exp(rng.normal(0.0, 0.15))]
    for _ in range(60 * want):
        if len(centers) == want:
            break
        r = r0 * math.exp(rng.normal(0.0, 0.15))
        j = rng.integers(len(centers))
        v = rng.standard_normal(dim)
        c = centers[j] + v / np.linalg.norm(v) * (radii[j] + r - overlap)
        if np.any(c - 0.7 * r < 0) or np.any(c + 0.7 * r > ext):
            continue
        if np.all(np.linalg.norm(np.array(centers) - c, axis=1) >= np.array(radii) + r - overlap - 1e-9):
            centers.append(c)
            radii.append(r)
    colours = []
    for i, c in enumerate(centers):
        gap = [math.inf] * case["grains"]
        for j in range(i):
            gap[colours[j]] = min(gap[colours[j]], float(np.linalg.norm(c - centers[j])) - radii[i] - radii[j])
        colours.append(int(np.argmax(gap)))
    return centers, radii, colours


def _state(case, seed):
    """(C, nodes) FP64 state of a packing with tanh profiles (width 2) and a
    smooth chemical potential, on the GPU; and a generator for what follows."""
    rng = np.random.default_rng([seed, 17])
    gen = torch.Generator("cuda").manual_seed(seed)
    cells, h, G = _cells_of(case), case["h"], case["grains"]
    dim, width = len(cells), 2.0
    shape = [n + 1 for n in reversed(cells)]
    u = torch.zeros([G + 2] + shape, dtype=torch.float64, device="cuda")
    xs = [torch.arange(n + 1, dtype=torch.float64, device="cuda") * h for n in cells]
    for c, r, col in zip(*_particles(case, rng)):
        lo = [max(0, int((c[d] - r - 10 * width) / h)) for d in range(dim)]
        hi = [min(cells[d] + 1, int((c[d] + r + 10 * width) / h) + 2) for d in range(dim)]
        d2 = torch.zeros([], dtype=torch.float64, device="cuda")
        for d in range(dim):
            x2 = (xs[d][lo[d]:hi[d]] - c[d]) ** 2
            d2 = d2 + x2.view([-1] + [1] * d)
        box = (2 + col,) + tuple(slice(lo[d], hi[d]) for d in reversed(range(dim)))
        u[box] = torch.maximum(u[box], 0.5 * (1.0 - torch.tanh(2.0 * (d2.sqrt() - r) / width)))
    u[0] = u[2:].amax(0).clamp(0.0, 1.0)
    if case["kind"] != "steps":
        k = torch.as_tensor(rng.uniform(0.02, 0.1, dim), device="cuda")
        wave = sum(torch.sin(k[d] * xs[d] / h + 0.7 * d).view([-1] + [1] * d) for d in range(dim))
        u[1] = 0.1 * wave + 0.2 * u[0] * (1 - u[0])
    u = u.view(G + 2, -1)
    if case.get("noise"):
        u += case["noise"] * (2.0 * torch.rand(u.shape, generator=gen, dtype=torch.float64, device="cuda") - 1.0)
    return u, gen


def _uniform(like, gen, dtype=torch.float64):
    return 2.0 * torch.rand(like.shape, generator=gen, dtype=dtype, device="cuda") - 1.0


def _history(case, u, gen):
    """Earlier states: u with small relative changes."""
    return [u * (1.0 - 1e-3 * (i + 1) * torch.rand(u.shape, generator=gen, dtype=torch.float64, device="cuda"))
            for i in range(case.get("order", 1))]


def _weights(case):
    dt = 1e-3
    return hb.bdf_weights(case.get("order", 1), [dt, 0.8 * dt][:case.get("order", 1)])


def _vec(op, x):
    v = op.initialize_dof_vector(x.dtype)
    v[:, :op.N] = x
    return v


def prepare(case, seed):
    u, gen = _state(case, seed)
    cells = _cells_of(case)
    op = hb.SinteringOperatorGeneric(
        hb.Mesh(len(cells), tuple(cells), (case["h"],) * 3),
        hb.Params(case["grains"], A, B, KAPPA_C, KAPPA_P, MVOL, MVAP, MSURF, MGB, L, case["tensorial"]))
    s = {"kind": case["kind"], "op": op}
    kind = case["kind"]
    if kind in ("jvp", "residual", "precond"):
        w = _weights(case)
        op.set_time_weights(w[0], w[1:], 1.0)
    if kind == "jvp":
        ud = _vec(op, u)
        op.fill_quadrature_point_values(ud)
        if case.get("cut_off"):
            op.set_component_mask(ud, case["cut_off"])
        dtype = torch.float32 if case["precision"] == 32 else torch.float64
        s["src"] = _vec(op, _uniform(u, gen, dtype))
        s["dst"] = op.initialize_dof_vector(dtype)
    elif kind == "residual":
        s["src"], s["dst"] = _vec(op, u), op.initialize_dof_vector()
        s["hist"] = [_vec(op, x) for x in _history(case, u, gen)]
    elif kind == "precond":
        dtype = torch.float32 if case["precision"] == 32 else torch.float64
        op.fill_quadrature_point_values(_vec(op, u))
        s["pc"] = hb.BlockPreconditioner2(op, case["block_0"])
        s["setup"] = case["setup"]
        if not case["setup"]:
            s["pc"].do_update()
        s["src"], s["dst"] = _vec(op, _uniform(u, gen, dtype)), op.initialize_dof_vector(dtype)
    elif kind == "steps":
        op.set_preconditioner_type(case["block_0"])
        nl = hb.NonLinearData(nl_rel_tol=1e-8, inner_precision=case["precision"],
                              right_preconditioning=case["block_0"] == "ch_gauss_seidel")
        s["integrator"] = TimeIntegrator(op, nl, TimeIntegrationData(time_step_init=case["dt"]),
                                         grain_cut_off_tolerance=case["cut_off"] if case.get("cut_off") else 0.0)
        s["u0"], s["dts"] = _vec(op, u), [case["dt"]] * case["steps"]
    else:
        from hpsint_b200 import learned_guess as LG
        from hpsint_b200 import learned_guess3d as LG3
        net, norm = LG.load_predictor(WEIGHTS)
        s["predictor"] = LG3.LearnedPredictor3D(op, net, norm)
        s["hist"] = [_vec(op, u), _vec(op, _history(case, u, gen)[0])]
    return s


def run(s):
    kind = s["kind"]
    if kind == "jvp":
        s["op"].vmult(s["dst"], s["src"])
        return s["dst"]
    if kind == "residual":
        s["op"].evaluate_nonlinear_residual(s["dst"], s["src"], 2, s["hist"])
        return s["dst"]
    if kind == "precond":
        if s["setup"]:
            s["pc"].do_update()
        s["pc"].vmult(s["dst"], s["src"])
        return s["dst"]
    if kind == "steps":
        s["integrator"].initialize(s["u0"])
        return s["integrator"].run(len(s["dts"]), dt_schedule=s["dts"])
    return s["predictor"](s["hist"], [1e-3], 1.2e-3)


# --- work of one pass -----------------------------------------------------------

def _cell_flops(dim, G, tens, jvp):
    """Operations per cell of the operator: sum-factorised evaluation and
    integration (n points and nodes per cell) and the point formulas."""
    n = 2 ** dim
    val, grad = dim * n * 5 // 2, dim * n * 5 // 2 + (42 if dim == 3 else 13)
    n_grad = (4 + G if jvp else 2 + G) if tens else (2 if jvp else 1)
    n_val = (G if jvp else 1 + G) if tens else (2 + 2 * G if jvp else 2 + 2 * G)
    pair = (8 * dim + 12 if jvp else 6 * dim + 7) if tens else 2
    point = (60 + 16 * dim if tens else 50) + 24 * G + pair * G * (G - 1) // 2
    rows = (G + 2) * (val + n) + (grad - val) + (G + 1) * 2 * n * n
    return n_grad * grad + n_val * val + n * point + rows


def work(case):
    cells = _cells_of(case)
    dim, G = len(cells), case["grains"]
    C = G + 2
    N, n_cells = math.prod(n + 1 for n in cells), math.prod(cells)
    kind, tens = case["kind"], case["tensorial"]
    b = 4 if case.get("precision") == 32 else 8
    if kind == "jvp":
        # with the cut-off most cells keep c and mu only
        g = 0 if case.get("cut_off") else G
        return {"bytes": b * N * C * 3 if not case.get("cut_off") else b * N * (6 + G),
                "flops": n_cells * _cell_flops(dim, g, tens, True)}
    if kind == "residual":
        return {"bytes": 8 * N * C * (2 + case["order"]), "flops": n_cells * _cell_flops(dim, G, tens, False)}
    if kind == "precond":
        nk = 3 ** dim
        gs = case["block_0"] == "ch_gauss_seidel"
        mat = nk * 4 if gs else 4
        apply_b, apply_f = b * N * (2 * C + G + mat), N * (2 * mat + 8 + G)
        if not case["setup"]:
            return {"bytes": apply_b, "flops": apply_f}
        n = 2 ** dim
        assemble = n_cells * n * ((n * n * 16 if gs else n * 24) + 6 * n * G + 40 * G + 20 * G * (G - 1) // 2 + 150)
        return {"bytes": 8 * N * (C + mat + G) + apply_b, "flops": assemble + apply_f}
    if kind == "steps":
        # per step about four Newton and forty Krylov iterations: product, preconditioner, orthogonalisation
        its = 40 * case["steps"]
        return {"bytes": its * N * C * b * 12, "flops": its * n_cells * _cell_flops(dim, G, tens, True)}
    w = 8
    taps = 2 * 27 * (G * (2 * w + w * w + w) + (6 * w + 2 * w * w + 3 * w) + (6 * w + 2 * w * w + 4 * w))
    return {"bytes": 8 * N * C * 3, "flops": N * taps}


# --- the same in plain FP64 torch ---------------------------------------------------

X1 = 0.5 + 0.5 / math.sqrt(3.0)
X0 = 1.0 - X1


class _Q1:
    """Uniform Q1 mesh: 2-point Gauss rule, shape values and cell views."""

    def __init__(self, case):
        self.cells, self.h = _cells_of(case), case["h"]
        self.dim = len(self.cells)
        self.n = 2 ** self.dim
        self.shape = [c + 1 for c in reversed(self.cells)]
        self.N = math.prod(self.shape)
        self.ld = (self.N + 31) // 32 * 32
        self.jxw = (0.5 * self.h) ** self.dim
        per_layer = math.prod(self.cells[:-1])
        step = max(1, 1_500_000 // per_layer)
        self.chunks = [(a, min(a + step, self.cells[-1])) for a in range(0, self.cells[-1], step)]

    def bits(self, l):
        return [(l >> d) & 1 for d in range(self.dim)]

    def phi(self, l, q):
        return math.prod(X1 if a == b else X0 for a, b in zip(self.bits(l), self.bits(q)))

    def dphi(self, l, q):
        lb, qb = self.bits(l), self.bits(q)
        return [(1.0 if lb[d] else -1.0) / self.h *
                math.prod(X1 if lb[e] == qb[e] else X0 for e in range(self.dim) if e != d) for d in range(self.dim)]

    def view(self, F, l, chunk):
        """Local node l of every cell of the chunk (layers of the slowest direction)."""
        lb = self.bits(l)
        idx = [slice(lb[d], lb[d] + self.cells[d]) for d in range(self.dim)]
        idx[-1] = slice(chunk[0] + lb[-1], chunk[1] + lb[-1])
        return F[(Ellipsis,) + tuple(reversed(idx))]

    def at(self, F, q, chunk, grad=True):
        """Values (and gradients, one per direction) of the fields at point q."""
        v, g = 0.0, [0.0] * self.dim
        for l in range(self.n):
            f = self.view(F, l, chunk)
            v = v + self.phi(l, q) * f
            if grad:
                dp = self.dphi(l, q)
                g = [a + p * f for a, p in zip(g, dp)]
        return v, g

    def add(self, out, row, q, chunk, val, flux=None):
        for l in range(self.n):
            r = self.phi(l, q) * val
            if flux is not None:
                for p, f in zip(self.dphi(l, q), flux):
                    r = r + p * f
            self.view(out[row], l, chunk).add_(r, alpha=self.jxw)

    def padded(self, x):
        out = torch.zeros((x.shape[0], self.ld), dtype=torch.float64, device="cuda")
        out[:, :self.N] = x.reshape(x.shape[0], -1)
        return out


def _dot(a, b):
    return sum(x * y for x, y in zip(a, b))


def _normal(gc):
    n2 = _dot(gc, gc)
    inv = torch.where(n2 > 1e-20, 1.0 / n2.clamp_min(1e-300).sqrt(), torch.zeros_like(n2))
    return [x * inv for x in gc], n2, inv


def _phi_c(c):
    return (c ** 3 * (10.0 - 15.0 * c + 6.0 * c * c)).clamp(0.0, 1.0)


def _pairs(eta, geta, tens):
    """(i, j, d_ij, 1/|d_ij|^2) over the grain pairs, d_ij = grad eta_i - grad eta_j."""
    for i in range(eta.shape[0]):
        for j in range(i):
            if not tens:
                yield i, j, None, None
                continue
            d = [g[i] - g[j] for g in geta]
            n2 = _dot(d, d)
            yield i, j, d, torch.where(n2 > 1e-20, 1.0 / n2.clamp_min(1e-300), torch.zeros_like(n2))


def _fcc(c):
    return 2 * A * c * c + 4 * A * c * (2 * c - 2) + 2 * A * (1 - c) ** 2 + 2 * B


def _fee(c, e, s2):
    return B * (12 - 12 * c + 2 * e * (12 * c - 24) + 24 * e * e + 12 * s2)


def _mobility_coefs(c, gc, gmu, tens):
    """fvv, fsurf, unit normal, dM/dc grad mu coefficients (a, b: a grad mu - b n (n . grad mu)),
    the surface part and 1/|grad c| of dM/dgrad c."""
    omc = 1 - c
    phi = _phi_c(c)
    fvv = MVOL * phi + MVAP * (1 - phi)
    c2 = 4 * c * c * omc * omc
    if not tens:
        dmdc = (MVOL - MVAP) * 30 * c * c * omc * omc + MSURF * 8 * c * (1 - 3 * c + 2 * c * c)
        return fvv, MSURF * c2, None, dmdc, None, None, None
    nc, n2, rs = _normal(gc)
    fsurf = MSURF * c2
    zero = torch.zeros_like(c)
    dfs = torch.where(fsurf < 1e-6, zero, MSURF * 8 * c * omc * (1 - 2 * c))
    fs3 = torch.where(fsurf < 1e-6, zero, fsurf)
    inrm = torch.where(n2 < 1e-8, torch.ones_like(c), rs)
    return fvv, fsurf, nc, (MVOL - MVAP) * 30 * c2 + 1.001 * dfs, dfs, fs3, inrm


def _masks(m, u, case, chunk):
    if not case.get("cut_off"):
        return None
    mx = None
    for l in range(m.n):
        a = m.view(u[2:], l, chunk).abs()
        mx = a if mx is None else torch.maximum(mx, a)
    return (mx > case["cut_off"]).double()


def _exact_jvp(case, u, v):
    m, tens = _Q1(case), case["tensorial"]
    u, v = u.view([-1] + m.shape), v.double().view([-1] + m.shape)
    out = torch.zeros_like(u)
    w0 = _weights(case)[0]
    for ch in m.chunks:
        mask = _masks(m, u, case, ch)
        for q in range(m.n):
            uq, gu = m.at(u, q, ch)
            vq, gv = m.at(v, q, ch)
            c, eta, dc, dmu, deta = uq[0], uq[2:], vq[0], vq[1], vq[2:]
            gc, gmu, geta = [g[0] for g in gu], [g[1] for g in gu], [g[2:] for g in gu]
            gdc, gdmu, gdeta = [g[0] for g in gv], [g[1] for g in gv], [g[2:] for g in gv]
            if mask is not None:
                eta, deta = eta * mask, deta * mask
                geta, gdeta = [g * mask for g in geta], [g * mask for g in gdeta]
            fvv, fsurf, nc, am, dfs, fs3, inrm = _mobility_coefs(c, gc, gmu, tens)
            if tens:
                n_dmu, n_mu, n_dc = _dot(nc, gdmu), _dot(nc, gmu), _dot(nc, gdc)
                t = [a - b * n_dc for a, b in zip(gdc, nc)]
                k3, mu_t = -fs3 * inrm, _dot(gmu, t)
                flux = [(fvv + fsurf) * gdmu[d] - nc[d] * fsurf * n_dmu + am * dc * gmu[d] -
                        nc[d] * dfs * n_mu * dc + k3 * (n_mu * t[d] + nc[d] * mu_t) for d in range(m.dim)]
            else:
                flux = [(fvv + fsurf) * gdmu[d] + am * dc * gmu[d] for d in range(m.dim)]
            for i, j, d, f in _pairs(eta, geta, tens):
                p1, p2 = eta[i] * eta[j], eta[j] * deta[i] + eta[i] * deta[j]
                if tens:
                    s = f * (p1 * _dot(d, gdmu) + p2 * _dot(d, gmu))
                    flux = [x + 2 * MGB * (p1 * a + p2 * b - s * e) for x, a, b, e in zip(flux, gdmu, gmu, d)]
                else:
                    flux = [x + 2 * MGB * (p1 * a + p2 * b) for x, a, b in zip(flux, gdmu, gmu)]
            m.add(out, 0, q, ch, w0 * dc, flux)
            s2, sd = (eta * eta).sum(0), (eta * deta).sum(0)
            fce = 12 * B * (eta * eta - eta)
            m.add(out, 1, q, ch, dmu - _fcc(c) * dc - (fce * deta).sum(0), [-KAPPA_C * g for g in gdc])
            row = w0 * deta + L * (fce * dc + _fee(c, eta, s2) * deta + 24 * B * eta * (sd - eta * deta))
            gfl = [L * KAPPA_P * g for g in gdeta]
            if mask is not None:
                row, gfl = row * mask, [g * mask for g in gfl]
            m.add(out, slice(2, None), q, ch, row, gfl)
    return m.padded(out)


def _exact_residual(case, u, hist):
    m, tens = _Q1(case), case["tensorial"]
    w = _weights(case)
    hw = sum(x * wi for x, wi in zip(hist, w[1:])).view([-1] + m.shape)
    u = u.view([-1] + m.shape)
    out = torch.zeros_like(u)
    for ch in m.chunks:
        for q in range(m.n):
            uq, gu = m.at(u, q, ch)
            hq, _ = m.at(hw, q, ch, grad=False)
            c, mu, eta = uq[0], uq[1], uq[2:]
            gc, gmu, geta = [g[0] for g in gu], [g[1] for g in gu], [g[2:] for g in gu]
            fvv, fsurf, nc = _mobility_coefs(c, gc, gmu, tens)[:3]
            if tens:
                n_mu = _dot(nc, gmu)
                flux = [(fvv + 1.001 * fsurf) * g - fsurf * n_mu * x for g, x in zip(gmu, nc)]
            else:
                flux = [(fvv + fsurf) * g for g in gmu]
            for i, j, d, f in _pairs(eta, geta, tens):
                p1 = eta[i] * eta[j]
                s = f * _dot(d, gmu) if tens else None
                flux = [x + 2 * MGB * p1 * (g - s * d[k] if tens else g) for k, (x, g) in enumerate(zip(flux, gmu))]
            m.add(out, 0, q, ch, w[0] * c + hq[0], flux)
            s2, s3 = (eta ** 2).sum(0), (eta ** 3).sum(0)
            df = A * c * c * (2 * c - 2) + 2 * A * c * (1 - c) ** 2 + B * (2 * c - 6 * s2 + 4 * s3)
            m.add(out, 1, q, ch, mu - df, [-KAPPA_C * g for g in gc])
            row = 12 * B * L * eta * (eta * (c - 2) + (1 - c) + s2) + w[0] * eta + hq[2:]
            m.add(out, slice(2, None), q, ch, row, [L * KAPPA_P * g for g in geta])
    return m.padded(out)


def _exact_precond(case, u, r):
    m, tens, G = _Q1(case), case["tensorial"], case["grains"]
    u = u.view([-1] + m.shape)
    w0 = _weights(case)[0]
    nk = 3 ** m.dim
    mat = torch.zeros([nk, 4] + m.shape, dtype=torch.float64, device="cuda")
    diag = torch.zeros([G] + m.shape, dtype=torch.float64, device="cuda")
    gs = case["block_0"] == "ch_gauss_seidel"
    dims = range(m.dim)
    for ch in m.chunks:
        for q in range(m.n):
            uq, gu = m.at(u, q, ch)
            c, eta = uq[0], uq[2:]
            gc, gmu, geta = [g[0] for g in gu], [g[1] for g in gu], [g[2:] for g in gu]
            fvv, fsurf, nc, am, dfs, fs3, inrm = _mobility_coefs(c, gc, gmu, tens)
            if tens:
                n_mu = _dot(nc, gmu)
                M = [[(fvv + 1.001 * fsurf if a == b else 0.0) - fsurf * nc[a] * nc[b] for b in dims] for a in dims]
                mv = [am * gmu[a] - dfs * nc[a] * n_mu for a in dims]
                # dM/dgrad c = -f (n.grad mu I + n grad mu^T) (I - n n^T) / |grad c|
                K = [[-fs3 * inrm * ((n_mu if a == b else 0.0) + nc[a] * gmu[b] - 2 * n_mu * nc[a] * nc[b])
                      for b in dims] for a in dims]
            else:
                M = [[(fvv + fsurf if a == b else 0.0 * c) for b in dims] for a in dims]
                mv, K = [am * g for g in gmu], None
            for i, j, d, f in _pairs(eta, geta, tens):
                p1 = 2 * MGB * eta[i] * eta[j]
                for a in dims:
                    M[a][a] = M[a][a] + p1
                    if tens:
                        for b in dims:
                            M[a][b] = M[a][b] - p1 * f * d[a] * d[b]
            fcc = _fcc(c)
            fee = _fee(c, eta, (eta * eta).sum(0))
            for l in range(m.n):
                p, dp = m.phi(l, q), m.dphi(l, q)
                m.view(diag, l, ch).add_((w0 + L * fee) * (p * p) + L * KAPPA_P * _dot(dp, dp), alpha=m.jxw)
            for b in range(m.n):  # column: local node b
                ps, ds = m.phi(b, q), m.dphi(b, q)
                mg = [_dot(M[a], ds) for a in dims]
                fl = [mv[a] * ps + (_dot(K[a], ds) if K else 0.0) for a in dims]
                for l in range(m.n):
                    if not gs and l != b:
                        continue
                    p, dp = m.phi(l, q), m.dphi(l, q)
                    off = [x - y for x, y in zip(m.bits(b), m.bits(l))]
                    k = sum((o + 1) * 3 ** d for d, o in enumerate(off))
                    for e, val in enumerate((w0 * ps * p + _dot(fl, dp), _dot(mg, dp),
                                             -fcc * (ps * p) - KAPPA_C * _dot(ds, dp), None)):
                        if e == 3:
                            m.view(mat[k, 3], l, ch).add_(ps * p * m.jxw)
                        else:
                            m.view(mat[k, e], l, ch).add_(val, alpha=m.jxw)
    r = r.double().view([-1] + m.shape)
    z = torch.empty_like(r)
    z[2:] = r[2:] / diag
    ctr = mat[nk // 2]
    det = ctr[0] * ctr[3] - ctr[1] * ctr[2]
    inv = torch.stack([ctr[3] / det, -ctr[1] / det, -ctr[2] / det, ctr[0] / det])
    if not gs:
        z[0], z[1] = inv[0] * r[0] + inv[1] * r[1], inv[2] * r[0] + inv[3] * r[1]
        return m.padded(z)
    zp = torch.zeros([2] + [s + 2 for s in m.shape], dtype=torch.float64, device="cuda")

    def lattice(F, col, off=None):
        """The nodes of colour col (parity per direction), shifted by off in the padded field."""
        idx = []
        for d in dims:
            start = (col >> d) & 1
            if off is None:
                idx.append(slice(start, None, 2))
            else:
                cnt = (m.cells[d] + 1 - start + 1) // 2
                idx.append(slice(start + 1 + off[d], start + 1 + off[d] + 2 * cnt - 1, 2))
        return F[(Ellipsis,) + tuple(reversed(idx))]

    def sweep(col, forward):
        s = [0.0, 0.0]
        for k in range(nk):
            off = [k // 3 ** d % 3 - 1 for d in dims]
            nc = col ^ sum((o & 1) << d for d, o in enumerate(off))
            if not (nc < col if forward else nc > col):
                continue
            a, x = lattice(mat[k], col), lattice(zp, col, off)
            s = [s[0] + a[0] * x[0] + a[1] * x[1], s[1] + a[2] * x[0] + a[3] * x[1]]
        i, here = lattice(inv, col), lattice(zp, col, [0] * m.dim)
        if here.numel() == 0:
            return
        if forward:
            b = lattice(r[:2], col)
            s = [b[0] - s[0], b[1] - s[1]]
            here[0], here[1] = i[0] * s[0] + i[1] * s[1], i[2] * s[0] + i[3] * s[1]
        else:
            here[0] -= i[0] * s[0] + i[1] * s[1]
            here[1] -= i[2] * s[0] + i[3] * s[1]

    for col in range(m.n):
        sweep(col, True)
    for col in reversed(range(m.n - 1)):
        sweep(col, False)
    z[:2] = zp[(slice(None),) + (slice(1, -1),) * m.dim]
    return m.padded(z)


def _conv(x, w):
    """3x3x3 convolution, x [samples][Cin][D][H][W], w [3][Cout][Cin][3][3], zero boundary, FP64."""
    S, _, D, H, W = x.shape
    xp = torch.nn.functional.pad(x, (1, 1, 1, 1, 1, 1))
    out = torch.zeros((S, w.shape[1], D * H * W), dtype=torch.float64, device="cuda")
    for dz in range(3):
        for dy in range(3):
            for dx in range(3):
                t = xp[:, :, dz:dz + D, dy:dy + H, dx:dx + W].reshape(S, x.shape[1], -1)
                out += torch.matmul(w[dz, :, :, dy, dx], t)
    return out.view(S, w.shape[1], D, H, W)


def _exact_guess(case, un, um, dt_old, dt):
    m, G = _Q1(case), case["grains"]
    with np.load(WEIGHTS) as f:
        width, layers, gi, si, so, _ = (int(x) for x in f["cfg"])
        flat = torch.as_tensor(f["params"], dtype=torch.float64, device="cuda")
        base, slope = [float(x) for x in f["base"]], float(f["slope"])
    r = dt / dt_old
    inc = r * (un - um)
    groups = (slice(0, 1), slice(1, 2), slice(2, None))
    mags = [float(inc[g].abs().max()) for g in groups]
    grid = lambda t: t.view(m.shape)
    hg = torch.stack([torch.stack([grid(un[2 + i]) * base[2], grid(inc[2 + i]) / mags[2]]) for i in range(G)])
    hs = torch.stack([grid(un[0]) * base[0], grid(inc[0]) / mags[0], grid(un[1]) * base[1], grid(inc[1]) / mags[1]])[None]
    cg, cs, at = gi, si, 0
    for layer in range(layers):
        last = layer == layers - 1
        go, sh = (1, so) if last else (width, width)
        w = {}
        for key, shape in (("A", (3, go, cg, 3, 3)), ("B", (3, go, cg, 3, 3)), ("C", (3, go, cs, 3, 3)),
                           ("D", (3, sh, cs, 3, 3)), ("E", (3, sh, cg, 3, 3)), ("a", (go,)), ("d", (sh,))):
            w[key] = flat[at:at + math.prod(shape)].view(shape)
            at += math.prod(shape)
        pool = hg.sum(0, keepdim=True)
        zg = _conv(hg, w["A"]) + w["a"].view(1, -1, 1, 1, 1) + _conv(pool, w["B"]) + _conv(hs, w["C"])
        zs = _conv(hs, w["D"]) + w["d"].view(1, -1, 1, 1, 1) + _conv(pool, w["E"])
        act = (lambda t: t) if last else (lambda t: torch.where(t > 0, t, slope * t))
        hg, hs, cg, cs = act(zg), act(zs), go, sh
    corr = torch.cat([hs[0], hg[:, 0]]).view(G + 2, -1)
    guess = un + inc
    for k, g in enumerate(groups):
        guess[g] += corr[g] * (mags[k] * dt / base[3 + k])
    return m.padded(guess)


def exact(case, seed):
    if case["kind"] == "steps":
        return None  # an iterative solve: its value depends on where each iteration stops
    u, gen = _state(case, seed)
    dtype = torch.float32 if case.get("precision") == 32 else torch.float64
    if case["kind"] == "jvp":
        return _exact_jvp(case, u, _uniform(u, gen, dtype))
    if case["kind"] == "residual":
        return _exact_residual(case, u, _history(case, u, gen))
    if case["kind"] == "precond":
        return _exact_precond(case, u, _uniform(u, gen, dtype))
    return _exact_guess(case, u, _history(case, u, gen)[0], 1e-3, 1.2e-3)
