"""The measured workloads: what a user of the solver has it do.

Four kinds of case, each through the package's public entry points:

  step   a solver handle advanced by `steps` time steps (Solver.run); the
         conserved state it leaves is handed on as device tensors: FP64 from
         the FP64 form, single precision from the mixed form (whose arithmetic
         is FP32)
  op     the compact first derivative, second derivative and filter along one
         direction of a device field (Operator.apply)
  adj    the discrete adjoint: record `steps` time steps, take them back
         (Solver.adjoint_record, Solver.adjoint_backward)
  post   vorticity magnitude and Q-criterion of a state (Solver.vorticity_q)

exact() restates the method in plain torch in 64 bits: dense line operators
A^-1 B applied by matrix products.
"""
import importlib
import math

import numpy as np
import torch

pkg = importlib.import_module("3dcompactsolver_gb300")
abi = importlib.import_module("3dcompactsolver_gb300._abi")

GAMMA = 1.4
RGAS = 1.0 / GAMMA


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _step(name, n, precision, flow="vortex", rk="rk4", filter_step=1, steps=1):
    c = {"kind": "step", "nx": n[0], "ny": n[1], "nz": n[2], "precision": precision, "flow": flow,
         "rk": rk, "filter_step": filter_step, "steps": steps}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest grid a user starts from (the package's own smoke run)
        _step("vortex16_fp64", (16, 16, 16), "fp64"),
        # Taylor-Green 64^3 and 128^3, the solver's benchmark grids; three
        # steps go through the three orders of the filter's passes
        _step("vortex64_mixed", (64, 64, 64), "mixed", steps=3),
        _step("vortex128_mixed", (128, 128, 128), "mixed", steps=3),
        # isotropic turbulence on the largest benchmark grid
        _step("turbulence256_mixed", (256, 256, 256), "mixed", "turbulence", steps=3),
        # the plain form on the same grids: validation and reference runs
        _step("vortex128_fp64", (128, 128, 128), "fp64"),
        _step("turbulence256_fp64", (256, 256, 256), "fp64", "turbulence"),
        # a box whose sides divide nothing, the other integrator, filtered
        # every second step
        _step("ragged_mixed", (101, 90, 77), "mixed", rk="tvdrk3", filter_step=2, steps=2),
        # the temporal shear layer: walls, sponge bands, filtered every fifth step
        _step("shear_mixed", (256, 128, 42), "mixed", "shear", rk="tvdrk3", filter_step=5, steps=5),
        # single operators on device arrays: a cube, and long odd wall lines
        {"name": "operators128", "kind": "op", "nx": 128, "ny": 128, "nz": 128, "dir": 2, "bc": "periodic"},
        {"name": "operators_wall301", "kind": "op", "nx": 301, "ny": 77, "nz": 50, "dir": 0, "bc": "wall"},
        # gradient of the final kinetic energy with respect to the initial state
        {"name": "adjoint64_mixed", "kind": "adj", "nx": 64, "ny": 64, "nz": 64, "precision": "mixed",
         "rk": "rk4", "steps": 4, "every": 2},
        # post-processing of a state
        {"name": "vorticity128", "kind": "post", "nx": 128, "ny": 128, "nz": 128},
    ]


def draw(rng):
    def side(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def box(lo, hi, most):
        # half of the boxes are near-cubes, half have unequal sides
        if rng.random() < 0.5:
            s = side(lo, min(hi, int(most ** (1.0 / 3.0))))
            n = [min(hi, max(lo, s + rng.randint(-3, 3))) for _ in range(3)]
        else:
            n = [side(lo, hi) for _ in range(3)]
        while n[0] * n[1] * n[2] > most:
            k = n.index(max(n))
            n[k] = max(lo, int(n[k] * 0.8))
        return n

    kind = rng.choice(["step"] * 6 + ["op"] * 2 + ["adj", "post"])
    if kind == "step":
        flow = rng.choice(["vortex", "vortex", "turbulence", "shear"])
        precision = rng.choice(["mixed", "mixed", "fp64"])
        rk = "tvdrk3" if flow == "shear" else rng.choice(["rk4", "rk4", "tvdrk3"])
        n = box(24 if flow == "shear" else 12, 320, 8_000_000 if precision == "mixed" else 4_000_000)
        fs = 5 if flow == "shear" else rng.choice([1, 1, 2])
        return _step(None, n, precision, flow, rk, fs, rng.randint(1, 3))
    if kind == "op":
        n = box(12, 512, 12_000_000)
        return {"kind": "op", "nx": n[0], "ny": n[1], "nz": n[2], "dir": rng.randint(0, 2),
                "bc": rng.choice(["periodic", "periodic", "wall"])}
    if kind == "adj":
        n = box(12, 96, 500_000)
        return {"kind": "adj", "nx": n[0], "ny": n[1], "nz": n[2], "precision": rng.choice(["mixed", "fp64"]),
                "rk": rng.choice(["rk4", "rk4", "tvdrk3"]), "steps": rng.randint(2, 4), "every": 2}
    n = box(16, 256, 6_000_000)
    return {"kind": "post", "nx": n[0], "ny": n[1], "nz": n[2]}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _shape(case):
    return case["nz"], case["ny"], case["nx"]


def _config(case):
    n = (case["nx"], case["ny"], case["nz"])
    prec = abi.FP32_MIXED if case.get("precision") == "mixed" else abi.FP64
    rk = abi.TVDRK3 if case.get("rk") == "tvdrk3" else abi.RK4
    if case.get("flow") == "shear":
        return abi.make_config(
            n, tuple(0.5 * (k - 1) for k in n),
            bc_type=(abi.PERIODIC_SOLVE, abi.DIRICHLET_SOLVE, abi.PERIODIC_SOLVE),
            bc_kind=(abi.PERIODIC, abi.PERIODIC, abi.ADIABATIC_WALL, abi.ADIABATIC_WALL, abi.PERIODIC,
                     abi.PERIODIC),
            alphaF=0.495, mu_ref=0.00375, CFL=0.5, filter_step=case["filter_step"], rk=rk, precision=prec,
            sponge_mode=abi.SPONGE_BANDS, sponge_frac=(0.0, 0.0, 0.15, 0.15, 0.0, 0.0))
    L = tuple(2.0 * math.pi * (1.0 - 1.0 / k) for k in n)
    if case["kind"] == "op":
        bc = [abi.PERIODIC_SOLVE] * 3
        if case["bc"] == "wall":
            bc[case["dir"]] = abi.DIRICHLET_SOLVE
        return abi.make_config(n, L, bc_type=tuple(bc), alphaF=0.49)
    if case.get("flow") == "turbulence":
        mu = 2.0e-4
    else:
        mu = 1.0 / (1600.0 * (100.0 ** 0.76))
    # the adjoint's frozen time step: CFL 0.5 of the vortex (Mach 0.1)
    dt = 0.5 * min(L[d] / (n[d] - 1.0) for d in range(3)) / 33.0 if case["kind"] == "adj" else 0.0
    return abi.make_config(n, L, alphaF=0.49, mu_ref=mu, CFL=0.5, filter_step=case.get("filter_step", 1), rk=rk,
                           precision=prec, dt_fixed=dt)


def _mesh(case, cfg):
    ax = [torch.arange(k, dtype=torch.float64, device="cuda") * (L / (k - 1.0))
          for k, L in ((cfg.Nx, cfg.Lx), (cfg.Ny, cfg.Ly), (cfg.Nz, cfg.Lz))]
    return ax[0].view(1, 1, -1), ax[1].view(1, -1, 1), ax[2].view(-1, 1, 1)


def _modes(rng, cfg, kmin, kmax, count, amplitude):
    """Three velocity components: a sum of `count` random Fourier modes with
    kmin <= |k| <= kmax, solenoidal, of rms `amplitude`."""
    ax = [2.0 * math.pi * torch.arange(k, dtype=torch.float64, device="cuda") / k for k in (cfg.Nx, cfg.Ny, cfg.Nz)]
    u = torch.zeros((3, cfg.Nz, cfg.Ny, cfg.Nx), dtype=torch.float64, device="cuda")
    top = [max(1, min(kmax, k // 4)) for k in (cfg.Nx, cfg.Ny, cfg.Nz)]
    for _ in range(count):
        while True:
            k = np.array([rng.integers(-t, t + 1) for t in top], dtype=np.float64)
            if kmin <= math.sqrt(float(k @ k)) <= kmax:
                break
        a = rng.standard_normal(3)
        a -= k * (a @ k) / (k @ k)
        ph = rng.uniform(0.0, 2.0 * math.pi)
        ex = torch.exp(1j * (k[0] * ax[0] + ph))
        ey, ez = torch.exp(1j * (k[1] * ax[1])), torch.exp(1j * (k[2] * ax[2]))
        w = ((ez.view(-1, 1) * ey.view(1, -1)).unsqueeze(-1) * ex).real
        for c in range(3):
            u[c] += float(a[c]) * w
    rms = float((u * u).sum(0).mean().sqrt())
    return u * (amplitude / max(rms, 1e-30))


def _flow(case, cfg, seed):
    """rho0, p0, U0, V0, W0 of the case on the device, (Nz, Ny, Nx) each."""
    rng = np.random.default_rng(seed)
    x, y, z = _mesh(case, cfg)
    one = torch.ones(_shape(case), dtype=torch.float64, device="cuda")
    flow = case.get("flow", "vortex")
    if flow == "turbulence":
        # decaying isotropic turbulence, turbulent Mach number 0.3, sound speed 1
        u = _modes(rng, cfg, 1.0, 10.0, 24, 0.3)
        return one, one / GAMMA, u[0], u[1], u[2]
    if flow == "shear":
        du, delta = 0.6, 2.0
        g = torch.Generator(device="cuda")
        g.manual_seed(int(seed))
        noise = 2.0 * torch.rand((3,) + _shape(case), dtype=torch.float64, device="cuda", generator=g) - 1.0
        s = y - cfg.Ly / 2.0
        pert = 0.1 * du / 2.0 * torch.exp(-s * s) * noise
        return one, one / GAMMA, du / 2.0 * torch.tanh(s / delta) + pert[0], pert[1], pert[2]
    # Taylor-Green vortex at Mach 0.1 with its phases drawn and a few weak modes
    a, b, c = rng.uniform(0.0, 2.0 * math.pi, 3)
    x, y, z = x + a, y + b, z + c
    u = _modes(rng, cfg, 1.0, 4.0, 6, 0.03)
    p = 100.0 / GAMMA + (torch.cos(2 * x) + torch.cos(2 * y)) * (torch.cos(2 * z) + 2.0) / 16.0
    return (one, p * one, torch.sin(x) * torch.cos(y) * torch.cos(z) + u[0],
            -torch.cos(x) * torch.sin(y) * torch.cos(z) + u[1], u[2])


def _field(case, seed):
    """One smooth field with some noise, in the direction's contiguous layout."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    cfg = _config(case)
    u = _modes(np.random.default_rng(seed), cfg, 1.0, 6.0, 6, 1.0)[0]
    u = u + 0.01 * torch.randn(u.shape, dtype=torch.float64, device="cuda", generator=g)
    order = {0: (0, 1, 2), 1: (2, 0, 1), 2: (1, 2, 0)}[case["dir"]]  # XYZ, YZX, ZXY
    return u.permute(order).contiguous()


class _Device:
    """A device array of a solver, for torch.as_tensor; the tensor keeps this
    object, and with it the solver that owns the memory."""

    def __init__(self, solver, ptr, shape):
        self.solver = solver
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": tuple(shape), "typestr": "<f8", "version": 3}


def prepare(case, seed):
    cfg = _config(case)
    if case["kind"] == "op":
        field = _field(case, seed)
        op = pkg.Operator(cfg, case["dir"])
        torch.cuda.synchronize()
        return {"case": case, "op": op, "in": field, "out": [torch.empty_like(field) for _ in range(3)]}
    ic = [f.cpu().numpy() for f in _flow(case, cfg, seed)]
    solver = pkg.Solver(cfg)
    solver.set_initial_conditions(*ic)
    state = {"case": case, "solver": solver, "views": {}}
    if case["kind"] == "step" and case["precision"] == "mixed":
        state["stream"] = torch.cuda.ExternalStream(solver.stream())
        state["out"] = [torch.empty(_shape(case), dtype=torch.float32, device="cuda") for _ in range(5)]
        torch.cuda.synchronize()
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "op":
        src = state["in"].data_ptr()
        for kind in (pkg.OP_DERIV1, pkg.OP_DERIV2, pkg.OP_FILTER):
            state["op"].apply(kind, src, state["out"][kind - 1].data_ptr())
        return state["out"]
    solver = state["solver"]
    if case["kind"] == "adj":
        solver.adjoint_record(case["steps"], case["every"])
        grad, J = solver.adjoint_backward()
        if case["precision"] == "mixed":  # single-precision Jacobians: the optimiser takes FP32
            return [torch.from_numpy(grad).float(), float(J)]
        return [grad, float(J)]
    if case["kind"] == "post":
        return list(solver.vorticity_q())
    solver.run(case["steps"])
    out = []
    for f in range(5):
        ptr = solver.field_ptr(f)
        if ptr not in state["views"]:
            state["views"][ptr] = torch.as_tensor(_Device(solver, ptr, _shape(case)), device="cuda")
        out.append(state["views"][ptr])
    if case["precision"] == "mixed":
        with torch.cuda.stream(state["stream"]):
            for single, q in zip(state["out"], out):
                single.copy_(q)
        return state["out"]
    return out


def work(case):
    n = float(case["nx"]) * case["ny"] * case["nz"]
    if case["kind"] == "op":  # one field in, three out; 10 and 16 operations a row and stencil kind
        return {"bytes": 8.0 * 4 * n, "flops": 40.0 * n}
    if case["kind"] == "post":  # state in, two fields out; nine derivatives
        return {"bytes": 8.0 * 7 * n, "flops": 150.0 * n}
    stages = 3 if case["rk"] == "tvdrk3" else 4
    if case["kind"] == "adj":  # state in; state and gradient out; a forward and about two more back
        return {"bytes": 8.0 * 15 * n, "flops": 3.0 * case["steps"] * stages * 1000.0 * n}
    flops = case["steps"] * (stages * 1000.0 + 375.0 / case["filter_step"]) * n
    return {"bytes": 8.0 * 10 * n, "flops": flops}


# ---------------------------------------------------------------------------
# the same in 64 bits, in plain torch
# ---------------------------------------------------------------------------
def _dense(kind, N, periodic, h, alphaF=0.49):
    """A^-1 B of one compact operator on N points, dense, in 64 bits: the
    sixth-order first derivative (1) and second derivative (2), the eighth-order
    filter (3), with the solver's one-sided closures at walls."""
    A = np.eye(N)
    B = np.zeros((N, N))
    if kind == 1:
        al, half = 1.0 / 3.0, 2
        taps = np.array([-1.0 / 36.0, -7.0 / 9.0, 0.0, 7.0 / 9.0, 1.0 / 36.0]) / h
    elif kind == 2:
        al, half = 2.0 / 11.0, 2
        a, b = 12.0 / 11.0, 3.0 / 11.0
        taps = np.array([b / 4.0, a, -2.0 * a - b / 2.0, a, b / 4.0]) / (h * h)
    else:
        al, half = alphaF, 4
        c = [(93.0 + 70.0 * al) / 128.0, (7.0 + 18.0 * al) / 32.0, (-7.0 + 14.0 * al) / 64.0,
             (1.0 - 2.0 * al) / 32.0, (-1.0 + 2.0 * al) / 256.0]
        taps = np.array([c[4], c[3], c[2], c[1], c[0], c[1], c[2], c[3], c[4]])
    for i in range(N):
        if periodic or half <= i < N - half:
            for k in range(-half, half + 1):
                B[i, (i + k) % N] += taps[k + half]
            A[i, (i - 1) % N] += al
            A[i, (i + 1) % N] += al
    if not periodic:
        if kind == 1:
            rows = [[-197 / 60, -5 / 12, 5, -5 / 3, 5 / 12, -1 / 20], [-43 / 96, -5 / 6, 9 / 8, 1 / 6, -1 / 96]]
            off, sign, sc = [(0.0, 5.0), (1.0 / 8.0, 3.0 / 4.0)], -1.0, 1.0 / h
        elif kind == 2:
            rows = [[145 / 12, -76 / 3, 29 / 2, -4 / 3, 1 / 12],
                    [177 / 88, -507 / 44, 783 / 44, -201 / 22, 81 / 88, -3 / 44]]
            off, sign, sc = [(0.0, 10.0), (2.0 / 11.0, -131.0 / 22.0)], 1.0, 1.0 / (h * h)
        else:
            s = [(11 + 10 * al) / 16, (15 + 34 * al) / 64, (-3 + 6 * al) / 32, (1 - 2 * al) / 64]
            rows = [[15 / 16, 4 / 16, -6 / 16, 4 / 16, -1 / 16], [1 / 16, 3 / 4, 6 / 16, -4 / 16, 1 / 16],
                    [-1 / 16, 4 / 16, 5 / 8, 4 / 16, -1 / 16], [s[3], s[2], s[1], s[0], s[1], s[2], s[3]]]
            off, sign, sc = [(0.0, 0.0)] * 3 + [(al, al)], 1.0, 1.0
        for r, row in enumerate(rows):
            lo, up = off[r]
            B[r, :] = 0.0
            B[N - 1 - r, :] = 0.0
            for k, v in enumerate(row):
                B[r, k] = v * sc
                B[N - 1 - r, N - 1 - k] = sign * v * sc
            if r > 0:
                A[r, r - 1] = lo
                A[N - 1 - r, N - r] = lo
            A[r, r + 1] = up
            A[N - 1 - r, N - 2 - r] = up
    return torch.from_numpy(np.linalg.solve(A, B)).cuda()


class _Exact:
    """The solver's step in plain torch, 64 bits."""

    def __init__(self, case, cfg):
        n, L = (cfg.Nx, cfg.Ny, cfg.Nz), (cfg.Lx, cfg.Ly, cfg.Lz)
        self.cfg, self.case = cfg, case
        self.h = [L[d] / (n[d] - 1.0) for d in range(3)]
        self.per = [cfg.bc_type[d] == abi.PERIODIC_SOLVE for d in range(3)]
        self.M = [[_dense(k, n[d], self.per[d], self.h[d], cfg.alphaF) for k in (1, 2, 3)] for d in range(3)]
        self.walls = not self.per[1]
        self.sigma = None
        if any(f > 0.0 for f in cfg.sponge_frac):
            s = torch.zeros(cfg.Ny, dtype=torch.float64, device="cuda")
            y = torch.arange(cfg.Ny, dtype=torch.float64, device="cuda") * self.h[1]
            for hi in (0, 1):
                band = cfg.sponge_frac[2 + hi] * cfg.Ly
                r = ((band - y) if hi == 0 else (y - (cfg.Ly - band))) / band
                s = torch.maximum(s, torch.where(r > 0, 6.0 * (0.068 * r ** 2 + 0.845 * r.clamp(min=0) ** 8), 0 * r))
            self.sigma = s.view(1, -1, 1)

    def ap(self, u, d, k):
        M = self.M[d][k - 1]
        if d == 0:
            return u @ M.T
        if d == 1:
            return torch.matmul(M, u)
        return (M @ u.reshape(u.shape[0], -1)).reshape(u.shape)

    @staticmethod
    def prim(q):
        U, V, W = q[1] / q[0], q[2] / q[0], q[3] / q[0]
        p = (GAMMA - 1.0) * (q[4] - 0.5 * q[0] * (U * U + V * V + W * W))
        return U, V, W, p, p / (q[0] * RGAS)

    def bc(self, q):
        """Adiabatic no-slip walls at the y faces: Neumann temperature."""
        if not self.walls:
            return q
        T = self.prim(q)[4]
        w = (360.0, -450.0, 400.0, -225.0, 72.0, -10.0)
        q = q.clone()
        for face, s in ((0, 1), (self.cfg.Ny - 1, -1)):
            Tw = sum(w[m] * T[:, face + s * (m + 1), :] for m in range(6)) / 147.0
            q[1:4, :, face, :] = 0.0
            q[4, :, face, :] = q[0, :, face, :] * RGAS * Tw / (GAMMA - 1.0)
        return q

    def rhs(self, q, savg):
        U, V, W, p, T = self.prim(q)
        mu = self.cfg.mu_ref * T ** 0.76
        amu = 0.76 * mu / T
        c43, k = 4.0 / 3.0, (RGAS * GAMMA / (GAMMA - 1.0)) / 0.7
        d, u = [[self.ap(f, e, 1) for e in range(3)] for f in (U, V, W, T)], (U, V, W)
        dd = [[self.ap(f, e, 2) for e in range(3)] for f in (U, V, W, T)]
        grad, m = d[:3], [amu * d[3][e] for e in range(3)]
        Uxy, Vxy = self.ap(d[0][0], 1, 1), self.ap(d[1][0], 1, 1)
        S = self.ap(d[0][0] + d[1][1], 2, 1)
        Wxz, Wyz = self.ap(d[2][0], 2, 1), self.ap(d[2][1], 2, 1)
        div = grad[0][0] + grad[1][1] + grad[2][2]
        # divergence of the viscous stress, with its cross derivatives
        cross = (Vxy + Wxz, Uxy + Wyz, S)
        visc, diss = [], 0.0
        for a in range(3):
            t = mu * (dd[a][0] + dd[a][1] + dd[a][2] + dd[a][a] / 3.0 + cross[a] / 3.0)
            for b in range(3):
                tau = grad[a][b] + grad[b][a] - (2.0 / 3.0 * div if a == b else 0.0)
                t = t + m[b] * tau
                diss = diss + mu * tau * grad[a][b]
            visc.append(t)
        heat = k * (sum(m[e] * d[3][e] for e in range(3)) + mu * (dd[3][0] + dd[3][1] + dd[3][2]))
        conv = [0.0] * 5
        for e in range(3):
            mass = self.ap(q[1 + e], e, 1)
            conv[0] = conv[0] + mass
            if e == 1:
                dv = mass  # what is left of continuity at a y wall
            for a in range(3):
                conv[1 + a] = conv[1 + a] + self.ap(q[1 + a] * u[e] + (p if a == e else 0.0), e, 1)
            conv[4] = conv[4] + self.ap((q[4] + p) * u[e], e, 1)
        R = [-conv[0], visc[0] - conv[1], visc[1] - conv[2], visc[2] - conv[3],
             heat + U * visc[0] + V * visc[1] + W * visc[2] + diss - conv[4]]
        if self.sigma is not None:
            for f in range(5):
                R[f] = R[f] + (2.0 if f == 4 else 1.0) * self.sigma * (savg[f] - q[f])
        R = torch.stack(R)
        if self.walls:
            edge = torch.zeros((1, self.cfg.Ny, 1), dtype=torch.bool, device="cuda")
            edge[:, 0], edge[:, -1] = True, True
            R = torch.stack([torch.where(edge, -dv if f == 0 else 0.0 * R[f], R[f]) for f in range(5)])
        return R

    def cfl(self, q):
        U, V, W, p, T = self.prim(q)
        c = torch.sqrt(GAMMA * p / q[0])
        return self.cfg.CFL / float(((U.abs() + c) / self.h[0] + (V.abs() + c) / self.h[1]
                                     + (W.abs() + c) / self.h[2]).max())

    def steps(self, q, count):
        cfg, savg, filtered = self.cfg, q.clone() if self.sigma is not None else None, 0
        for ts in range(1, count + 1):
            dt = cfg.dt_fixed if cfg.dt_fixed > 0.0 else self.cfl(q)
            q = self.bc(q)
            if cfg.rk == abi.TVDRK3:
                y = self.bc(q + dt * self.rhs(q, savg))
                y = self.bc(0.75 * q + 0.25 * y + 0.25 * dt * self.rhs(y, savg))
                q = q / 3.0 + (2.0 / 3.0) * y + (2.0 / 3.0) * dt * self.rhs(y, savg)
            else:
                k = dt * self.rhs(q, savg)
                q2 = q + k / 6.0
                for b, a in ((0.5, 3.0), (0.5, 3.0), (1.0, 6.0)):
                    k = dt * self.rhs(self.bc(q + b * k), savg)
                    q2 = q2 + k / a
                q = q2
            if ts % cfg.filter_step == 0:
                filtered += 1
                for e in ((0, 1, 2), (1, 2, 0), (2, 0, 1))[(filtered - 1) % 3]:
                    q = torch.stack([self.ap(q[f], e, 3) for f in range(5)])
            if savg is not None:
                eps = 1.0 / (15.0 / dt + 1.0)
                savg = savg + eps * (q - savg)
                ke = 0.5 * (savg[1] ** 2 + savg[2] ** 2 + savg[3] ** 2) / savg[0]
                savg[4] = 0.005 * savg[4] + 0.995 * (1.0 / GAMMA / (GAMMA - 1.0) + ke)
        return q

    def initial(self, seed):
        r, p, U, V, W = _flow(self.case, self.cfg, seed)
        if self.walls:
            # the walls' Neumann temperature, then rhoE from p = rho R T everywhere
            T = p / (r * RGAS)
            w = (360.0, -450.0, 400.0, -225.0, 72.0, -10.0)
            U, V, W = U.clone(), V.clone(), W.clone()
            for face, s in ((0, 1), (self.cfg.Ny - 1, -1)):
                T[:, face, :] = sum(w[m] * T[:, face + s * (m + 1), :] for m in range(6)) / 147.0
                for v in (U, V, W):
                    v[:, face, :] = 0.0
            p = r * RGAS * T
        return torch.stack([r, r * U, r * V, r * W, p / (GAMMA - 1.0) + 0.5 * r * (U * U + V * V + W * W)])


def exact(case, seed):
    cfg = _config(case)
    if case["kind"] == "op":
        n, L = (cfg.Nx, cfg.Ny, cfg.Nz)[case["dir"]], (cfg.Lx, cfg.Ly, cfg.Lz)[case["dir"]]
        u = _field(case, seed)
        return [u @ _dense(k, n, case["bc"] == "periodic", L / (n - 1.0), 0.49).T for k in (1, 2, 3)]
    e = _Exact(case, cfg)
    q = e.initial(seed)
    if case["kind"] == "post":
        vel = [q[1 + c] / q[0] for c in range(3)]
        g = [[e.ap(vel[c], d, 1) for d in range(3)] for c in range(3)]
        w = (g[2][1] - g[1][2], g[0][2] - g[2][0], g[1][0] - g[0][1])
        vort = torch.sqrt(w[0] ** 2 + w[1] ** 2 + w[2] ** 2)
        S2 = sum(((g[a][b] + g[b][a]) / 2.0) ** 2 for a in range(3) for b in range(3))
        W2 = sum(((g[a][b] - g[b][a]) / 2.0) ** 2 for a in range(3) for b in range(3))
        return [vort.cpu().numpy(), (0.5 * W2 - 0.5 * S2).cpu().numpy()]
    if case["kind"] == "adj":
        q.requires_grad_(True)
        r = e.steps(q, case["steps"])
        J = (0.5 * (r[1] ** 2 + r[2] ** 2 + r[3] ** 2) / r[0]).mean()
        J.backward()
        grad = q.grad.cpu()
        return [grad if case["precision"] == "mixed" else grad.numpy(), float(J.detach())]
    return [f.clone() for f in e.steps(q, case["steps"])]
