"""The mixed form's segmented line solves (csrc/cs3d_seg.cuh) at the line
lengths where their plan changes: the shortest and longest of each segment
count, full and ragged segments, lines split over a cluster of blocks and
lines in one block, and the lengths left to the Thomas solves."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# clusters of one-segment blocks: 20..32, 40..256; of two-segment blocks:
# 257..512; one block: the others
LENGTHS = [9, 15, 16, 17, 18, 19, 20, 21, 22, 31, 32, 33, 39, 40, 41, 42, 43, 44, 60, 61, 63, 64, 65, 66, 77, 96, 97, 101, 127, 128, 129, 131, 176, 192, 193,
           256, 257, 263, 264, 320, 511, 512, 513]

# One RK4 step plus filter of a state of order one at CFL 0.5: each of the four
# stages and the filter adds at most about four FP32 roundings (2^-24) of terms
# (dt/h) * flux of order one, weighted by the operators' row sums (below 4).
TOL = 5 * 4 * 4 * 2.0 ** -24


def _noise(shape, seed):
    rng = np.random.default_rng(seed)
    one = np.ones(shape)
    u = [0.2 * np.cos(rng.uniform(0, 6.28) + sum(2 * np.pi * rng.integers(0, 3) * np.arange(n).reshape(
        [-1 if a == b else 1 for b in range(3)]) / n for a, n in enumerate(shape)))
        + 0.02 * rng.standard_normal(shape) for _ in range(4)]
    return one + 0.1 * u[3], one / 1.4 + 0.05 * u[0] ** 2, u[0], u[1], u[2]


@pytest.mark.parametrize("N", LENGTHS)
@pytest.mark.parametrize("d", [0, 1, 2])
def test_mixed_step_tracks_fp64_at_plan_edges(gpu_pkg, N, d):
    abi = gpu_pkg._abi
    n = [12, 12, 12]
    n[d] = N
    n[(d + 1) % 3] = 19  # a tile that is not full
    ic = _noise((n[2], n[1], n[0]), 100 * d + N)
    out = []
    for prec in (abi.FP64, abi.FP32_MIXED):
        L = [6.283185307179586 * (1.0 - 1.0 / k) for k in n]
        s = gpu_pkg.Solver(gpu_pkg.make_config(tuple(n), tuple(L), mu_ref=1e-3, CFL=0.5, precision=prec))
        s.set_initial_conditions(*ic)
        s.step()
        s.sync()
        out.append(s.conserved())
        s.close()
    scale = np.maximum(np.abs(out[0]).reshape(5, -1).max(1), 1.0).reshape(5, 1, 1, 1)
    assert float((np.abs(out[1] - out[0]) / scale).max()) <= TOL


@pytest.mark.parametrize("rk", ["RK4", "TVDRK3"])
@pytest.mark.parametrize("prec", ["FP64", "FP32_MIXED"])
@pytest.mark.parametrize("n", [(32, 64, 32), (33, 45, 101), (12, 12, 12)])
def test_steps_do_not_depend_on_what_is_stored(gpu_pkg, n, prec, rk):
    """The sweeps' instances without the code of diagnostics and increments
    compute what the general instances do: the same operations in the same
    order but for contractions, a rounding of the working type a stage."""
    abi = gpu_pkg._abi
    ic = _noise((n[2], n[1], n[0]), 7)
    out = []
    for store in (0, 1):
        s = gpu_pkg.Solver(gpu_pkg.make_config(n, tuple(6.283185307179586 * (1.0 - 1.0 / k) for k in n), mu_ref=1e-3, CFL=0.5,
                                               rk=getattr(abi, rk), precision=getattr(abi, prec)))
        s.set_option(gpu_pkg.OPT_STORE_DIAGNOSTICS, store)
        s.set_option(gpu_pkg.OPT_STORE_INCREMENTS, store)
        s.set_initial_conditions(*ic)
        s.step()
        s.sync()
        out.append(s.conserved())
        s.close()
    eps = 2.0 ** -24 if prec == "FP32_MIXED" else 2.0 ** -53
    scale = np.maximum(np.abs(out[0]).reshape(5, -1).max(1), 1.0).reshape(5, 1, 1, 1)
    assert float((np.abs(out[1] - out[0]) / scale).max()) <= 5 * 4 * 4 * eps


@pytest.mark.parametrize("kind", ["mixed", "fp64", "sponge"])
def test_repeated_steps_equal_single_handles(gpu_pkg, kind):
    """Steps launched as a recorded graph (small grids, after eight of a form)
    leave the same bits as the sub-step calls, which are never recorded."""
    cases = __import__("importlib").import_module("3dcompactsolver_gb300.cases")
    abi = gpu_pkg._abi
    if kind == "sponge":
        cfg, ic = cases.wall_box(rk=abi.TVDRK3, moving=True, sponge=True)
        cfg = cfg.copy(filter_step=2)
    else:
        cfg, ic = cases.tgv(16, precision=abi.FP32_MIXED if kind == "mixed" else abi.FP64, filter_step=2)
    a, b = gpu_pkg.Solver(cfg), gpu_pkg.Solver(cfg)
    for s in (a, b):
        s.set_initial_conditions(*ic)
    n = 70
    a.run(n)
    for _ in range(n):
        b.pre_step()
        ns = 3 if cfg.rk == abi.TVDRK3 else 4
        for st in range(1, ns + 1):
            b.sub_step(st, st == ns)
        b.post_step()
    assert a.scalars() == b.scalars()
    assert a.launch_count() == b.launch_count()
    assert np.array_equal(a.conserved(), b.conserved())
    a.set_initial_conditions(*ic)  # (the graphs of the old state are dropped)
    a.run(3)
    c = gpu_pkg.Solver(cfg)
    c.set_initial_conditions(*ic)
    c.run(3)
    assert np.array_equal(a.conserved(), c.conserved())
    for s in (a, b, c):
        s.close()


@pytest.mark.parametrize("N", [39, 40, 41, 43, 44, 45, 60, 61, 63, 64, 65, 66, 101, 127, 128, 176, 255, 256, 257])
@pytest.mark.parametrize("d", [1, 2])
def test_mixed_step_tracks_fp64_between_walls(gpu_pkg, N, d):
    """Wall lines over a cluster (40..256 points; the others by the Thomas
    solves).  The one-sided rows' taps sum to about ten times the
    interior's, and the walls' no-slip rows drive the largest increments."""
    abi = gpu_pkg._abi
    n = [19, 12, 12]
    n[d] = N
    n[3 - d] = 13
    rho, p, U, V, W = _noise((n[2], n[1], n[0]), 500 * d + N)
    shape = [1, 1, 1]
    shape[2 - d] = N
    ramp = np.sin(np.pi * np.arange(N) / (N - 1.0)).reshape(shape)
    ic = (rho, p, U * ramp, V * ramp, W * ramp)
    bt = [abi.PERIODIC_SOLVE] * 3
    bt[d] = abi.DIRICHLET_SOLVE
    kind = [abi.PERIODIC] * 6
    kind[2 * d] = abi.ADIABATIC_WALL
    kind[2 * d + 1] = abi.MOVING_ADIABATIC_WALL if N % 2 else abi.ADIABATIC_WALL
    out = []
    for prec in (abi.FP64, abi.FP32_MIXED):
        L = [6.283185307179586 * (1.0 - 1.0 / k) for k in n]
        s = gpu_pkg.Solver(gpu_pkg.make_config(
            tuple(n), tuple(L), bc_type=tuple(bt), bc_kind=tuple(kind), mu_ref=1e-3, CFL=0.3, precision=prec,
            wall_vel=(0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.05, -0.02, 0.0, 0.0, 0.03, 0.01)))
        s.set_initial_conditions(*ic)
        s.step()
        s.sync()
        out.append(s.conserved())
        s.close()
    scale = np.maximum(np.abs(out[0]).reshape(5, -1).max(1), 1.0).reshape(5, 1, 1, 1)
    assert float((np.abs(out[1] - out[0]) / scale).max()) <= 10 * TOL


@pytest.mark.parametrize("N", [19, 20, 21, 22, 31, 32, 33, 39, 40, 41, 42, 44, 65, 101, 256, 257, 511])
@pytest.mark.parametrize("d", [0, 1, 2])
def test_mixed_transposed_sweep_tracks_fp64_at_plan_edges(gpu_pkg, N, d):
    """The transposed sweeps use the same plans.  FP32 rounds each of about
    forty products of a seed of order one and a coefficient at 2^-24, against the
    largest entry of a field; 2e-3 leaves the cancellation of the second
    derivatives' taps (four orders), a wrong neighbour is of order one."""
    abi = gpu_pkg._abi
    n = [20, 20, 20]
    n[d] = N
    n[(d + 1) % 3] = 19
    rho, p, U, V, W = _noise((n[2], n[1], n[0]), 900 * d + N)
    q = np.stack([rho, rho * U, rho * V, rho * W, p / 0.4 + 0.5 * rho * (U * U + V * V + W * W)])
    w = np.random.default_rng(N).standard_normal(q.shape)
    out = []
    for prec in (abi.FP64, abi.FP32_MIXED):
        s = gpu_pkg.Solver(gpu_pkg.make_config(tuple(n), tuple(6.283185307179586 * (1.0 - 1.0 / k) for k in n), mu_ref=1e-3, CFL=0.5,
                                               precision=prec))
        s.set_initial_conditions(rho, p, U, V, W)
        out.append(s.rhs_vjp(q, w))
        s.close()
    for f in range(5):
        assert np.abs(out[1][f] - out[0][f]).max() <= 2e-3 * np.abs(out[0][f]).max(), f
