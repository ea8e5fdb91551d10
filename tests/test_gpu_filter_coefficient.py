"""The filter at coefficients alphaF from the explicit filter (0) on, at line
lengths whose segments are and are not all full: single operators and full
steps against the oracle, the mixed form against the plain one, the adjoint
against finite differences."""
import numpy as np
import pytest

from conftest import rel_err, state_errors

pytestmark = pytest.mark.gpu

# one segment (9), ragged segments, full ones (48, 64)
LENGTHS = [9, 24, 33, 48, 64, 77, 90, 100, 101, 301, 1000]


@pytest.mark.parametrize("N", LENGTHS)
@pytest.mark.parametrize("bc", [0, 1])
@pytest.mark.parametrize("alphaF", [0.0, 0.02, -0.02])
def test_operator_matches_oracle(gpu_pkg, oracle, N, bc, alphaF):
    lines = np.random.default_rng(N + bc).standard_normal((35, N)) + 3.0
    bt = [gpu_pkg.PERIODIC_SOLVE] * 3
    bt[0] = bc
    op = gpu_pkg.Operator(gpu_pkg.make_config((N, 5, 7), (1.0, 1.0, 1.0), bc_type=tuple(bt), alphaF=alphaF), 0)
    out = op.apply_host(3, lines)
    op.close()
    # FP64, as the operators' other comparisons with the oracle
    assert rel_err(out, oracle.line_op_port(3, bc, N, 1.0 / (N - 1.0), alphaF, lines)) <= 1e-13


@pytest.mark.parametrize("alphaF", [1e-12, 1e-9, -1e-7, 1e-6, 1e-5, 1e-4, -1e-3, 1e-2])
@pytest.mark.parametrize("N", [33, 64, 77, 100])
def test_operator_at_small_coefficients(gpu_pkg, oracle, N, alphaF):
    """The root l of a = l / (1 + l^2) keeps its relative accuracy down to l = a."""
    test_operator_matches_oracle(gpu_pkg, oracle, N, 0, alphaF)


def _steps(gpu_pkg, cfg, ic, n):
    s = gpu_pkg.Solver(cfg)
    s.set_initial_conditions(*ic)
    s.run(n)
    s.sync()
    q = s.conserved()
    s.close()
    return q


@pytest.mark.parametrize("alphaF", [0.0, 1e-6, -1e-5, 0.011, -0.02])
@pytest.mark.parametrize("n", [(24, 33, 77), (90, 9, 24), (20, 100, 64)])
def test_filtered_steps_of_both_forms(gpu_pkg, oracle, n, alphaF):
    """Three steps, so that each direction's filter comes first once.  Mixed
    form: tolerance as tests/test_gpu_segments.py, for three steps."""
    rng = np.random.default_rng(n[0])
    shape = n[::-1]
    u = [0.2 * np.cos(rng.uniform(0, 6.28) + sum(2 * np.pi * rng.integers(0, 3) * np.arange(k).reshape(
        [-1 if a == b else 1 for b in range(3)]) / k for a, k in enumerate(shape)))
        + 0.02 * rng.standard_normal(shape) for _ in range(4)]
    ic = (1.0 + 0.1 * u[3], 1 / 1.4 + 0.05 * u[0] ** 2, u[0], u[1], u[2])
    L = tuple(6.283185307179586 * (1.0 - 1.0 / k) for k in n)
    cfg = gpu_pkg.make_config(n, L, mu_ref=1e-3, CFL=0.5, alphaF=alphaF)
    q = _steps(gpu_pkg, cfg, ic, 3)
    r = oracle.OraclePort(cfg)
    r.set_initial_conditions(*ic)
    r.run(3)
    if alphaF == 0.0:
        assert max(state_errors(q, r.conserved())) <= 1e-12
    mixed = _steps(gpu_pkg, cfg.copy(precision=gpu_pkg.FP32_MIXED), ic, 3)
    scale = np.maximum(np.abs(q).reshape(5, -1).max(1), 1.0).reshape(5, 1, 1, 1)
    assert float((np.abs(mixed - r.conserved()) / scale).max()) <= 3 * 5 * 4 * 4 * 2.0 ** -24


def test_adjoint_of_the_explicit_filter(gpu_pkg, cases):
    N, nsteps, eps = 24, 4, 1e-5
    cfg, ic = cases.tgv(N)
    cfg = cfg.copy(alphaF=0.0)
    s = gpu_pkg.Solver(cfg)
    s.set_initial_conditions(*ic)
    s.step()
    cfg = cfg.copy(dt_fixed=s.scalars()[0])
    s.close()
    rho0, p0, U0, V0, W0 = ic
    grads = []
    for prec in (gpu_pkg.FP64, gpu_pkg.FP32_MIXED):
        s = gpu_pkg.Solver(cfg.copy(precision=prec))
        s.set_initial_conditions(*ic)
        s.adjoint_record(nsteps, 2)
        g, _ = s.adjoint_backward(gpu_pkg.ADJ_KE_MEAN)
        grads.append(np.stack(gpu_pkg.ic_velocity_gradient(g, rho0, U0, V0, W0)))
        s.close()
    # (bounds as tests/test_gpu_adjoint.py)
    assert np.linalg.norm(grads[1] - grads[0]) <= 1e-6 * np.linalg.norm(grads[0])
    rng = np.random.default_rng(6)
    for _ in range(3):
        d = rng.standard_normal((3,) + U0.shape)
        J = []
        for e in (eps, -eps):
            q = _steps(gpu_pkg, cfg, (rho0, p0, U0 + e * d[0], V0 + e * d[1], W0 + e * d[2]), nsteps)
            J.append(float(np.mean(0.5 * (q[1] ** 2 + q[2] ** 2 + q[3] ** 2) / q[0])))
        fd = (J[0] - J[1]) / (2 * eps)
        assert abs(float(np.sum(grads[0] * d)) - fd) <= 1e-6 * abs(fd)
