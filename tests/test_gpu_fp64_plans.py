"""The plain form's step against the oracle at the line lengths where the plan
of its sequential solves or of its filter's segments changes: x lines in one,
two and four segments, y and z lines in one block and in clusters of two to
eight, rows divided evenly and not, and the first length whose filter is left
to the Thomas solves (513)."""
import numpy as np
import pytest

from conftest import state_errors

pytestmark = pytest.mark.gpu
TOL = 1e-12  # as the form's other comparisons with the oracle


@pytest.mark.parametrize("N", [63, 65, 79, 80, 81, 97, 119, 120, 121, 127, 129, 159, 160, 161, 163, 193, 255, 257, 511, 513])
@pytest.mark.parametrize("d", [0, 1, 2])
def test_step_matches_oracle_at_plan_edges(gpu_pkg, oracle, N, d):
    n = [9, 10, 9]
    n[d] = N
    n[(d + 1) % 3] = 11
    shape = tuple(n[::-1])
    rng = np.random.default_rng(1000 * d + N)
    u = [0.2 * np.cos(rng.uniform(0, 6.28) + sum(2 * np.pi * rng.integers(0, 3) * np.arange(k).reshape(
        [-1 if a == b else 1 for b in range(3)]) / k for a, k in enumerate(shape)))
        + 0.02 * rng.standard_normal(shape) for _ in range(4)]
    ic = (1.0 + 0.1 * u[3], 1 / 1.4 + 0.05 * u[0] ** 2, u[0], u[1], u[2])
    cfg = gpu_pkg.make_config(tuple(n), tuple(6.283185307179586 * (1.0 - 1.0 / k) for k in n), mu_ref=1e-3, CFL=0.5)
    s = gpu_pkg.Solver(cfg)
    s.set_initial_conditions(*ic)
    s.step()
    s.sync()
    r = oracle.OraclePort(cfg)
    r.set_initial_conditions(*ic)
    r.run(1)
    errs = state_errors(s.conserved(), r.conserved())
    s.close()
    assert max(errs) <= TOL, errs
