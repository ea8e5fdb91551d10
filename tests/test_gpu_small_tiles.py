"""The plain form's step against the oracle on small grids, where the number of
lines a tile takes depends on how many blocks a launch has: two, four and eight
lines, tiles that are not full, thin plates."""
import numpy as np
import pytest

from conftest import state_errors
from test_gpu_segments import _noise

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(16, 16, 16), (18, 18, 18), (20, 21, 20), (24, 24, 24), (32, 32, 32), (16, 32, 16), (64, 16, 16),
                               (33, 16, 17), (40, 9, 40), (9, 40, 39), (40, 41, 9), (12, 40, 40), (8, 8, 100)])
def test_step_matches_oracle(gpu_pkg, oracle, n):
    ic = _noise(n[::-1], sum(n))
    cfg = gpu_pkg.make_config(n, tuple(6.283185307179586 * (1.0 - 1.0 / k) for k in n), mu_ref=1e-3, CFL=0.5)
    s = gpu_pkg.Solver(cfg)
    s.set_initial_conditions(*ic)
    s.step()
    s.sync()
    r = oracle.OraclePort(cfg)
    r.set_initial_conditions(*ic)
    r.run(1)
    errs = state_errors(s.conserved(), r.conserved())
    s.close()
    assert max(errs) <= 1e-12, errs  # as the form's other comparisons with the oracle
