"""Vorticity and Q either side of the rules that choose how the derivatives
along x are launched (64 points a line, 2^18 in all), against the oracle."""
import numpy as np
import pytest

from test_gpu_segments import _noise

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(8, 9, 10), (16, 16, 16), (17, 9, 12), (33, 20, 9), (64, 9, 10), (65, 9, 10), (64, 64, 64),
                               (63, 65, 65)])
@pytest.mark.parametrize("wall", [False, True])
def test_vorticity_q(gpu_pkg, oracle, n, wall):
    kw = {}
    if wall:
        kw = {"bc_type": (gpu_pkg.DIRICHLET_SOLVE, gpu_pkg.PERIODIC_SOLVE, gpu_pkg.PERIODIC_SOLVE),
              "bc_kind": (gpu_pkg.ADIABATIC_WALL,) * 2 + (gpu_pkg.PERIODIC,) * 4}
    cfg = gpu_pkg.make_config(n, tuple(6.283185307179586 * (1.0 - 1.0 / k) for k in n), mu_ref=1e-3, CFL=0.3, **kw)
    ic = _noise(n[::-1], sum(n) + wall)
    s = gpu_pkg.Solver(cfg)
    s.set_initial_conditions(*ic)
    r = oracle.OraclePort(cfg)
    r.set_initial_conditions(*ic)
    # (FP64, as tests/test_gpu_post.py)
    for a, b in zip(s.vorticity_q(), r.vorticity_q()):
        assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max()
    s.close()
