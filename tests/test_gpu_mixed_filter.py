"""The mixed TVD-RK3 form's filter where one direction is between walls: its
first and its last pass take the unfiltered value from q2 by different kernels
and must form the same number.  Where the state is constant along every line
the filter then leaves it as it is."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c", [0.137, 0.2113, 0.0529, 0.1106])
def test_unfiltered_value_is_the_same_in_every_pass(gpu_pkg, c):
    """A shear flow u = +c on 160 z planes and -c on 240, brought to zero at
    the y walls.  Sixty points from both, the derivatives are zero and what
    they (0.382^60 = 8e-26) and the filter (1/3^60 = 2e-29 at alphaF = 0.3) carry
    there is below 1e-12 after nine stages and nine passes (60^8 / 8! = 4e9
    ways).  The filter's correction of a constant is the rounding of taps below
    0.11 and of their sum, less than half of the fluctuation's last place.  So
    filtered steps, each order of the passes once, leave the unfiltered steps'
    values; 1e-12 is a thousand times less than the last place of 0.05.  (For
    these c one rounding of q2 - ref and two give different numbers.)"""
    n = (20, 160, 400)
    s = np.where(np.arange(400) < 160, 1.0, -1.0).reshape(-1, 1, 1)
    t = np.minimum(1.0, np.minimum(np.arange(160), 159 - np.arange(160)) / 5.0).reshape(1, -1, 1)
    one = np.ones((400, 160, 20))
    h = []
    for filter_step in (1, 100):
        h.append(gpu_pkg.Solver(gpu_pkg.make_config(
            n, (2.5, 20.0, 50.0), bc_type=(gpu_pkg.PERIODIC_SOLVE, gpu_pkg.DIRICHLET_SOLVE, gpu_pkg.PERIODIC_SOLVE),
            bc_kind=(gpu_pkg.PERIODIC, gpu_pkg.PERIODIC, gpu_pkg.ADIABATIC_WALL, gpu_pkg.ADIABATIC_WALL,
                     gpu_pkg.PERIODIC, gpu_pkg.PERIODIC),
            alphaF=0.3, mu_ref=1e-3, CFL=0.3, filter_step=filter_step, rk=gpu_pkg.TVDRK3_KIND,
            precision=gpu_pkg.FP32_MIXED)))
        h[-1].set_initial_conditions(one, one / 1.4, c * s * t * one, 0 * one, 0 * one)
    for _ in range(3):
        out = []
        for x in h:
            x.step()
            x.sync()
            q = x.conserved()[:, :, 70:90]
            out.append(np.concatenate([q[:, 60:100], q[:, 220:340]], axis=1))
        assert np.abs(out[0] - out[1]).max() <= 1e-12
    for x in h:
        x.close()
