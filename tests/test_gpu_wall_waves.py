"""Mixed steps between walls either side of the rule that leaves lines to the
Thomas solves where clusters would take a second wave of blocks."""
import numpy as np
import pytest

from test_gpu_segments import TOL, _noise

pytestmark = pytest.mark.gpu


# (Nx, N, planes): Thomas (48, 100, 50), (83, 129, 25), (20, 256, 76); clusters: one plane
# more or three blocks, few idle columns
@pytest.mark.parametrize("Nx,N,planes", [(48, 100, 50), (48, 100, 51), (48, 96, 50), (83, 129, 25), (85, 129, 25),
                                         (20, 256, 76), (20, 256, 77), (20, 128, 76)])
@pytest.mark.parametrize("d", [1, 2])
def test_mixed_step_tracks_fp64_between_walls(gpu_pkg, Nx, N, planes, d):
    n = [Nx, planes, planes]
    n[d] = N
    rho, p, U, V, W = _noise((n[2], n[1], n[0]), N + planes + d)
    shape = [1, 1, 1]
    shape[2 - d] = N
    ramp = np.sin(np.pi * np.arange(N) / (N - 1.0)).reshape(shape)
    bt = [gpu_pkg.PERIODIC_SOLVE] * 3
    bt[d] = gpu_pkg.DIRICHLET_SOLVE
    kind = [gpu_pkg.PERIODIC] * 6
    kind[2 * d] = kind[2 * d + 1] = gpu_pkg.ADIABATIC_WALL
    out = []
    for prec in (gpu_pkg.FP64, gpu_pkg.FP32_MIXED):
        s = gpu_pkg.Solver(gpu_pkg.make_config(tuple(n), tuple(6.283185307179586 * (1.0 - 1.0 / k) for k in n),
                                               bc_type=tuple(bt), bc_kind=tuple(kind), mu_ref=1e-3, CFL=0.3, precision=prec))
        s.set_initial_conditions(rho, p, U * ramp, V * ramp, W * ramp)
        s.step()
        s.sync()
        out.append(s.conserved())
        s.close()
    scale = np.maximum(np.abs(out[0]).reshape(5, -1).max(1), 1.0).reshape(5, 1, 1, 1)
    assert float((np.abs(out[1] - out[0]) / scale).max()) <= 10 * TOL  # (as between walls in tests/test_gpu_segments.py)
