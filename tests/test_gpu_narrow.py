"""Mixed steps of grids narrow in x, whose y and z lines go by clusters, by
segments in one block or by the Thomas solves depending on their length."""
import numpy as np
import pytest

from test_gpu_segments import TOL, _noise

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Nx,N", [(9, 128), (9, 129), (12, 192), (16, 200), (16, 204), (16, 205), (9, 257), (16, 320),
                                  (12, 400), (13, 400), (16, 410), (17, 39), (17, 40), (17, 200), (17, 300)])
@pytest.mark.parametrize("d", [1, 2])
def test_mixed_step_tracks_fp64_on_narrow_grids(gpu_pkg, Nx, N, d):
    n = [Nx, 10, 10]
    n[d] = N
    ic = _noise((n[2], n[1], n[0]), 10 * N + Nx + d)
    out = []
    for prec in (gpu_pkg.FP64, gpu_pkg.FP32_MIXED):
        s = gpu_pkg.Solver(gpu_pkg.make_config(tuple(n), tuple(6.283185307179586 * (1.0 - 1.0 / k) for k in n),
                                               mu_ref=1e-3, CFL=0.5, precision=prec))
        s.set_initial_conditions(*ic)
        s.step()
        s.sync()
        out.append(s.conserved())
        s.close()
    scale = np.maximum(np.abs(out[0]).reshape(5, -1).max(1), 1.0).reshape(5, 1, 1, 1)
    assert float((np.abs(out[1] - out[0]) / scale).max()) <= TOL
