"""Single operators in register segments (csrc/cs3d_lineop.cu) against the
oracle at the line lengths where the cut changes: the shortest and longest of
each segment count, full and ragged, a partly filled last warp, and the lengths
left to the Thomas solve (8, 1025)."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu
TOL = 1e-13  # FP64, as the operators' other comparisons with the oracle


@pytest.mark.parametrize("N", [8, 9, 15, 16, 17, 18, 31, 32, 34, 41, 47, 48, 49, 65, 66, 96, 97, 127, 129, 193, 255, 257, 301,
                               512, 513, 767, 1023, 1024, 1025])
@pytest.mark.parametrize("bc", [0, 1])
@pytest.mark.parametrize("alphaF", [0.49, -0.3])
def test_operator_handle_at_plan_edges(gpu_pkg, oracle, N, bc, alphaF):
    rng = np.random.default_rng(N * 2 + bc)
    lines = rng.standard_normal((7, 5, N)) + 3.0
    bt = [gpu_pkg.PERIODIC_SOLVE] * 3
    bt[0] = bc
    L = 2.0 * np.pi * (1 - 1.0 / N)
    op = gpu_pkg.Operator(gpu_pkg.make_config((N, 5, 7), (L, 1.0, 1.0), bc_type=tuple(bt), alphaF=alphaF), 0)
    dh = (1.0 / (N - 1.0)) * L
    for kind in (1, 2, 3):
        out = op.apply_host(kind, lines)
        ref = oracle.line_op_port(kind, bc, N, dh, alphaF, lines.reshape(-1, N))
        assert rel_err(out.reshape(-1, N), ref) <= TOL, kind
    op.close()
