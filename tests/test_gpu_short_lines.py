"""Single operators on short lines either side of the number of points from
which they are solved in segments, against the oracle."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [9, 10, 11, 12, 15, 16, 17, 20, 21, 24, 25])
@pytest.mark.parametrize("bc,points", [(0, 1 << 17), (1, 1 << 18)])
def test_operators_either_side_of_the_switch(gpu_pkg, oracle, N, bc, points):
    bt = [gpu_pkg.PERIODIC_SOLVE] * 3
    bt[0] = bc
    for nl in ((points - 1) // N // 8 * 8, ((points - 1) // N // 8 + 1) * 8):
        lines = np.random.default_rng(N + bc).standard_normal((nl, N)) + 3.0
        op = gpu_pkg.Operator(gpu_pkg.make_config((N, nl // 8, 8), (1.0, 1.0, 1.0), bc_type=tuple(bt)), 0)
        for kind in (1, 2, 3):
            out = op.apply_host(kind, lines)
            # FP64, as the operators' other comparisons with the oracle
            assert rel_err(out, oracle.line_op_port(kind, bc, N, 1.0 / (N - 1.0), 0.49, lines)) <= 1e-13, (nl, kind)
        op.close()
