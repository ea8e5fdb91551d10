"""A constant has no derivative, exactly: the taps of the plain form's
sequential solves sum to zero (compiled for the host; 1 and its sums with the
taps are exact), and single operators take differences before products."""
import ctypes

import numpy as np
import pytest

from test_seq_tasks_cpu import seq_lib  # noqa: F401  (a fixture)


@pytest.mark.parametrize("d,N", [(0, 9), (0, 81), (0, 163), (1, 64), (1, 83), (2, 161)])
@pytest.mark.parametrize("dh", [0.01, 0.037, 0.07, 2.0 * np.pi / 97, 2.0 * np.pi / 128])
def test_sequential_solves(seq_lib, d, N, dh):  # noqa: F811
    n1, L = (9, 11, 12)[d], 4
    f = np.ones((n1, L, N))
    out = np.empty((n1 + 4, L, N))
    dp = ctypes.POINTER(ctypes.c_double)
    seq_lib.solve(N, d, L, n1, 256 if d == 0 else 128, dh, f.ctypes.data_as(dp), out.ctypes.data_as(dp))
    assert not out.any()


@pytest.mark.gpu
@pytest.mark.parametrize("bc", [0, 1])
@pytest.mark.parametrize("N", [12, 16, 33, 64, 77, 100, 128, 130, 301, 1000])
def test_single_operators(gpu_pkg, N, bc):
    """(Short lines in segments from 2^17 points on, between walls from 2^18.)"""
    planes = 400 if N <= 16 else 8
    bt = [gpu_pkg.PERIODIC_SOLVE] * 3
    bt[0] = bc
    op = gpu_pkg.Operator(gpu_pkg.make_config((N, 100, planes), (1.0, 1.0, 1.0), bc_type=tuple(bt)), 0)
    for kind in (1, 2):
        assert not op.apply_host(kind, np.full((100 * planes, N), 1.1)).any()
    op.close()
