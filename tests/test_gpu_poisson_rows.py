"""Row transforms of the power-of-two lengths, whole and cut last blocks of rows, through one flow step.

A thread pairs the modes k and N - k of a row (N = itot/2 = 32 .. 256), the
middle one by itself; the last block's missing rows are left out.  The levels
are those at which the eliminations' sixteen segments hold one or two levels or
none.  Both sides work in FP64 and differ by roundings: within 1e-10 of the
largest value, as the other flow-step tests ask.
"""
import numpy as np
import pytest

import oracle as O
from test_gpu_flow_solver import _ctx, _state

pytestmark = pytest.mark.gpu


# lengths with odd composite factors above 10 (21, 27, 35, 45, 63), which are passes of several small radices
ODD = [(294, 108, 6), (126, 27, 5), (70, 63, 9), (90, 135, 4)]


@pytest.mark.parametrize("n", ODD)
def test_flow_step_odd_composites(cuda, n):
    test_flow_step_power_rows(cuda, n)


@pytest.mark.parametrize("n", [(64, 13, 5), (64, 16, 16), (128, 13, 15), (128, 8, 32), (256, 11, 16), (256, 8, 4),
                               (512, 12, 31), (512, 8, 18)])
def test_flow_step_power_rows(cuda, n):
    grid = (*n, 1 / 32, 1 / 24, 1 / 20)
    vel, p, f = _state(grid, sum(n))
    dt, rep = 1e-3, 0.8
    ref = O.flow_step(grid, dt, rep, *vel, p, *f)
    cs = _ctx(grid)
    cs.set_flow_params(rep)
    pg = p.copy()
    got = cs.flow_step(dt, *vel, pg, *f)
    for g, r in zip((*got, pg), ref):
        assert np.abs(g - r).max() <= 1e-10 * np.abs(r).max()
