"""solver1d's transforms and eliminations at their edges, through one flow step against the oracle.

The rows' complex length itot/2 and the y length jtot go through every
radix of the mixed-radix passes (composite ones up to 16, primes up to 61),
lengths of one to three passes and the register transforms of 32 to 256; the
eliminations through tiles of every width with a remainder of columns, few and
many levels, and columns too long for a tile.  Both sides work in FP64 and
differ by roundings: within 1e-10 of the largest value, as the other flow-step
tests ask.
"""
import numpy as np
import pytest

import oracle as O
from test_gpu_flow_solver import _ctx, _state

pytestmark = pytest.mark.gpu

MIXED = [(22, 13, 7), (38, 15, 5), (54, 23, 33), (118, 36, 6), (28, 45, 12), (150, 150, 99), (70, 77, 21),
         (96, 96, 64), (160, 60, 17), (40, 231, 11), (288, 100, 4), (36, 253, 5), (12, 59, 9), (180, 28, 150)]
REGISTER = [(64, 32, 40), (64, 64, 100), (12, 128, 65), (12, 256, 130), (512, 256, 33)]
LEVELS = [(12, 13, 10), (12, 15, 11), (12, 13, 128), (12, 15, 129), (12, 13, 188), (12, 13, 375), (12, 13, 783),
          (12, 12, 2347)]


@pytest.mark.parametrize("n", MIXED + REGISTER + LEVELS)
def test_flow_step_lengths(cuda, n):
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
