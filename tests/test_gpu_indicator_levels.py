"""The indicator on columns of every length that the elimination treats differently.

Tiles of sixteen, eight and four columns in shared memory (to 198, 396 and 2338 levels), sweeps over
global memory beyond, and as many levels as launches with a block row per level had room for; on narrow
planes with a remainder of columns.  Neumann rows, whose mean mode has an exactly zero pivot.  One capsule, radial
normals; indic, visc and the centrifugal terms within 1e-10 of their largest value, the cells within ten
times the tolerance of a threshold left out, as the other indicator tests ask.
"""
import numpy as np
import pytest

import oracle as O
from suguru_b200 import workloads as W
from suguru_b200.coupling import CouplingStep
from test_gpu_indicator import PARAMS

pytestmark = pytest.mark.gpu

TOL = 1e-10


@pytest.mark.parametrize("n", [(16, 13, 198), (16, 13, 199), (16, 13, 396), (16, 13, 397), (16, 13, 2338),
                               (16, 13, 2339), (8, 8, 65534)])
def test_levels(cuda, n):
    d = 1 / 16
    grid = (*n, d, d, d)
    R = 3.1 * d
    rng = np.random.default_rng(sum(n))
    ca, cb = W.random_shape(rng, 9, 0.03 * R)
    x, y, z = W.capsule_points(9, R, (n[0] * d / 2, n[1] * d / 2, 0.4 * n[2] * d), ca, cb)
    _, nrm, area = O.complagrforces(9, R, x, y, z)
    shape = (n[2] + 2, n[1] + 2, n[0] + 2)
    fy0, fz0 = rng.normal(size=shape), rng.normal(size=shape)
    ref = O.indicator(grid, x, y, z, *nrm, area, fy=fy0, fz=fz0, **PARAMS)
    cs = CouplingStep(grid, np.array([9], np.int32), np.array([R]))
    cs.set_indicator_params(**PARAMS)
    fy, fz = fy0.copy(), fz0.copy()
    indic, visc = cs.indicator(x, y, z, *nrm, area, fy=fy, fz=fz)
    assert ref["indic"].max() == 1.0
    kt, q = n[2], n[2] // 4
    raw = np.zeros(shape)
    raw[1:kt - q + 1, 1:-1, 1:-1] = ref["indi"][1 + q:kt + 1, 1:-1, 1:-1]
    O.boundp(raw)
    near = (np.abs(raw - 0.01) < 10 * TOL) | (np.abs(raw - 0.9) < 10 * TOL)
    near_y, near_z = near.copy(), near.copy()
    near_y[:, :-1] |= near[:, 1:]
    near_z[:-1] |= near[1:]
    for g, r, skip in ((indic, ref["indic"], near), (visc, ref["visc"], near), (fy, ref["fy"], near_y),
                       (fz, ref["fz"], near_z)):
        assert np.abs(g - r)[~skip].max() <= TOL * np.abs(r).max()
    assert near.mean() < 1e-3
