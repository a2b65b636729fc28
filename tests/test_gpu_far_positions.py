"""Positions far outside the domain, as a run that has blown up leaves them.

Up to 2^52 cells they wrap exactly; beyond that the cell they are given means nothing but lies in the
grid.  The other points' velocities are those of the call without them, bit for bit; with zero forces they
change the field by no more than the fixed-point step, which follows a tile's entries (1e-12, mixed 1e-6).
"""
import numpy as np
import pytest

from suguru_b200 import workloads as W
from suguru_b200.coupling import CouplingStep
from util import rel_l2

pytestmark = pytest.mark.gpu

FAR = [2.0 ** 51 + 7, -2.0 ** 51 - 5, 2.0 ** 56 + 2.0 ** 20, -3.1e17, 2.7e18, -1e19, 1e22, -4e40, 1e300]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("grid", [(64, 48, 40), (100, 43, 37)])
def test_other_points_are_untouched(cuda, precision, grid):
    wl = W.small_config(grid=grid)
    dt = np.float64 if precision == "fp64" else np.float32
    cs = CouplingStep(wl.grid, wl.degree, wl.radius, precision=precision)
    rng = np.random.default_rng(2)
    far = rng.choice(wl.npts, 6 * len(FAR), replace=False)
    f = rng.normal(size=(3, wl.npts)).astype(dt)
    f[:, far] = 0
    area = rng.uniform(0.5, 1.0, wl.npts).astype(dt)
    u = [a.astype(dt) for a in wl.velocity()]
    near = [a.copy() for a in (wl.x, wl.y, wl.z)]
    away = [a.copy() for a in near]
    for q, p in enumerate(far):
        for c in ([0], [1], [2], [0, 1], [1, 2], [0, 1, 2])[q % 6]:
            away[c][p] = FAR[q // 6] * wl.grid[3 + c]
    others = np.setdiff1d(np.arange(wl.npts), far)
    for a, b in zip(cs.eulr2lagr(*u, *near), cs.eulr2lagr(*u, *away)):
        assert np.array_equal(a[others], b[others])
    for a, b in zip(cs.lagr2eulr(*near, *f, area), cs.lagr2eulr(*away, *f, area)):
        assert rel_l2(b, a) <= (1e-12 if precision == "fp64" else 1e-6)
