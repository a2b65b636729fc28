"""The FP64 spread's fixed-point step against the forces of the tile, where it is easiest to lose bits.

All points of a tile (but one, in the dense tiles) sit at one place with one force, so that every
contribution to a cell is rounded alike and the roundings add up instead of averaging out.  With M the largest magnitude F A / dV of a
tile's n <= 4096 points, the step is at most 2^e / 2^56, 2^e the power of two above n M; a cell's sum of n
equal contributions is off from n times the oracle's field of one point by at most n / 2 steps, and by 4
roundings in 64 bits of a contribution below 0.3 M on either side.
"""
import math

import numpy as np
import pytest

import oracle as O
from suguru_b200.coupling import CouplingStep

pytestmark = pytest.mark.gpu

GRID = (64, 32, 16, 1 / 16, 1 / 16, 1 / 16)
D = GRID[3]
AT = (8.3, 4.4, 2.2)  # in the first tile


def points(n, m, big):
    """n points of magnitude m at one place of the first tile and one of magnitude big far from them in it;
    the capsules' other points in another tile, without force."""
    degree = np.full(-(-(n + 1) // 3872), 21, np.int32)
    npts = 3872 * degree.size
    k = np.arange(npts)
    pos = [D * np.where(k < n, AT[0], 44.5), np.full(npts, D * AT[1]), np.full(npts, D * AT[2])]
    f = np.where(k < n, m, 0.0)
    if big:
        pos[0][n], f[n] = D * 22.7, big
    return degree, pos, [f, -f, 0.5 * f], np.full(npts, D ** 3)  # F A / dV = F


def errors(n, m, big=0.0):
    """Largest difference around the n points from n times the field of one, per component."""
    degree, pos, f, area = points(n, m, big)
    one = O.spread(GRID, *(np.array([D * a]) for a in AT), *(np.array([q[0]]) for q in f), area[:1])
    cs = CouplingStep(GRID, degree, np.full(degree.size, 0.3))
    got = cs.lagr2eulr(*pos, *f, area)
    near = np.s_[:, :, :17]
    return [np.abs(g[near] - n * r[near]).max() for g, r in zip(got, one)]


def bound(n, step, m):
    return n * (step / 2 + 8 * 0.3 * m * 2.0 ** -53)


@pytest.mark.parametrize("n", [1, 3, 7, 60, 127, 128, 130, 136, 140, 146, 150, 153, 200, 255, 256, 400, 1000, 4000])
def test_even_tile(cuda, n):
    for m in np.random.default_rng(n).uniform(0.835, 0.95, 12):
        for err, s in zip(errors(n, m), (1.0, 1.0, 0.5)):
            assert err <= bound(n, math.ldexp(1.0, math.frexp(n * s * m)[1] - 56), s * m), m


@pytest.mark.parametrize("n", [4095, 4096, 5000, 20000])
@pytest.mark.parametrize("ratio", [1.0, 1e-2, 1e-4, 1e-6])
def test_dense_tile_with_one_large_force(cuda, n, ratio):
    """Above 4096 entries: 2^-56 of 0.3 times the sum of their magnitudes, each rounded up to 2^-12 of the
    power of two above the largest, the product rounded up to a power of two."""
    for m in ratio * np.random.default_rng(n).uniform(0.5, 1.0, 4):
        for err, s in zip(errors(n, m, big=1.0), (1.0, 1.0, 0.5)):
            unit = math.ldexp(1.0, math.frexp(s)[1] - 12)
            total = s + n * math.ceil(s * m / unit) * unit
            top = 0.3 * total if n + 1 > 4096 else (n + 1) * s
            assert err <= bound(n, math.ldexp(1.0, math.frexp(top)[1] - 56), s * m), m
