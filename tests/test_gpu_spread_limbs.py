"""The FP64 spread's two-limb sums at the edges of a pass, against the oracle.

The force points are gathered around one cell, so that one tile's entries are
one, a whole pass (255 entries), one more or less, a power of two, several
passes or more than 2^15, with forces of mixed sign whose magnitudes span many
orders, all one sign, or tiny.  The limbs' step is 2^-48 of the largest
magnitude or finer, so a cell's sum of n contributions is off by at most
n 2^-48 of it: 1e-12 in the relative 2-norm, as the other spread tests ask.
"""
import numpy as np
import pytest

import oracle as O
from suguru_b200.coupling import CouplingStep

pytestmark = pytest.mark.gpu

GRID = (64, 32, 16, 1 / 16, 1 / 16, 1 / 16)


@pytest.mark.parametrize("n", [1, 2, 31, 127, 128, 254, 255, 256, 511, 1020, 4097, 40000])
@pytest.mark.parametrize("kind", ["mixed", "same", "tiny"])
def test_entry_counts(cuda, n, kind):
    degree = np.full(max(1, -(-n // 3872)), 21, np.int32)
    npts = 3872 * degree.size
    rng = np.random.default_rng(n)
    d = GRID[3]
    # n points inside cells 12..13, 12..13, 6..7 (one tile), the others far away in x
    x = np.where(np.arange(npts) < n, 12.5, 44.5)
    pos = [d * (c + rng.uniform(0.0, 1.0, npts)) for c in (x, 12.5, 6.0)]
    if kind == "mixed":
        f = [rng.normal(size=npts) * 10.0 ** rng.uniform(-6, 2, npts) for _ in range(3)]
    elif kind == "same":
        f = [np.full(npts, s) for s in (1.0, -1.0, 0.75)]
    else:
        f = [1e-30 * rng.normal(size=npts) for _ in range(3)]
    area = rng.uniform(0.5, 1.0, npts) * d * d
    ref = O.spread(GRID, *pos, *f, area)
    cs = CouplingStep(GRID, degree, np.full(degree.size, 0.3))
    got = cs.lagr2eulr(*pos, *f, area)
    again = cs.lagr2eulr(*pos, *f, area)
    for g, a, r in zip(got, again, ref):
        assert np.linalg.norm(g - r) <= 1e-12 * np.linalg.norm(r)
        assert np.array_equal(g, a)
