"""The chained FP64 contractions at the edges of their tiles, against the oracle.

A tile holds 32 data rows, six or eight per capsule: one capsule, tiles that
end inside a capsule and on its last row, more than one tile; degrees with
even and odd row lengths, below and above the 16 and 32 lanes of a row.
Force, normals and area within 1e-10, the tolerance of the FP64 parity tests.
"""
import numpy as np
import pytest

import oracle as O
from suguru_b200 import workloads as W
from suguru_b200.coupling import CouplingStep

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("degree", [2, 3, 7, 8, 15, 16, 17, 31])
@pytest.mark.parametrize("ncap", [1, 4, 5, 11])
def test_force(cuda, degree, ncap):
    rng = np.random.default_rng(100 * degree + ncap)
    dx = 1.0 / 16
    R = 4.0 * dx
    pts = []
    for _ in range(ncap):
        ca, cb = W.random_shape(rng, degree, 0.05 * R)
        pts.append(W.capsule_points(degree, R, rng.uniform(1.0, 1.5, 3), ca, cb))
    x, y, z = (np.concatenate([p[c] for p in pts]) for c in range(3))
    cs = CouplingStep((48, 40, 40, dx, dx, dx), np.full(ncap, degree, np.int32), np.full(ncap, R))
    f, n, a = cs.complagrforces(x, y, z)
    m = W.npts_of(degree)
    for k in range(ncap):
        s = slice(k * m, (k + 1) * m)
        rf, rn, ra = O.complagrforces(degree, R, x[s], y[s], z[s])
        rel = lambda g, r: np.linalg.norm(g - r) / np.linalg.norm(r)
        assert rel(np.stack([q[s] for q in f]), rf) <= 1e-10
        assert rel(np.stack([q[s] for q in n]), rn) <= 1e-10
        assert rel(a[s], ra) <= 1e-10
