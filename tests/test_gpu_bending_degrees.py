"""The bending kernels at the ends of their degree range, against the oracle.

Degrees 2 and 3 (many rows per chunk), odd and even row lengths, a last m
pair of one, and 31 (the most shared memory), beside each other; per capsule
within the tolerances of the bending tests: FP64 1e-10, mixed 1e-4.
"""
import numpy as np
import pytest

import oracle as O
from suguru_b200 import workloads as W
from suguru_b200.coupling import CouplingStep

pytestmark = pytest.mark.gpu

DEGREES = [2, 3, 8, 15, 16, 31]


@pytest.mark.parametrize("precision, tol", [("fp64", 1e-10), ("mixed", 1e-4)])
@pytest.mark.parametrize("law", [0, 1])
def test_degrees(cuda, precision, tol, law):
    rng = np.random.default_rng(5 + law)
    dx = 1.0 / 16
    pts, radius = [], []
    for L in DEGREES:
        R = (3.0 + 0.2 * L) * dx
        # the whole spectrum of the degree: a smoother shape's force is so small beside the rounding
        # of its fourth derivatives that the oracle itself is off by 1e-9 at degree 31
        ca, cb = W.random_shape(rng, L, 0.03 * R)
        pts.append(W.capsule_points(L, R, rng.uniform(1.2, 1.6, 3), ca, cb))
        radius.append(R)
    x, y, z = (np.concatenate([p[c] for p in pts]) for c in range(3))
    radius = np.array(radius)
    eb = 0.3 * radius ** 2
    cs = CouplingStep((48, 48, 48, dx, dx, dx), np.array(DEGREES, np.int32), radius, precision=precision)
    cs.set_capsule_law([law] * len(DEGREES))
    cs.set_capsule_bending(eb)
    f, n, a = cs.complagrforces(x, y, z)
    off = 0
    for k, L in enumerate(DEGREES):
        s = slice(off, off + W.npts_of(L))
        off = s.stop
        rf, rn, ra = O.complagrforces(L, radius[k], x[s], y[s], z[s], law=law, eb=eb[k])
        rel = lambda g, r: np.linalg.norm(g - r) / np.linalg.norm(r)
        assert rel(np.stack([q[s] for q in f]), rf) <= tol, L
        assert rel(np.stack([q[s] for q in n]), rn) <= tol, L
        assert rel(a[s], ra) <= tol, L
