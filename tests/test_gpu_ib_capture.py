"""The coupled solver's buffers under captures: three rotate in an eager loop and in run()'s own graph of three
steps, a caller's own capture of a pair of steps finds every buffer back in its place.  The kernels and their
inputs are the same on every path, so the states are equal bit for bit, the velocity levels included.
"""
import numpy as np
import pytest

import oracle as O
from suguru_b200 import workloads as W
from suguru_b200.ib_solver import IBSolver
from test_gpu_ib_solver import IND

pytestmark = pytest.mark.gpu


def _solver(precision):
    wl = W.small_config()
    u0 = list(wl.velocity())
    O.bounduvw(*u0)
    return IBSolver(wl, 0.01 * wl.grid[3], 0.5, u0, indicator=IND, precision=precision)


def _levels(s):
    s.torch.cuda.synchronize()
    st = s.state()
    return [*st["X"], *st["u"], st["p"], *st["force"], *(t.cpu().numpy() for t in (*s.uo, *s.uoo))]


@pytest.mark.parametrize("precision,steps,how", [("fp64", 2, "run"), ("fp64", 8, "run"), ("fp64", 6, "pair"),
                                                 ("mixed", 6, "pair"), ("mixed", 5, "run")])
def test_captured_steps_equal_the_eager_loop(cuda, precision, steps, how):
    import torch
    a, b = _solver(precision), _solver(precision)
    a.run(steps)
    if how == "run":
        b.run(steps, graph=True)
    else:
        b.run(2)  # first launches outside the capture
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=b.st):
            b.step()
            b.step()
        with torch.cuda.stream(b.st):
            for _ in range((steps - 2) // 2):
                g.replay()
        torch.cuda.synchronize()
        del g
    for x, y in zip(_levels(a), _levels(b)):
        assert np.array_equal(x, y)
