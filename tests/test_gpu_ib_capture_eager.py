"""Eager steps of the coupled solver beside a caller's captured pair of steps.

A captured pair reads and writes the buffers that held the velocity levels when it was captured, so an
even number of steps taken in any other way in between must leave every level where the pair finds it.
The kernels and their inputs are the same on every path: equal bit for bit to the eager loop, levels
included.
"""
import numpy as np
import pytest

from test_gpu_ib_capture import _levels, _solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("before", [1, 2, 3])
def test_eager_steps_between_replays_of_a_captured_pair(cuda, precision, before):
    import torch
    a, b = _solver(precision), _solver(precision)
    b.run(before)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=b.st):
        b.step()
        b.step()

    def replay():
        with torch.cuda.stream(b.st):
            g.replay()
        torch.cuda.synchronize()

    for between in (lambda: None, lambda: b.run(2), lambda: b.run(4), lambda: b.run(4, graph=True),
                    lambda: b.stage_times(2), lambda: b.run(6, graph=True)):
        between()
        replay()
    a.run(before + 2 + (2 + 2) + (4 + 2) + (4 + 2) + (2 + 2) + (6 + 2))
    for x, y in zip(_levels(a), _levels(b)):
        assert np.array_equal(x, y)
    del g
