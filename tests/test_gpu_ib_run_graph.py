"""run(graph=True) of the coupled solver takes its steps from graphs, whatever their number, and they are the
eager loop's, velocity levels included, bit for bit.
"""
import numpy as np
import pytest

from test_gpu_ib_capture import _levels, _solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps", [1, 2, 3, 4, 5, 8])
@pytest.mark.parametrize("captured", [False, True])
def test_every_step_is_replayed(cuda, steps, captured, monkeypatch):
    import torch
    a, b = _solver("fp64"), _solver("fp64")
    a.run(1 + steps)
    b.run(1)
    if captured:  # a caller's own pair, not replayed
        own = torch.cuda.CUDAGraph()
        with torch.cuda.graph(own, stream=b.st):
            b.step()
            b.step()
    eager = []
    step = b.step

    def counted(*args, **kw):
        if not torch.cuda.is_current_stream_capturing():
            eager.append(1)
        return step(*args, **kw)

    monkeypatch.setattr(b, "step", counted)
    b.run(steps, graph=True)
    assert len(eager) == (1 if steps == 1 else 0)
    for x, y in zip(_levels(a), _levels(b)):
        assert np.array_equal(x, y)
