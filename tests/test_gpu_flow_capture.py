"""Flow steps captured in CUDA graphs beside eager ones with other time steps.

The solver keeps the pivots of its eliminations for the shift Rep / dt that they were made with.  A graph
must find those of its own shift whatever was solved in between, and an eager step must not take what a
replay has left: every result within 1e-10 of the oracle's step with the same dt, as the other flow-step
tests ask.
"""
import numpy as np
import pytest

import oracle as O
from suguru_b200.coupling import CouplingStep
from test_gpu_flow_solver import GRID, _state

pytestmark = pytest.mark.gpu

REP = 0.7


class Case:
    def __init__(self, torch):
        self.torch = torch
        self.vel, self.p, self.f = _state(GRID, 12)
        self.st = torch.cuda.Stream()
        self.cs = CouplingStep(GRID, np.array([3], np.int32), np.array([0.1]), mem="device",
                               stream=self.st.cuda_stream, async_=True)
        self.cs.set_flow_params(REP)
        dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
        self.d = [dev(a) for a in (*self.vel, *self.f)]
        self.p0, self.pd = dev(self.p), dev(self.p)
        self.out = [torch.zeros_like(self.pd) for _ in range(3)]
        self.ref = {}

    def call(self, dt):
        self.pd.copy_(self.p0)
        self.cs.flow_step(dt, *self.d[:6], self.pd, *self.d[6:], out=self.out)

    def eager(self, dt):
        with self.torch.cuda.stream(self.st):
            self.call(dt)
        self.check(dt)

    def capture(self, dt):
        g = self.torch.cuda.CUDAGraph()
        with self.torch.cuda.graph(g, stream=self.st):
            self.call(dt)
        return lambda: self.replay(g, dt)

    def replay(self, g, dt):
        for o in self.out:
            o.zero_()
        self.torch.cuda.synchronize()
        with self.torch.cuda.stream(self.st):
            g.replay()
        self.check(dt)

    def check(self, dt):
        self.torch.cuda.synchronize()
        if dt not in self.ref:
            self.ref[dt] = O.flow_step(GRID, dt, REP, *self.vel, self.p, *self.f)
        for g, r in zip((*self.out, self.pd), self.ref[dt]):
            assert np.abs(g.cpu().numpy() - r).max() <= 1e-10 * np.abs(r).max(), dt


def test_graph_of_a_step_already_taken(cuda):
    c = Case(cuda)
    c.eager(1e-3)
    g = c.capture(1e-3)
    c.eager(3e-3)
    g()
    c.eager(3e-3)
    g()
    c.eager(1e-3)


def test_graph_of_a_step_not_taken_before(cuda):
    c = Case(cuda)
    c.eager(1e-3)
    g = c.capture(2e-3)
    c.eager(3e-3)
    g()
    c.eager(3e-3)
    c.eager(2e-3)
    g()
    c.eager(3e-3)


def test_capture_before_any_step(cuda):
    c = Case(cuda)
    g = c.capture(1e-3)
    c.eager(3e-3)
    g()
    c.eager(3e-3)
    c.eager(1e-3)
    g()


@pytest.mark.parametrize("taken", [True, False])
def test_many_graphs(cuda, taken):
    c = Case(cuda)
    c.eager(9e-3)
    dts = [1e-3 * (1 + q) for q in range(6)]
    gs = []
    for dt in dts:
        if taken:
            c.eager(dt)
        gs.append(c.capture(dt))
    for order in (range(6), (5, 0, 3, 3, 1, 4, 2)):
        for q in order:
            gs[q]()
            if q % 2:
                c.eager(7e-3)
    for dt in (*dts, 9e-3):
        c.eager(dt)
    for g in gs:
        g()


def test_indicator_captured_before_any_call(cuda):
    """The indicator's Neumann rows have one table: a graph of the first call and eager calls around it agree."""
    torch = cuda
    from suguru_b200 import workloads as W
    d = GRID[3]
    R = 5.0 * d
    x, y, z = W.capsule_points(9, R, (1.0, 0.8, 0.6))
    _, n, a = O.complagrforces(9, R, x, y, z)
    res = []
    for order in ("eager", "graph first"):
        st = torch.cuda.Stream()
        cs = CouplingStep(GRID, np.array([9], np.int32), np.array([R]), mem="device", stream=st.cuda_stream, async_=True)
        cs.set_indicator_params()
        dev = [torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (x, y, z, *n, a)]
        out = [torch.zeros((GRID[2] + 2, GRID[1] + 2, GRID[0] + 2), dtype=torch.float64, device="cuda") for _ in range(2)]
        torch.cuda.synchronize()
        if order == "graph first":
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=st):
                cs.indicator(*dev, out=out)
        else:
            g = None
        for run in (lambda: cs.indicator(*dev, out=out),) + ((g.replay, lambda: cs.indicator(*dev, out=out)) if g else ()):
            for o in out:
                o.zero_()
            torch.cuda.synchronize()
            with torch.cuda.stream(st):
                run()
            torch.cuda.synchronize()
            res.append([o.cpu().numpy() for o in out])
    for r in res[1:]:
        for p, q in zip(r, res[0]):
            assert np.array_equal(p, q)
