"""The SIR step (src/Vahana.jl's apply! over Person and Contact) whose neighbours
come from the infected mask of the step before, against the same steps with
the state bytes (a column's device pointer was handed out: no mask is used):
bit-identical states and days, for populations at the ends of a mask word and of
a block, rows longer than a batch of loads, both sides of the rule that
prefetches the rows, and with everything that may come between two steps."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def build(vh, n, degree, seed):
    from vahana_gb300 import models
    run = models.build_sir(n=n, degree=degree, seed=seed)
    vh.finish_init(run.sim)
    return run


def same(vh, a, b):
    for x, y in zip(vh.read_agents(a.sim, "Person")[0].values(),
                    vh.read_agents(b.sim, "Person")[0].values()):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("n,degree", [(2, 1), (31, 3), (32, 3), (33, 20), (255, 5), (256, 5),
                                      (257, 40), (8191, 7), (40_000, 30), (150_000, 6),
                                      (150_000, 9)])
@pytest.mark.parametrize("queued", [False, True])
def test_mask(vh, n, degree, queued):
    from vahana_gb300._lib import check, lib
    rng = np.random.default_rng(n)
    a, b = build(vh, n, degree, 7), build(vh, n, degree, 7)
    p = C.c_void_p()
    check(lib().vg_agent_field_device_ptr(b.sim._h, b.sim.T("Person").index, 0, C.byref(p)))
    for r in (a, b):
        vh.set_async(r.sim, queued)

    def both(f):
        for r in (a, b):
            f(r)

    def steps(k):
        both(lambda r: [r.step() for _ in range(k)])

    steps(1)
    steps(9)
    same(vh, a, b)
    steps(3)
    new = {"state": rng.choice([0, 0, 0, 1, 2], n).astype(np.uint8),
           "days": rng.integers(0, 3, n).astype(np.int32)}
    both(lambda r: vh.write_agents(r.sim, "Person", **new))   # between two steps
    steps(4)
    both(lambda r: vh.synchronize(r.sim))
    steps(2)
    both(lambda r: vh.mapreduce(r.sim, "state", "max", "Person"))
    steps(2)
    same(vh, a, b)
    # another transition writes the states (kind 1: the agent's number is odd)
    both(lambda r: vh.apply_(r.sim, "set_field", ["Person"], ["Person"], ["Person"],
                             params=[0, 1, 0]))
    steps(5)
    same(vh, a, b)
    # a step that fails leaves the states, and the mask must not run ahead
    for r in (a, b):
        with pytest.raises(Exception):
            vh.apply_(r.sim, "sir", ["Person"], ["Person"], ["Person"], params=[])
    steps(3)
    same(vh, a, b)
    # a copy and a snapshot start without a mask
    c = vh.copy_simulation(a.sim)
    steps(1)
    same(vh, a, b)
    vh.write_agents(a.sim, "Person", **dict(zip(("state", "days"),
                                                vh.read_agents(c, "Person")[0].values())))
    vh.write_agents(b.sim, "Person", **dict(zip(("state", "days"),
                                                vh.read_agents(c, "Person")[0].values())))
    steps(2)
    same(vh, a, b)


def test_recorded_steps(vh):
    """Two steps recorded in a CUDA graph and replayed after the states were
    written, then steps again: as the same steps made directly."""
    import torch
    n = 40_000
    rng = np.random.default_rng(5)
    a, b = build(vh, n, 12, 9), build(vh, n, 12, 9)
    stream = torch.cuda.Stream()
    vh.set_stream(a.sim, stream.cuda_stream)
    for r in (a, b):
        vh.set_async(r.sim, True)
        for _ in range(4):
            r.step()
        vh.synchronize(r.sim)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        a.step()
        a.step()
    new = {"state": rng.choice([0, 0, 0, 1, 2], n).astype(np.uint8),
           "days": rng.integers(0, 3, n).astype(np.int32)}
    for r in (a, b):
        vh.write_agents(r.sim, "Person", **new)
        vh.synchronize(r.sim)
    graph.replay()
    torch.cuda.synchronize()
    b.step()
    b.step()
    same(vh, a, b)
    for r in (a, b):
        r.step()
        r.step()
    same(vh, a, b)
