"""A recorded CUDA graph is replayed without the library's knowledge: SIR steps
made directly before and after a replay that writes the states count their
neighbours from the states as they are, whatever transitions were recorded."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,degree", [(1000, 6), (40_000, 12), (120_000, 12)])
def test_replay_between_two_steps(vh, n, degree):
    import torch
    from vahana_gb300 import models
    a, b = (models.build_sir(n=n, degree=degree, seed=3) for _ in range(2))
    stream = torch.cuda.Stream()
    for r in (a, b):
        vh.finish_init(r.sim)
        vh.set_async(r.sim, True)
    vh.set_stream(a.sim, stream.cuda_stream)
    odd = ["Person"], ["Person"], ["Person"]
    a.step()  # (its tables are uploaded)
    b.step()
    vh.synchronize(a.sim)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        for _ in range(2):  # agents of odd number are infected, the others susceptible
            vh.apply_(a.sim, "set_field", *odd, params=[0, 1, 0])
    for _ in range(2):  # (as many transitions)
        vh.apply_(b.sim, "keep", *odd)
    # the recording swapped the columns without writing them
    same = dict(zip(("state", "days"), vh.read_agents(b.sim, "Person")[0].values()))
    vh.write_agents(a.sim, "Person", **same)
    for _ in range(2):
        a.step()
        b.step()
    vh.synchronize(a.sim)
    graph.replay()
    torch.cuda.synchronize()
    vh.write_agents(b.sim, "Person", state=(np.arange(1, n + 1) % 2).astype(np.uint8))
    a.step()
    b.step()
    for x, y in zip(vh.read_agents(a.sim, "Person")[0].values(),
                    vh.read_agents(b.sim, "Person")[0].values()):
        np.testing.assert_array_equal(x, y)
    for r in (a, b):
        r.close()
