"""read_edges on both sides of the sizes from which rows and sources are widened
on the device (2^14): row pointers, agent ids of one source type and of two, and
payload, exactly as they were added."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("n,ne", [(3, 16_383), (3, 16_384), (3, 16_385), (16_382, 40),
                                  (16_383, 40), (16_384, 16_385), (1, 0), (20_000, 0)])
def test_sizes(vh, n, ne, mixed):
    rng = np.random.default_rng(n + ne)
    m = (vh.ModelTypes().register_agenttype("P", [], ":Immortal").register_agenttype("Q", [])
         .register_edgetype("E", [("w", "i32")]).register_edgetype("S", [], ":Stateless")
         .register_edgetype("N", [], ":NumEdgesOnly").create_model("Sizes"))
    sim = vh.create_simulation(m)
    p, q = vh.add_agents(sim, "P", n), vh.add_agents(sim, "Q", 5)
    frm = rng.choice(np.concatenate([p, q]) if mixed else p, ne)
    row = np.sort(rng.integers(0, n, ne))
    w = rng.integers(-9, 9, ne).astype(np.int32)
    if ne:
        vh.add_edges(sim, "E", frm, p[row], w=w)
        vh.add_edges(sim, "S", frm, p[row])
        vh.add_edges(sim, "N", frm, p[row])
    vh.finish_init(sim)
    rp = np.concatenate([[0], np.cumsum(np.bincount(row, minlength=n))])
    for E in "ESN":
        got_rp, got_from, cols = vh.read_edges(sim, E, "P")
        np.testing.assert_array_equal(got_rp, rp[:got_rp.size])
        assert got_rp.size == n + 1 or ne == 0
        np.testing.assert_array_equal(got_from[:ne], 0 if E == "N" else frm)
        if E == "E":
            np.testing.assert_array_equal(cols["w"][:ne], w)
    sim.close()
