"""The bounded-confidence gather's blocks for long slices and long hub rows
(k_opinion_long) against the oracle, at the in-degrees where rounds, slices
and the choice of the block begin and end: rows up to the hub threshold
bit-exact, rows above it within 1e-12 relative, for weights on and off the
2^-53 grid; the same step through the host exchange and through the
serving-sized launch is covered by their own tests."""
import numpy as np
import pytest

from oracle import models as om

pytestmark = pytest.mark.gpu

DEGREES = [0, 1, 2, 31, 32, 33, 63, 64, 65, 95, 96, 97, 127, 128, 129, 160, 1023, 1024, 1025,
           1535, 1536, 1537, 3071, 3072, 3073, 4096, 4129, 9000]


@pytest.mark.parametrize("grid", [True, False])
@pytest.mark.parametrize("hub", [1536, 64, 4294967295])
@pytest.mark.parametrize("n", [61, 8192, 8211])
def test_long_rows(vh, n, hub, grid):
    rng = np.random.default_rng(n + hub % 1000)
    deg = np.full(n, 3)
    at = rng.permutation(n)[:2 * len(DEGREES)]
    deg[at] = np.resize(DEGREES, at.size)
    to_row = rng.permutation(np.repeat(np.arange(n), deg))
    E = to_row.size
    m = (vh.ModelTypes().register_agenttype("Opinion", [("x", "f64")], ":Immortal")
         .register_edgetype("Weight", [("w", "f64")], target="Opinion").create_model("Long"))
    sim = vh.create_simulation(m)
    x0 = rng.random(n)
    ids = vh.add_agents(sim, "Opinion", n, x=x0)
    frm, to = ids[rng.integers(0, n, E)], ids[to_row]
    w = 1.0 - rng.random(E) if grid else rng.random(E) * 0.7 + 1e-3
    vh.add_edges(sim, "Weight", frm, to, w=w)
    vh.finish_init(sim)
    exact = deg <= hub
    x = x0
    for _ in range(3):
        vh.apply_(sim, "bounded_confidence", ["Opinion"], ["Opinion", "Weight"], ["Opinion"],
                  params=[m["Weight"].index, 0.3, 0.5, 0.5, hub])
        ref = om.run_opinion(n, frm, to, w, x, 0.3, 1)  # from the library's own last state
        x = vh.read_agents(sim, "Opinion")[0]["x"].copy()
        np.testing.assert_array_equal(x[exact].view(np.uint64), ref[exact].view(np.uint64))
        np.testing.assert_allclose(x[~exact], ref[~exact], rtol=1e-12, atol=0)
    # the host exchange reports the long blocks with the hub rows
    out = vh.apply_host(sim, "bounded_confidence", ["Opinion"], ["Opinion", "Weight"],
                        ["Opinion"], "Opinion", {"x": x},
                        params=[m["Weight"].index, 0.3, 0.5, 0.5, hub])["x"]
    ref = om.run_opinion(n, frm, to, w, x, 0.3, 1)
    np.testing.assert_array_equal(out[exact].view(np.uint64), ref[exact].view(np.uint64))
    np.testing.assert_allclose(out[~exact], ref[~exact], rtol=1e-12, atol=0)
    sim.close()
