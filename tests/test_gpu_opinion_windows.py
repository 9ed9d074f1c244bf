"""Bounded confidence on both sides of the rule that lets the first blocks of
every window of 2^13 rows run ahead: heavy rows in the first windows only, in
the last only, spread over all, and none -- every row bit-exact with the oracle,
for whole and broken windows, with and without hub rows among them."""
import numpy as np
import pytest

from oracle import models as om

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hub", [1536, 90])
@pytest.mark.parametrize("where", ["first", "last", "spread", "none"])
@pytest.mark.parametrize("n", [8191, 24_576 + 129, 140_001])
def test_heavy_rows(vh, n, where, hub):
    rng = np.random.default_rng(n + len(where))
    deg = rng.integers(0, 8, n)
    k = n // 100
    at = {"first": np.arange(k), "last": np.arange(n - k, n),
          "spread": rng.permutation(n)[:k], "none": np.arange(0)}[where]
    deg[at] = rng.integers(30, 120, at.size)  # slices below and above 96 slots
    to_row = rng.permutation(np.repeat(np.arange(n), deg))
    m = (vh.ModelTypes().register_agenttype("Opinion", [("x", "f64")], ":Immortal")
         .register_edgetype("Weight", [("w", "f64")], target="Opinion").create_model("Windows"))
    sim = vh.create_simulation(m)
    x = rng.random(n)
    ids = vh.add_agents(sim, "Opinion", n, x=x)
    frm, to = ids[rng.integers(0, n, to_row.size)], ids[to_row]
    w = 1.0 - rng.random(to_row.size)
    vh.add_edges(sim, "Weight", frm, to, w=w)
    vh.finish_init(sim)
    args = (["Opinion"], ["Opinion", "Weight"], ["Opinion"])
    params = [m["Weight"].index, 0.3, 0.5, 0.5, hub]
    exact = deg <= hub
    # hub rows sum up to 120 positive terms in another order: two sums of
    # (120 + 1) 2^-53 relative each, on both sides
    for host in (False, False, True):
        if host:
            got = vh.apply_host(sim, "bounded_confidence", *args, "Opinion", {"x": x},
                                params=params)["x"].copy()
        else:
            vh.apply_(sim, "bounded_confidence", *args, params=params)
            got = vh.read_agents(sim, "Opinion")[0]["x"].copy()
        ref = om.run_opinion(n, frm, to, w, x, 0.3, 1)
        np.testing.assert_array_equal(got[exact].view(np.uint64), ref[exact].view(np.uint64))
        np.testing.assert_allclose(got[~exact], ref[~exact], rtol=4 * 122 * 2.0 ** -53, atol=0)
        x = got
    sim.close()
