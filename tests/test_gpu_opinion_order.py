"""The order in which a bounded-confidence launch takes its slice blocks when
the first blocks of every window of 2^13 rows run ahead: every row written
once and bit-exact with the oracle, for one to five full windows, with and
without a part of another and of a block, resident and through the host
exchange (whose ranges of rows are reported as they finish)."""
import numpy as np
import pytest

from oracle import models as om

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8192, 8193, 16_384, 16_384 + 127, 24_576 + 129, 40_960, 40_960 + 8191])
@pytest.mark.parametrize("longest", [96, 700])
def test_every_row_once(vh, n, longest):
    rng = np.random.default_rng(n + longest)
    deg = rng.integers(0, 6, n)
    deg[rng.permutation(n)[:n // 500]] = rng.integers(20, 97, n // 500)
    deg[rng.integers(0, n)] = longest  # a slice with a block of its own
    to_row = rng.permutation(np.repeat(np.arange(n), deg))
    m = (vh.ModelTypes().register_agenttype("Opinion", [("x", "f64")], ":Immortal")
         .register_edgetype("Weight", [("w", "f64")], target="Opinion").create_model("Order"))
    sim = vh.create_simulation(m)
    x = rng.random(n)
    ids = vh.add_agents(sim, "Opinion", n, x=x)
    frm, to = ids[rng.integers(0, n, to_row.size)], ids[to_row]
    w = 1.0 - rng.random(to_row.size)
    vh.add_edges(sim, "Weight", frm, to, w=w)
    vh.finish_init(sim)
    args = (["Opinion"], ["Opinion", "Weight"], ["Opinion"])
    params = [m["Weight"].index, 0.3, 0.5, 0.5, 4294967295]
    for _ in range(3):
        vh.apply_(sim, "bounded_confidence", *args, params=params)
    x = om.run_opinion(n, frm, to, w, x, 0.3, 3)
    np.testing.assert_array_equal(vh.read_agents(sim, "Opinion")[0]["x"].view(np.uint64),
                                  x.view(np.uint64))
    for _ in range(2):
        out = vh.apply_host(sim, "bounded_confidence", *args, "Opinion", {"x": x},
                            params=params)["x"]
        x = om.run_opinion(n, frm, to, w, x, 0.3, 1)
        np.testing.assert_array_equal(out.view(np.uint64), x.view(np.uint64))
