"""Bounded confidence where no row is left for the slices: every agent's row is
a hub, and those of 3072 in-edges or more take a block of the long launch each
(the complete graph of a few thousand agents is such a graph).  Resident,
through the host exchange, and as the only job of a serving tick."""
import numpy as np
import pytest

from oracle import models as om

pytestmark = pytest.mark.gpu

# Terms are positive, so n additions and the n products under them are off by
# at most (n + 1) 2^-53 relative, in the library's order and in the oracle's:
# for n <= 4100 a quotient of two such sums differs by less than 4 (n + 2) 2^-53
RTOL = 4 * 4102 * 2.0 ** -53


def run(vh, n, frm, to, hub):
    rng = np.random.default_rng(n)
    m = (vh.ModelTypes().register_agenttype("Opinion", [("x", "f64")], ":Immortal")
         .register_edgetype("Weight", [("w", "f64")], target="Opinion").create_model("Hubs"))
    sim = vh.create_simulation(m)
    x = rng.random(n)
    ids = vh.add_agents(sim, "Opinion", n, x=x)
    w = 1.0 - rng.random(frm.size)
    vh.add_edges(sim, "Weight", ids[frm], ids[to], w=w)
    vh.finish_init(sim)
    args = ["Opinion"], ["Opinion", "Weight"], ["Opinion"]
    params = [m["Weight"].index, 0.3, 0.5, 0.5, hub]
    for k in range(4):
        if k < 2:
            vh.apply_(sim, "bounded_confidence", *args, params=params)
            got = vh.read_agents(sim, "Opinion")[0]["x"].copy()
        else:  # the host exchange
            got = vh.apply_host(sim, "bounded_confidence", *args, "Opinion", {"x": x},
                                params=params)["x"].copy()
        ref = om.run_opinion(n, ids[frm], ids[to], w, x, 0.3, 1)
        np.testing.assert_allclose(got, ref, rtol=RTOL, atol=0)
        assert n < 30 or not np.array_equal(got, x)
        x = got
    sim.close()


def test_complete_graph(vh):
    n = 3200
    frm, to = np.divmod(np.arange(n * n), n)
    away = frm != to
    run(vh, n, frm[away], to[away], 1536)


@pytest.mark.parametrize("hub", [0, 1536])
@pytest.mark.parametrize("degrees", [[3072], [3073, 4100], [3072] * 33, [3071, 3072, 3073],
                                     [1537, 3071], [1537, 4000] * 20])
def test_hubs_only(vh, degrees, hub):
    n = len(degrees)
    rng = np.random.default_rng(sum(degrees))
    to = rng.permutation(np.repeat(np.arange(n), degrees))
    run(vh, n, rng.integers(0, n, to.size), to, hub)


@pytest.mark.parametrize("n", [5, 40])
def test_alone_at_a_server(vh, n):
    from vahana_gb300 import models, serve
    spec = serve.opinion_job(n, mean_degree=10_000, steps=3, seed=4, wmax=1e3, keep_state=True)
    _, to, _ = om.gen_chung_lu(n, 10_000 * n, 10_000, 2.5, 1e3, 4)
    assert np.bincount((to & np.uint64((1 << 36) - 1)).astype(np.int64))[1:].min() >= 3072
    alone = models.build_opinion(n=n, mean_degree=10_000, gamma=2.5, wmax=1e3, eps=spec.eps,
                                 seed=4, hub_threshold=models.OPINION_HUB_THRESHOLD)
    vh.finish_init(alone.sim)
    x0 = vh.read_agents(alone.sim, "Opinion")[0]["x"].copy()
    for _ in range(spec.steps):
        alone.step()
    want = vh.read_agents(alone.sim, "Opinion")[0]["x"]
    assert not np.array_equal(want, x0)
    with serve.Server() as S:
        i = S.submit(spec)
        S.drain()
        S.poll()
        np.testing.assert_array_equal(S.job_state(i, spec).view(np.uint64), want.view(np.uint64))
    alone.close()
