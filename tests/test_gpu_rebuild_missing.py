"""Records to agents that do not exist are refused, and nothing is stored for
them: walkers on a raster whose cells were written anew (a mortal type in
`write` without add_existing starts empty), and agents linked with a source
that was never added.  The simulation goes on."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("queued", [False, True])
@pytest.mark.parametrize("before", [0, 3])
@pytest.mark.parametrize("dims,n", [((10, 10), 50), ((300, 257), 5000)])
def test_cells_written_anew(vh, dims, n, before, queued):
    m = (vh.ModelTypes().register_agenttype("Cell", [("a", "i32")])
         .register_agenttype("Walker", [("x", "i32"), ("y", "i32")], ":Immortal")
         .register_edgetype("On", [], ":Stateless", target="Cell")
         .register_edgetype("Sees", [], ":Stateless")
         .register_edgetype("Self", [], ":Stateless").create_model("Anew"))
    sim = vh.create_simulation(m)
    vh.add_raster(sim, "r", dims, "Cell", a=0)
    rng = np.random.default_rng(n)
    vh.add_agents(sim, "Walker", n, x=rng.integers(1, dims[0] + 1, n),
                  y=rng.integers(1, dims[1] + 1, n))
    vh.finish_init(sim)
    on, sees, own = (m[x].index for x in ("On", "Sees", "Self"))
    vh.set_async(sim, queued)

    def walk():
        vh.apply_(sim, "random_walk", ["Walker"], ["Walker"], ["Walker", "On"],
                  params=[on, 0, 7])

    def move():
        vh.apply_(sim, "move_to", ["Walker"], ["Walker"], ["Walker", "Sees"],
                  params=[0, -1, sees, 1, 0, 1, 0, 0])

    for _ in range(before):  # (workspaces of an earlier rebuild are there or not)
        walk()
        move()
    vh.apply_(sim, "keep", ["Walker"], ["Walker"], ["Walker", "Cell"])
    vh.synchronize(sim)
    assert vh.num_agents(sim, "Cell") == 0
    for f in (walk, move):
        with pytest.raises((AssertionError, vh.VahanaError)):
            f()
            vh.synchronize(sim)
    vh.apply_(sim, "self_edge", ["Walker"], ["Walker"], ["Walker", "Self"], params=[own])
    vh.synchronize(sim)
    rp, frm, _ = vh.read_edges(sim, "Self", "Walker")
    np.testing.assert_array_equal(rp, np.arange(n + 1))
    sim.close()


@pytest.mark.parametrize("n", [5, 4096, 40_000])
def test_sources_never_added(vh, n):
    m = (vh.ModelTypes().register_agenttype("P", [("v", "i64")], ":Immortal")
         .register_edgetype("E", [("w", "i64")]).register_edgetype("F", [("w", "i64")], target="P")
         .create_model("Never"))
    sim = vh.create_simulation(m)
    ids = vh.add_agents(sim, "P", n, v=3)
    frm = np.roll(ids, 1)
    frm[n // 2] = ids[-1] + np.uint64(1 + n)
    vh.add_edges(sim, "E", frm, ids, w=1)
    vh.finish_init(sim)
    for _ in range(3):
        with pytest.raises(AssertionError, match="does not exist"):
            vh.apply_(sim, "link_neighbors", ["P"], ["P", "E"], ["P", "F"],
                      params=[m["E"].index, m["F"].index])
    np.testing.assert_array_equal(vh.read_agents(sim, "P")[0]["v"], np.full(n, 3))
    assert vh.num_edges(sim, "F") == 0
    sim.close()
