"""Typed rebuilds where slots of the call stay empty (csrc/vg_bucket.cuh): agents
that died and whose rows hold edges all the same (walkers move onto dead
cells, add_edges! takes any target), and positions outside the raster in queued
transitions.  The containers equal a numpy filter of the records (order kept,
tolerance 0), at row counts where the key of an empty slot needs one bit more
than the rows (256, 65 536) and others, over several rebuilds in both forms."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def check(vh, sim, E, T, n, row, src, **pl):
    rp, frm, got = vh.read_edges(sim, E, T)
    o = np.argsort(row, kind="stable")
    np.testing.assert_array_equal(rp.astype(np.int64),
                                  np.concatenate([[0], np.cumsum(np.bincount(row, minlength=n))]))
    nr = (frm & np.uint64((1 << 36) - 1)).astype(np.int64) - 1
    np.testing.assert_array_equal(nr[:row.size], src[o])
    assert vh.num_edges(sim, E) == row.size
    for name, col in pl.items():
        np.testing.assert_array_equal(got[name][:row.size], col[o])


@pytest.mark.parametrize("walkers", [100, 3000, 70_000])
@pytest.mark.parametrize("dims", [(40, 25), (16, 16), (256, 256)])
def test_cells_that_died(vh, dims, walkers):
    rng = np.random.default_rng(dims[0] + walkers)
    W, H = dims
    cells = W * H
    m = (vh.ModelTypes().register_agenttype("Cell", [("a", "i32")])
         .register_agenttype("Walker", [("x", "i32"), ("y", "i32")], ":Immortal")
         .register_edgetype("On", [("w", "i32")], target="Cell")
         .register_edgetype("At", [("u", "f64"), ("b", "u8")]).create_model("DeadCells"))
    sim = vh.create_simulation(m)
    a = (rng.random(dims) < 0.3).astype(np.int32)
    a[-1, -1] = a[0, 0] = 0
    vh.add_raster(sim, "r", dims, "Cell", a=a)
    vh.add_agents(sim, "Walker", walkers, x=1, y=1)
    vh.finish_init(sim)
    dead = a.ravel(order="F") > 0
    vh.apply_(sim, "die_if", ["Cell"], ["Cell"], ["Cell"], params=[1, 0, 1.0])
    who = np.arange(walkers)
    for _ in range(4):
        x, y = rng.integers(1, W + 1, walkers), rng.integers(1, H + 1, walkers)
        vh.write_agents(sim, "Walker", x=x, y=y)
        row = (x - 1) + (y - 1) * W
        for E in ("On", "At"):
            e = m[E].index
            vh.apply_(sim, "move_to", ["Walker"], ["Walker"], ["Walker", E],
                      params=[0, -1, e, 0, 0, 1, 0, 0])
            check(vh, sim, E, "Cell", cells, row, who)
            # the living cells add their edges again, the dead ones do not
            live = ~dead[row]
            o = np.argsort(row[live], kind="stable")
            r, s = row[live][o], who[live][o]
            for _ in range(3):
                vh.apply_(sim, "readd_edges", ["Cell"], ["Cell", E], ["Cell", E], params=[e])
                check(vh, sim, E, "Cell", cells, r, s)
    sim.close()


@pytest.mark.parametrize("n", [256, 1000, 65_536])
def test_edges_to_agents_that_died(vh, n):
    rng = np.random.default_rng(n)
    m = (vh.ModelTypes().register_agenttype("P", [("v", "i64")])
         .register_edgetype("E", [("w", "i64")]).register_edgetype("F", [("w", "i64")], target="P")
         .register_edgetype("G", [], ":Stateless").create_model("LateEdges"))
    sim = vh.create_simulation(m)
    v = rng.integers(0, 4, n)
    ids = vh.add_agents(sim, "P", n, v=v)
    vh.finish_init(sim)
    e, f, g = (m[x].index for x in "EFG")
    vh.apply_(sim, "die_if", ["P"], ["P"], ["P"], params=[1, 0, 3.0])
    dead = v >= 3
    living = np.nonzero(~dead)[0]
    src, row = rng.choice(living, 5 * n), rng.integers(0, n, 5 * n)
    w = rng.integers(0, 1 << 40, 5 * n)
    vh.disable_transition_checks(sim, True)
    vh.add_edges(sim, "E", ids[src], ids[row], w=w)
    vh.disable_transition_checks(sim, False)
    check(vh, sim, "E", "P", n, row, src, w=w)
    keep = ~dead[row]
    o = np.argsort(row[keep], kind="stable")
    r, s = row[keep][o], src[keep][o]
    to, frm = np.stack([r, s], 1).ravel(), np.stack([s, r], 1).ravel()
    for _ in range(4):  # linked along the living agents' edges
        vh.apply_(sim, "link_neighbors", ["P"], ["P", "E"], ["P", "F"], params=[e, f])
        check(vh, sim, "F", "P", n, to, frm, w=np.repeat(v[r], 2))
        vh.apply_(sim, "link_neighbors", ["P"], ["P", "E"], ["P", "G"], params=[e, g])
        check(vh, sim, "G", "P", n, to, frm)
    for _ in range(4):
        vh.apply_(sim, "readd_edges", ["P"], ["P", "E"], ["P", "E"], params=[e])
        check(vh, sim, "E", "P", n, r, s, w=w[keep][o])
    sim.close()


@pytest.mark.parametrize("how", ["queued", "host", "checked"])
@pytest.mark.parametrize("dims,n", [((10, 7), 300), ((16, 16), 256), ((256, 256), 65_536)])
def test_positions_outside(vh, dims, n, how):
    rng = np.random.default_rng(n)
    W, H = dims
    m = (vh.ModelTypes().register_agenttype("Cell", [("a", "i32")], ":Immortal")
         .register_agenttype("Walker", [("x", "i32"), ("y", "i32")], ":Immortal")
         .register_edgetype("In", [], ":Stateless").register_edgetype("Out", [], ":Stateless")
         .create_model("Outside"))
    sim = vh.create_simulation(m)
    vh.add_raster(sim, "r", dims, "Cell", a=0)
    vh.add_agents(sim, "Walker", n, x=1, y=1)
    vh.finish_init(sim)
    args = ["Walker"], ["Walker"], ["Walker", "In", "Out"]
    params = [0, m["In"].index, m["Out"].index, 0, 0, 1, 0, 0]
    vh.set_async(sim, how == "queued")
    for _ in range(4):
        x = rng.integers(1, W + 1, n).astype(np.int32)
        y = rng.integers(1, H + 1, n).astype(np.int32)
        vh.write_agents(sim, "Walker", x=x, y=y)
        vh.apply_(sim, "move_to", *args, params=params)
        vh.synchronize(sim)
        row, who = (x - 1) + (y - 1) * W, np.arange(n)
        check(vh, sim, "Out", "Cell", W * H, row, who)
        check(vh, sim, "In", "Walker", n, who, row)
        x[rng.integers(0, n, 3)] = W + 1
        y[rng.integers(0, n, 3)] = 0
        if how == "host":
            with pytest.raises(vh.VahanaError):
                vh.apply_host(sim, "move_to", *args, "Walker", {"x": x, "y": y}, params=params)
        else:
            vh.write_agents(sim, "Walker", x=x, y=y)
            with pytest.raises(vh.VahanaError):
                vh.apply_(sim, "move_to", *args, params=params)
                vh.synchronize(sim)
        if how != "checked":  # the rebuild ran before the error was read
            ok = (x <= W) & (y >= 1)
            row, who = row[ok], who[ok]
        check(vh, sim, "Out", "Cell", W * H, row, who)
        check(vh, sim, "In", "Walker", n, who, row)
    sim.close()
