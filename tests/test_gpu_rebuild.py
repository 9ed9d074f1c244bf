"""The typed rebuild of an edge type's container (csrc/vg_bucket.cuh): records
in known slots, sorted by bucket tile by tile and placed bucket by bucket.
Every container equals the one a stable sort of the records by target row
gives (tolerance 0), over sizes at the edges of tiles (4096 slots), buckets
and staged chunks (1024 and 2048 records), containers of up to several spans
of 8192 rows, records crowded into one row or bucket, payload of every width,
rows left out by with_edge, old edges kept by add_existing, and agents that
died."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def container(vh, sim, E, T):
    rp, frm, pl = vh.read_edges(sim, E, T)
    nr = (frm & np.uint64((1 << 36) - 1)).astype(np.int64) - 1
    return rp.astype(np.int64), nr, pl


def expect(n, row, src, pl=()):
    """(row pointers, sources, payload columns) of records in call order."""
    o = np.argsort(row, kind="stable")
    return (np.concatenate([[0], np.cumsum(np.bincount(row, minlength=n))]), src[o],
            [p[o] for p in pl])


def check(vh, sim, E, T, n, row, src, **pl):
    rp, nr, got = container(vh, sim, E, T)
    wrp, wsrc, wpl = expect(n, row, src, pl.values())
    np.testing.assert_array_equal(rp, wrp)
    np.testing.assert_array_equal(nr, wsrc)
    for name, w in zip(pl, wpl):
        np.testing.assert_array_equal(got[name], w)


def test_records_that_crowd_after_spreading(vh):
    """A rebuild planned for evenly spread records meets buckets that hold far
    more than their block stages, and the ones after it; then spread again."""
    rng = np.random.default_rng(4)
    n, size = 30_000, 60_000
    m = (vh.ModelTypes().register_agenttype("P", [("v", "f64")], ":Immortal")
         .register_edgetype("A", []).register_edgetype("B", [])
         .register_edgetype("F", [("v", "f64")], target="P")
         .register_edgetype("G", [], ":Stateless")
         .create_model("Crowd"))
    sim = vh.create_simulation(m)
    v = rng.random(n)
    ids = vh.add_agents(sim, "P", n, v=v)
    ends = {"A": (rng.integers(0, n, size), rng.integers(0, n, size)),
            "B": (np.full(size, 3), np.minimum((n * rng.random(size) ** 30).astype(np.int64), n - 1))}
    for E, (src, row) in ends.items():
        vh.add_edges(sim, E, ids[src], ids[row])
    vh.finish_init(sim)
    for E in "AAABBBAAAB":
        src, row = ends[E]
        o = np.argsort(row, kind="stable")
        to, frm = np.stack([row[o], src[o]], 1).ravel(), np.stack([src[o], row[o]], 1).ravel()
        for F in "FG":
            vh.apply_(sim, "link_neighbors", ["P"], ["P", E], ["P", F],
                      params=[m[E].index, m[F].index])
            check(vh, sim, F, "P", n, to, frm, **({"v": np.repeat(v[row[o]], 2)} if F == "F" else {}))
    sim.close()


def skewed(rng, n, size, how):
    if how == "uniform":
        return rng.integers(0, n, size)
    if how == "one":  # every record in one row
        return np.full(size, n // 2)
    return np.minimum((n * rng.random(size) ** 8).astype(np.int64), n - 1)  # crowded


@pytest.mark.parametrize("how", ["uniform", "one", "crowded"])
@pytest.mark.parametrize("n,deg", [(1, 1), (3, 2), (1000, 4), (1024, 4), (1365, 3), (2049, 2),
                                   (70_000, 1), (40_000, 30), (300_001, 2)])
def test_readd_and_link(vh, n, deg, how):
    rng = np.random.default_rng(n + deg)
    m = (vh.ModelTypes().register_agenttype("P", [("v", "f64"), ("k", "i32")], ":Immortal")
         .register_edgetype("E", [("a", "f64"), ("b", "i32"), ("c", "u8"), ("d", "i16")])
         .register_edgetype("F", [("v", "f32")], target="P")
         .register_edgetype("G", [], ":IgnoreFrom")
         .create_model("Rebuild"))
    sim = vh.create_simulation(m)
    v = rng.random(n)
    ids = vh.add_agents(sim, "P", n, v=v, k=0)
    size = n * deg
    src, row = rng.integers(0, n, size), skewed(rng, n, size, how)
    pl = {"a": rng.random(size), "b": rng.integers(-9, 9, size).astype(np.int32),
          "c": rng.integers(0, 9, size).astype(np.uint8),
          "d": rng.integers(-9, 9, size).astype(np.int16)}
    vh.add_edges(sim, "E", ids[src], ids[row], **pl)
    vh.finish_init(sim)
    e, f, g = (m[x].index for x in "EFG")
    for _ in range(3):  # sorted first, then by buckets in the same buffers
        vh.apply_(sim, "readd_edges", ["P"], ["P", "E"], ["P", "E"], params=[e])
        check(vh, sim, "E", "P", n, row, src, **pl)
        vh.apply_(sim, "link_neighbors", ["P"], ["P", "E"], ["P", "F"], params=[e, f])
        o = np.argsort(row, kind="stable")
        to = np.stack([row[o], src[o]], 1).ravel()
        frm = np.stack([src[o], row[o]], 1).ravel()
        check(vh, sim, "F", "P", n, to, frm, v=np.repeat(v[row[o]], 2).astype(np.float32))
    vh.apply_(sim, "link_neighbors", ["P"], ["P", "E"], ["P", "G"], params=[e, g])
    rp, _, _ = container(vh, sim, "G", "P")
    np.testing.assert_array_equal(np.diff(rp), np.bincount(to, minlength=n))
    # add_existing: the old edges stay ahead in their rows
    for k in range(2, 4):
        vh.apply_(sim, "link_neighbors", ["P"], ["P", "E"], ["P", "F"], add_existing=["F"],
                  params=[e, f])
        check(vh, sim, "F", "P", n, np.tile(to, k), np.tile(frm, k),
              v=np.tile(np.repeat(v[row[o]], 2), k).astype(np.float32))
    sim.close()


@pytest.mark.parametrize("n", [5, 4096, 50_000])
def test_with_edge_deaths_and_newcomers(vh, n):
    rng = np.random.default_rng(n)
    m = (vh.ModelTypes().register_agenttype("P", [("v", "i64")])
         .register_edgetype("E", [("w", "i64")])
         .register_edgetype("H", [], ":Stateless")
         .register_edgetype("S", [("w", "i64")], target="P")
         .create_model("Turnover"))
    sim = vh.create_simulation(m)
    v = rng.integers(0, 10, n)
    ids = vh.add_agents(sim, "P", n, v=v)
    src, row = rng.integers(0, n, 3 * n), rng.integers(0, n, 3 * n)
    w = rng.integers(0, 1 << 40, 3 * n)
    vh.add_edges(sim, "E", ids[src], ids[row], w=w)
    hosts = np.sort(rng.permutation(n)[:(n + 2) // 3])
    vh.add_edges(sim, "H", ids[hosts], ids[hosts])
    vh.finish_init(sim)
    e, s = m["E"].index, m["S"].index
    # only hosts re-add their edges
    vh.apply_(sim, "readd_edges", ["P"], ["P", "E", "H"], ["P", "E"], with_edge="H", params=[e])
    keep = np.isin(row, hosts)
    src, row, w = src[keep], row[keep], w[keep]
    check(vh, sim, "E", "P", n, row, src, w=w)
    # agents with v == 3 die while they would link; their slots stay empty
    vh.apply_(sim, "self_edge", ["P"], ["P"], ["P", "S"], params=[s, 7])
    check(vh, sim, "S", "P", n, np.arange(n), np.arange(n), w=np.full(n, 7))
    vh.apply_(sim, "link_neighbors", ["P"], ["P", "E"], ["P", "S"], params=[e, s, 3])
    dead = v == 3
    o = np.argsort(row, kind="stable")
    to = np.stack([row[o], src[o]], 1).ravel()
    frm = np.stack([src[o], row[o]], 1).ravel()
    by = np.repeat(row[o], 2)
    ok = ~dead[by] & ~dead[to] & ~dead[frm]
    check(vh, sim, "S", "P", n, to[ok], frm[ok], w=v[by[ok]])
    ok = ~dead[row] & ~dead[src]
    row, src, w = row[ok], src[ok], w[ok]
    check(vh, sim, "E", "P", n, row, src, w=w)
    # newcomers linked with their makers, old edges kept
    vh.apply_(sim, "spawn", ["P"], ["P", "H"], ["P", "E"], add_existing=["E"], with_edge="H",
              params=[1, 100, e])
    makers = hosts[~dead[hosts]]
    pop = list(np.nonzero(dead)[0])  # slots of the dead are reused last in, first out
    total = n
    to, frm, pay = list(row[np.argsort(row, kind="stable")]), None, None
    o = np.argsort(row, kind="stable")
    to, frm, pay = list(row[o]), list(src[o]), list(w[o])
    for h in makers:
        if pop:
            t = pop.pop()
        else:
            t, total = total, total + 1
        to += [h, t]
        frm += [t, h]
        pay += [(1 << 56) + t + 1] * 2
    check(vh, sim, "E", "P", total, np.array(to, np.int64), np.array(frm, np.int64),
          w=np.array(pay, np.int64))
    # self edges of the living only
    vh.apply_(sim, "self_edge", ["P"], ["P"], ["P", "S"], params=[s, 1])
    _, died = vh.read_agents(sim, "P")
    alive = np.nonzero(~died)[0]
    check(vh, sim, "S", "P", total, alive, alive, w=np.ones(alive.size, np.int64))
    sim.close()


@pytest.mark.parametrize("W,H,walkers", [(3, 3, 1), (90, 91, 4097), (128, 64, 500),
                                         (4100, 4099, 20_000), (300, 300, 200_000)])
def test_walkers_crowded_or_sparse(vh, W, H, walkers):
    """Walkers that all start on one cell: one bucket holds every record."""
    m = (vh.ModelTypes().register_agenttype("C", [("a", "bool")], ":Immortal")
         .register_agenttype("Wk", [("x", "i32"), ("y", "i32")], ":Immortal")
         .register_edgetype("On", [], ":Stateless", target="C").create_model("Walk"))
    sim = vh.create_simulation(m)
    vh.add_raster(sim, "r", (W, H), "C", a=False)
    vh.add_agents(sim, "Wk", walkers, x=W, y=1)
    vh.finish_init(sim)
    for _ in range(4):
        vh.apply_(sim, "random_walk", ["Wk"], ["Wk"], ["Wk", "On"],
                  params=[m["On"].index, 0, 11])
        c = vh.read_agents(sim, "Wk")[0]
        row = (c["x"].astype(np.int64) - 1) + (c["y"].astype(np.int64) - 1) * W
        assert ((c["x"] >= 1) & (c["x"] <= W) & (c["y"] >= 1) & (c["y"] <= H)).all()
        check(vh, sim, "On", "C", W * H, row, np.arange(walkers))
    sim.close()
