"""neighbor_sum and neighbor_or over sources of one type (a kernel per column
type, eight edges of a row in flight) and of several (the general kernel):
against the fold of each row in its order, for every column type, into
integer and Float columns, rows around a batch of eight and longer ones, empty
rows, mortal sources, with two target rows' worth of rows behind the last edge.
Exact: the order of the additions is the row's (tolerance 0)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
DT = ["bool", "u8", "i8", "u16", "i16", "u32", "i32", "u64", "i64", "f32", "f64"]
NP = {"bool": bool, "f32": np.float32, "f64": np.float64}


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("kinds", ["one", "two"])
@pytest.mark.parametrize("mortal", [False, True])
def test_rows(vh, dt, kinds, mortal):
    rng = np.random.default_rng(DT.index(dt))
    t = NP.get(dt) or np.dtype(dt.replace("u", "uint") if dt[0] == "u" else dt.replace("i", "int"))
    n = 700

    def column(k):
        if dt[0] == "f":
            return (rng.standard_normal(k) * 10.0 ** rng.integers(-6, 7, k)).astype(t)
        if dt == "bool":
            return rng.random(k) < 0.1
        info = np.iinfo(t)
        x = rng.integers(max(info.min, -10 ** 9), min(info.max, 10 ** 9), k).astype(t)
        x[rng.random(k) < 0.5] = 0
        return x

    hints = [] if mortal else [":Immortal"]
    m = (vh.ModelTypes()
         .register_agenttype("P", [("v", dt), ("i", "i64"), ("f", "f64")], *hints)
         .register_agenttype("Q", [("v", dt)], *hints)
         .register_edgetype("E", []).create_model("Neighbors"))
    sim = vh.create_simulation(m)
    pv, qv = column(n), column(50)
    p = vh.add_agents(sim, "P", n, v=pv, i=rng.integers(0, 2, n), f=np.zeros(n))
    q = vh.add_agents(sim, "Q", 50, v=qv)
    own = vh.read_agents(sim, "P")[0]["i"].copy()
    lens = np.concatenate([np.arange(34), rng.integers(0, 20, n - 40), [1000, 0, 0, 7, 8, 0]])
    ids, vals = (p, pv) if kinds == "one" else (np.concatenate([p, q]), np.concatenate([pv, qv]))
    pick = rng.integers(0, ids.size, lens.sum())
    vh.add_edges(sim, "E", ids[pick], np.repeat(p, lens))
    vh.finish_init(sim)
    read = ["P", "Q", "E"]
    e = m["E"].index
    rows = np.split(vals[pick], np.cumsum(lens)[:-1])
    vh.apply_(sim, "neighbor_or", ["P"], read, ["P"], params=[e, 0, 1])
    want = (own != 0) | np.array([(r.astype(np.int64) != 0).any() for r in rows])
    np.testing.assert_array_equal(vh.read_agents(sim, "P")[0]["i"], want.astype(np.int64))
    vh.apply_(sim, "neighbor_sum", ["P"], read, ["P"], params=[e, 0, 2])
    want = np.array([np.add.accumulate(np.concatenate([[0.0], r.astype(np.float64)]))[-1]
                     for r in rows])
    got = vh.read_agents(sim, "P")[0]["f"]
    np.testing.assert_array_equal(got.view(np.uint64), want.view(np.uint64))
    if dt[0] != "f":
        vh.apply_(sim, "neighbor_sum", ["P"], read, ["P"], params=[e, 0, 1])
        with np.errstate(over="ignore"):
            want = np.array([r.astype(np.int64).sum() for r in rows])
        np.testing.assert_array_equal(vh.read_agents(sim, "P")[0]["i"], want)
