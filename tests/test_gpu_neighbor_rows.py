"""neighbor_sum and neighbor_or over rows of few and of many edges: a rest of
every length in one warp, rows of none, a long row beside empty ones, the
columns' types and both kinds of sum against sums in edge order."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

COLUMNS = [("i", "i32"), ("b", "u8"), ("f", "f32"), ("d", "f64")]


def degrees(form, n, rng):
    if form == "sparse":                       # a warp with one edge or none
        return (rng.random(n) < 0.03).astype(np.int64)
    if form == "rests":                        # 0..11: every rest of 4 and of 8
        return np.arange(n) % 12
    if form == "sixteen":                      # just at the change of form
        return np.full(n, 16)
    if form == "fifteen":
        return np.full(n, 15) + (np.arange(n) % 3 == 0) - (np.arange(n) % 3 == 1)
    d = np.zeros(n, np.int64)                  # one row beyond the others
    d[n // 2] = {"hub": 1024, "below": 1023}[form]
    return d


@pytest.mark.parametrize("form", ["sparse", "rests", "fifteen", "sixteen", "hub", "below"])
@pytest.mark.parametrize("mortal", [False, True])
def test_sums_in_edge_order(vh, form, mortal):
    n = 1000
    rng = np.random.default_rng(11)
    hints = [] if mortal else [":Immortal"]
    fields = COLUMNS + [("si", "i64"), ("sd", "f64"), ("any", "i32")]
    m = (vh.ModelTypes()
         .register_agenttype("P", fields, *hints)
         .register_edgetype("S", [], ":Stateless", target="P").create_model("rows"))
    values = {"i": rng.integers(-9, 9, n).astype(np.int32),
              "b": rng.integers(0, 2, n).astype(np.uint8),
              "f": rng.normal(0, 1e3, n).astype(np.float32),
              "d": rng.normal(0, 1e9, n) * 10.0 ** rng.integers(-8, 8, n)}
    own = (np.arange(n) % 7 == 0).astype(np.int32)
    sim = vh.create_simulation(m)
    ids = vh.add_agents(sim, "P", n, si=0, sd=0.0, any=own, **values)
    deg = degrees(form, n, rng)
    row = np.repeat(np.arange(n), deg)
    src = rng.integers(0, n, row.size)
    vh.add_edges(sim, "S", ids[src], ids[row])
    vh.finish_init(sim)
    e = m["S"].index
    for k, (name, _) in enumerate(COLUMNS):
        for out in (4, 5):
            if name in "fd" and out == 4:
                continue
            vh.apply_(sim, "neighbor_sum", ["P"], ["P", "S"], ["P"], params=[e, k, out])
            got = vh.read_agents(sim, "P")[0][fields[out][0]]
            want = np.zeros(n, np.int64 if out == 4 else np.float64)
            np.add.at(want, row, values[name][src].astype(want.dtype))   # in edge order
            np.testing.assert_array_equal(got, want)
    # a binary64 column into whole numbers: truncated, then added
    vh.apply_(sim, "neighbor_sum", ["P"], ["P", "S"], ["P"], params=[e, 2, 4])
    want = np.zeros(n, np.int64)
    np.add.at(want, row, values["f"][src].astype(np.int64))
    np.testing.assert_array_equal(vh.read_agents(sim, "P")[0]["si"], want)
    vh.apply_(sim, "neighbor_or", ["P"], ["P", "S"], ["P"], params=[e, 1, 6])
    hit = np.zeros(n, bool)
    np.logical_or.at(hit, row, values["b"][src] != 0)
    np.testing.assert_array_equal(vh.read_agents(sim, "P")[0]["any"], (own != 0) | hit)
    sim.close()
