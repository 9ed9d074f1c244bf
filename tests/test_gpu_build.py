"""finish_init!'s edge containers (src/Simulation.jl:440-480,
src/EdgeMethods.jl:440-520) against a stable numpy sort of the records by
target: row pointers, sources, payload and order exactly, for row counts at
the edges of a block's span of rows (8192), empty first and last rows, one
crowded row, several target types, mixed sources, edges staged by the program
in several pieces, and the errors a build reports."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def targets(shape, n, ne, rng):
    if shape == "crowded":
        to = rng.integers(0, n, ne)
        to[: ne // 2] = n - 1
        return to
    if shape == "inner":  # the first and last third of the rows stay empty
        return rng.integers(n // 3, max(n // 3 + 1, 2 * n // 3), ne)
    return rng.integers(0, n, ne)


@pytest.mark.parametrize("shape", ["uniform", "crowded", "inner"])
@pytest.mark.parametrize("n,ne", [(1, 1), (1, 5000), (33, 7), (8191, 20_000), (8192, 20_000),
                                  (16_385, 300_000), (100_000, 9000)])
@pytest.mark.parametrize("both", [False, True])
def test_containers(vh, n, ne, shape, both):
    rng = np.random.default_rng(n + ne + len(shape))
    m = (vh.ModelTypes().register_agenttype("P", []).register_agenttype("Q", [])
         .register_edgetype("E", [("w", "f64"), ("k", "u8"), ("h", "i16")])
         .register_edgetype("S", [], ":Stateless", target="P")
         .register_edgetype("I", [("w", "i32")], ":IgnoreFrom")
         .register_edgetype("N", [], ":NumEdgesOnly")
         .register_edgetype("X", [("w", "i32")], ":SingleEdge")
         .create_model("Build"))
    sim = vh.create_simulation(m)
    ids = {T: vh.add_agents(sim, T, n) for T in "PQ"}
    every = np.concatenate([ids["P"], ids["Q"]])
    recs = {}
    for E in "ESIN":
        to = ids["P"][targets(shape, n, ne, rng)]
        if both and E != "S":
            to = np.where(rng.random(ne) < 0.3, ids["Q"][targets(shape, n, ne, rng)], to)
        frm = (every if both and E == "E" else ids["P"])
        frm = frm[rng.integers(0, frm.size, ne)]
        pl = {"E": {"w": rng.random(ne), "k": rng.integers(0, 9, ne).astype(np.uint8),
                    "h": rng.integers(-9, 9, ne).astype(np.int16)},
              "I": {"w": rng.integers(0, 99, ne).astype(np.int32)}}.get(E, {})
        cut = sorted(rng.integers(0, ne + 1, 2).tolist()) if both else [0, ne]
        for a, b in ((0, cut[0]), (cut[0], cut[1]), (cut[1], ne)):
            if b > a:
                vh.add_edges(sim, E, frm[a:b], to[a:b], **{k: v[a:b] for k, v in pl.items()})
        recs[E] = (frm, to, pl)
    some = rng.permutation(n)[: max(1, n // 2)]
    vh.add_edges(sim, "X", ids["P"][some], ids["P"][some], w=some.astype(np.int32))
    recs["X"] = (ids["P"][some], ids["P"][some], {"w": some.astype(np.int32)})
    vh.finish_init(sim)
    for E, (frm, to, pl) in recs.items():
        for T in ("P", "Q"):
            if E in "SX" and T == "Q":
                continue
            mine = (to >> np.uint64(56)) == np.uint64(m[T].index)
            rows = ((to[mine] & np.uint64((1 << 36) - 1)) - np.uint64(1)).astype(np.int64)
            order = np.argsort(rows, kind="stable")
            rp, got, cols = vh.read_edges(sim, E, T)
            if not rows.size:
                assert got.size == 0 and rp[-1] == 0
                continue
            want = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))])
            np.testing.assert_array_equal(rp, want.astype(np.uint64))
            if E in "ESX":
                np.testing.assert_array_equal(got, frm[mine][order])
            for k, v in pl.items():
                np.testing.assert_array_equal(cols[k], v[mine][order])


@pytest.mark.parametrize("bad", ["target", "single"])
def test_errors(vh, bad):
    m = (vh.ModelTypes().register_agenttype("P", [])
         .register_edgetype("X", [("w", "i32")], *([":SingleEdge"] if bad == "single" else []))
         .create_model("Errors"))
    sim = vh.create_simulation(m)
    p = vh.add_agents(sim, "P", 10)
    to = p[[0, 3, 3]] if bad == "single" else np.array([p[0], p[9] + np.uint64(1)], np.uint64)
    with pytest.raises(AssertionError):
        vh.add_edges(sim, "X", p[: to.size], to, w=np.zeros(to.size, np.int32))
        vh.finish_init(sim)
