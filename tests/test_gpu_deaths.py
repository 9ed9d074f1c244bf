"""Deaths and the removal of their edges (src/AgentMethods.jl:300-345,
src/EdgeMethods.jl:606-631, :897-920): the packed containers of every kind of
edge type against a numpy filter of the records (order kept, tolerance 0), for
populations at the edges of a scan tile (4096 agents) and of a warp's rows,
rows longer than a warp, two agent types that die in one transition, mixed
sources, and repeated deaths with reused slots."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
NR = np.uint64((1 << 36) - 1)


@pytest.mark.parametrize("share", [0.0, 0.02, 0.5, 1.0])
@pytest.mark.parametrize("n", [1, 31, 33, 4096, 4097, 40_000])
def test_packed_containers(vh, n, share):
    rng = np.random.default_rng(n + int(100 * share))
    m = (vh.ModelTypes()
         .register_agenttype("P", [("die", "i32")]).register_agenttype("Q", [("die", "i32")])
         .register_edgetype("E", [("w", "f64"), ("k", "u8")])   # mixed sources
         .register_edgetype("S", [], ":Stateless", target="P")
         .register_edgetype("I", [("w", "i32")], ":IgnoreFrom")
         .register_edgetype("N", [], ":NumEdgesOnly")
         .create_model("Deaths"))
    sim = vh.create_simulation(m)
    die = {T: (rng.random(n) < share).astype(np.int32) for T in "PQ"}
    ids = {T: vh.add_agents(sim, T, n, die=die[T]) for T in "PQ"}
    both = np.concatenate([ids["P"], ids["Q"]])
    dead_of = dict(zip(both.tolist(), np.concatenate([die["P"], die["Q"]]).tolist()))
    size = 5 * n
    edges = {}
    for E, frm, to in (("E", both, both), ("S", ids["P"], ids["P"]), ("I", both, both),
                       ("N", both, both)):
        f, t = frm[rng.integers(0, frm.size, size)], to[rng.integers(0, to.size, size)]
        t[:size // 5] = to[0]  # one long row
        pl = {"E": {"w": rng.random(size), "k": rng.integers(0, 9, size).astype(np.uint8)},
              "I": {"w": rng.integers(0, 99, size).astype(np.int32)}}.get(E, {})
        vh.add_edges(sim, E, f, t, **pl)
        edges[E] = (f, t, pl)
    vh.finish_init(sim)
    vh.apply_(sim, "die_if", ["P", "Q"], ["P", "Q"], ["P", "Q"], params=[1, 0, 1.0])
    for T in "PQ":
        _, died = vh.read_agents(sim, T)
        np.testing.assert_array_equal(died, die[T] > 0)
    for E, (f, t, pl) in edges.items():
        gone = np.array([dead_of[x] for x in t.tolist()], bool)
        if E in "ES":
            gone |= np.array([dead_of[x] for x in f.tolist()], bool)
        for T in ("P",) if E == "S" else ("P", "Q"):
            mine = ((t >> np.uint64(56)) == np.uint64(m[T].index)) & ~gone
            row = (t[mine] & NR).astype(np.int64) - 1
            o = np.argsort(row, kind="stable")
            rp, frm, got = vh.read_edges(sim, E, T)
            if not ((t >> np.uint64(56)) == np.uint64(m[T].index)).any():
                assert rp.size == 1 and frm.size == 0  # no container of that target type
                continue
            np.testing.assert_array_equal(rp.astype(np.int64),
                                          np.concatenate([[0], np.cumsum(np.bincount(row, minlength=n))]))
            if E in "ES":
                np.testing.assert_array_equal(frm, f[mine][o])
            for name, col in pl.items():
                np.testing.assert_array_equal(got[name], col[mine][o])
    sim.close()


def test_deaths_and_newcomers_again_and_again(vh):
    """Slots of the dead are reused last in, first out, wave after wave."""
    n = 5000
    m = (vh.ModelTypes().register_agenttype("P", [("v", "i64")])
         .register_edgetype("H", [], ":Stateless").create_model("Waves"))
    sim = vh.create_simulation(m)
    ids = vh.add_agents(sim, "P", n, v=np.arange(n) % 7 - 8)  # residents below 0
    hosts = np.arange(0, n, 3)
    vh.add_edges(sim, "H", ids[hosts], ids[hosts])
    vh.finish_init(sim)
    stack, total, alive = [], n, set(range(n))
    for wave in range(4):
        vh.apply_(sim, "spawn", ["P"], ["P", "H"], ["P"], with_edge="H", params=[1, 100])
        new = []
        for _ in hosts:
            t = stack.pop() if stack else total
            total = max(total, t + 1)
            new.append(t)
        alive |= set(new)
        cols, died = vh.read_agents(sim, "P")
        assert died.size == total and set(np.nonzero(~died)[0]) == alive
        np.testing.assert_array_equal(cols["v"][new], cols["v"][hosts] + 100)
        vh.apply_(sim, "die_if", ["P"], ["P"], ["P"], params=[1, 0, 92.0 + wave])
        gone = [t for t in sorted(alive) if cols["v"][t] >= 92 + wave]
        stack += gone
        alive -= set(gone)
        assert set(np.nonzero(~vh.read_agents(sim, "P")[1])[0]) == alive
        assert vh.num_agents(sim, "P") == len(alive)
    sim.close()
