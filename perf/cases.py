"""The work a user of the framework has it do, as timed cases.

A case is a simulation of one of the kinds below, built once (`prepare`),
and one pass of its step loop with the results a user reads (`run`).  Every
call goes through the Python mirror of the API (`vahana_gb300.api`), the
test-model builders, the ensemble and the serving client.

  sir         contagion: the initial state is written, `steps` transitions
              run, the final state is read (a replicate of an experiment)
  opinion     bounded confidence with the state kept on the device
  host        bounded confidence for a program that keeps the opinions in its
              own (pinned) memory: one apply_host per step
  life        Life on a raster with walkers whose walker -> cell edges are
              rebuilt every step
  stencil     a cellular automaton on a raster of any size, dimension,
              metric and distance, periodic or bounded
  ensemble    many SIR instances of uneven size stepped together
  serve       jobs of both models submitted to a running server
  turnover    mortal agents: newcomers are added with their ties, look at
              their neighbours, die, and their edges go
  rewire      a contact network rebuilt every step from the friendships
              (with two columns of payload), then read by the agents
  foragers    mobile agents that move, look at the cells around them
              (move_to with a distance) and collect what they see
  statistics  mapreduce over the agents' columns after a step
"""
import ctypes as C
import math
import os
import sys
import time

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "vahana.jl_gb300"))

from vahana_gb300 import api, models, serve  # noqa: E402
from vahana_gb300._lib import check, lib  # noqa: E402


def listed():
    return [
        # one small replicate, checked at every step: launches and latency
        {"name": "sir_small", "kind": "sir", "n": 1000, "degree": 7, "steps": 50,
         "async": False},
        # the contagion model at its stated size, steps queued
        {"name": "sir_100k", "kind": "sir", "n": 100_000, "degree": 10, "steps": 100,
         "async": True},
        # an ordinary opinion network driven from host memory
        {"name": "opinion_host_1m", "kind": "host", "n": 1_000_003, "degree": 20, "steps": 5,
         "graph": "host"},
        # the headline size: power-law graph, 2e8 weighted edges
        {"name": "opinion_10m", "kind": "opinion", "n": 10_000_000, "degree": 20, "steps": 10,
         "graph": "device"},
        # the raster workload with a million walkers
        {"name": "life_walkers_4096", "kind": "life", "w": 4096, "h": 4096,
         "walkers": 1_000_000, "steps": 20, "edges": False},
        # a bounded raster of odd size and a wider neighbourhood
        {"name": "stencil_odd", "kind": "stencil", "d0": 2047, "d1": 1531, "d2": 0,
         "metric": "euclidean", "distance": 2.0, "periodic": False, "steps": 10},
        # the ensemble of the parameter sweep
        {"name": "ensemble_512", "kind": "ensemble", "instances": 512, "lo": 1000, "hi": 100_000,
         "steps": 200},
        # a burst of small and middling jobs at a running server
        {"name": "serve_24", "kind": "serve", "jobs": 24, "lo": 1000, "hi": 100_000,
         "steps_lo": 50, "steps_hi": 200},
        # births, deaths and their edges in a population of 2e5
        {"name": "turnover_200k", "kind": "turnover", "n": 200_000, "degree": 5,
         "newcomers": 20_000, "steps": 2},
        # a contact network of 2e6 edges made anew each step
        {"name": "rewire_100k", "kind": "rewire", "n": 100_000, "degree": 10, "steps": 2},
        # mobile agents that look one cell around themselves
        {"name": "foragers_100k", "kind": "foragers", "w": 1000, "h": 800, "n": 100_000,
         "distance": 1.0, "steps": 2},
        # the statistics taken after a step, four columns of 5e6 agents
        {"name": "statistics_5m", "kind": "statistics", "n": 5_000_000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sir", "opinion", "host", "life", "stencil", "ensemble", "serve",
                       "turnover", "rewire", "foragers", "statistics"])
    if kind == "sir":
        return {"kind": kind, "n": _log(rng, 500, 1_000_000), "degree": rng.randint(5, 30),
                "steps": rng.randint(20, 100), "async": rng.random() < 0.5}
    if kind in ("opinion", "host"):
        # graphs made by the program up to 1e6 agents, larger ones on the device
        n = _log(rng, 1000, 6_000_000 if kind == "opinion" else 3_000_000)
        return {"kind": kind, "n": n, "degree": rng.randint(5, 30), "steps": rng.randint(2, 10),
                "graph": "host" if n <= 1_000_000 else "device"}
    if kind == "life":
        w, h = _log(rng, 60, 4096), _log(rng, 60, 4096)
        walkers = max(1, int(w * h * rng.choice([0.01, 0.06, 0.3])))
        return {"kind": kind, "w": w, "h": h, "walkers": min(walkers, 1_000_000),
                "steps": rng.randint(5, 20), "edges": w * h <= 1_000_000}
    if kind == "stencil":
        d2 = rng.choice([0, 0, rng.randint(3, 90)])
        d0, d1 = _log(rng, 30, 300 if d2 else 3000), _log(rng, 30, 300 if d2 else 3000)
        return {"kind": kind, "d0": d0, "d1": d1, "d2": d2,
                "metric": rng.choice(["chebyshev", "euclidean", "manhatten"]),
                "distance": float(rng.choice([1, 1, 2])), "periodic": rng.random() < 0.6,
                "steps": rng.randint(5, 10)}
    if kind == "ensemble":
        return {"kind": kind, "instances": rng.randint(8, 256), "lo": 1000,
                "hi": _log(rng, 5000, 100_000), "steps": rng.randint(50, 200)}
    if kind == "serve":
        return {"kind": kind, "jobs": rng.randint(4, 32), "lo": 1000,
                "hi": _log(rng, 5000, 100_000), "steps_lo": 50,
                "steps_hi": rng.randint(60, 200)}
    if kind == "turnover":
        n = _log(rng, 2000, 500_000)
        return {"kind": kind, "n": n, "degree": rng.randint(2, 8),
                "newcomers": max(1, int(n * rng.uniform(0.02, 0.2))), "steps": rng.randint(1, 3)}
    if kind == "rewire":
        return {"kind": kind, "n": _log(rng, 2000, 300_000), "degree": rng.randint(3, 15),
                "steps": rng.randint(1, 3)}
    if kind == "foragers":
        return {"kind": kind, "w": _log(rng, 50, 1500), "h": _log(rng, 50, 1500),
                "n": _log(rng, 1000, 200_000), "distance": float(rng.choice([1, 1, 2])),
                "steps": rng.randint(1, 3)}
    return {"kind": kind, "n": _log(rng, 1000, 5_000_000)}


# ------------------------------------------------------------------ helpers
class Device:
    """A field of an agent type in device memory, for a consumer that takes
    device arrays; keeps the simulation alive."""

    def __init__(self, sim, T, field, typestr):
        t = sim.T(T)
        p = C.c_void_p()
        check(lib().vg_agent_field_device_ptr(sim._h, t.index, t.field_index(field), C.byref(p)))
        self.sim = sim
        self.__cuda_array_interface__ = {
            "shape": (api.agent_slots(sim, T),), "typestr": typestr, "data": (p.value, False),
            "version": 2, "strides": None}


def device_column(sim, T, field, typestr):
    return torch.as_tensor(Device(sim, T, field, typestr), device="cuda")


class State:
    """What a program holds: the simulation (or server) and its step calls."""

    def __init__(self, case, **kw):
        self.case = case
        self.__dict__.update(kw)


class Held:
    """Closes an ensemble or a server with the program's last reference."""

    def __init__(self, obj):
        self.obj = obj

    def __del__(self):
        self.obj.close()


def _rng(seed, salt):
    return np.random.default_rng([int(seed), salt])


def _pinned(a):
    t = torch.from_numpy(a).pin_memory()
    return t, t.numpy()


def _opinion_inputs(case, seed):
    """Opinions, and for graphs made by the program its power-law edges
    (sources and targets proportional to i^(-2/3), capped near 1 % of the
    agents' mean; weights in (0, 1])."""
    n, ne = case["n"], case["n"] * case["degree"]
    x = _rng(seed, 1).random(n)
    if case["graph"] == "device":
        return x, None
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 7 + 3)
    w = torch.arange(1, n + 1, device="cuda", dtype=torch.float64).pow_(-2.0 / 3.0)
    w = torch.clamp(w, max=float(w[min(n - 1, max(1, n // 2000))]))
    cdf = torch.cumsum(w, 0)
    perm = torch.randperm(n, device="cuda", generator=g)
    u = torch.rand(2, ne, device="cuda", dtype=torch.float64, generator=g) * cdf[-1]
    ends = torch.searchsorted(cdf, u).clamp_(max=n - 1)
    frm, to = perm[ends[0]], perm[ends[1]]
    wt = 1.0 - torch.rand(ne, device="cuda", dtype=torch.float64, generator=g)
    return x, (frm, to, wt)


def _ids(T, idx):
    """Agent ids of 0-based indices (device tensor) as a host array."""
    return (idx + ((T.index << 56) + 1)).cpu().numpy().view(np.uint64)


def _opinion_sim(case, seed):
    model = models.opinion_model()
    sim = api.create_simulation(model)
    x, edges = _opinion_inputs(case, seed)
    api.add_agents(sim, "Opinion", case["n"], x=x)
    T, E = model["Opinion"], model["Weight"]
    if edges is None:
        check(lib().vg_gen_chung_lu_edges(sim._h, E.index, T.index, case["n"] * case["degree"],
                                          float(case["degree"]), 2.5, 1e4, int(seed), 0))
    else:
        api.add_edges(sim, "Weight", _ids(T, edges[0]), _ids(T, edges[1]),
                      w=edges[2].cpu().numpy())
    api.finish_init(sim)
    params = [E.index, 0.3, 0.5, 0.5, models.OPINION_HUB_THRESHOLD]
    return sim, x, (["Opinion"], ["Opinion", "Weight"], ["Opinion"]), params


def _random_graph(seed, salt, n, degree):
    """degree in-edges per agent on average, ends uniform."""
    r = _rng(seed, salt)
    frm = r.integers(0, n, n * degree)
    to = r.integers(0, n, n * degree)
    return frm, to


def _np_ids(T, idx):
    return (idx.astype(np.uint64) + np.uint64(1)) | np.uint64(T.index << 56)


# ------------------------------------------------------------------ prepare
def _prepare_sir(case, seed):
    run = models.build_sir(n=case["n"], degree=case["degree"], seed=seed)
    api.finish_init(run.sim)
    api.set_async(run.sim, case["async"])
    state, days = models.sir_initial_state(case["n"], seed)
    return State(case, sim=run.sim, step=run.step, state=state, days=days)


def _prepare_opinion(case, seed):
    sim, x, args, params = _opinion_sim(case, seed)
    api.set_async(sim, True)
    return State(case, sim=sim, step=api.prepare_apply(sim, "bounded_confidence", *args,
                                                       params=params))


def _prepare_host(case, seed):
    sim, x, args, params = _opinion_sim(case, seed)
    t0, x0 = _pinned(x)
    t1, x1 = _pinned(np.empty_like(x))
    t2, x2 = _pinned(np.empty_like(x))
    return State(case, sim=sim, args=args, params=params, bufs=(x0, x1, x2), keep=(t0, t1, t2))


def _prepare_life(case, seed):
    w, h, n = case["w"], case["h"], case["walkers"]
    r = _rng(seed, 2)
    model = models.life_model()
    sim = api.create_simulation(model)
    api.add_raster(sim, "raster", (w, h), "Cell", alive=r.random(w * h, dtype=np.float32) < 0.3)
    api.connect_raster_neighbors(sim, "raster", "Neighbor", implicit=True)
    x = r.integers(1, w + 1, n).astype(np.int32)
    y = r.integers(1, h + 1, n).astype(np.int32)
    ids = api.add_agents(sim, "Walker", n, x=x, y=y)
    api.add_edges(sim, "OnCell", ids, _np_ids(model["Cell"], (x - 1) + (y.astype(np.int64) - 1) * w))
    api.finish_init(sim)
    api.set_async(sim, True)
    life = api.prepare_apply(sim, "life", ["Cell"], ["Cell", "Neighbor"], ["Cell"],
                             params=[model["Neighbor"].index])
    walk = api.prepare_apply(sim, "random_walk", ["Walker"], ["Walker"], ["Walker", "OnCell"],
                             params=[model["OnCell"].index, 0, seed])
    return State(case, sim=sim, life=life, walk=walk)


def _dims(case):
    return tuple(d for d in (case["d0"], case["d1"], case["d2"]) if d)


def _prepare_stencil(case, seed):
    dims = _dims(case)
    model = (api.ModelTypes().register_agenttype("Cell", [("alive", "bool")], ":Immortal")
             .register_edgetype("Neighbor", [], ":Stateless", target="Cell")
             .create_model("Automaton"))
    sim = api.create_simulation(model)
    api.add_raster(sim, "raster", dims, "Cell",
                   alive=_rng(seed, 3).random(int(np.prod(dims)), dtype=np.float32) < 0.35)
    api.connect_raster_neighbors(sim, "raster", "Neighbor", distance=case["distance"],
                                 metric=case["metric"], periodic=case["periodic"], implicit=True)
    api.finish_init(sim)
    api.set_async(sim, True)
    # birth on 3, survival on 2 and 3; wider neighbourhoods also 4..6
    moore = len(dims) == 2 and case["distance"] == 1 and case["metric"] == "chebyshev"
    masks = [8, 12] if moore else [0b1101000, 0b1111100]
    step = api.prepare_apply(sim, "life", ["Cell"], ["Cell", "Neighbor"], ["Cell"],
                             params=[model["Neighbor"].index] + masks)
    return State(case, sim=sim, step=step)


def _sizes(case, k):
    """k sizes spread evenly over the logarithm of lo..hi, in a mixed order."""
    q = (np.arange(k) + 0.5) / k
    n = (case["lo"] * (case["hi"] / case["lo"]) ** q).astype(np.int64)
    return n[np.random.default_rng(k).permutation(k)]


def _prepare_ensemble(case, seed):
    k, r = case["instances"], _rng(seed, 4)
    n = _sizes(case, k)
    batch = models.Batch(n, r.integers(5, 31, k), r.uniform(0.01, 0.1, k), r.integers(5, 11, k),
                         r.integers(1, 1 << 31, k))
    batch.tuning()
    return State(case, batch=batch, held=Held(batch))


def _prepare_serve(case, seed):
    r = _rng(seed, 5)
    specs = []
    for j, n in enumerate(int(x) for x in _sizes(case, case["jobs"])):
        deg = int(r.integers(5, 31))
        steps = int(r.integers(case["steps_lo"], case["steps_hi"] + 1))
        s = int(r.integers(1, 1 << 31))
        if j % 2 == 0:
            specs.append(serve.sir_job(n, degree=deg, steps=steps, seed=s,
                                       beta=float(r.uniform(0.01, 0.1)),
                                       recovery=int(r.integers(5, 11)), keep_state=True))
        else:
            specs.append(serve.opinion_job(n, mean_degree=deg, steps=steps, seed=s, wmax=1e3,
                                           keep_state=True))
    server = serve.Server(budget_bytes=32 << 30)
    return State(case, server=server, held=Held(server), specs=specs)


def _prepare_turnover(case, seed):
    n, m = case["n"], case["newcomers"]
    model = (api.ModelTypes()
             .register_agenttype("Person", [("gen", "i64"), ("sum", "i64")])
             .register_edgetype("Tie", [("id", "i64")])
             .register_edgetype("Host", [], ":Stateless")
             .create_model("Turnover"))
    sim = api.create_simulation(model)
    gen = -_rng(seed, 6).integers(1, 50, n)  # residents below 0, newcomers above
    ids = api.add_agents(sim, "Person", n, gen=gen, sum=0)
    frm, to = _random_graph(seed, 7, n, case["degree"])
    api.add_edges(sim, "Tie", ids[frm], ids[to], id=frm)
    hosts = ids[_rng(seed, 8).permutation(n)[:m]]
    api.add_edges(sim, "Host", hosts, hosts)
    api.finish_init(sim)
    tie = model["Tie"].index
    birth = api.prepare_apply(sim, "spawn", ["Person"], ["Person", "Host"], ["Person", "Tie"],
                              add_existing=["Tie"], with_edge="Host", params=[1, 100, tie])
    look = api.prepare_apply(sim, "neighbor_sum", ["Person"], ["Person", "Tie"], ["Person"],
                             params=[tie, 0, 1])
    death = api.prepare_apply(sim, "die_if", ["Person"], ["Person"], ["Person"],
                              params=[1, 0, 1.0])
    return State(case, sim=sim, birth=birth, look=look, death=death)


def _rewire_inputs(case, seed):
    frm, to = _random_graph(seed, 9, case["n"], case["degree"])
    return frm, to, _rng(seed, 10).random(case["n"])


def _prepare_rewire(case, seed):
    model = (api.ModelTypes()
             .register_agenttype("Person", [("v", "f64"), ("s", "f64")], ":Immortal")
             .register_edgetype("Friend", [("w", "f64"), ("since", "i32")])
             .register_edgetype("Contact", [("v", "f64")], target="Person")
             .create_model("Rewire"))
    sim = api.create_simulation(model)
    frm, to, v = _rewire_inputs(case, seed)
    ids = api.add_agents(sim, "Person", case["n"], v=v, s=0.0)
    api.add_edges(sim, "Friend", ids[frm], ids[to], w=0.5, since=frm.astype(np.int32))
    api.finish_init(sim)
    friend, contact = model["Friend"].index, model["Contact"].index
    meet = api.prepare_apply(sim, "link_neighbors", ["Person"], ["Person", "Friend"],
                             ["Person", "Contact"], params=[friend, contact])
    look = api.prepare_apply(sim, "neighbor_sum", ["Person"], ["Person", "Contact"], ["Person"],
                             params=[contact, 0, 1])
    again = api.prepare_apply(sim, "readd_edges", ["Person"], ["Person", "Friend"],
                              ["Person", "Friend"], params=[friend])
    return State(case, sim=sim, meet=meet, look=look, again=again)


def _prepare_foragers(case, seed):
    w, h, n = case["w"], case["h"], case["n"]
    r = _rng(seed, 11)
    model = (api.ModelTypes()
             .register_agenttype("Cell", [("food", "i64")], ":Immortal")
             .register_agenttype("Forager", [("x", "i32"), ("y", "i32"), ("seen", "i64")],
                                 ":Immortal")
             .register_edgetype("OnCell", [], ":Stateless", target="Cell")
             .register_edgetype("Sees", [], ":Stateless")
             .create_model("Foragers"))
    sim = api.create_simulation(model)
    api.add_raster(sim, "raster", (w, h), "Cell", food=r.integers(0, 1 << 40, w * h))
    api.add_agents(sim, "Forager", n, x=r.integers(1, w + 1, n).astype(np.int32),
                   y=r.integers(1, h + 1, n).astype(np.int32), seen=0)
    api.finish_init(sim)
    sees, on = model["Sees"].index, model["OnCell"].index
    walk = api.prepare_apply(sim, "random_walk", ["Forager"], ["Forager"], ["Forager", "OnCell"],
                             params=[on, 0, seed])
    move = api.prepare_apply(sim, "move_to", ["Forager"], ["Forager"], ["Forager", "Sees"],
                             params=[0, sees, -1, case["distance"], 0, 1, 0, 0])
    look = api.prepare_apply(sim, "neighbor_sum", ["Forager"], ["Cell", "Forager", "Sees"],
                             ["Forager"], params=[sees, 0, 2])
    return State(case, sim=sim, walk=walk, move=move, look=look)


def _statistics_inputs(case, seed):
    r = _rng(seed, 12)
    n = case["n"]
    return {"x": r.random(n), "wealth": np.exp(r.standard_normal(n)),
            "state": r.integers(0, 3, n).astype(np.uint8),
            "age": r.integers(0, 100, n).astype(np.int32)}


def _prepare_statistics(case, seed):
    model = (api.ModelTypes()
             .register_agenttype("Person", [("x", "f64"), ("wealth", "f64"), ("state", "u8"),
                                            ("age", "i32")], ":Immortal")
             .create_model("Statistics"))
    sim = api.create_simulation(model)
    api.add_agents(sim, "Person", case["n"], **_statistics_inputs(case, seed))
    api.finish_init(sim)
    return State(case, sim=sim)


def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, int(seed))


# ---------------------------------------------------------------------- run
def _run_sir(s):
    api.write_agents(s.sim, "Person", state=s.state, days=s.days)
    for _ in range(s.case["steps"]):
        s.step()
    cols, _ = api.read_agents(s.sim, "Person")
    return cols


def _run_opinion(s):
    for _ in range(s.case["steps"]):
        s.step()
    api.synchronize(s.sim)
    return device_column(s.sim, "Opinion", "x", "<f8")


def _run_host(s):
    x0, a, b = s.bufs
    src = x0
    for _ in range(s.case["steps"]):
        dst = b if src is a else a
        api.apply_host(s.sim, "bounded_confidence", *s.args, "Opinion", {"x": src},
                       out={"x": dst}, params=s.params)
        src = dst
    return src


def _run_life(s):
    for _ in range(s.case["steps"]):
        s.life()
        s.walk()
    api.synchronize(s.sim)
    out = {"alive": device_column(s.sim, "Cell", "alive", "|u1")}
    out["x"] = device_column(s.sim, "Walker", "x", "<i4")
    out["y"] = device_column(s.sim, "Walker", "y", "<i4")
    if s.case["edges"]:
        rp, frm, _ = api.read_edges(s.sim, "OnCell", "Cell")
        out["row_ptr"], out["from"] = rp.view(np.int64), frm.view(np.int64)
    return out


def _run_stencil(s):
    for _ in range(s.case["steps"]):
        s.step()
    api.synchronize(s.sim)
    return device_column(s.sim, "Cell", "alive", "|u1")


def _run_ensemble(s):
    b = s.batch
    b.step(s.case["steps"], mode=3)
    got = [b.states(i) for i in range(b.n)]
    return {"state": np.concatenate([g[0] for g in got]),
            "days": np.concatenate([g[1] for g in got])}


def _run_serve(s):
    ids = [s.server.submit(spec) for spec in s.specs]
    done = 0
    while done < len(ids):
        got = s.server.poll()
        if not got:
            time.sleep(1e-4)
        done += len(got)
    states = [s.server.job_state(i, spec) for i, spec in zip(ids, s.specs)]
    return {"state": np.concatenate([g[0] for g in states[0::2]]),
            "days": np.concatenate([g[1] for g in states[0::2]]),
            "x": np.concatenate(states[1::2])}


def _run_turnover(s):
    for _ in range(s.case["steps"]):
        s.birth()
        s.look()
        s.death()
    cols, died = api.read_agents(s.sim, "Person")
    rp, frm, pl = api.read_edges(s.sim, "Tie", "Person")
    return {"gen": cols["gen"], "sum": cols["sum"], "died": died, "row_ptr": rp.view(np.int64),
            "from": frm.view(np.int64), "id": pl["id"]}


def _run_rewire(s):
    for _ in range(s.case["steps"]):
        s.meet()
        s.look()
        s.again()
    cols, _ = api.read_agents(s.sim, "Person")
    rp, frm, pl = api.read_edges(s.sim, "Contact", "Person")
    return {"s": cols["s"], "row_ptr": rp.view(np.int64), "from": frm.view(np.int64),
            "v": pl["v"]}


def _run_foragers(s):
    for _ in range(s.case["steps"]):
        s.walk()
        s.move()
        s.look()
    cols, _ = api.read_agents(s.sim, "Forager")
    rp, frm, _ = api.read_edges(s.sim, "Sees", "Forager")
    return {"x": cols["x"], "y": cols["y"], "seen": cols["seen"], "row_ptr": rp.view(np.int64),
            "from": frm.view(np.int64)}


def _run_statistics(s):
    mr = api.mapreduce
    return {"x": mr(s.sim, "x", "+", "Person"), "wealth": mr(s.sim, "wealth", "+", "Person"),
            "richest": mr(s.sim, "wealth", "max", "Person"),
            "infected": mr(s.sim, ("==", "state", 1), "+", "Person"),
            "years": mr(s.sim, "age", "+", "Person")}


def run(state):
    return globals()["_run_" + state.case["kind"]](state)


# ---------------------------------------------------------------- exact, work
def _exact_opinion(case, seed):
    x, edges = _opinion_inputs(case, seed)
    if edges is None:
        return None
    frm, to, w = edges
    x = torch.from_numpy(x).cuda()
    for _ in range(case["steps"]):
        xj = x[frm]
        q = (xj - x[to]).abs() < 0.3
        wq = torch.where(q, w, torch.zeros_like(w))
        sw = torch.zeros_like(x).index_add_(0, to, wq)
        swx = torch.zeros_like(x).index_add_(0, to, wq * xj)
        x = torch.where(sw > 0, 0.5 * x + 0.5 * (swx / torch.where(sw > 0, sw, 1.0)), x)
    return x


def exact(case, seed):
    kind = case["kind"]
    if kind == "opinion":
        return _exact_opinion(case, seed)
    if kind == "host":
        x = _exact_opinion(case, seed)
        return None if x is None else x.cpu().numpy()
    if kind == "rewire":
        frm, to, v = _rewire_inputs(case, seed)
        s = np.bincount(to, v[frm], case["n"]) + np.bincount(frm, v[to], case["n"])
        return {"s": s, "row_ptr": None, "from": None, "v": None}
    if kind == "statistics":
        c = _statistics_inputs(case, seed)
        return {"x": math.fsum(c["x"]), "wealth": math.fsum(c["wealth"]),
                "richest": float(c["wealth"].max()), "infected": None, "years": None}
    return None


def work(case):
    kind, steps = case["kind"], case.get("steps", 1)
    if kind == "sir":
        n, e = case["n"], case["n"] * case["degree"]
        # row bounds, sources, state and days in; state and days out
        return {"bytes": steps * (4 * e + 14 * n), "flops": steps * e}
    if kind in ("opinion", "host"):
        n, e = case["n"], case["n"] * case["degree"]
        return {"bytes": steps * (12 * e + 20 * n), "flops": 4 * steps * e}
    if kind == "life":
        c, w = case["w"] * case["h"], case["walkers"]
        # cells in and out; walkers in and out; the new row pointers and sources
        return {"bytes": steps * (2 * c + 16 * w + 4 * c + 4 * w), "flops": steps * 9 * c}
    if kind == "stencil":
        c = int(np.prod(_dims(case)))
        return {"bytes": steps * 2 * c, "flops": steps * 9 * c}
    if kind == "ensemble":
        # mean of a log-uniform size, mean out-degree 17.5
        n = case["instances"] * (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])
        return {"bytes": steps * n * (4 * 17.5 + 16), "flops": steps * n * 17.5}
    if kind == "serve":
        n = case["jobs"] * (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])
        k = (case["steps_lo"] + case["steps_hi"]) / 2
        e = 17.5 * n
        return {"bytes": k * (0.5 * (4 * e + 14 * n) + 0.5 * (12 * e + 20 * n)) + 2 * 24 * e,
                "flops": k * 2.5 * e}
    if kind == "turnover":
        n, m = case["n"] + case["newcomers"], case["newcomers"]
        e = case["n"] * case["degree"] + 2 * m
        # three sweeps of the persons' columns and died flags; the ties read
        # by the sum, written with the newcomers' and written without them
        return {"bytes": steps * (3 * 34 * n + 5 * (12 * e + 4 * n)), "flops": steps * e}
    if kind == "rewire":
        n, e = case["n"], case["n"] * case["degree"]
        # friends read twice and written once, contacts written and read
        return {"bytes": steps * (3 * 32 * n + 3 * 16 * e + 2 * 2 * 12 * e),
                "flops": steps * 2 * e}
    if kind == "foragers":
        n, c = case["n"], case["w"] * case["h"]
        k = (2 * int(case["distance"]) + 1) ** 2
        return {"bytes": steps * (3 * 32 * n + 8 * c + 4 * c + 4 * n + 2 * (4 * n * k + 4 * n)),
                "flops": steps * n * k}
    return {"bytes": case["n"] * 21.0, "flops": case["n"] * 5.0}
