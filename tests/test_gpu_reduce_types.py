"""mapreduce by the parallel tree (src/AgentMethods.jl:533-565) over every
column type, operator and comparison, against numpy: NaN, infinities, both
zeros, subnormal and extreme values, thresholds between and beyond the values,
columns shorter than a warp and at the edges of a thread's batch (8 x 256) and
of the 1024 blocks, with and without died agents.  Exact (Float + and * of
integers small enough that no sum or product rounds)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SIZES = [1, 31, 257, 2049, 1024 * 256 + 1, 1024 * 2048 + 3]


def column(dt, n, rng, special):
    if dt in ("f64", "f32"):
        x = rng.integers(-50, 50, n).astype(dt.replace("f", "float"))
        if special:
            pool = np.array([0.0, -0.0, np.inf, -np.inf, 1e-310, -1e-310, 2.5, -2.5, 1e30],
                            x.dtype)
            at = rng.integers(0, n, max(1, n // 3))
            x[at] = pool[rng.integers(0, pool.size, at.size)]
        return x
    info = np.iinfo(dt.replace("u", "uint") if dt[0] == "u" else dt.replace("i", "int"))
    x = rng.integers(max(info.min, -50), min(info.max, 50), n).astype(info.dtype)
    if special:
        x[rng.integers(0, n, max(1, n // 5))] = info.max
        x[rng.integers(0, n, max(1, n // 5))] = info.min
    return x


def jl(op, x):  # Julia's max and min: NaN wins, -0.0 is below +0.0
    if np.isnan(x).any():
        return np.nan
    m = x.max() if op == "max" else x.min()
    if m == 0:
        signs = np.signbit(x[x == 0])
        return (-0.0 if signs.all() else 0.0) if op == "max" else (-0.0 if signs.any() else 0.0)
    return m


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("dt", ["u8", "i8", "u16", "i16", "u32", "i32", "i64", "f32", "f64"])
def test_types(vh, dt, n):
    rng = np.random.default_rng(n + len(dt))
    special = n % 2 == 1
    x = column(dt, n, rng, special)
    nan = x.copy()
    if dt[0] == "f":
        nan[n // 2] = np.nan
    dead = (rng.random(n) < 0.2).astype(np.int32)
    m = (vh.ModelTypes().register_agenttype("A", [("x", dt), ("y", dt), ("dead", "i32")])
         .create_model("Reduce"))
    sim = vh.create_simulation(m)
    vh.add_agents(sim, "A", n, x=x, y=nan, dead=dead)
    vh.finish_init(sim)
    for alive in (np.ones(n, bool), dead == 0):
        if not alive.all():
            vh.apply_(sim, "die_if", ["A"], ["A"], ["A"], params=[1, 2, 1.0])
        for name, col in (("x", x[alive]), ("y", nan[alive])):
            for op in ("max", "min"):
                if not col.size:
                    continue
                got = vh.mapreduce(sim, name, op, "A")
                if dt[0] == "f":
                    lim = float(2 ** 63 - 1)
                    ref = jl(op, np.append(col.astype(np.float64), -lim if op == "max" else lim))
                    assert np.isnan(got) == np.isnan(ref)
                    assert np.isnan(ref) or np.float64(got).view(np.uint64) == \
                        np.float64(ref).view(np.uint64), (op, got, ref)
                else:
                    # (the fold starts from the operator's identity, -+typemax(Int64))
                    assert got == (max(int(col.max()), 1 - 2 ** 63) if op == "max" else
                                   min(int(col.min()), 2 ** 63 - 1))
            for arg in (0.0, -0.0, 2.5, 3.0, -7.0, 255.0, 1e300, -1e300, np.inf, np.nan):
                with np.errstate(all="ignore"):
                    c = col.astype(np.float64)
                    for cmp, ref in (("==", c == arg), ("!=", c != arg), ("<", c < arg),
                                     (">", c > arg)):
                        assert vh.mapreduce(sim, (cmp, name, arg), "+", "A") == ref.sum(), \
                            (cmp, arg)
        if dt[0] != "f":
            c = [int(v) for v in x[alive][:100_000]]
            if alive.sum() <= 100_000:
                wrap = lambda v: (v + 2 ** 63) % 2 ** 64 - 2 ** 63
                p = 1
                for v in c:
                    p = wrap(p * v)
                assert vh.mapreduce(sim, "x", "*", "A") == p
            with np.errstate(all="ignore"):
                assert vh.mapreduce(sim, "x", "+", "A") == x[alive].astype(np.int64).sum()
        elif not special:
            assert vh.mapreduce(sim, "x", "+", "A", ordered=False) == x[alive].sum(dtype=np.float64)
