"""The sequential Float sum of mapreduce computed in parallel (csrc/vg_fold.cuh)
against the loop itself, reduced = x + reduced (src/AgentMethods.jl:533-565):
bit-identical (tolerance 0) at the edges of its tiles, chunks and rounds and
on the data where an addition can round up, down or to even, cross a power of
two, cancel, overflow or stay subnormal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 31, 33, 128, 4095, 4096, 8192, 8193, 3 * 4096 + 1, 1024 * 4096 + 4097]


def data(kind, n, rng):
    if kind == "grid":  # multiples of 2^-53: ties in the first binades
        return rng.integers(0, 1 << 53, n) * 2.0 ** -53
    if kind == "halves":  # a tie at nearly every addition once the sum is 2^53 or more
        x = rng.integers(0, 4, n) * 1.0
        x[0] = 2.0 ** 53
        return x
    if kind == "signs":
        return rng.standard_normal(n)
    if kind == "spread":
        return rng.standard_normal(n) * np.exp(rng.uniform(-300, 300, n))
    if kind == "cancel":  # the sum returns to zero, or nearly, all the time
        x = rng.random(n)
        x[1::2] = -x[0:n - 1:2]
        return x
    if kind == "negative":
        return -np.exp(rng.standard_normal(n))
    if kind == "tiny":
        return rng.random(n) * 2.0 ** -1060
    if kind == "huge":  # overflows to infinity on the way
        return rng.random(n) * 2.0 ** 1014
    x = rng.random(n)
    x[n // 2] = np.nan
    return x


@pytest.mark.parametrize("kind", ["grid", "halves", "signs", "spread", "cancel", "negative",
                                  "tiny", "huge", "nan"])
@pytest.mark.parametrize("n", SIZES)
def test_parallel_fold_equals_the_loop(vh, n, kind):
    rng = np.random.default_rng(n * 31 + len(kind))
    m = (vh.ModelTypes().register_agenttype("Val", [("x", "f64"), ("h", "f32")], ":Immortal")
         .create_model("Fold"))
    sim = vh.create_simulation(m)
    with np.errstate(all="ignore"):
        x = data(kind, n, rng)
        h = x.astype(np.float32)
        vh.add_agents(sim, "Val", n, x=x, h=h)
        vh.finish_init(sim)
        for col, init in ((x, 0.0), (x, -0.75), (h.astype(np.float64), 0.0)):
            ref = np.add.accumulate(np.concatenate([[init], col]))[-1]
            got = np.float64(vh.mapreduce(sim, "x" if col is x else "h", "+", "Val",
                                          init=init if init else None))
            if np.isnan(ref):
                assert np.isnan(got)
            else:
                assert got.view(np.uint64) == ref.view(np.uint64), (n, kind, init, got, ref)
    sim.close()


@pytest.mark.parametrize("dt", ["bool", "u8", "i8", "u16", "i16", "u32", "i32", "u64", "i64",
                                "f32", "f64"])
@pytest.mark.parametrize("n", [1, 255, 2048, 300_001])
def test_typed_reductions_equal_numpy(vh, n, dt):
    """Sums, extremes and comparisons (integral, fractional and NaN
    arguments) of every column type, exact."""
    rng = np.random.default_rng(n)
    np_dt = "bool" if dt == "bool" else {"u": "uint", "i": "int", "f": "float"}[dt[0]] + dt[1:]
    x = (rng.integers(0, 2, n) if dt == "bool" else
         rng.integers(0 if dt[0] == "u" else -100, 101, n)).astype(np_dt)
    m = (vh.ModelTypes().register_agenttype("Val", [("x", dt), ("u", "f64")])
         .create_model("Typed"))
    sim = vh.create_simulation(m)
    u = rng.random(n)
    vh.add_agents(sim, "Val", n, x=x, u=u)
    vh.finish_init(sim)
    for dead in (False, True):
        if dead:
            vh.apply_(sim, "die_if", ["Val"], ["Val"], ["Val"], params=[1, 1, 0.5])
        y = x[u < 0.5] if dead else x
        assert vh.mapreduce(sim, "x", "+", "Val") == y.sum(dtype="f8" if dt[0] == "f" else "i8")
        if y.size and dt != "bool":
            assert vh.mapreduce(sim, "x", "max", "Val") == y.max()
            assert vh.mapreduce(sim, "x", "min", "Val") == y.min()
        for arg in (1, -3, 0.5, float("nan"), 1e300, -1e300):
            z = y.astype("f8")
            for cmp, want in (("==", z == arg), ("!=", z != arg), ("<", z < arg), (">", z > arg)):
                assert vh.mapreduce(sim, (cmp, "x", arg), "+", "Val") == want.sum(), (cmp, arg)
    sim.close()
