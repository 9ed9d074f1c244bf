"""The parallel sequential Float sum (csrc/vg_fold.cuh) where the sum changes
its binade: in more tiles (2048 elements) than have chunk maps, several times
in a chunk of 64 elements or by many binades at once, at the ends of tiles
and chunks, through zero and to infinity.  Bit-identical to the loop
(tolerance 0)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TILE = 2048


def data(kind, n, rng):
    i = np.arange(n)
    if kind == "swing":      # up and down over a power of two, tile by tile
        x = np.where((i // TILE) % 2 == 0, 1.0, -1.0) * rng.random(n) * 2 ** -4
        x[0] = 1000.0
    elif kind == "jumps":    # several binades in a chunk, up and down again
        x = rng.random(n)
        x[i % 1000 == 777] = 1e9
        x[i % 1000 == 779] = -1e9 + 3.0
    elif kind == "ends":     # the first or last element of a tile or chunk crosses
        x = rng.random(n) * 2.0 ** -30
        for k, at in enumerate((1, TILE - 1, TILE, 2 * TILE, 2 * TILE + 63, 3 * TILE + 64,
                                n - 1)):
            x[at % n] = 4.0 ** k
    elif kind == "zero":     # through zero, once per tile
        x = rng.random(n) - 0.5
        x[::TILE] = 0.0
        s = np.add.accumulate(x)
        x[TILE - 1::TILE] -= s[TILE - 1::TILE] - np.concatenate([[0.0], s[TILE - 1:-1:TILE]])[
            :s[TILE - 1::TILE].size]
    elif kind == "infinite":
        x = rng.random(n) * 2.0 ** 1013
    else:                    # steady: one crossing every 1, 2, 4, ... tiles
        x = 1.0 + rng.random(n)
        x[rng.random(n) < 0.01] *= -1
    return x


@pytest.mark.parametrize("kind", ["swing", "jumps", "ends", "zero", "infinite", "steady"])
@pytest.mark.parametrize("n", [3 * TILE, 3 * TILE + 1, 33 * TILE + 63, 300 * TILE - 1,
                               1025 * TILE + 65])
@pytest.mark.parametrize("mortal", [False, True])
def test_crossings(vh, n, kind, mortal):
    rng = np.random.default_rng(n + len(kind))
    with np.errstate(all="ignore"):
        x = data(kind, n, rng)
        dead = (rng.random(n) < 0.1).astype(np.int32)
        m = (vh.ModelTypes().register_agenttype("V", [("x", "f64"), ("dead", "i32")],
                                                *([] if mortal else [":Immortal"]))
             .create_model("Crossings"))
        sim = vh.create_simulation(m)
        vh.add_agents(sim, "V", n, x=x, dead=dead)
        vh.finish_init(sim)
        if mortal:
            vh.apply_(sim, "die_if", ["V"], ["V"], ["V"], params=[1, 1, 1.0])
            x = x[dead == 0]
        ref = np.add.accumulate(np.concatenate([[0.0], x]))[-1]
        got = np.float64(vh.mapreduce(sim, "x", "+", "V"))
    assert got.view(np.uint64) == ref.view(np.uint64) or (np.isnan(got) and np.isnan(ref)), \
        (n, kind, got, ref)
