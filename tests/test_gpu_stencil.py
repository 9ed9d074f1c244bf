"""Cellular automata on implicit raster edges of every metric
(connect_raster_neighbors!, src/Raster.jl:82-167): the row kernel for Bool
cells (k_life_rows) and the general one behind it (UInt8 cells, distances
beyond its reach, dimensions no larger than the reach) against a direct numpy
count of the offsets, for 1 to 4 dimensions, row lengths of every remainder
modulo a word, and sizes below, at and above its tiles of 128 x 32 cells."""
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def offsets(nd, metric, distance):
    d = int(distance)
    for off in itertools.product(range(-d, d + 1), repeat=nd):
        r = {"chebyshev": 0, "euclidean": np.sqrt(sum(v * v for v in off)),
             "manhatten": sum(abs(v) for v in off)}[metric]
        if any(off) and r <= distance:
            yield off


def count(a, offs, periodic):
    c = np.zeros(a.shape, np.int64)
    for off in offs:
        s = np.roll(a, off, axis=range(a.ndim))
        if not periodic:  # nothing comes in over the border
            for ax, v in enumerate(off):
                idx = [slice(None)] * a.ndim
                idx[ax] = slice(0, v) if v > 0 else slice(a.shape[ax] + v, None) if v < 0 \
                    else slice(0, 0)
                s[tuple(idx)] = 0
        c += s
    return c


CASES = [((n, 7), "chebyshev", 1.5) for n in (9, 10, 11, 123, 124, 125, 126, 127, 129, 249)] + [
    ((n, 900), "chebyshev", 1) for n in (5, 9, 713, 1001)] + [
    ((n, 1100), "manhatten", 1) for n in (17, 18, 301)] + [
    ((129, 31), "manhatten", 1), ((130, 32), "euclidean", 2), ((127, 33), "chebyshev", 2),
    ((133, 65), "manhatten", 3), ((64, 34), "euclidean", 3.5), ((66, 40), "chebyshev", 4),
    ((70, 40), "manhatten", 5), ((300,), "chebyshev", 2), ((3,), "chebyshev", 1),
    ((2, 9), "manhatten", 2), ((33, 18, 5), "euclidean", 1), ((35, 18, 6), "chebyshev", 1),
    ((130, 34, 7), "manhatten", 2), ((17, 9, 4, 3), "chebyshev", 1),
    ((18, 9, 5, 4), "euclidean", 1.5)]


@pytest.mark.parametrize("dtype", ["bool", "u8"])
@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("dims,metric,distance", CASES)
def test_automaton(vh, dims, metric, distance, periodic, dtype):
    rng = np.random.default_rng(sum(dims) + int(periodic))
    birth, survive = 0b1101000, 0b1111100 | 1 << 30
    if metric == "chebyshev" and distance == 1 and len(dims) == 2:
        birth, survive = 8, 12
    a = (rng.random(dims) < 0.35).astype(np.uint8)
    m = (vh.ModelTypes().register_agenttype("Cell", [("alive", dtype)], ":Immortal")
         .register_edgetype("Neighbor", [], ":Stateless", target="Cell").create_model("Automaton"))
    sim = vh.create_simulation(m)
    vh.add_raster(sim, "raster", dims, "Cell", alive=a.astype("bool" if dtype == "bool" else "u1"))
    vh.connect_raster_neighbors(sim, "raster", "Neighbor", distance=distance, metric=metric,
                                periodic=periodic, implicit=True)
    vh.finish_init(sim)
    offs = list(offsets(len(dims), metric, distance))
    for _ in range(3):
        vh.apply_(sim, "life", ["Cell"], ["Cell", "Neighbor"], ["Cell"],
                  params=[m["Neighbor"].index, birth, survive])
        c = count(a, offs, periodic)
        rule = np.where(a > 0, survive, birth)
        a = np.where(c < 31, (rule >> np.minimum(c, 31)) & 1, 0).astype(np.uint8)
        got = vh.rastervalues(sim, "raster", "alive").astype(np.uint8)
        np.testing.assert_array_equal(got, a)
    sim.close()
