"""Automata on rasters of one dimension, which have no neighbouring rows: lengths
of every remainder modulo a word, below, at and above the row kernel's tiles, as
long as its rule asks for, distances 1 to 4, against a numpy count."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (in two dimensions 8 offsets go by rows from 9 cells on, fewer from 10^6 cells x offsets on)
CASES = [(n, 4) for n in (9, 10, 11, 12, 123, 124, 125, 126, 130, 131, 132, 133, 249, 1000,
                          1_000_001)] + \
        [(166_667, 3), (166_670, 3), (250_000, 2), (250_003, 2), (500_002, 1)]


@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("n,distance", CASES)
def test_one_dimension(vh, n, distance, periodic):
    rng = np.random.default_rng(n + distance)
    birth, survive = 0b1101010, 0b0011100
    a = rng.random(n) < 0.4
    m = (vh.ModelTypes().register_agenttype("Cell", [("alive", "bool")], ":Immortal")
         .register_edgetype("Neighbor", [], ":Stateless", target="Cell").create_model("Line"))
    sim = vh.create_simulation(m)
    vh.add_raster(sim, "raster", (n,), "Cell", alive=a)
    vh.connect_raster_neighbors(sim, "raster", "Neighbor", distance=distance, periodic=periodic,
                                implicit=True)
    vh.finish_init(sim)
    for _ in range(3):
        vh.apply_(sim, "life", ["Cell"], ["Cell", "Neighbor"], ["Cell"],
                  params=[m["Neighbor"].index, birth, survive])
        p = np.pad(a.astype(np.int64), distance, mode="wrap" if periodic else "constant")
        c = sum(p[distance + k:distance + k + n] for k in range(-distance, distance + 1)) - a
        a = (np.where(a, survive, birth) >> c & 1).astype(bool)
        np.testing.assert_array_equal(vh.rastervalues(sim, "raster", "alive").astype(bool), a)
    sim.close()
