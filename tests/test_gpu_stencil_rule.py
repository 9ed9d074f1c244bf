"""Automata at the sizes where the choice between rows and a cell per thread turns
(estimates of both forms' time): rasters of 2 to 4 dimensions with short, long, few
and many rows, stencils of one plane and of several, bounded and periodic, against a
numpy count.  Each shape lies beside another that takes the other form."""
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PAIRS = [  # (dims, metric, distance)
    ((9, 16), "manhatten", 1), ((9, 5000), "manhatten", 1), ((17, 5000), "manhatten", 1),
    ((100_001, 2), "manhatten", 1), ((10_001, 2), "manhatten", 1), ((1001, 3), "euclidean", 2),
    ((20, 8, 300), "manhatten", 1), ((20, 8, 30), "manhatten", 1), ((124, 32, 20), "manhatten", 1),
    ((125, 33, 20), "manhatten", 1), ((40, 12, 60), "chebyshev", 1), ((9, 8, 900), "chebyshev", 1),
    ((61, 24, 20), "euclidean", 2), ((3, 3, 2000), "manhatten", 2), ((2, 2, 2, 900), "chebyshev", 1),
    ((20, 12, 8, 8), "manhatten", 1), ((130, 8, 3, 3), "manhatten", 1), ((3, 3, 30, 40), "manhatten", 2),
    ((10, 40), "chebyshev", 1.5), ((33, 31), "chebyshev", 4), ((7, 900), "manhatten", 3)]


@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("dims,metric,distance", PAIRS)
def test_shapes(vh, dims, metric, distance, periodic):
    rng = np.random.default_rng(sum(dims))
    birth, survive = 0b1101000, 0b1111100 | 1 << 9
    a = rng.random(dims) < 0.3
    m = (vh.ModelTypes().register_agenttype("Cell", [("alive", "bool")], ":Immortal")
         .register_edgetype("Neighbor", [], ":Stateless", target="Cell").create_model("Rule"))
    sim = vh.create_simulation(m)
    vh.add_raster(sim, "raster", dims, "Cell", alive=a)
    vh.connect_raster_neighbors(sim, "raster", "Neighbor", distance=distance, metric=metric,
                                periodic=periodic, implicit=True)
    vh.finish_init(sim)
    d = int(distance)
    offs = [o for o in itertools.product(range(-d, d + 1), repeat=len(dims)) if any(o) and
            {"chebyshev": 0, "euclidean": np.sqrt(sum(v * v for v in o)),
             "manhatten": sum(abs(v) for v in o)}[metric] <= distance]
    for _ in range(2):
        vh.apply_(sim, "life", ["Cell"], ["Cell", "Neighbor"], ["Cell"],
                  params=[m["Neighbor"].index, birth, survive])
        p = np.pad(a.astype(np.int64), d, mode="wrap" if periodic else "constant")
        c = sum(p[tuple(slice(d + v, d + v + n) for v, n in zip(o, dims))] for o in offs)
        a = np.where(c < 31, np.where(a, survive, birth) >> np.minimum(c, 31) & 1, 0).astype(bool)
        np.testing.assert_array_equal(vh.rastervalues(sim, "raster", "alive").astype(bool), a)
    sim.close()
