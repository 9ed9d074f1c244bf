"""Life (B3/S23) on UInt8 cells that hold other values than 0 and 1: the
neighbours' values are summed, a sum of 3 makes a cell alive, a sum of 2 keeps
one that is not 0 -- at widths that take four cells per word and that do not,
against numpy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("dims", [(64, 40), (65, 40), (4, 5), (132, 17), (128, 8), (1000, 800),
                                  (1001, 800)])
@pytest.mark.parametrize("top", [2, 4])
def test_values_are_summed(vh, dims, periodic, top):
    rng = np.random.default_rng(dims[0] + top)
    m = (vh.ModelTypes().register_agenttype("Cell", [("v", "u8")], ":Immortal")
         .register_edgetype("Neighbor", [], ":Stateless", target="Cell").create_model("Values"))
    sim = vh.create_simulation(m)
    vh.add_raster(sim, "raster", dims, "Cell", v=np.zeros(dims, np.uint8))
    vh.connect_raster_neighbors(sim, "raster", "Neighbor", periodic=periodic, implicit=True)
    vh.finish_init(sim)
    for share in (0.1, 0.3, 0.6):
        a = np.where(rng.random(dims) < share, rng.integers(0, top, dims), 0).astype(np.uint8)
        vh.write_agents(sim, "Cell", v=a.ravel(order="F"))
        vh.apply_(sim, "life", ["Cell"], ["Cell", "Neighbor"], ["Cell"],
                  params=[m["Neighbor"].index])
        p = np.pad(a.astype(np.int64), 1, mode="wrap" if periodic else "constant")
        c = sum(p[1 + x:1 + x + dims[0], 1 + y:1 + y + dims[1]]
                for x in (-1, 0, 1) for y in (-1, 0, 1)) - a
        want = ((c == 3) | ((a != 0) & (c == 2))).astype(np.uint8)
        np.testing.assert_array_equal(vh.rastervalues(sim, "raster", "v"), want)
    sim.close()
