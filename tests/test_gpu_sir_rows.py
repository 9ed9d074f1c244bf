"""SIR steps around the edge count from which rows are read after the agent's own
state (4*10^5): states and days equal the oracle's, from the mask and from the
state bytes, for rows shorter than a batch of sources, as long, and longer."""
import ctypes as C

import numpy as np
import pytest

from oracle import models as om

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shared", [False, True])
@pytest.mark.parametrize("n,degree", [(39_999, 10), (40_000, 10), (133_333, 3), (133_334, 3),
                                      (24_999, 16), (25_000, 16), (13_333, 30), (13_334, 30),
                                      (70_001, 15)])
def test_steps(vh, n, degree, shared):
    from vahana_gb300 import models
    from vahana_gb300._lib import check, lib
    run = models.build_sir(n=n, degree=degree, seed=n)
    state, days = models.sir_initial_state(n, n)
    vh.finish_init(run.sim)
    if shared:
        p = C.c_void_p()
        check(lib().vg_agent_field_device_ptr(run.sim._h, run.sim.T("Person").index, 0, C.byref(p)))
    frm, to = om.gen_uniform_out(n, degree, n)
    for _ in range(25):
        run.step()
    ref = om.run_sir(n, frm, to, state, days, 0.05, 7, n, 25)
    for got, want in zip(vh.read_agents(run.sim, "Person")[0].values(), ref):
        np.testing.assert_array_equal(got, want)
    run.close()
