"""Read-backs and the error word: edges that are widened on the device piece by
piece (pieces of 2^21), batch states read through pinned memory or past it,
and the kernels' error code, reported and cleared, with and without a line of
mapped memory.  Exact values, tolerance 0."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
NR = np.uint64((1 << 36) - 1)


@pytest.mark.parametrize("n,ne", [(1, 0), (1, 1), (7, 1 << 21), (300, (1 << 21) + 1),
                                  ((1 << 21) - 1, 5), (1 << 21, 4_200_000)])
@pytest.mark.parametrize("single", [False, True])
def test_edges(vh, n, ne, single):
    rng = np.random.default_rng(n + ne)
    m = (vh.ModelTypes().register_agenttype("P", []).register_agenttype("Q", [])
         .register_edgetype("E", [("w", "i32")], *([":SingleType"] if single else []),
                            **({"target": "P"} if single else {}))
         .create_model("Read"))
    sim = vh.create_simulation(m)
    p, q = vh.add_agents(sim, "P", n), vh.add_agents(sim, "Q", 3)
    both = p if single else np.concatenate([p, q])
    to = np.sort(rng.integers(0, n, ne))
    frm = both[rng.integers(0, both.size, ne)]
    w = rng.integers(-9, 9, ne).astype(np.int32)
    if ne:
        vh.add_edges(sim, "E", frm, p[to], w=w)
    vh.finish_init(sim)
    rp, got, cols = vh.read_edges(sim, "E", "P")
    want = np.concatenate([[0], np.cumsum(np.bincount(to, minlength=n))]).astype(np.uint64)
    k = rp.size
    np.testing.assert_array_equal(rp, want[:k])
    assert k == n + 1 or want[k - 1:].min() == ne
    np.testing.assert_array_equal(got[:ne], frm)
    np.testing.assert_array_equal(cols["w"][:ne], w)


@pytest.mark.parametrize("n", [40, 209_715, 209_716])  # 5 bytes an agent, 2^20 at a time
def test_batch_states(vh, n):
    from vahana_gb300 import models
    from vahana_gb300._lib import check, lib
    b = models.Batch([n, 33], [6, 6], [0.3, 0.3], [5, 5], [1, 2])
    b.step(3, mode=1)
    for i in (0, 1):
        b.step_one(i, 3)
        s, d = b.states(i)
        for x, y in zip((s, d), b.states(i, which=1)):
            np.testing.assert_array_equal(x, y)
        half, out = len(s) // 2, C.c_uint64()
        for want_s, want_d in ((True, False), (False, True), (True, True)):
            gs, gd = np.full(len(s), 77, np.uint8), np.full(len(s), 77, np.int32)
            check(lib().vg_batch_read_states2(
                b._h, i, 0, gs.ctypes.data_as(C.POINTER(C.c_uint8)) if want_s else None,
                gd.ctypes.data_as(C.POINTER(C.c_int32)) if want_d else None, half, C.byref(out)))
            assert out.value == len(s)
            for g, full, want in ((gs, s, want_s), (gd, d, want_d)):
                np.testing.assert_array_equal(g[:half], full[:half] if want else 77)
                assert (g[half:] == 77).all()


def _immortal(vh, m):
    sim = vh.create_simulation(m)
    vh.add_agents(sim, "A", 5, x=[0, 1, 0, 0, 1])
    vh.finish_init(sim)
    return sim


def _error_is_reported_once(vh, sim):
    for queued in (False, True):
        vh.set_async(sim, queued)
        with pytest.raises(Exception, match="device status 201"):
            vh.apply_(sim, "die_if", ["A"], ["A"], ["A"], params=[1, 0, 1.0])
            vh.synchronize(sim)
        vh.set_async(sim, False)
        vh.apply_(sim, "die_if", ["A"], ["A"], ["A"], params=[1, 0, 9.0])  # none dies
        vh.synchronize(sim)


def test_error_word(vh):
    m = vh.ModelTypes().register_agenttype("A", [("x", "i32")], ":Immortal").create_model("Imm")
    _error_is_reported_once(vh, _immortal(vh, m))
    # 4096 simulations hold a mapped line; the others read the word by a copy
    held = [_immortal(vh, m) for _ in range(4100)]
    for i in (0, 4095, 4096, 4099):
        _error_is_reported_once(vh, held[i])
    for sim in held:
        sim.close()
    _error_is_reported_once(vh, _immortal(vh, m))
