"""Deaths of a type that `call` names twice are put on the reuse stack once:
newcomers take exactly the numbers that are there, then new ones."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,share", [(1, 1.0), (100, 0.2), (5000, 0.45), (5000, 1.0)])
def test_type_called_twice(vh, n, share):
    rng = np.random.default_rng(n)
    die = (rng.random(n) < share).astype(np.int64)
    m = (vh.ModelTypes().register_agenttype("P", [("die", "i64")])
         .create_model("Twice"))
    sim = vh.create_simulation(m)
    vh.add_agents(sim, "P", n, die=die)
    vh.finish_init(sim)
    vh.apply_(sim, "die_if", ["P", "P"], ["P"], ["P"], params=[1, 0, 1.0])
    callers = int((~vh.read_agents(sim, "P")[1]).sum())
    vh.apply_(sim, "spawn", ["P"], ["P"], ["P"], params=[1, 100])
    cols, _ = vh.read_agents(sim, "P")
    reused = min(callers, int(die.sum()))
    assert cols["die"].size == n + callers - reused
    assert (cols["die"] >= 100).sum() == callers
    np.testing.assert_array_equal(np.sort(cols["die"][:n] >= 100)[::-1],
                                  np.arange(n) < reused)
    sim.close()


@pytest.mark.parametrize("n", [1, 33, 5000, 70_000])
def test_more_numbers_than_agents(vh, n):
    """Agents whose numbers are on the stack already die again and again: the
    stack grows with them."""
    m = (vh.ModelTypes().register_agenttype("P", [("die", "i64")]).create_model("Again"))
    sim = vh.create_simulation(m)
    vh.add_agents(sim, "P", n, die=1)
    vh.finish_init(sim)
    for _ in range(3):
        vh.apply_(sim, "die_if", ["P", "P"], ["P"], ["P"], params=[1, 0, 1.0])
        assert not vh.read_agents(sim, "P")[1].any()
    # 3 n numbers are on the stack: n callers with 4 newcomers each take them all
    vh.apply_(sim, "spawn", ["P"], ["P"], ["P"], params=[4, 1, 1, 1, 1])
    cols, died = vh.read_agents(sim, "P")
    assert cols["die"].size == 2 * n and not died.any()
    sim.close()
