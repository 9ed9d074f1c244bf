"""The ensemble's persistent and cluster forms (states in one buffer,
instances without an infected agent skipped) against the per-step launches:
bit-identical states and days after odd and even numbers of steps, while
epidemics run, when they end within a run and when they ended before it, for
instances smaller than a mask word and larger than a block's range, with
agents taken by a warp each."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def batch(models, kind):
    rng = np.random.default_rng(3)
    if kind == "tiny":       # several instances share a mask word
        N = rng.integers(2, 40, 300)
    elif kind == "mixed":
        N = np.concatenate([rng.integers(2, 64, 40), rng.integers(500, 9000, 20), [70_001]])
    else:
        N = rng.integers(2000, 5000, 12)
    n = len(N)
    deg = np.minimum(rng.integers(1, 12, n), np.maximum(N - 1, 0))
    # some epidemics die out at once, some burn out, some last
    beta = rng.choice([0.0, 0.01, 0.15, 0.5], n)
    rec = rng.integers(1, 12, n)
    return models.Batch(N, deg, beta, rec, np.arange(n) + 11, infected_per_1000=30)


@pytest.mark.parametrize("kind", ["tiny", "mixed", "plain"])
@pytest.mark.parametrize("mode,bucket", [(2, 0), (2, 8), (3, 0), (4, 0)])
def test_forms(vh, kind, mode, bucket):
    from vahana_gb300 import models
    a, b = batch(models, kind), batch(models, kind)
    if bucket:  # a warp for each agent above 8 in-edges
        a.set_launch(1, tpb=256, bucket_threshold=bucket)
    total = 0
    for steps in (1, 2, 7, 20, 33, 80, 1, 6):
        try:
            a.step(steps, mode=mode)
        except vh.VahanaError as e:  # the cluster form may not fit an arena
            assert mode == 4 and "cluster" in str(e)
            pytest.skip(str(e))
        b.step(steps, mode=0)
        total += steps
        for i in range(a.n):
            for x, y in zip(a.states(i), b.states(i)):
                np.testing.assert_array_equal(x, y, err_msg="instance %d after %d steps" % (i, total))
    # the forms may follow one another at any point
    a.step(3, mode=0)
    a.step(4, mode=2)
    a.step(5, mode=1)
    b.step(12, mode=0)
    for i in range(a.n):
        for x, y in zip(a.states(i), b.states(i)):
            np.testing.assert_array_equal(x, y)
    a.close()
    b.close()
