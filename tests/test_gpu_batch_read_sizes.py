"""Batch states on both sides of the size that is read through pinned memory
(128 KB, 5 bytes an agent) equal the instance stepped by itself; results that are
kept are not overwritten by later reads."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_sizes(vh):
    from vahana_gb300 import models
    N = [2, 26_213, 26_214, 26_215, 30_000, 33]
    k = len(N)
    b = models.Batch(N, [5] * k, [0.2] * k, [6] * k, list(range(1, k + 1)))
    kept = []
    for steps in (0, 2, 3):
        if steps:
            b.step(steps, mode=1)
            for i in range(k):
                b.step_one(i, steps)
        for i in range(k):
            got = b.states(i)
            for x, y in zip(got, b.states(i, which=1)):
                np.testing.assert_array_equal(x, y)
            kept.append((got, [x.copy() for x in got]))
    for got, want in kept:
        for x, y in zip(got, want):
            np.testing.assert_array_equal(x, y)
    b.close()
