"""What a program pays that makes a context for a few calls: a receptor's, then the next one's."""
import time

import numpy as np
import pytest

from conftest import random_poses
from gpu_helpers import engine_for

pytestmark = pytest.mark.gpu


def test_first_call_of_a_new_context(small_system):
    """A context's first small batch allocates its device buffer and no more: of twelve contexts, one at a time,
    it takes (in the median) under ten times a later call (twice; 30 times where it allocated page-locked
    memory)."""
    first, later = [], []
    lig, rng = small_system["ligs"][2], np.random.default_rng(1)
    xs = random_poses(lig, small_system["box"], rng, 8)
    c, rv = np.array([x.mean(0) for x in xs]), np.zeros((8, 3))
    for _ in range(12):
        eng, _ = engine_for(small_system)
        for times in (first, later, later):
            t = time.perf_counter()
            eng.score_batch([2] * 8, xs, c, rv)
            times.append(time.perf_counter() - t)
        eng.close()
    assert np.median(first) < 10 * np.median(later), (np.median(first), np.median(later))
