"""What a program pays that makes a context for a few calls: a receptor's, then the next one's."""
import time

import numpy as np
import pytest

from conftest import random_poses
from gpu_helpers import engine_for

pytestmark = pytest.mark.gpu


def test_first_call_of_a_new_context(small_system):
    """A context's first small batch allocates its device buffer and no more: of twelve contexts, one at a time,
    it takes (at best, for a busy host's sake) under ten times a later call (twice; 18 times where it allocated
    page-locked memory)."""
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
    assert min(first) < 10 * np.median(later), (first, later)


def test_first_direct_search_on_a_receptor(small_system):
    """The neighbour lists of a new receptor, built by its first direct search, cost little beside a search of one
    chain: of ten receptors it takes (at best) under five times a later one (twice; ten times where the lists
    were built on the host)."""
    from ud2b200 import Engine, MODE_DIRECT
    from ud2b200.model import Box
    rng = np.random.default_rng(5)
    box = Box.from_center_size([20.0] * 3, [30.0] * 3)
    eng = Engine(box)
    eng.add_ligands([small_system["ligs"][2]])
    first, later = [], []
    for _ in range(10):
        eng.set_receptor(rng.uniform(-3.0, 43.0, (8000, 3)).astype(np.float32), rng.choice([2, 3, 5, 10], 8000))
        for times in (first, later, later):
            t = time.perf_counter()
            eng.search(seed=1, nchain=1, mc_steps=0, opt_steps=0, mode=MODE_DIRECT)
            times.append(time.perf_counter() - t)
    eng.close()
    assert min(first) < 5 * np.median(later), (first, later)
