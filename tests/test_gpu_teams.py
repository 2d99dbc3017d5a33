"""A launch with few chains takes a team of warps per chain; its chains, counts and poses are those of
one warp per chain (a fixed packing), bit for bit."""
import numpy as np
import pytest

from gpu_helpers import engine_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,constraint,retain,opt_steps", [
    ("grid", False, 1, 12), ("grid", True, 4, 6), ("direct", False, 4, 3), ("grid", False, 1, 1)])
def test_team_search_is_the_search_of_one_warp(small_system, mode, constraint, retain, opt_steps):
    from ud2b200 import MODE_DIRECT, MODE_GRID
    m = MODE_GRID if mode == "grid" else MODE_DIRECT
    eng, _ = engine_for(small_system)
    eng.set_flags(constraint=constraint)
    eng.set_retain(retain)
    got = {}
    for packing in ((0, 0), (8, 1)):
        eng.set_packing(*packing)
        ne = eng.search(seed=17, nchain=20, mc_steps=9, opt_steps=opt_steps, randomize=True, mode=m)
        got[packing] = (ne, [eng.chain_poses(l).copy() for l in range(len(small_system["ligs"]))], eng.search_shape())
    assert got[(0, 0)][2]["warps_per_cta"] == 4 and got[(8, 1)][2]["warps_per_cta"] == 8
    assert got[(0, 0)][0] == got[(8, 1)][0]
    for a, b in zip(got[(0, 0)][1], got[(8, 1)][1]):
        assert np.array_equal(a, b, equal_nan=True)
    eng.close()


@pytest.mark.parametrize("max_steps,rounds", [(0, 1), (2, 5), (9, 1)])
def test_team_refinement_is_that_of_one_warp(small_system, max_steps, rounds):
    """The same poses in a batch of ten (teams) and of 1200 (one warp each)."""
    from ud2b200 import MODE_DIRECT, make_record
    eng, _ = engine_for(small_system)
    rng = np.random.default_rng(4)
    ligs = small_system["ligs"]
    pl = np.arange(1200) % len(ligs)
    recs = []
    for l in pl[:10]:
        x = ligs[l].coords + rng.uniform(-2, 2, 3).astype(np.float32)
        recs.append(make_record(ligs[l], x, x.mean(0)))
    kw = dict(max_steps=max_steps, rounds=rounds, vcap=1000.0, slope0=100.0, ramp=True, mode=MODE_DIRECT)
    few, ne = eng.bfgs_batch(pl[:10], recs, **kw)
    many, ne2 = eng.bfgs_batch(pl, [recs[i % 10] for i in range(1200)], **kw)
    eng.close()
    for i in range(1200):
        assert ne2[i] == ne[i % 10] and np.array_equal(many[i], few[i % 10], equal_nan=True)
