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


@pytest.mark.parametrize("bias", ["pos", "align"])
def test_team_search_with_bias_records(small_system, bias):
    """The same with bias records on some of the atoms."""
    import copy
    rng = np.random.default_rng(6)
    ligs = []
    for lig in small_system["ligs"]:
        lig = copy.copy(lig)
        lig.bias_atoms = np.sort(rng.integers(0, lig.natom, 5)).astype(np.int32)
        site = np.asarray(small_system["center"]) + rng.uniform(-3, 3, (5, 3))
        lig.bias_params = np.column_stack([site, rng.uniform(-2, -0.5, 5), rng.uniform(0.5, 2, 5)]).astype(np.float32)
        ligs.append(lig)
    eng, _ = engine_for(dict(small_system, ligs=ligs))
    got = {}
    for kind in (0, 1 if bias == "pos" else 2):
        eng.set_flags(bias_type=kind, bias_k=0.5)
        for packing in ((0, 0), (8, 1)):
            eng.set_packing(*packing)
            ne = eng.search(seed=23, nchain=16, mc_steps=6, opt_steps=8, randomize=True)
            got[bool(kind), packing] = (ne, [eng.chain_poses(l).copy() for l in range(len(ligs))])
            assert eng.search_shape()["warps_per_cta"] == (8 if packing[0] else 4)
    eng.close()
    (na, a), (nb, b) = got[True, (0, 0)], got[True, (8, 1)]
    assert na == nb and all(np.array_equal(x, y, equal_nan=True) for x, y in zip(a, b))
    assert not any(np.array_equal(x, y, equal_nan=True) for x, y in zip(a, got[False, (0, 0)][1]))


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


@pytest.fixture(scope="module")
def large_sys(small_system):
    """Ligands on both sides of the pair buffer's 4096 pairs (3813, 4215 and 4774), in a box that holds them."""
    from ud2b200 import synth
    from ud2b200.model import Box, parse_ligands
    ligs = parse_ligands({f"p{i}": synth.make_ligand(n, t, seed=s, center=small_system["center"])
                          for i, (n, t, s) in enumerate([(100, 10, 1), (100, 12, 2), (110, 10, 3)])})
    return dict(small_system, ligs=ligs, box=Box.from_center_size(small_system["center"], [44.0] * 3))


@pytest.mark.parametrize("which,team", [([0], True), ([1], False), ([2], False), ([0, 2], False)])
def test_no_team_without_a_pair_buffer(large_sys, which, team):
    """Atomic sums have no fixed order, a team needs equal bits: a launch that holds a ligand of more pairs
    than the buffer takes one warp per chain.  Its recorded energies are those of its poses."""
    from ud2b200 import MODE_GRID, split_record
    ligs = [large_sys["ligs"][k] for k in which]
    eng, _ = engine_for(dict(large_sys, ligs=ligs))
    eng.search(seed=3, nchain=12, mc_steps=3, opt_steps=4, randomize=True)
    assert (eng.search_shape()["register_class"] == 4) == team       # such a blob leaves one warp per chain no 64 registers
    for l, lig in enumerate(ligs):
        recs = [split_record(lig, r) for r in eng.chain_poses(l)]
        recs = [r for r in recs if r["energy"] < 1e9]             # the others: no accepted pose
        e, _ = eng.score_batch([l] * len(recs), [r["coords"] for r in recs], [r["center"] for r in recs],
                               [r["rot_vec"] for r in recs], mode=MODE_GRID, vcap=1000.0)
        assert len(recs) >= 4 and np.allclose([r["energy"] for r in recs], e, rtol=1e-4, atol=1e-4)
    eng.close()


def test_refinement_without_a_pair_buffer(large_sys):
    """Few poses, those of ligands beyond the pair buffer among them: every pose's energy falls to that of
    the pose returned."""
    from ud2b200 import MODE_DIRECT, make_record, split_record
    eng, _ = engine_for(large_sys)
    ligs = large_sys["ligs"]
    pl = [0, 1, 2, 0, 1, 2]
    recs = [make_record(ligs[l], ligs[l].coords, ligs[l].center) for l in pl]
    out, ne = eng.bfgs_batch(pl, recs, max_steps=5, rounds=2, vcap=1000.0, slope0=100.0, ramp=False, mode=MODE_DIRECT)
    out = [split_record(ligs[l], r) for l, r in zip(pl, out)]
    kw = dict(mode=MODE_DIRECT, vcap=1000.0, slope=100.0)
    pose = lambda rs: ([r["coords"] for r in rs], [r["center"] for r in rs], [r["rot_vec"] for r in rs])  # noqa: E731
    e, _ = eng.score_batch(pl, *pose(out), **kw)
    e0, _ = eng.score_batch(pl, *pose([split_record(ligs[l], r) for l, r in zip(pl, recs)]), **kw)
    eng.close()
    assert (np.asarray(ne) > 2).all() and np.allclose([r["energy"] for r in out], e, rtol=1e-4, atol=1e-4)
    assert (e <= e0).all() and (e < e0).any()
