"""GPU parity of the map build and of the search's sums where their loops change: bricks of grid points
with remainders, receptors that overflow a brick's atom list, direct sums over neighbour lists,
and evaluations that leave the forces out."""
import numpy as np
import pytest

from gpu_helpers import MAP_TYPES_ALL, engine_for, rel_err

pytestmark = pytest.mark.gpu

TOL = 1e-4


@pytest.mark.parametrize("size,spacing,natom", [
    ((2.9, 3.0, 1.4), 0.375, 60),       # one brick and a point more along y: 9 x 9 x 5 points
    ((0.3, 6.0, 9.0), 0.375, 300),      # the smallest extent: 2 points along x
    ((8.0, 8.0, 8.0), 1.0, 0),          # no receptor
    ((6.0, 6.0, 6.0), 0.5, 3000),       # more atoms near every brick than its list holds at once
    ((20.0, 14.0, 11.0), 0.6, 900)])
def test_grid_bricks_match_oracle(oracle64, size, spacing, natom):
    from ud2b200 import Engine
    from ud2b200.model import Box, parse_receptor
    rng = np.random.default_rng(7)
    box = Box.from_center_size([30.0, 31.0, 32.0], size)
    xyz = rng.uniform(box.lo - 8.5, box.hi + 8.5, (natom, 3)).astype(np.float32)
    types = rng.choice([2, 3, 5, 10, 11, 15], natom).astype(np.int32)
    eng = Engine(box)
    eng.set_receptor(xyz, types)
    eng.build_grid(spacing, MAP_TYPES_ALL)
    maps, gd, org = eng.get_grid()
    eng.close()
    rec = parse_receptor([[*map(float, x), int(t), 0, 0.0] for x, t in zip(xyz, types)], box)
    want = oracle64.grid_build(rec, MAP_TYPES_ALL, org.astype(np.float64), spacing, gd)
    assert list(gd) == [max(2, int(np.ceil(s / spacing - 1e-4)) + 1) for s in size]
    assert np.all(np.abs(maps - want) <= TOL * np.maximum(1.0, np.abs(want)))


@pytest.fixture(scope="module")
def sums_sys(small_system):
    from ud2b200 import synth
    from ud2b200.model import parse_ligands
    ligs = parse_ligands({f"s{i}": synth.make_ligand(n, t, seed=700 + i, center=small_system["center"])
                          for i, (n, t) in enumerate([(8, 0), (31, 5), (33, 6), (65, 12)])})
    sysd = dict(small_system, ligs=ligs)
    eng, _ = engine_for(sysd)
    yield dict(sysd, eng=eng)
    eng.close()


@pytest.mark.parametrize("mode", ["grid", "direct"])
@pytest.mark.parametrize("opt_steps", [0, 3])
def test_search_energies_are_those_of_the_scoring(sums_sys, mode, opt_steps):
    """Every chain's best energy (neighbour-list sums or maps; with and without forces) is the batch
    scoring's energy (cell rows or maps) of its pose; randomised starts (0 MC steps) stick out of
    the box and of the cells."""
    from ud2b200 import MODE_DIRECT, MODE_GRID, split_record
    eng, m = sums_sys["eng"], MODE_GRID if mode == "grid" else MODE_DIRECT
    for steps in (0, 4):
        eng.search(seed=5, nchain=24, mc_steps=steps, opt_steps=opt_steps, randomize=True, mode=m)
        for li, lig in enumerate(sums_sys["ligs"]):
            recs = [split_record(lig, r) for r in eng.chain_poses(li)]
            recs = [r for r in recs if r["energy"] < 1e8 and np.isfinite(r["rot_vec"]).all()]
            assert len(recs) > 12
            # a refined new best is optimised again with curl 1000
            vcap = 1000.0 if steps and opt_steps else 10.0
            e, _ = eng.score_batch([li] * len(recs), [r["coords"] for r in recs], [r["center"] for r in recs],
                                   [r["rot_vec"] for r in recs], mode=m, vcap=vcap)
            got = np.array([r["energy"] for r in recs])
            # every one of them: the pose stored is the one the energy is of (the same code on maps; on direct
            # sums the same terms in another order)
            near = np.abs(got - e) <= TOL * np.maximum(1.0, np.abs(e))
            assert near.all(), (li, steps, got[~near], e[~near])


def test_direct_search_follows_the_receptor(sums_sys, oracle64):
    """The neighbour lists belong to the current receptor: a direct search after a new receptor scores
    on that one, also where it is empty."""
    from ud2b200 import Engine, MODE_DIRECT, split_record
    box, lig = sums_sys["box"], sums_sys["ligs"][1]
    rows = np.asarray([r[:4] for r in sums_sys["rows"]])
    eng = Engine(box)
    eng.add_ligands([lig])
    for keep in (len(rows), len(rows) // 2, 0):
        eng.set_receptor(rows[:keep, :3].astype(np.float32), rows[:keep, 3].astype(np.int32))
        eng.search(seed=9, nchain=8, mc_steps=0, opt_steps=0, mode=MODE_DIRECT)
        recs = [split_record(lig, r) for r in eng.chain_poses(0)]
        e, _ = eng.score_batch([0] * 8, [r["coords"] for r in recs], [r["center"] for r in recs],
                               [r["rot_vec"] for r in recs], mode=MODE_DIRECT, vcap=10.0)
        assert rel_err([r["energy"] for r in recs], e) <= TOL
    eng.close()


def test_direct_sums_at_the_faces_of_the_cells(oracle64):
    """A ligand atom a hair to either side of a face between cells, at the outermost ones and up to 8 A beyond
    them, along each axis: the rows and end cells left out hold nothing within the cutoff."""
    from ud2b200 import Engine, MODE_DIRECT, synth
    from ud2b200.model import Box, parse_ligands, parse_receptor
    rng = np.random.default_rng(12)
    box = Box.from_center_size([30.0, 31.0, 32.0], [6.0, 7.0, 9.0])
    xyz = rng.uniform(box.lo - 8.5, box.hi + 8.5, (1500, 3)).astype(np.float32)
    types = rng.choice([2, 3, 5, 10, 11, 15], len(xyz)).astype(np.int32)
    lig = parse_ligands({"a": synth.make_ligand(8, 0, seed=5, center=[30.0, 31.0, 32.0])})[0]
    eng = Engine(box)
    eng.set_receptor(xyz, types)
    eng.add_ligands([lig])
    cell, lo = 8.0625, box.lo - 8.0
    poses = []
    for axis in range(3):
        for face in range(int((box.hi - box.lo)[axis] + 16) // 8 + 2):
            for off in (-7.99, -1e-3, -1e-6, 0.0, 1e-6, 1e-3, 4.0):
                at = rng.uniform(box.lo - 8.0, box.hi + 8.0)
                at[axis] = lo[axis] + cell * face + off
                poses.append(lig.coords - lig.coords[rng.integers(8)] + at)
    poses = np.asarray(poses, np.float32)
    c, rv = poses.mean(1), np.zeros((len(poses), 3))
    e, g = eng.score_batch([0] * len(poses), poses, c, rv, mode=MODE_DIRECT, vcap=10.0, slope=0.0)
    t, _ = eng.score_terms([0] * len(poses), poses)
    eng.close()
    rec = parse_receptor([[*map(float, x), int(k), 0, 0.0] for x, k in zip(xyz, types)], box)
    env = oracle64.make_env(rec, box, mode="direct")
    olig = oracle64.ligand(lig)
    we, wg = oracle64.e_grad_batch(olig, env, poses.astype(np.float64), c.astype(np.float64), rv, 10.0, 0.0)
    wt = np.array([oracle64.score_terms(olig, env, p) for p in poses])
    assert (np.abs(we) > 1e-3).sum() > len(poses) / 2
    assert np.all(np.abs(e - we) <= TOL * np.maximum(1.0, np.abs(we)))
    assert np.all(np.abs(t[:, 1] - wt[:, 1]) <= TOL * np.maximum(1.0, np.abs(wt[:, 1])))
    assert all(rel_err(a, b) <= TOL for a, b in zip(g, wg))


@pytest.mark.parametrize("mode", ["grid", "direct"])
def test_scoring_workspace_of_the_largest_ligand(small_system, mode):
    """Ligands at both ends of the sizes, alone (a workspace of their own) and beside the largest: the
    same numbers."""
    from conftest import random_poses
    from ud2b200 import MODE_DIRECT, MODE_GRID, synth
    from ud2b200.model import parse_ligands
    ligs = parse_ligands({f"w{i}": synth.make_ligand(n, t, seed=720 + i, center=small_system["center"])
                          for i, (n, t) in enumerate([(8, 0), (32, 1), (64, 14), (80, 20)])})
    eng, _ = engine_for(dict(small_system, ligs=ligs))
    m = MODE_DIRECT if mode == "direct" else MODE_GRID
    rng = np.random.default_rng(3)
    pl = np.arange(36) % 4
    xs = [random_poses(ligs[l], small_system["box"], rng, 1)[0] for l in pl]
    c, rv = np.array([x.mean(0) for x in xs]), rng.uniform(-1, 1, (36, 3)).astype(np.float32)
    e, g = eng.score_batch(pl, xs, c, rv, mode=m, vcap=10.0)
    for l in range(4):
        at = np.flatnonzero(pl == l)
        e1, g1 = eng.score_batch(pl[at], [xs[i] for i in at], c[at], rv[at], mode=m, vcap=10.0)
        assert np.array_equal(e1, e[at]) and all(np.array_equal(a, g[i]) for a, i in zip(g1, at))
        assert all(len(a) == 6 + ligs[l].ntors and np.isfinite(a).all() for a in g1)
    eng.close()
