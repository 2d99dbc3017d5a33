"""Ligands at the limits of size: what is refused as too large depends on the ligand, not on how the kernels
lay out its workspace and topology; what those cannot hold takes the far forms of the search and of the
refinement (topology, or start pose, in global memory), with the results of the near ones."""
import numpy as np
import pytest

from gpu_helpers import engine_for

pytestmark = pytest.mark.gpu


def _ligand(natom, small=()):
    """natom carbons in a ball; the atoms of `small` are a second fragment, turned by the one torsion and
    paired with all others."""
    from ud2b200.model import Ligand
    rng = np.random.default_rng(natom)
    x = rng.normal(size=(natom, 3))
    x *= 6.0 * rng.random((natom, 1)) ** (1 / 3) / np.linalg.norm(x, axis=1, keepdims=True)
    a = np.zeros(natom, bool)
    a[list(small)] = True
    pairs = [np.flatnonzero(a != a[i]).astype(np.int32) if a.any() else np.zeros(0, np.int32) for i in range(natom)]
    off = np.concatenate([[0], np.cumsum([len(p) for p in pairs])]).astype(np.int32)
    tors = bool(a.any())
    return Ligand(name="x%d" % natom, coords=x.astype(np.float32), types=np.full(natom, 3, np.int32),
                  ff_types=np.zeros(natom, np.int32), charges=np.zeros(natom, np.float32),
                  axis=np.array([[int(np.flatnonzero(~a)[0]), small[0]]] if tors else np.zeros((0, 2)), np.int32),
                  dihedrals=np.zeros(int(tors), np.float32),
                  ranges=[np.array([[-np.pi, np.pi]], np.float32)] if tors else [],
                  rotated=[np.array(sorted(small), np.int32)] if tors else [], pair_off=off,
                  pairs=np.concatenate(pairs).astype(np.int32))


@pytest.fixture(scope="module")
def wide(small_system):
    from ud2b200.model import Box
    return dict(small_system, box=Box.from_center_size(small_system["center"], [40.0] * 3))


def _centred(lig, system):
    lig.coords = (lig.coords + np.asarray(system["center"], np.float32)).astype(np.float32)
    return lig


@pytest.mark.parametrize("mode,retain", [("grid", 1), ("direct", 3)])
@pytest.mark.parametrize("which", ["rigid", "hub"])
def test_search_with_a_very_large_or_uneven_ligand(wide, mode, retain, which):
    """2408 atoms, whose topology cannot be staged, and 13 atoms spread over the list that pair with 287, whose
    gather lists all have a tail: the others of the batch keep their chains bit for bit, its own energies are
    those of its poses."""
    from ud2b200 import MODE_DIRECT, MODE_GRID, split_record
    m = MODE_GRID if mode == "grid" else MODE_DIRECT
    big = _centred(_ligand(2408) if which == "rigid" else _ligand(300, list(range(0, 299, 23))), wide)
    ligs = [wide["ligs"][1], wide["ligs"][3]]
    got = []
    for batch in (ligs, ligs + [big]):
        eng, _ = engine_for(dict(wide, ligs=batch))
        eng.set_retain(retain)
        eng.set_packing(4, 1)                          # one warp per chain in both
        eng.search(seed=8, nchain=5, mc_steps=4, opt_steps=5, randomize=True, mode=m)
        got.append([eng.chain_poses(l).copy() for l in range(len(batch))])
        if len(batch) == 3:
            recs = [split_record(big, r) for r in got[1][2] if r[0] < 1e9]
            assert len(recs) >= 4
            e, _ = eng.score_batch([2] * len(recs), [r["coords"] for r in recs], [r["center"] for r in recs],
                                   [r["rot_vec"] for r in recs], mode=m, vcap=1000.0)
            assert np.allclose([r["energy"] for r in recs], e, rtol=1e-4, atol=1e-3)
        eng.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("mode", ["grid", "direct"])
def test_refinement_with_a_ligand_beyond_the_near_workspace(wide, mode):
    """3700 atoms: scored and refined, and the poses of other ligands in the call with it as without."""
    from ud2b200 import MODE_DIRECT, MODE_GRID, make_record, split_record
    m = MODE_GRID if mode == "grid" else MODE_DIRECT
    big = _centred(_ligand(3700), wide)
    ligs = list(wide["ligs"]) + [big]
    eng, _ = engine_for(dict(wide, ligs=ligs))
    rng = np.random.default_rng(2)
    pl = [0, 3, 4, 5, 2, 5]
    recs = []
    for l in pl:
        x = ligs[l].coords + rng.uniform(-2, 2, 3).astype(np.float32)
        recs.append(make_record(ligs[l], x, x.mean(0)))
    kw = dict(max_steps=6, rounds=3, vcap=1000.0, slope0=100.0, ramp=True, mode=m)
    out, ne = eng.bfgs_batch(pl, recs, **kw)
    near = [k for k, l in enumerate(pl) if l != 5]
    alone, ne2 = eng.bfgs_batch([pl[k] for k in near], [recs[k] for k in near], **kw)
    for k, a, n2 in zip(near, alone, ne2):
        assert np.array_equal(out[k], a) and ne[k] == n2
    at = [k for k, l in enumerate(pl) if l == 5]
    r = [split_record(big, out[k]) for k in at]
    e, _ = eng.score_batch([5] * len(r), [q["coords"] for q in r], [q["center"] for q in r], [q["rot_vec"] for q in r],
                           mode=m, vcap=1000.0)
    eng.close()
    assert np.allclose([q["energy"] for q in r], e, rtol=1e-4, atol=1e-3)


@pytest.mark.parametrize("natom,small", [(300, range(0, 299, 23)), (120, [7]), (33, [0, 32]), (64, range(0, 64, 3))])
def test_gather_lists_of_uneven_lengths_match_oracle(wide, oracle64, natom, small):
    """Atoms that pair with most others, one or more in a group of 32: rows of the lists and their tail."""
    from ud2b200 import MODE_DIRECT
    lig = _centred(_ligand(natom, list(small)), wide)
    eng, _ = engine_for(dict(wide, ligs=[lig]))
    rng = np.random.default_rng(natom)
    x = lig.coords[None] * (1 + 0.02 * rng.normal(size=(3,) + lig.coords.shape)).astype(np.float32)
    c, rv = x.mean(1), rng.uniform(-1, 1, (3, 3)).astype(np.float32)
    e, g = eng.score_batch([0] * 3, x, c, rv, mode=MODE_DIRECT, vcap=10.0)
    eng.close()
    we, wg = oracle64.e_grad_batch(oracle64.ligand(lig), oracle64.make_env(wide["rec"], wide["box"], mode="direct"),
                                   x.astype(np.float64), c.astype(np.float64), rv.astype(np.float64), 10.0, 1e6)
    assert np.all(np.abs(e - we) <= 1e-4 * np.maximum(1.0, np.abs(we)))
    for a, b in zip(g, wg):
        assert np.abs(a - b).max() <= 1e-4 * max(1.0, np.abs(b).max())


def test_topologies_stay_within_the_predicted_bytes(wide):
    """What a launch's memory budget counts for a ligand's topology is an upper bound, also where padded
    gather lists would take several times as much (2000 of each of four kinds, 4 MB for the rest)."""
    from ud2b200 import MODE_DIRECT
    from ud2b200.batching import predict_dock_bytes
    kinds = [_centred(_ligand(*a), wide) for a in ((120, [7]), (40, [0, 39]), (200, [1, 60, 100, 150]))] + [wide["ligs"][4]]
    ligs = kinds * 2000
    count = lambda f: np.array([f(l) for l in kinds])  # noqa: E731
    want = predict_dock_bytes(count(lambda l: l.natom), count(lambda l: l.ntors), count(lambda l: len(l.pairs)),
                              count(lambda l: sum(map(len, l.rotated))), count(lambda l: sum(map(len, l.ranges))),
                              np.zeros(4, int), nchain=0, retain=0, num_pose=0).sum() * 2000
    eng, _ = engine_for(dict(wide, ligs=kinds))
    x = [kinds[0].coords]
    score = lambda: eng.score_batch([0], x, x[0].mean(0), np.zeros(3), mode=MODE_DIRECT)  # noqa: E731
    score()
    free = eng.device_memory()[0]
    eng.add_ligands(ligs)
    score()
    used = free - eng.device_memory()[0]
    eng.close()
    assert 0.3 * want < used <= want + (4 << 20), (used, want)


def test_too_large_is_refused_before_any_work(wide):
    """The same limits with and without BFGS, for the batch calls and for a dock, whose refinement would come
    after the search."""
    from ud2b200 import make_record
    from ud2b200.engine import EngineError
    for natom, search_only in ((2500, True), (3900, False)):
        big = _centred(_ligand(natom), wide)
        eng, _ = engine_for(dict(wide, ligs=[big]))
        x, c, rv = [big.coords], big.coords.mean(0, keepdims=True), np.zeros((1, 3))
        for opt in (0, 3):
            with pytest.raises(EngineError, match="too large"):
                eng.search(seed=1, nchain=2, mc_steps=2, opt_steps=opt)
            with pytest.raises(EngineError, match="too large"):
                eng.dock(1, 2, 2, opt, 3, 1, 1.0, 10.0)
        rec = make_record(big, big.coords, big.coords.mean(0))
        if search_only:
            assert np.isfinite(eng.score_batch([0], x, c, rv)[0]).all()
            eng.bfgs_batch([0], [rec], max_steps=1)
        else:
            for call in (lambda: eng.score_batch([0], x, c, rv), lambda: eng.bfgs_batch([0], [rec], max_steps=1)):
                with pytest.raises(EngineError, match="too large"):
                    call()
        eng.close()
