"""The batch calls' copies where they change: calls that travel in one page-locked block, calls that
do not fit it, and a small one after a large one; the forms in which poses are passed."""
import numpy as np
import pytest

from conftest import random_poses
from gpu_helpers import engine_for

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def io_sys(small_system):
    eng, _ = engine_for(small_system)
    yield dict(small_system, eng=eng)
    eng.close()


def _poses(sysd, n):
    rng = np.random.default_rng(n)
    pl = np.arange(n) % len(sysd["ligs"])
    some = [random_poses(l, sysd["box"], rng, 4) for l in sysd["ligs"]]
    return pl, [some[l][i % 4] for i, l in enumerate(pl)]


@pytest.mark.parametrize("n", [1, 3000, 20000])
def test_batches_of_any_size_give_each_pose_its_own_result(io_sys, n):
    """Every pose's energy, gradient, terms, decomposition and refinement in a batch are those of the
    same pose in a batch of twenty."""
    eng = io_sys["eng"]
    pl, xs = _poses(io_sys, n)
    c = np.array([x.mean(0) for x in xs])
    rv = np.full((n, 3), 0.3, np.float32)
    e, g = eng.score_batch(pl, xs, c, rv, vcap=10.0)
    t, d = eng.score_terms(pl, xs, decomp=True)
    recs = [np.concatenate([[0.0], a, np.zeros(4), x.reshape(-1), io_sys["ligs"][l].dihedrals]).astype(np.float32)
            for a, x, l in zip(c, xs, pl)]
    r, ne = eng.bfgs_batch(pl, recs, max_steps=1)
    at = np.unique(np.linspace(0, n - 1, 20).astype(int))
    pick = lambda v: [v[i] for i in at]  # noqa: E731
    e2, g2 = eng.score_batch(pl[at], pick(xs), c[at], rv[at], vcap=10.0)
    t2, d2 = eng.score_terms(pl[at], pick(xs), decomp=True)
    r2, ne2 = eng.bfgs_batch(pl[at], pick(recs), max_steps=1)
    assert np.array_equal(e[at], e2) and np.array_equal(t[at], t2) and np.array_equal(ne[at], ne2)
    assert all(np.array_equal(a, b) for a, b in zip(pick(g), g2))
    assert all(np.array_equal(a, b, equal_nan=True) for a, b in zip(pick(r), r2))
    off = np.concatenate([[0], np.cumsum([5 * io_sys["ligs"][l].natom for l in pl])])
    assert np.array_equal(np.concatenate([d[off[i]:off[i + 1]] for i in at]), d2)


def test_forms_of_the_coordinates(io_sys):
    """Lists, flat arrays, doubles, mixtures, one array for equal ligands and a generator all pass."""
    eng = io_sys["eng"]
    pl, xs = _poses(io_sys, 10)
    c, rv = np.array([x.mean(0) for x in xs]), np.zeros((10, 3))
    want, _ = eng.score_batch(pl, xs, c, rv)
    forms = [[x.tolist() for x in xs], [x.reshape(-1) for x in xs], [x.astype(np.float64) for x in xs],
             [x if i % 2 else x.reshape(-1) for i, x in enumerate(xs)], (x for x in xs), np.concatenate([x.reshape(-1) for x in xs])]
    for f in forms:
        assert np.array_equal(eng.score_batch(pl, f, c, rv)[0], want)
    same = np.stack([xs[0], xs[5]])
    assert np.array_equal(eng.score_batch([0, 0], same, c[[0, 5]], rv[:2])[0], want[[0, 5]])
    with pytest.raises(IndexError):
        eng.score_batch([99], xs[:1], c[:1], rv[:1])


def test_batches_before_and_after_the_page_locked_block(small_system):
    """Calls of several sizes again and again, until their copies go through page-locked memory: the same
    numbers all along."""
    eng, _ = engine_for(small_system)
    sizes, first = (3, 700, 1600, 9000), {}
    for rnd in range(60):
        for n in sizes if rnd % 20 == 0 else sizes[1:3]:
            if n not in first:
                pl, xs = _poses(small_system, n)
                first[n] = [pl, xs, np.array([x.mean(0) for x in xs]), np.full((n, 3), 0.2, np.float32), None]
            pl, xs, c, rv, want = first[n]
            e, g = eng.score_batch(pl, xs, c, rv, vcap=10.0)
            got = np.concatenate([e, *g])
            if want is None:
                first[n][4] = got
            else:
                assert np.array_equal(got, want), (rnd, n)
    eng.close()
