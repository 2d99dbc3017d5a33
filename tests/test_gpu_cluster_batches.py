"""Clustering, 32 poses of the ranking at a time, against a plain greedy pass around the batch's edges and
from no two poses alike to all alike."""
import numpy as np
import pytest

from gpu_helpers import engine_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nchain", [1, 31, 32, 33, 200, 300])
@pytest.mark.parametrize("rmsd", [0.0, 1.0, 3.0, 99.0])
def test_leaders_match_a_plain_greedy_pass(small_system, nchain, rmsd):
    """Torsion moves alone about a fixed root, so that the limits split the poses in every way."""
    eng, _ = engine_for(small_system)
    eng.set_flags(constraint=True)
    eng.search(seed=3, nchain=nchain, mc_steps=0, opt_steps=0, randomize=True)
    lead, cnt = eng.cluster(rmsd)
    for l, lig in enumerate(small_system["ligs"]):
        recs = eng.chain_poses(l)
        x = recs[:, 8:8 + 3 * lig.natom].reshape(nchain, lig.natom, 3)[:, lig.types != 0].astype(np.float32)
        e = np.where(np.isnan(recs[:, 0]), np.inf, recs[:, 0])
        thr = np.float32(np.float32(rmsd) * np.float32(rmsd)) * np.float32(x.shape[1])
        want = []
        for c in np.argsort(e, kind="stable"):
            # squares summed in order with one rounding each, for all leaders at once
            d = np.zeros(len(want), np.float32)
            diff = (x[c] - x[want]).reshape(len(want), 3 * x.shape[1]).astype(np.float64)
            for k in range(diff.shape[1]):
                d = (diff[:, k] ** 2 + d).astype(np.float32)
            if not (d < thr).any():
                want.append(int(c))
        assert list(lead[l, :cnt[l]]) == want and (lead[l, cnt[l]:] == -1).all()
    eng.close()


def test_as_many_chains_as_shared_memory_ranks(small_system):
    """12 bytes per pose, and all but 32 bytes of the CTA's 227 KB for them."""
    eng, _ = engine_for(dict(small_system, ligs=small_system["ligs"][:1]))
    eng.search(seed=3, nchain=19368, mc_steps=0, opt_steps=0, randomize=True)
    lead, cnt = eng.cluster(99.0)
    e = eng.chain_poses(0)[:, 0]
    eng.close()
    assert cnt[0] == 1 and lead[0, 0] == np.argsort(np.where(np.isnan(e), np.inf, e), kind="stable")[0]
