"""GPU parity of the BFGS inverse-Hessian rows at the sizes where their split over the lanes changes:
two lanes per row up to 16 rows (10 torsions), one per row up to 32 (26 torsions), several rows per
lane above."""
import numpy as np
import pytest

from gpu_helpers import engine_for, oracle_grid, perturbed_poses

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("natom,ntors", [(30, 9), (32, 10), (34, 11), (66, 26), (68, 27)])
def test_bfgs_rows_match_oracle(small_system, oracle32, oracle64, natom, ntors):
    """Two BFGS steps from random poses end at the FP32 restatement's energy (1e-3) as often as the
    FP32 and FP64 restatements agree with each other (less 15 % of the starts)."""
    from ud2b200 import MODE_GRID, make_record, synth
    from ud2b200.model import parse_ligands
    lig = parse_ligands({"a": synth.make_ligand(natom, ntors, seed=900 + ntors, center=small_system["center"])})[0]
    assert lig.ntors == ntors
    sysd = dict(small_system, ligs=[lig])
    eng, _ = engine_for(sysd)
    grid, _ = oracle_grid(oracle64, sysd, eng)
    env = {o: o.make_env(sysd["rec"], sysd["box"], grid=grid, mode="grid") for o in (oracle32, oracle64)}
    starts = perturbed_poses(oracle64, oracle64.ligand(lig), env[oracle64], lig, np.random.default_rng(3), 16, sysd["box"])
    recs = [make_record(lig, p["coords"], p["center"], p["rot_vec"], p["dihedrals"]) for p in starts]
    out, _ = eng.bfgs_batch([0] * len(recs), recs, max_steps=2, rounds=1, vcap=10.0, slope0=1e6, mode=MODE_GRID)
    eng.close()
    want = {o: [o.bfgs(o.ligand(lig), env[o], {k: v.astype(np.float64) for k, v in p.items()}, 2, 10.0, 1e6)[0]["energy"]
                for p in starts] for o in (oracle32, oracle64)}
    near = lambda a, b: sum(abs(x - y) <= 1e-3 * max(1.0, abs(y)) for x, y in zip(a, b))  # noqa: E731
    got = near([r[0] for r in out], want[oracle32])
    assert got >= near(want[oracle32], want[oracle64]) - 0.15 * len(recs), got
    assert got >= 1
