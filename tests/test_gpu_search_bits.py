"""The search's arithmetic, operation by operation: chains recorded once, compared bit for bit.

A BFGS search amplifies rounding until its chains part, so that one sum taken in another order (the
FP64 products of the inverse Hessian among them) moves about one chain in 10^4 visibly and no tolerance
tells it from a wrong one.  The digests were taken on a B200 with the library built by CUDA 12.9, with
a lane summing whole rows of the inverse Hessian; another compiler may round differently."""
import hashlib
import json
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "ref_5s8i.json")
DIGESTS = {                              # (seed, chains): a warp per chain; the last two by teams of warps
    (1, 8192): "ea1f7c6e19296b7782ed1efc3546534bc12c4b91f2939c9a420bfa8a751b5b28",
    (2, 8192): "1960c75dc10d2fc15fe07af2f8ad401b818948a94d8cdeb56a9c62bada7ccb97",
    (3, 256): "7ef264c1b432c1cdaeffdd587ddde59b55b644c617f867061153cdd62d6ffc81",
    (4, 256): "613843757a4040a06bf458df62b7d8548ec6a69b2ec1bf5e898df9db13f4ddbf",
}


@pytest.fixture(scope="module")
def redock():
    from ud2b200 import Engine
    from ud2b200.model import Box, parse_ligands
    with open(GOLDEN) as f:
        case = json.load(f)
    ligs = parse_ligands(case["ligands"])
    eng = Engine(Box.from_center_size(case["settings"]["center"], case["settings"]["size"]))
    rows = np.asarray([r[:4] for r in case["receptor"]])
    eng.set_receptor(rows[:, :3].astype(np.float32), rows[:, 3].astype(np.int32))
    eng.build_grid(0.375, sorted(set(int(t) for t in ligs[0].types if t)))
    eng.add_ligands(ligs)
    yield eng
    eng.close()


@pytest.mark.parametrize("seed,nchain", DIGESTS)
def test_chains_are_the_recorded_ones(redock, seed, nchain):
    redock.search(seed, nchain, 20, 20)
    assert hashlib.sha256(redock.chain_poses(0).tobytes()).hexdigest() == DIGESTS[seed, nchain]
