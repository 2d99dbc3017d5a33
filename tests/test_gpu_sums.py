"""GPU parity of the map build where its loops change: bricks of grid points with remainders, receptors
that overflow a brick's atom list."""
import numpy as np
import pytest

from gpu_helpers import MAP_TYPES_ALL

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
