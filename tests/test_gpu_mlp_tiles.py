"""GPU parity of the network's tcgen05 GEMMs and column sums at batch sizes around their tiles: one
row, a full and a started 128-row tile, and contractions shorter and longer than the stage ring and its
splits."""
import numpy as np
import pytest

import mlp_oracle as M
from test_gpu_learned import _data, bare_engine  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 128, 129, 4097])
def test_loss_and_gradient_match_oracle_at_tile_edges(bare_engine, n):  # noqa: F811
    """Gradient blocks within 3e-2 of their norm (BF16 operands and activations), biases included."""
    rng = np.random.default_rng(n)
    p = M.init_params(21)
    p = (p + rng.normal(0, 0.01, p.size)).astype(np.float32)
    bare_engine.mlp_set_params(p)
    X, Y, mask = _data(rng, n)
    loss, g = bare_engine.mlp_loss_grad(X, Y, mask)
    want_loss, want = M.loss_grad(p, X, Y, mask)
    assert abs(loss - want_loss) <= 1e-3 * max(1.0, abs(want_loss))
    off = 0
    for shape in M.SHAPES:
        k = int(np.prod(shape))
        a, b = g[off:off + k].astype(np.float64), want[off:off + k]
        assert np.linalg.norm(a - b) <= 3e-2 * max(np.linalg.norm(b), 1e-12), (shape, n)
        off += k
