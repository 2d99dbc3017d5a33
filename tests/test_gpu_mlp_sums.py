"""The training gradients' sums over the batch, in their order: biases row by row, weights in partial sums
over a cut that depends on the batch and the layer alone.  FP32 sums in another order differ in their last
bits, which Adam's first steps turn into other weights.  Inputs are chosen so that every product and every
partial sum is exact, and the expected bits follow from the order alone."""
import numpy as np
import pytest

import mlp_oracle as M
from test_gpu_learned import bare_engine  # noqa: F401

pytestmark = pytest.mark.gpu


def _blocks(g):
    out, off = [], 0
    for s in M.SHAPES:
        out.append(g[off:off + int(np.prod(s))].reshape(s))
        off += int(np.prod(s))
    return out


def _in_order(v):
    return np.add.accumulate(np.asarray(v, np.float32), axis=0, dtype=np.float32)[-1]


@pytest.mark.parametrize("n", [1, 127, 128, 129, 1024, 4097])
def test_bias_gradient_adds_the_rows_in_order(bare_engine, n):  # noqa: F811
    """With all parameters zero the means' output gradient is -y / n."""
    rng = np.random.default_rng(n)
    y = rng.standard_normal((n, 26), np.float32)
    bare_engine.mlp_set_params(np.zeros(bare_engine.mlp_param_count(), np.float32))
    _, g = bare_engine.mlp_loss_grad(rng.standard_normal((n, 672), np.float32), y, np.ones((n, 26), np.float32))
    want = _in_order(-y * (np.float32(1) / np.float32(n)))
    assert np.array_equal(_blocks(g)[-1][:26], want)


@pytest.mark.parametrize("n", [64, 1024, 4096])
def test_weight_gradient_adds_the_batch_in_its_parts(bare_engine, n):  # noqa: F811
    """One path of unit weights leads from the first output to the first layer, so that its gradient is
    the sum of x times whole numbers v: exact in every part, rounded where the parts are added."""
    rng = np.random.default_rng(n)
    v = rng.integers(1, 128, n).astype(np.float64)
    v[::16] = 2.0 ** 19
    p = [np.zeros(s, np.float32) for s in M.SHAPES]
    p[1][0], p[2][0, 0], p[4][0, 0], p[6][0, 0], p[7][0] = 1, 1, 1, 1, -1
    bare_engine.mlp_set_params(np.concatenate([a.reshape(-1) for a in p]))
    x = rng.integers(1, 3, (n, 672)).astype(np.float32)
    y, mask = np.zeros((n, 26), np.float32), np.zeros((n, 26), np.float32)
    y[:, 0], mask[:, 0] = -v * n, 1
    _, g = bare_engine.mlp_loss_grad(x, y, mask)
    g = _blocks(g)

    def parts(h, rows):                                # h: what the layer's input multiplies v by
        splits = max(1, min(n // 64, 296 // -(-rows // 128))) if n >= 128 else 1
        step = -(-(-(-n // splits)) // 32) * 32
        s = np.stack([(h[k:k + step] * v[k:k + step, None]).sum(0) for k in range(0, n, step)])
        assert np.abs(s).max() < 2.0 ** 24
        return _in_order(s)

    assert np.array_equal(g[0][:, 0], parts(x.astype(np.float64), 672))
    one = parts(np.ones((n, 1)), 256)
    assert g[2][0, 0] == one[0] and g[4][0, 0] == one[0] and g[6][0, 0] == one[0]
    for b in (1, 3, 5):
        assert g[b][0] == _in_order(v)
