"""The training kernel at the edges of its 128-row tiles and beyond one tile for each SM (where a CTA keeps its weight
gradients over several), against the FP64 oracle with the same BF16 operand rounding.

Tolerance: as for the full-size gradient check, 1 % of each tensor's norm (FP32 sums of the same BF16 products; a
pre-rounding difference of one FP32 ulp may move an operand by one BF16 ulp, 0.4 %)."""
import numpy as np
import pytest

import oracle
from botheadstudios_b200 import learned_h

pytestmark = pytest.mark.gpu

BLOCKS = dict(W1=(learned_h.W1, learned_h.B1), b1=(learned_h.B1, learned_h.W2), W2=(learned_h.W2, learned_h.B2),
              b2=(learned_h.B2, learned_h.W3), W3=(learned_h.W3, learned_h.B3), b3=(learned_h.B3, learned_h.B3 + 1))


def _case(n):
    rng = np.random.default_rng(n)
    p = learned_h.init_params(rng.normal(0, 0.3, 8), rng.uniform(0.5, 2.0, 8), 0.004, 0.01, seed=n)
    p[learned_h.W3:learned_h.B3] *= 10.0
    p[learned_h.B1:learned_h.W2] = rng.normal(0, 0.1, 64)
    p[learned_h.B2:learned_h.W3] = rng.normal(0, 0.1, 64)
    x = rng.normal(size=(n, 8)).astype(np.float32)
    # targets on one side of the network's outputs: the sums do not cancel, so a tensor's norm is a fair scale
    t = (0.06 + 0.01 * np.tanh(x[:, 2])).astype(np.float32)
    return p, x, t


@pytest.mark.parametrize("n", [1, 127, 128, 129, 1000, 148 * 128, 148 * 128 + 1, 40_001])
def test_gradient_at_the_edges_of_the_tiles(n):
    p, x, t = _case(n)
    loss, g = learned_h.grad(p, x, t)
    want_loss, want = oracle.mlp_grad(p, x, t, bf16=True)
    assert abs(loss - want_loss) <= 1e-3 * want_loss
    for name, (a, b) in BLOCKS.items():
        assert np.linalg.norm(g[a:b] - want[a:b]) <= 1e-2 * np.linalg.norm(want[a:b]), name


def test_training_is_repeatable():
    p, x, t = _case(5000)
    a, la = learned_h.train(p, x, t, epochs=2, batch=1000, seed=3)
    b, lb = learned_h.train(p, x, t, epochs=2, batch=1000, seed=3)
    assert np.array_equal(a, b) and np.array_equal(la, lb)
