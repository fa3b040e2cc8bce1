"""The subtree-size model's kernels work on tiles of 64 samples, one block per SM
taking several: sample counts at the edges of a tile, of one round of blocks and
of the next, against the float64 restatement."""
import numpy as np
import pytest

from gmkbe_b200 import learned as L
from oracle import mlp_ref

pytestmark = pytest.mark.gpu

# Weights and inputs are the same FP16 values on both sides; a gradient component
# is a sum over n samples of products of two FP32 sums of at most 64 terms, kept
# in FP32 over at most ceil(n / 64 / 148) * 64 terms in a row and 148 block sums:
# (64 + 64 + 192 + 148) roundings of 2^-24 are below 3e-5 of the sum of absolute
# terms, which is at most about ten times the largest component.
RTOL = 3e-4


@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 127, 129, 148 * 64, 148 * 64 + 1, 2 * 148 * 64 + 63])
def test_gradient_and_prediction_at_tile_edges(n):
    rng = np.random.default_rng(n)
    x = rng.uniform(0, 4, (n, 16)).astype(np.float32)
    y = (0.5 * x[:, 2] + np.sin(x[:, 6]) + 0.1 * rng.standard_normal(n)).astype(np.float32)
    m = L.SubtreeModel(seed=5)
    got, loss = m.gradient(x, y)
    want_loss, want = mlp_ref.loss_and_gradient(m.params(), x, y)
    assert abs(loss - want_loss) <= RTOL * max(1.0, abs(want_loss))
    assert np.abs(got - want).max() <= RTOL * np.abs(want).max()
    out = m.predict(x)
    ref = mlp_ref.forward(m.params(), x)[0]
    assert out.shape == (n,) and np.abs(out - ref).max() <= 1e-4 * max(1.0, np.abs(ref).max())
    again, loss2 = m.gradient(x, y)
    assert np.array_equal(got, again) and loss == loss2      # sums in a fixed order
