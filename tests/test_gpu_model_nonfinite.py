"""The gradient of the subtree-size model where an input or a weight is infinite
(past FP16's range): a unit that is off, and an output that is right, have no part
in it, so a zero factor leaves its term out instead of making it NaN.  Against the
restatement of that rule in float64, in one tile of 64 samples and over several."""
import numpy as np
import pytest

from gmkbe_b200 import learned as L
from oracle import mlp_ref as R

pytestmark = pytest.mark.gpu


def _times(a, b, both=True):
    """a * b with a zero factor (both: either, else a only) leaving 0."""
    z = (a == 0) | (b == 0) if both else np.broadcast_to(a == 0, np.broadcast(a, b).shape)
    return np.where(z, 0.0, a * b)


def _gradient(p, x, y):
    w1, b1, w2, b2, w3, b3 = R._unpack(p)
    x = x.astype(np.float16).astype(np.float64)
    a1 = (x[:, None, :] * w1).sum(2) + b1
    h1 = np.where(a1 > 0, a1, 0.0)
    a2 = (h1[:, None, :] * w2).sum(2) + b2
    h2 = np.where(a2 > 0, a2, 0.0)
    out = (h2 * w3).sum(1) + b3
    d = 2.0 * (out - y) / y.size
    dh2 = np.where(h2 > 0, d[:, None] * w3, 0.0)
    dh1 = np.where(h1 > 0, _times(dh2[:, :, None], w2, both=False).sum(1), 0.0)
    g = np.zeros(R.NP)
    g[R.OFF_B3] = d.sum()
    g[R.OFF_W3:R.OFF_B3] = (d[:, None] * h2).sum(0)
    g[R.OFF_B2:R.OFF_W3] = dh2.sum(0)
    g[R.OFF_W2:R.OFF_B2] = _times(dh2[:, :, None], h1[:, None, :]).sum(0).ravel()
    g[R.OFF_B1:R.OFF_W2] = dh1.sum(0)
    g[R.OFF_W1:R.OFF_B1] = _times(dh1[:, :, None], x[:, None, :], both=False).sum(0).ravel()
    return g


# The tolerance of the tile tests: (64 + 64 + 192 + 148) roundings of 2^-24 are below 3e-5 of the sum of
# absolute terms, which is at most about ten times the largest component.
RTOL = 3e-4


@pytest.mark.filterwarnings("ignore::RuntimeWarning")
@pytest.mark.parametrize("n", [1, 64, 100, 300])
@pytest.mark.parametrize("what", ["none", "inputs", "weight", "target"])
def test_zero_factors_leave_their_terms_out(what, n):
    rng = np.random.default_rng(n)
    x = rng.uniform(0, 4, (n, 16)).astype(np.float32)
    y = (x[:, 2] + 0.1 * rng.standard_normal(n)).astype(np.float32)
    m = L.SubtreeModel(seed=3)
    p = m.params()
    if what == "inputs":          # one sample each: a feature above 65 504, one below
        x[n // 2, 5] = 1e6
        x[n // 3, 9] = -1e6
    elif what == "weight":        # a unit that every sample keeps off, with an infinite outgoing weight
        p[R.OFF_W1 + 7 * 16:R.OFF_W1 + 8 * 16] = -1.0
        p[R.OFF_W2 + 11 * 64 + 7] = 1e6
        m.set_params(p)
    elif what == "target":
        y[n // 2] = np.inf
    got, _ = m.gradient(x, y)
    want = _gradient(p, x, y)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert np.array_equal(np.isposinf(got), np.isposinf(want)) and np.array_equal(np.isneginf(got), np.isneginf(want))
    ok = np.isfinite(want)
    assert np.abs(got[ok] - want[ok]).max() <= RTOL * np.abs(want[ok]).max()
    if what == "inputs":
        assert ok.all()
