"""Loss and gradients of the fused training pass (GB300) against a float64 numpy
forward and backward pass, at the sizes where its tiles end: one sample, around one
64-sample tile, a block that does one tile more than the others, several tiles a block.

The pass is FP32: about six chained sums of 64 terms (forward, data gradients) and one
over the samples, each rounded to 2^-24 of its running value, so the 2-norm of the error
stays near 6 sqrt(64) 2^-24 = 3e-6 of the gradient's; 1e-5 is allowed.  The sigmoid's
hardware exponential and division add 2 ulp each, within the same figure."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _reference(p, x, y, w_tau):
    shapes = [(64, 2), (64,), (64, 64), (64,), (64, 64), (64,), (2, 64), (2,)]
    W, at = [], 0
    for s in shapes:
        k = int(np.prod(s))
        W.append(p[at:at + k].astype(np.float64).reshape(s))
        at += k
    h, z = [x.astype(np.float64)], []
    for k in range(3):
        z.append(h[k] @ W[2 * k].T + W[2 * k + 1])
        h.append(z[k] / (1 + np.exp(-z[k])))
    d = h[3] @ W[6].T + W[7] - y
    wc = np.array([1.0, w_tau])
    loss = float((wc * d * d).sum() / len(x))
    g, dz = [None] * 8, 2 * wc * d / len(x)
    for k in (3, 2, 1, 0):
        g[2 * k], g[2 * k + 1] = dz.T @ h[k], dz.sum(0)
        if k:
            s = 1 / (1 + np.exp(-z[k - 1]))
            dz = (dz @ W[2 * k]) * (s * (1 + z[k - 1] * (1 - s)))
    return loss, np.concatenate([v.ravel() for v in g])


@pytest.mark.parametrize("n", [1, 63, 64, 65, 9727, 9728, 9729, 20000])
def test_gradients_at_tile_edges(gpu_engine, n):
    rng = np.random.default_rng(n)
    p = rng.uniform(-0.3, 0.3, 8642).astype(np.float32)
    x = rng.uniform(-1, 1, (n, 2)).astype(np.float32)
    y = rng.uniform(-1, 1, (n, 2)).astype(np.float32)
    loss, g = gpu_engine.surrogate_gradients(p, x, y, w_tau=0.1)
    want_loss, want = _reference(p, x, y, 0.1)
    assert abs(loss - want_loss) <= 1e-5 * want_loss
    assert np.linalg.norm(g - want) <= 1e-5 * np.linalg.norm(want)
