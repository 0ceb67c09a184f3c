"""The fused training pass (GB300) at the edges of each of its tiles: 28 samples (batches up
to 4256 on 152 SMs, and 9729 to 12,768), 56 (to 8512, 12,769 to 17,024, and the default
batch of 16,384) and 64 (8513 to 9728, 17,025 to 19,456); and whole training steps, with
the samples' weights, batches that wrap round the training set and BF16-rounded hidden
layers, against the same steps in float64 numpy.

Gradients: about six chained sums of 64 terms and one over the samples, each rounded to
2^-24 of its running value: 1e-5 of the gradient's 2-norm is allowed.  Training: a loss is
within 1e-4 (parameters off by some 1e-5 of their change; BF16 roundings that fall on the
other side, one in 10^4, each worth 5e-6).  Adam divides a gradient by its own size, so a
parameter whose gradient is below the error may step the other way: with errors of 1e-5
to 5e-5 of the mean size that is a 2-norm of up to sqrt(5e-5) = 7e-3 of the change; 2e-2 is
allowed."""
import math

import numpy as np
import pytest

from test_gpu_training_pass import _reference

pytestmark = pytest.mark.gpu

SHAPES = [(64, 2), (64,), (64, 64), (64,), (64, 64), (64,), (2, 64), (2,)]
SCALE = {0: 1.2, 2: 0.3, 4: 0.3, 6: 0.2}


@pytest.mark.parametrize("n", [27, 28, 29, 4255, 4256, 4257, 8511, 8512, 8513, 12768, 12769, 16384, 17023, 17024,
                               17025, 19456, 19457])
def test_gradients_at_the_tiles_edges(gpu_engine, n):
    rng = np.random.default_rng(n)
    p = rng.uniform(-0.3, 0.3, 8642).astype(np.float32)
    x = rng.uniform(-1, 1, (n, 2)).astype(np.float32)
    y = rng.uniform(-1, 1, (n, 2)).astype(np.float32)
    loss, g = gpu_engine.surrogate_gradients(p, x, y, w_tau=0.1)
    want_loss, want = _reference(p, x, y, 0.1)
    assert abs(loss - want_loss) <= 1e-5 * want_loss
    assert np.linalg.norm(g - want) <= 1e-5 * np.linalg.norm(want)


def _philox(n, seed):
    """two 53-bit uniforms per sample: Philox4x32-10 (Salmon et al. 2011) at (i, 0, 0, 0x5347)"""
    m32, i = np.uint64(0xFFFFFFFF), np.arange(n, dtype=np.uint64)
    c = [i & m32, i >> np.uint64(32), np.zeros(n, np.uint64), np.full(n, 0x5347, np.uint64)]
    k = [seed & 0xFFFFFFFF, (seed >> 32) ^ 0x53474E4E]
    for _ in range(10):
        p0, p1 = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k[0]), p1 & m32,
             (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k[1]), p0 & m32]
        k = [(k[0] + 0x9E3779B9) & 0xFFFFFFFF, (k[1] + 0xBB67AE85) & 0xFFFFFFFF]
    return [(((c[a] << np.uint64(21)) ^ (c[a + 1] >> np.uint64(11))).astype(np.float64) + 0.5) / 2.0 ** 53
            for a in (0, 2)]


def _bf16(v):
    u = np.ascontiguousarray(v, dtype=np.float32).view(np.uint32).astype(np.uint64)
    u = (u + 0x7FFF + ((u >> np.uint64(16)) & np.uint64(1))) & np.uint64(0xFFFF0000)
    return u.astype(np.uint32).view(np.float32).astype(np.float64)


def _initial(seed):
    st, at, P = (seed * 6364136223846793005 + 1442695040888963407) % 2 ** 64, 0, []
    for k, s in enumerate(SHAPES):
        v = np.zeros(int(np.prod(s)))
        if k in SCALE:
            for j in range(len(v)):
                st = (st * 6364136223846793005 + 1442695040888963407) % 2 ** 64
                v[j] = float(np.float32((st >> 11) / 2.0 ** 53) * 2 - 1) * SCALE[k]
        P.append(v.reshape(s))
    return P


def _train(engine, n, B, steps, quant, seed):
    """last loss, initial and trained parameters; the targets through the engine's services"""
    u0, u1 = _philox(n, seed)
    le, b = -4.0 + 8.0 * u0, 12.0 * np.sqrt(u1)
    eps = 10.0 ** le
    s2 = engine.scatter(eps, b, precision="fp64")
    tau = engine.quadrature(eps, b)[1]
    base = -np.log(1 + (2 * eps * b) ** 2 * np.exp(2 * 0.20162 * b))
    X = np.stack([le * 0.25, b / 6 - 1], 1)
    Y = np.stack([(np.log(np.maximum(s2, 1e-300)) - base) / 4, tau / 10], 1)
    wts = s2 + 1e-6
    wts /= wts.mean()
    P = _initial(seed)
    start = np.concatenate([p.ravel() for p in P])
    M, V = [0 * p for p in P], [0 * p for p in P]
    rnd = _bf16 if quant else (lambda v: v)
    for it in range(steps):
        at = (it * B + np.arange(B)) % n
        x, y, w = X[at], Y[at], wts[at]
        h, z = [x], []
        for k in range(3):
            z.append((rnd(h[k]) @ rnd(P[2 * k]).T if k else h[0] @ P[0].T) + P[2 * k + 1])
            h.append(z[k] / (1 + np.exp(-z[k])))
        d = h[3] @ P[6].T + P[7] - y
        wc = np.stack([w, np.full_like(w, 0.1)], 1)
        loss = float((wc * d * d).sum() / B)
        g, dz = [None] * 8, 2 * wc * d / B
        for k in (3, 2, 1, 0):
            hid = k in (1, 2)
            g[2 * k], g[2 * k + 1] = dz.T @ (rnd(h[k]) if hid else h[k]), dz.sum(0)
            if k:
                s = 1 / (1 + np.exp(-z[k - 1]))
                dz = (dz @ (rnd(P[2 * k]) if hid else P[2 * k])) * (s * (1 + z[k - 1] * (1 - s)))
        t = it + 1
        lr = 2e-3 * (0.02 + 0.98 * 0.5 * (1 + math.cos(math.pi * min(1.0, t / steps))))
        for k in range(8):
            M[k] = 0.9 * M[k] + 0.1 * g[k]
            V[k] = 0.999 * V[k] + 0.001 * g[k] * g[k]
            P[k] = P[k] - lr * (M[k] / (1 - 0.9 ** t)) / (np.sqrt(V[k] / (1 - 0.999 ** t)) + 1e-8)
    return loss, start, np.concatenate([p.ravel() for p in P])


@pytest.mark.parametrize("quant", [0, 1])
@pytest.mark.parametrize("n,batch", [(1700, 1500), (8600, 8200), (9500, 9001)])
def test_weighted_wrapped_and_rounded_steps(gpu_engine, n, batch, quant):
    steps, seed = 3, 11
    got = gpu_engine.surrogate_train(n_train=n, batch=batch, epochs=steps, qat_epochs=steps * quant, seed=seed,
                                     target="magic", weighting="transfer")
    assert got["steps"] == steps
    loss, start, want = _train(gpu_engine, n, batch, steps, quant, seed)
    assert abs(got["final_loss"] - loss) <= 1e-4 * loss
    p = gpu_engine.surrogate_params()
    assert np.linalg.norm(p - want) <= 2e-2 * np.linalg.norm(want - start)
