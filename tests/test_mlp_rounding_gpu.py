"""Training in FP32, bit for bit where nothing depends on the order in which CTAs finish: an epoch's weights amplify the
last bits of its first gradients and moments, so their rounding is part of the result."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

M64 = (1 << 64) - 1
W3 = slice(4992, 5056)
DECAYED = (slice(0, 768), slice(832, 4928), W3)


def _pairs(n, seed):
    g = np.random.default_rng(seed)
    X = g.normal(0, 1, (n, 12)).astype(np.float32)
    return X, (X[:, 9] - X[:, 1] + 0.3 * np.tanh(X[:, 2] * X[:, 5])).astype(np.float32)


def _fma(a, b, c):
    """FP32 a b + c rounded once (the product is exact in FP64)"""
    return (np.asarray(a, np.float64) * np.asarray(b, np.float64) + np.asarray(c, np.float64)).astype(np.float32)


@pytest.mark.parametrize("n", [1, 31, 32, 33, 96, 127, 128])
def test_output_weights_gradient_adds_32_pairs_after_32(gpe_mod, cuda_ok, n):
    """The gradient of w3 over one tile is the sums of its 32-row groups added in their order. Each group's sum comes from
    a call of its own, in which the other rows have the network's own output as target: no error, exact zeros."""
    X, T = _pairs(128, 7)
    net = gpe_mod.Mlp(max_pairs=8, seed=4)

    def padded(rows):
        t = np.where(rows, T, out)
        return net.gradient(X, t)[0][W3]

    blob = net.blob()
    blob[5056:] = 0.0  # b3 = 0; standardisation by mean 0 and deviation 1
    blob[5057 + 12:5057 + 24] = 1.0
    blob[-1] = 1.0
    net.set_blob(blob)
    out = net.infer(X)
    rows = np.arange(128) < n
    parts = [padded(rows & (np.arange(128) // 32 == q)) for q in range(4)]
    want = np.float32(0) + parts[0]
    for q in range(1, 4):
        want = want + parts[q]
    assert np.abs(want).max() > 0
    assert np.array_equal(padded(rows), want)


def _orders(n, seed, epochs):
    s = (seed ^ 0xBB67AE8584CAA73B) & M64
    for _ in range(epochs):
        o = list(range(n))
        for q in range(n - 1, 0, -1):
            s = (s + 0x9E3779B97F4A7C15) & M64
            z = ((s ^ (s >> 30)) * 0xBF58476D1CE4E5B9) & M64
            z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & M64
            j = (z ^ (z >> 31)) % (q + 1)
            o[q], o[j] = o[j], o[q]
        yield np.array(o)


@pytest.mark.parametrize("weight_decay", [0.0, 0.3])
def test_adamw_rounds_as_stated(gpe_mod, cuda_ok, weight_decay):
    """Three epochs of one minibatch of 64 pairs (two groups of 32 rows, whose sum has no order): the weights after each
    are AdamW's of the engine's own gradients with m = fma(1 - beta1, g, beta1 m), v = fma((1 - beta2) g, g, beta2 v),
    the decay added unfused and the step subtracted fused."""
    f = np.float32
    n = 64
    X, T = _pairs(n, 3)
    net = gpe_mod.Mlp(max_pairs=n, seed=1)
    net.set_pairs(X, T)
    first = net.blob()
    tp = gpe_mod.make_train_params(batch=n, lr=2e-3, seed=3, val_fraction=0.0, weight_decay=weight_decay)
    W, norm = [first[:5057]], None
    for epochs in (1, 2, 3):
        tp.epochs = epochs
        net.set_blob(first)
        net.train(tp)
        W.append(net.blob()[:5057])
        norm = net.blob()[5057:]
    b1, b2, eps, lr, wd = (f(v) for v in (tp.beta1, tp.beta2, tp.adam_eps, tp.lr, weight_decay))
    decayed = np.zeros(5057, bool)
    for s in DECAYED:
        decayed[s] = True
    m, v = np.zeros(5057, f), np.zeros(5057, f)
    for t, order in enumerate(_orders(n, 3, 3), 1):
        w = W[t - 1]
        net.set_blob(np.concatenate([w, norm]))
        g = net.gradient(X[order], T[order])[0]
        m = _fma(f(1) - b1, g, b1 * m)
        v = _fma((f(1) - b2) * g, g, b2 * v)
        step = (m / (f(1) - f(float(b1) ** t))) / (np.sqrt(v / (f(1) - f(float(b2) ** t))) + eps)
        step = np.where(decayed, step + wd * w, step)
        assert np.array_equal(_fma(-lr, step, w), W[t]), f"step {t}"
