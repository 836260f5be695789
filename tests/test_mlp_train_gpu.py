"""The training run's order and step: with all features zero the network is its output bias alone, and AdamW with
beta1 = beta2 = 0 and a huge epsilon is plain gradient descent on it, b <- b - lr 2 (b - t) in FP32. At lr = 1/4 each pair
halves what the bias held before, so the bias after an epoch of single-pair batches tells the last pairs' order and the
epoch's mean loss that of all. They are compared with the sequential Fisher-Yates shuffle in Python; single steps
round at 1e-7 and epsilon shrinks each by a factor 1 - |g| / 1e6, far below the tolerance of 1e-4."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

M64 = (1 << 64) - 1


def _epochs(t, seed, epochs):
    s = (seed ^ 0xBB67AE8584CAA73B) & M64
    n, b = len(t), 0.0
    for _ in range(epochs):
        o = list(range(n))
        for q in range(n - 1, 0, -1):
            s = (s + 0x9E3779B97F4A7C15) & M64
            z = ((s ^ (s >> 30)) * 0xBF58476D1CE4E5B9) & M64
            z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & M64
            j = (z ^ (z >> 31)) % (q + 1)
            o[q], o[j] = o[j], o[q]
        loss = 0.0
        for i in o:
            loss += (b - t[i]) ** 2
            b -= 0.5 * (b - t[i])
    return b, loss / n


@pytest.mark.parametrize("n", [1, 2, 3, 64, 257, 1000])
def test_epoch_order_is_the_sequential_shuffle(gpe_mod, cuda_ok, n):
    t = np.random.default_rng(n).normal(0, 1, n).astype(np.float32)
    net = gpe_mod.Mlp(max_pairs=n + 5, seed=3)
    net.set_pairs(np.zeros((n, gpe_mod.MLP_FEATURES), np.float32), t)
    loss, _ = net.train(gpe_mod.make_train_params(epochs=2, batch=1, lr=0.25e6, weight_decay=0.0, beta1=0.0, beta2=0.0,
                                                  adam_eps=1e6, val_fraction=0.0, seed=11))
    t64 = t.astype(np.float64)
    sd = t64.std() if n > 1 else 1.0
    b, want = _epochs((t64 - t64.mean()) / sd, 11, 2)
    assert abs(net.blob()[gpe_mod.MLP_NUM_WEIGHTS - 1] - b) < 1e-4
    assert abs(loss - want) < 1e-4
