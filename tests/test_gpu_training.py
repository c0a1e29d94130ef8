"""GPU tests of the training step: the gradient at the edges of its blocks of 64
rows, and the chained launches of gradient and update against the same step made
one gradient at a time."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def hc():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from nemo_gb300 import build as B
    B.build()
    from nemo_gb300 import hackcode
    return hackcode


def _rows(n, seed):
    rng = np.random.default_rng(seed)
    x = rng.normal(0.0, 1.5, (n, 12)).astype(np.float32)
    y = (rng.random(n) < 0.4).astype(np.float32)
    return x, y, rng.uniform(0.5, 2.0, n).astype(np.float32)


@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 127, 128, 129])
def test_gradient_is_the_sum_over_its_rows(hc, n):
    """Each row's terms are computed alike wherever the row stands, so a batch's
    gradient differs from the sum of its rows' by the FP32 sums over 64 rows and
    the blocks: at most 2^-24 of the sum of magnitudes per addition."""
    ctx = hc.Context(1024)
    ctx.learn_init(7)
    x, y, w = _rows(n, n)
    loss, g = ctx.learn_gradient(x, y, w)
    ls, total, size = 0.0, np.zeros(len(g)), np.zeros(len(g))
    for i in range(n):
        l1, g1 = ctx.learn_gradient(x[i:i + 1], y[i:i + 1], w[i:i + 1])
        ls += float(l1)
        total += g1.astype(float) * w[i] / w.sum(dtype=float)
        size += np.abs(g1) * w[i] / w.sum(dtype=float)
    assert (np.abs(g - total) <= (64 + 8) * 2.0 ** -24 * size + 1e-30).all()
    assert abs(loss - ls) <= 1e-5 * ls


def test_gradient_of_the_largest_batch(hc):
    """64 rows repeated over all 128 blocks: the gradient of the 64."""
    ctx = hc.Context(1024)
    ctx.learn_init(7)
    x, y, w = _rows(64, 5)
    _, g = ctx.learn_gradient(x, y, w)
    _, g128 = ctx.learn_gradient(np.tile(x, (128, 1)), np.tile(y, 128), np.tile(w, 128))
    size = np.zeros(len(g))
    for i in range(64):
        size += np.abs(ctx.learn_gradient(x[i:i + 1], y[i:i + 1], w[i:i + 1])[1]) * w[i] / w.sum(dtype=float)
    assert (np.abs(g128 - g) <= (64 + 128) * 2.0 ** -24 * size + 1e-30).all()


@pytest.mark.parametrize("n,batch", [(64, 64), (1280, 64), (1337, 100), (5000, 4096), (20000, 8192)])
def test_training_is_gradients_and_adam_steps(hc, n, batch):
    x, y, w = _rows(n, n + batch)
    lr, seed = 1e-3, 3
    ctx, one = hc.Context(1024), hc.Context(1024)
    ctx.learn_init(5)
    p = ctx.learn_params().astype(np.float64)
    ctx.learn_load_samples(x, y, w)
    ctx.learn_train(epochs=1, batch=batch, lr=lr, seed=seed)
    perm, st, mask = np.arange(n), (seed * 2862933555777941757 + 3037000493) % 2 ** 64, 2 ** 64 - 1
    for i in range(n - 1, 0, -1):
        st = (st * 6364136223846793005 + 1442695040888963407) & mask
        j = (st >> 33) % (i + 1)
        perm[i], perm[j] = perm[j], perm[i]
    m, v, t = np.zeros(len(p)), np.zeros(len(p)), 0
    for b in range(0, n - 63, batch):
        r = perm[b:b + batch]
        one.learn_params(p.astype(np.float32))
        g = one.learn_gradient(x[r], y[r], w[r])[1].astype(np.float64)
        t += 1
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        p = p - lr * (m / (1 - 0.9 ** t)) / (np.sqrt(v / (1 - 0.999 ** t)) + 1e-8)
    # a weight whose last bit differs may round to another BF16 number, 2^-9 of it away, which moves gradients by
    # parts in a thousand: a twentieth of each step is far above that, and far below a step that read stale weights
    assert np.abs(ctx.learn_params() - p).max() <= 0.05 * lr * t
