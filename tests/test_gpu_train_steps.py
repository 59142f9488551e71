"""The trainer's batches and parameter steps one by one: the same rows of the epoch's
permutation through the stateless gradient, and Adam in FP64 on the host."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

M32, M64 = 0xFFFFFFFF, (1 << 64) - 1


def keys(seed):
    out = []
    for _ in range(2):
        seed = (seed + 0x9E3779B97F4A7C15) & M64
        z = seed
        z = ((z ^ z >> 30) * 0xBF58476D1CE4E5B9) & M64
        z = ((z ^ z >> 27) * 0x94D049BB133111EB) & M64
        z ^= z >> 31
        out += [z & M32, z >> 32]
    return out


def permutation(n, seed):
    half = 0
    while 1 << 2 * half < n:
        half += 1
    mask, key = (1 << half) - 1, keys(seed)

    def mix(x):
        x = ((x ^ x >> 16) * 0x7FEB352D) & M32
        x = ((x ^ x >> 15) * 0x846CA68B) & M32
        return x ^ x >> 16

    def step(x):
        l, r = x >> half, x & mask
        for k in key:
            l, r = r, l ^ (mix(r ^ k) & mask)
        return l << half | r

    rows = []
    for i in range(n):
        x = step(i)
        while x >= n:
            x = step(x)
        rows.append(x)
    return np.array(rows)


# batches of several tiles with a short last one, one batch of part of a tile, a last batch
# of one row
@pytest.mark.parametrize("n,batch", [(3000, 777), (100, 4096), (513, 128)])
def test_epoch_is_its_batches(swc_mod, n, batch):
    from swc import learn

    rng = np.random.default_rng(n)
    f = rng.normal(size=(n, 8)).astype(np.float32)
    t = (f[:, 0] * f[:, 1] + 0.1 * rng.normal(size=n)).astype(np.float32)
    p0, norm, lr = learn.init_params(3), learn.normalisation(f, t), 1e-3
    tr = learn.Trainer(n, batch)
    tr.add(f, t)
    tr.set_params(p0, norm)
    tr.fit(epochs=1, lr=lr, seed=11)
    got = tr.params()[0]
    tr.close()

    order = permutation(n, 11)
    assert np.array_equal(np.sort(order), np.arange(n))
    p, m, v = p0.astype(np.float64), 0.0, 0.0
    steps = range(0, n, batch)
    for k, b in enumerate(steps, 1):
        rows = order[b:b + batch]
        g = learn.gradient(p.astype(np.float32), norm, f[rows], t[rows])[0].astype(np.float64)
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        p -= lr * (m / (1 - 0.9 ** k)) / (np.sqrt(v / (1 - 0.999 ** k)) + 1e-8)
    # a step is about lr a parameter whatever the gradient's size; FP32 against FP64 here
    # can turn the BF16 rounding of single weights (2^-8 of one term of a gradient)
    assert np.abs(got - p).max() < 0.02 * lr * len(steps)
