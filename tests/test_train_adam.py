"""Several Adam steps of the surrogate's training against numpy."""
import numpy as np
import pytest

from oracle import mlp_oracle as MO
from test_train_passes import _data

pytestmark = pytest.mark.gpu


def _shuffles(seed, n, count):
    """The training's row orders, one after another from one splitmix64 sequence."""
    state, mask = seed, (1 << 64) - 1
    for _ in range(count):
        q = list(range(n))
        for i in range(n - 1, 0, -1):
            state = (state + 0x9E3779B97F4A7C15) & mask
            z = state
            z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & mask
            z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
            k = (z ^ (z >> 31)) % (i + 1)
            q[i], q[k] = q[k], q[i]
        yield q


def test_adam_over_two_epochs_of_two_steps(cacg_lib):
    """Two members, two batches of 128 an epoch: the step sizes follow the cosine over the
    epochs, the bias corrections those of each epoch's first step (1, then 3).  Gradients
    are the device's own at numpy's parameters.  numpy's and the device's parameters differ
    by float32 roundings of an update (below 1e-6 of it) and of p (6e-8 |p|, |p| < 0.4:
    2.4e-8), 2.5e-5 lr a step; one that moves a parameter's BF16 copy by its last bit (2^-8
    of it) changes a later gradient by that share of one of 256 terms, far below 1 %, where a
    correction by step would change the second update by a third.  2 % of lr, for entries
    whose gradients are above 0.3 of their rms in all four steps."""
    n, batch, members, epochs, lr, seed = 256, 128, 2, 2, 1e-3, 11
    x, t = _data(n, 5)
    one = np.ones(MO.NIN, np.float32), np.ones(MO.NOUT, np.float32)
    nets = [cacg_lib.Mlp(0, members=members, seed=8) for _ in range(2)]
    try:
        for net in nets:
            net.set_normalization(0 * one[0], one[0], 0 * one[1], one[1], 1.0)
        net, ref = nets
        net.train(x, t, epochs=epochs, batch=batch, lr=lr, seed=seed)
        order = list(_shuffles(seed, n, epochs * members))
        for k in range(members):
            p = ref.params(k).astype(np.float64)
            m, v, clear = np.zeros_like(p), np.zeros_like(p), np.ones(p.size, bool)
            for ep in range(epochs):
                rate = lr * (0.05 + 0.95 * 0.5 * (1 + np.cos(np.pi * ep / epochs)))
                c1, c2 = 1 - 0.9 ** (2 * ep + 1), 1 - 0.999 ** (2 * ep + 1)
                for b in range(n // batch):
                    rows = order[ep * members + k][b * batch:(b + 1) * batch]
                    ref.set_params(k, p.astype(np.float32))
                    g = ref.loss_grad(k, x[rows], t[rows])[1].astype(np.float64)
                    m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
                    p = p - rate * (m / c1) / (np.sqrt(v / c2) + 1e-8)
                    clear &= np.abs(g) > 0.3 * np.sqrt((g * g).mean())
            assert clear.sum() > 1000
            assert np.abs(net.params(k) - p)[clear].max() <= 0.02 * lr
    finally:
        for net in nets:
            net.close()
