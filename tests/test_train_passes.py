"""The surrogate's training passes at the edges of their tiles,
against the numpy restatement."""
import numpy as np
import pytest

from oracle import mlp_oracle as MO

pytestmark = pytest.mark.gpu


def _data(n, seed):
    rng = np.random.default_rng(seed)
    x = rng.normal(size=(n, MO.NIN)).astype(np.float32)
    w = np.random.default_rng(0).normal(size=(MO.NIN, MO.NOUT)) / np.sqrt(MO.NIN)
    return x, np.tanh(x @ w).astype(np.float32)


# one row, a full tile, one row more, a last tile of 65 rows, and one of 8 rows behind 39
# full ones (the weight gradients run over 2, 2, 4, 10 and 80 k-tiles of 64 rows)
@pytest.mark.parametrize("n", [1, 128, 129, 577, 5000])
def test_loss_and_gradient(cacg_lib, n):
    x, t = _data(n, n)
    net = cacg_lib.Mlp(0, members=3, seed=n)
    try:
        # unit normalisation: one row has no spread of its own
        one = np.ones(MO.NIN, np.float32), np.ones(MO.NOUT, np.float32)
        net.set_normalization(0 * one[0], one[0], 0 * one[1], one[1], 1.0)
        for k in (0, 2):
            loss, g = net.loss_grad(k, x, t)
            l_ref, g_ref = MO.loss_grad(net.params(k).astype(np.float64), x.astype(np.float64),
                                        t.astype(np.float64))
            # bf16 operands: the bounds of the existing gradient test
            assert abs(loss - l_ref) <= 1e-3 * l_ref
            offs = np.cumsum([0] + [int(np.prod(s)) for _, s in MO.SHAPES])
            for b, (name, _) in enumerate(MO.SHAPES):
                gd, gr = g[offs[b]:offs[b + 1]], g_ref[offs[b]:offs[b + 1]]
                assert np.linalg.norm(gd - gr) < 2e-2 * max(np.linalg.norm(gr), 1e-30), (k, name)
    finally:
        net.close()


@pytest.mark.parametrize("members,batch", [(1, 128), (4, 640)])
def test_one_adam_step_moves_every_member_against_its_gradient(cacg_lib, members, batch):
    """n = batch, one epoch: one step, in which Adam moves each parameter by
    lr g / (|g| + 1e-8): by lr against the sign of g where g is not small (the
    gradient is within 2e-2 of its norm, so entries above 0.3 rms keep their
    sign; float32 rounding of the update and of p stays below 1e-3 lr)."""
    x, t = _data(batch, 3)
    lr = 1e-3
    net = cacg_lib.Mlp(0, members=members, seed=8)
    try:
        one = np.ones(MO.NIN, np.float32), np.ones(MO.NOUT, np.float32)
        net.set_normalization(0 * one[0], one[0], 0 * one[1], one[1], 1.0)
        before = [net.params(k) for k in range(members)]
        loss = net.train(x, t, epochs=1, batch=batch, lr=lr, seed=2)
        refs = [MO.loss_grad(p.astype(np.float64), x.astype(np.float64), t.astype(np.float64))
                for p in before]
        assert abs(loss - np.mean([r[0] for r in refs])) <= 1e-3 * loss
        offs = np.cumsum([0] + [int(np.prod(s)) for _, s in MO.SHAPES])
        for k in range(members):
            d, g = net.params(k).astype(np.float64) - before[k], refs[k][1]
            for b in range(len(MO.SHAPES)):
                gb, db = g[offs[b]:offs[b + 1]], d[offs[b]:offs[b + 1]]
                big = np.abs(gb) > max(0.3 * np.sqrt((gb ** 2).mean()), 1e-5)
                assert big.any()
                assert np.abs(db[big] + lr * np.sign(gb[big])).max() <= 2e-3 * lr, (k, b)
    finally:
        net.close()
