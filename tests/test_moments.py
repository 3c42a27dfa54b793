"""A data set's means, deviations and force scale on the device against NumPy's, to the
bit, at the edges of the kernel's chunks of 64 rows, and the forms that NumPy takes."""
import numpy as np
import pytest

from cac_code_gb300 import cacg

pytestmark = pytest.mark.gpu


def _numpy(x, t):
    sd, osd = x.std(axis=0), t.std(axis=0)
    fs = float(np.sqrt((t.astype(np.float64) ** 2).sum(axis=1).mean() / 8.0))
    return (x.mean(axis=0), np.where(sd > 0, sd, 1.0), t.mean(axis=0), np.where(osd > 0, osd, 1.0),
            max(fs, 1e-30))


@pytest.mark.parametrize("n", [1, 63, 64, 65, 256, 1023, 1024, 1087, 1088, 20001])
@pytest.mark.parametrize("form", ["plain", "double", "columns", "slice"])
def test_normalization_is_numpys(cacg_lib, monkeypatch, n, form):
    monkeypatch.setattr(cacg, "MOMENTS_MIN", 1)
    rng = np.random.default_rng(n)
    x = (rng.normal(0.3, 1.0, (n, 32)) * np.exp(rng.normal(0.0, 3.0, 32))).astype(np.float32)
    t = (rng.normal(0.0, 1.0, (n, 24)) * np.exp(rng.normal(0.0, 3.0, 24))).astype(np.float32)
    x[:, 5], t[:, 7] = 2.5, 0.0  # nothing to scale by
    x[:, 6] = -0.0
    if form == "double":
        x, t = x.astype(np.float64), t.astype(np.float64)
    if form == "columns":
        x, t = np.asfortranarray(x), np.asfortranarray(t)
    if form == "slice":
        x, t = np.repeat(x, 2, axis=0)[::2], np.repeat(t, 2, axis=0)[::2]
    net = cacg.Mlp(0, members=1, seed=1)
    try:
        net.fit_normalization(x, t)
        got = net.normalization()
    finally:
        net.close()
    net = cacg.Mlp(0, members=1, seed=1)
    try:
        net.set_normalization(*_numpy(x, t))
        want = net.normalization()
    finally:
        net.close()
    for g, w in zip(got, want):
        assert np.array_equal(np.asarray(g), np.asarray(w))
