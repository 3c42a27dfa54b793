"""The mixed EAM element passes over a shared stencil (32 elements a warp) against
the passes from the lists (one warp an element), at a number of elements that leaves
the last warp half full.

Sums are taken in another order, so the forces agree within the tolerance of the
mixed parity tests against bit-exact FP64 (1e-4); what culling leaves out changes no
bit.  Elements that are not alike run from the lists, to the bit.
"""
import os
import tempfile

import numpy as np
import pytest

from cac_code_gb300 import cacg
from cac_code_gb300 import workloads as W
from test_gpu_fused import rel_err

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eam_file():
    return W.write_eam(os.path.join(tempfile.mkdtemp(), "Cu_analytic_2000.eam"))


def _model(shape, vscale=1.0):
    m, cfg = W.c2_eam(cells=(4, 22, 22), layers=229, seed=17)  # 3,664 elements
    rng = np.random.default_rng(5)
    jitter = {"alike": 0.05, "shrunk": 0.05, "crooked": 1.0}[shape]
    m.nodex = m.nodex + rng.normal(0.0, jitter, m.nodex.shape)
    if shape == "shrunk":  # one element in 16 in a denser state
        x = m.nodex.reshape(-1, 8, 3)
        c = x.mean(axis=1, keepdims=True)
        x[::16] = c[::16] + 0.8 * (x[::16] - c[::16])
        m.nodex = x.reshape(m.nodex.shape)
    m.nodev = m.nodev * vscale
    m.atom_v = m.atom_v * vscale
    return m, cfg


def _forces(m, cfg, eam, mode, tune=(), steps=0):
    s = cacg.System(0)
    try:
        W.configure_system(s, m, cfg, eam)
        s.set_precision(mode)
        for t in tune:
            s.command("tune " + t)
        s.init()
        s.setup()
        s.neighbor_build()
        s.neighbor_ebuild()
        s.neighbor_nbuild()
        s.pair_compute()
        s.pair_ecompute()
        f = s.elements()["nodef"].copy()
        if steps:
            s.run(steps)
        return f, s.elements(), s.counts()
    finally:
        s.close()


@pytest.mark.parametrize("shape", ["alike", "shrunk", "crooked"])
def test_stencil_passes_match_the_lists(cacg_lib, eam_file, shape):
    m, cfg = _model(shape)
    lists, _, c0 = _forces(m, cfg, eam_file, cacg.MIXED, ["fused_variant 0"])
    sten, _, c1 = _forces(m, cfg, eam_file, cacg.MIXED)
    uncut, _, _ = _forces(m, cfg, eam_file, cacg.MIXED, ["cull no"])
    assert c0["elem_fused"] == 1 and c1["elem_fused"] == 1
    assert np.array_equal(sten.view(np.int64), uncut.view(np.int64))
    same = np.array_equal(sten.view(np.int64), lists.view(np.int64))
    assert same == (shape == "crooked")
    exact, _, _ = _forces(m, cfg, eam_file, cacg.FP64_EXACT)
    rms, mx = rel_err(sten, exact)
    assert rms <= 1e-4 and mx <= 1e-4, (rms, mx)


@pytest.mark.parametrize("vscale", [1.0, 40.0])
def test_stencil_run_follows_the_lists(cacg_lib, eam_file, vscale):
    """25 steps, at 40x the thermal speeds with list reorders (a new stencil each),
    within 1e-6 A of the run from the lists."""
    m, cfg = _model("alike", vscale)
    _, e0, _ = _forces(m, cfg, eam_file, cacg.MIXED, ["fused_variant 0"], 25)
    _, e1, c1 = _forces(m, cfg, eam_file, cacg.MIXED, [], 25)
    assert np.abs(e1["nodex"] - e0["nodex"]).max() < 1e-6
    if vscale > 1.0:
        assert c1["ip_reorders"] >= 2, c1["ip_reorders"]


def test_stencil_with_the_surrogate(cacg_lib, eam_file):
    """Elements that the surrogate evaluates are left as it wrote them, the others get the
    same bits as without it (an untrained net: every far element, then none)."""
    m, cfg = _model("alike")
    net = cacg_lib.Mlp(0, members=2, seed=3)
    s = cacg.System(0)
    try:
        net.set_normalization(np.zeros(32), np.ones(32), np.zeros(24), np.ones(24), 1.0)
        W.configure_system(s, m, cfg, eam_file)
        s.set_precision(cacg.MIXED)
        s.init()
        s.setup()
        s.neighbor_build()
        s.neighbor_ebuild()
        s.neighbor_nbuild()
        s.surrogate_reference(m.nodex)
        s.pair_ecompute()
        plain = s.elements()["nodef"].copy()
        s.surrogate_attach(net, tol=1e30, dist=11.0)
        s.pair_ecompute()
        far = s.counts()["surrogate_elements"]
        some = s.elements()["nodef"].copy()
        changed = np.any(some != plain, axis=(1, 2))
        assert 0 < far < m.nelements and changed.sum() == far
        assert np.array_equal(some[~changed], plain[~changed])
        s.command("tune fused_variant 0")  # from the lists
        s.pair_ecompute()
        assert np.array_equal(s.elements()["nodef"][changed], some[changed])
        s.command("tune fused_variant 1")
        s.surrogate_attach(net, tol=0.0, dist=11.0)
        s.pair_ecompute()
        assert np.array_equal(s.elements()["nodef"], plain)
    finally:
        s.close()
        net.close()
