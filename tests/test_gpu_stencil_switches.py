"""Switches that must not change a bit, above the number of elements from which the mixed
EAM element passes share one stencil (24 a multiprocessor: 3,664 elements here)."""
import numpy as np
import pytest

from cac_code_gb300 import cacg
from cac_code_gb300 import workloads as W
from test_gpu_fused import rel_err
from test_gpu_mixed import _host_array
from test_gpu_stencil import _model, eam_file  # noqa: F401  (eam_file: a fixture)

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def alike():
    return _model("alike")


def _system(m, cfg, eam, *tune):
    s = cacg.System(0)
    W.configure_system(s, m, cfg, eam)
    s.set_precision(cacg.MIXED)
    for t in tune:
        s.command("tune " + t)
    s.init()
    s.run(0)
    return s


@pytest.mark.parametrize("parts", [4, 8])
def test_run_host_in_small_parts_follows_run(cacg_lib, alike, eam_file, parts):  # noqa: F811
    """run_host with the force pass in parts of 916 and 458 elements (8 an SM and below are
    few enough for the passes from the lists) gives run's trajectory to the bit."""
    m, cfg = alike
    a, b = _system(m, cfg, eam_file, f"out_parts {parts}"), _system(m, cfg, eam_file)
    try:
        x0, e0 = a.atoms(), a.elements()
        hx, hv = _host_array(x0["x"], True), _host_array(x0["v"], True)
        hnx, hnv = _host_array(e0["nodex"], True), _host_array(e0["nodev"], True)
        for _ in range(12):
            a.run_host(1, hx, hv, hnx, hnv)
        b.run(12)
        xb, eb = b.atoms(), b.elements()
        assert b.counts()["elem_fused"] == 1
        for got, want in ((hx, xb["x"]), (hv, xb["v"]), (hnx, eb["nodex"]), (hnv, eb["nodev"])):
            assert np.array_equal(got, want)
    finally:
        a.close()
        b.close()


def _reorder_us(eam, layers, jitter):
    """Device time of a step's element list reorder, the least of six."""
    m, cfg = W.c2_eam(cells=(4, 22, 22), layers=layers, seed=17)
    m.nodex = m.nodex + np.random.default_rng(5).normal(0.0, jitter, m.nodex.shape)
    s = _system(m, cfg, eam)
    try:
        s.command("neigh_modify every 100000 delay 0 check yes")
        s.set_graphs(False)
        s.run(2)
        x, t = s.elements()["nodex"].copy(), []
        before = s.counts()["ip_reorders"]
        for k in range(6):
            s.put_nodes(x + (0.6 if k % 2 == 0 else 0.0), np.zeros_like(x))  # 0.6 A to and fro
            s.set_timing(True)
            s.run(1)
            t.append(1e3 * s.kernel_timing()[7])
        assert s.counts()["ip_reorders"] - before == 6
        return min(t)
    finally:
        s.close()


@pytest.mark.parametrize("jitter", [0.05, 1.0])
def test_reorder_with_the_stencil_costs_little_more(cacg_lib, eam_file, jitter):  # noqa: F811
    """A reorder of 3,664 elements builds and checks a stencil, whether it stands (alike) or
    not; one of 3,632 does not.  Both work on the same lists, so at most three times."""
    few, many = (_reorder_us(eam_file, n, jitter) for n in (227, 229))
    assert many <= 3.0 * few, (few, many)


@pytest.mark.parametrize("shape", ["alike", "shrunk", "crooked"])
def test_band_width_changes_no_bit(cacg_lib, eam_file, shape):  # noqa: F811
    """Widened to cutsq (1 +- 0.1), the guard band holds a lattice shell (at +8 %: scanned
    with the displacement culling off), so that every element is run again with FP64
    decisions, at every pass; these are the decisions of the default band, and the sums are
    taken in the same order: 8 steps to the bit, from the stencil (alike, shrunk) and from
    the lists (crooked)."""
    m, cfg = _model(shape)
    out = []
    for tune in ((), ("band 0.1",)):
        s = _system(m, cfg, eam_file, "cull no", *tune)
        try:
            s.pair_compute()
            s.pair_ecompute()
            f = s.elements()["nodef"].copy()
            s.run(8)
            out.append((f, s.elements(), s.counts()))
        finally:
            s.close()
    (f0, e0, c0), (f1, e1, c1) = out
    assert c1["elem_fused"] == 1 and c1["elem_stencil"] == (shape != "crooked")
    assert c1["band_reruns"] >= 2 * (1 + 8) * c1["enlocal"] > c0["band_reruns"]
    assert np.array_equal(f0.view(np.int64), f1.view(np.int64))
    for k in ("nodex", "nodev", "nodef"):
        assert np.array_equal(e0[k], e1[k]), k


def test_tables_that_fill_a_block(cacg_lib, alike, tmp_path):
    """Splines of 4,266 knots: the force pass from the lists takes all shared memory of a
    block but 16 bytes, more than the stencil's kernel can have beside its static part."""
    m, cfg = alike
    eam = W.write_eam(str(tmp_path / "Cu_4266.eam"), 4266)
    out = {}
    for mode in (cacg.MIXED, cacg.FP64_EXACT):
        s = cacg.System(0)
        try:
            W.configure_system(s, m, cfg, eam)
            s.set_precision(mode)
            s.init()
            s.run(0)
            s.pair_ecompute()
            out[mode] = s.elements()["nodef"].copy()
            c = s.counts()
            assert mode != cacg.MIXED or (c["elem_fused"], c["elem_stencil"]) == (1, 0)
        finally:
            s.close()
    rms, mx = rel_err(out[cacg.MIXED], out[cacg.FP64_EXACT])
    assert rms <= 1e-4 and mx <= 1e-4, (rms, mx)
