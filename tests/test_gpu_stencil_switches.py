"""Switches that must not change a bit, above the number of elements from which the mixed
EAM element passes share one stencil (24 a multiprocessor: 3,664 elements here)."""
import numpy as np
import pytest

from cac_code_gb300 import cacg
from cac_code_gb300 import workloads as W
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
