"""Mixed steps whose displacement flags need no memset: the first half-steps zero them
(atoms) or mark them (nodes).  The trajectory is the same to the bit however the steps
are issued -- replayed graphs, eager steps, the device loop, one run a step (which
starts the marks anew) and rebuild decisions in between -- and the lists are reordered
as often; and leaving out the far entries changes no bit, so no displacement is stale.
"""
import os
import tempfile

import numpy as np
import pytest

from cac_code_gb300 import cacg
from cac_code_gb300 import workloads as W

pytestmark = pytest.mark.gpu
STEPS = 60


@pytest.fixture(scope="module")
def eam_file():
    return W.write_eam(os.path.join(tempfile.mkdtemp(), "Cu_analytic_2000.eam"))


def _run(pair, eam, how, every):
    if pair == "eam":
        m, cfg = W.c2_eam(cells=(4, 22, 22), layers=8, seed=23)
        fast = 30.0  # the heavy nodes move far enough for reorders
    else:
        m, cfg = W.c1_lj(seed=23)
        fast = 14.0
    cfg["every"] = every
    s = cacg.System(0)
    try:
        W.configure_system(s, m, cfg, eam)
        s.command("neigh_modify every %d delay 0 check yes" % every)
        s.set_precision(cacg.MIXED)
        if how == "loop":
            s.command("tune loop device")
        if how == "uncut":
            s.command("tune cull no")
        if how == "eager":
            s.set_graphs(False)
        s.init()
        s.setup()
        a, e = s.atoms(), s.elements()
        s.put_atoms(a["x"], 3.0 * a["v"])
        s.put_nodes(e["nodex"], fast * e["nodev"])
        for n in ([1] * STEPS if how == "single" else [STEPS]):
            s.run(n)
        a, e, c = s.atoms(), s.elements(), s.counts()
        return (a["x"], a["v"], e["nodex"], e["nodev"]), (c["ip_reorders"], c["atom_reorders"])
    finally:
        s.close()


@pytest.mark.parametrize("every", [10, 100000])
@pytest.mark.parametrize("pair", ["lj", "eam"])
def test_steps_agree_however_issued(cacg_lib, eam_file, pair, every):
    want, reorders = _run(pair, eam_file, "graphs", every)
    assert reorders[0] >= 2 and (pair == "lj" or reorders[1] >= 2)
    for how in ("eager", "single", "loop", "uncut"):
        got, r = _run(pair, eam_file, how, every)
        assert r == reorders, how
        for x, y in zip(got, want):
            assert np.array_equal(x.view(np.int64), y.view(np.int64)), how
