"""Atom lists of atoms that have left a box with fixed boundaries."""
import numpy as np
import pytest

from cac_code_gb300 import cacg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [0.0, 90.0, 1500.0])
def test_atoms_far_outside_the_box(cacg_lib, shift):
    """6,000 atoms beside the box: a coordinate of 1,500 has a float spacing of 1.2e-4, so
    that float distances misplace some pairs about the list cutoff.  Entry for entry what
    FP64 arithmetic gives (the reference's: rsq <= cutneighmax^2)."""
    rng = np.random.default_rng(4)
    x = rng.uniform(0.0, 1.0, (6000, 3)) * [12.0, 12.0, 3.0] + [shift, 0.0, 0.0]
    s = cacg.System(0)
    try:
        s.command("units lj")
        s.command("boundary f p f")
        s.set_box(np.zeros(3), np.full(3, 12.0), (0, 1, 0))
        s.set_masses([1.0])
        s.set_atoms(x, np.zeros_like(x), np.ones(len(x), dtype=np.int32))
        for c in ("pair_style lj/cut 2.5", "pair_coeff 1 1 1.0 1.0", "neighbor 2.8 bin",
                  "neigh_modify every 1 delay 0 check yes", "timestep 0.005", "fix 1 all nve"):
            s.command(c)
        s.set_precision(cacg.FP64_EXACT)
        s.init()
        s.setup()
        s.neighbor_build()
        num, neigh = s.atom_list()
        xa = s.atoms(all_=True)["x"]
    finally:
        s.close()
    got = np.split(np.asarray(neigh), np.cumsum(num)[:-1])
    for i in range(len(x)):
        d = xa[i] - xa
        rsq = d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1] + d[:, 2] * d[:, 2]
        want = np.flatnonzero(rsq <= 2.8 * 2.8)
        assert np.array_equal(np.sort(got[i]), want[want != i]), i
