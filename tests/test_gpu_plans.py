"""Element passes whose plan no smaller system reaches, against the oracle: bit for bit in
the exact mode, within 1e-12 of the force scale with contraction."""
import os
import tempfile

import numpy as np
import pytest

import cases as C
from cac_code_gb300 import lattice as L
from cac_code_gb300 import workloads as W
from test_gpu_fp64_passes import FP64_TOL, _slab
from test_gpu_fused import rel_err

pytestmark = pytest.mark.gpu


def _long_elements(pair):
    """Elements of 3 x 3 x 66 sites (a line holds more than the line codes' 64), two abreast
    and one apart, in a box with fixed faces, beside a few atoms."""
    lj = pair == "lj/cut"
    a, mass = (C.A_LJ, 1.0) if lj else (C.A_CU, L.AnalyticEAM().mass)
    nae = np.array([3, 3, 66])
    t = (L.NODE_PARENT + 1) // 2
    edge = (nae - 1)[:, None] * a * L.PRIMITIVE
    at = np.array([[0.0, 0.0, 0.0], 3 * a * L.PRIMITIVE[0], 9 * a * L.PRIMITIVE[1]])
    nodex = at[:, None, :] + (t @ edge)[None]
    nodex = nodex + np.random.default_rng(9).normal(0.0, 0.02 if lj else 0.05, nodex.shape)
    gauss = [[i, j, k] for i in (0, 2) for j in (0, 2) for k in (14, 51)]
    intp = np.array([list(c * (nae - 1)) for c in t] + gauss)
    weight = np.array([0.0] * 8 + [3 * 3 * 66 / 8.0] * 8)
    atoms = L.fcc_sites((3, 3, 3), a) + nodex.reshape(-1, 3).max(axis=0) * [0.0, 0.0, 1.0] + [0.0, 0.0, 4 * a]
    every = np.concatenate([atoms, nodex.reshape(-1, 3)])
    return L.Model(boxlo=every.min(axis=0) - a, boxhi=every.max(axis=0) + a, periodic=(False,) * 3,
                   mass=mass, atom_x=atoms, atom_v=np.zeros_like(atoms),
                   etypes=[L.ElementType(tuple(int(n) for n in nae), intp, weight)],
                   elem_type=np.ones(3, dtype=np.int64), nodex=nodex, nodev=np.zeros_like(nodex),
                   lattice_a=a)


# more than an element an SM (positions by the integer units where the lists stay within
# the element, else by the FP64 unit), and elements that the line codes do not hold
CASES = {
    "lj_own_sites": lambda: ("lj/cut", _slab("lj/cut", (2, 32, 32), 8, 3, L.gauss_intp(8, False), 31, 0.02)),
    "lj_other_elements": lambda: ("lj/cut", _slab("lj/cut", (2, 25, 25), 5, 2, L.all_sites_intp(5), 31, 0.02)),
    "eam_other_elements": lambda: ("eam", _slab("eam", (2, 24, 24), 6, 3, L.gauss_intp(6, True), 31, 0.05)),
    "lj_long_lines": lambda: ("lj/cut", _long_elements("lj/cut")),
    "eam_long_lines": lambda: ("eam", _long_elements("eam")),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_forces_match_the_oracle(cacg_lib, oracle_lib, name):
    pair, m = CASES[name]()
    lj, long = pair == "lj/cut", "long" in name
    assert long or m.nelements > 152
    skin = 2.8 if lj else 7.5
    kw = dict(units="lj" if lj else "metal", pair=pair, skin=skin, every=1, delay=0, check=True,
              dt=0.005 if lj else 0.001, **(dict(lj=(1.0, 1.0, 2.5)) if lj else dict(eam_file=C.EAM_FILE)))
    o = oracle_lib.Oracle(m, **kw)
    o.setup()
    o.atom_list()
    ref = [o.atom_forces()]
    o.elem_lists()
    ref.append(o.elem_forces())
    assert np.abs(ref[1]).max() > 0
    for mode in (cacg_lib.FP64_EXACT, cacg_lib.FP64):
        s = cacg_lib.System(0)
        try:
            s.command(f"units {kw['units']}")
            s.command("boundary " + ("f f f" if long else "f p p"))
            s.load_model(m)
            s.command("pair_style " + ("lj/cut 2.5" if lj else "eam"))
            s.command("pair_coeff 1 1 " + ("1.0 1.0" if lj else C.EAM_FILE))
            s.command(f"neighbor {skin!r} bin")
            s.command("fix 1 all nve")
            s.set_precision(mode)
            s.init()
            s.run(0)
            s.pair_compute()
            s.pair_ecompute()
            got = [s.atoms()["f"], s.elements()["nodef"]]
        finally:
            s.close()
        for g, r in zip(got, ref):
            if mode == cacg_lib.FP64_EXACT:
                assert np.array_equal(g.view(np.int64), np.ascontiguousarray(r).view(np.int64))
            else:
                assert np.abs(g - r).max() <= FP64_TOL * np.abs(r).max()


@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_a_lost_node_beside_the_stencil(cacg_lib, value):
    """3,664 elements, one with a node that is no number: the other elements' forces stay
    those of bit-exact FP64, and with the node back all are the former ones, to the bit."""
    m, cfg = W.c2_eam(cells=(4, 22, 22), layers=229, seed=17)
    eam = W.write_eam(os.path.join(tempfile.mkdtemp(), "Cu_analytic_2000.eam"))
    exact = None
    for mode in (cacg_lib.FP64_EXACT, cacg_lib.MIXED):
        s = cacg_lib.System(0)
        try:
            W.configure_system(s, m, cfg, eam)
            s.command("neigh_modify every 100000 delay 0 check yes")
            s.set_precision(mode)
            s.init()
            s.run(0)
            s.pair_ecompute()
            f = s.elements()["nodef"].copy()
            if mode == cacg_lib.FP64_EXACT:
                exact = f
                continue
            x, v = s.elements()["nodex"].copy(), s.elements()["nodev"].copy()
            lost = x.copy()
            lost[1234, 5, 1] = value
            s.put_nodes(lost, v)
            others = np.arange(m.nelements) != 1234
            for _ in range(2):  # the second is the first reorder's successor
                s.pair_ecompute()
                rms, mx = rel_err(s.elements()["nodef"][others], exact[others])
                assert rms <= 1e-4 and mx <= 1e-4, (rms, mx)
            s.run(2)
            s.put_nodes(x, v)
            s.pair_ecompute()
            assert np.array_equal(s.elements()["nodef"].view(np.int64), f.view(np.int64))
        finally:
            s.close()
