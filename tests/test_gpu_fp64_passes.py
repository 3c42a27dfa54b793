"""The FP64 passes at the sizes where their blocks' edges lie, against the
oracle: bit for bit in the exact mode, within 1e-12 of the force scale with
contraction (the tolerance of the other FP64 parity tests)."""
import numpy as np
import pytest

import cases as C
from cac_code_gb300 import lattice as L

pytestmark = pytest.mark.gpu

FP64_TOL = 1e-12


def _slab(pair, cells, nae, layers, intp, seed, jitter):
    lj = pair == "lj/cut"
    a = C.A_LJ if lj else C.A_CU
    mass = 1.0 if lj else L.AnalyticEAM().mass
    rng = np.random.default_rng(seed)
    m = L.make_slab_model(a, mass, cells, nae, layers, intp)
    m.atom_x = m.atom_x + rng.normal(0.0, jitter, m.atom_x.shape)
    m.nodex = m.nodex + rng.normal(0.0, jitter, m.nodex.shape)
    L.remap_into_box(m)
    return m


# (the list radius is the skin) rows of an element in full and partial groups of 8 and none beyond its own
# sites or into others; rows with more entries in reach than a row's buffer
CASES = {
    "lj_gauss": dict(pair="lj/cut", cells=(4, 16, 16), nae=8, layers=2, rows="gauss", rc=2.5, skin=2.8),
    "lj_all_sites": dict(pair="lj/cut", cells=(4, 10, 10), nae=5, layers=2, rows="all", rc=2.5, skin=2.8),
    "lj_long_rows": dict(pair="lj/cut", cells=(4, 16, 16), nae=8, layers=2, rows="gauss", rc=4.4, skin=5.3),
    "eam_gauss_nodes": dict(pair="eam", cells=(3, 22, 22), nae=11, layers=2, rows="nodes"),
    "eam_near_elements": dict(pair="eam", cells=(3, 12, 12), nae=6, layers=3, rows="nodes"),
}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("mode", ["exact", "fp64"])
def test_forces_match_the_oracle(cacg_lib, oracle_lib, name, mode):
    c = CASES[name]
    lj = c["pair"] == "lj/cut"
    ip = {"gauss": lambda: L.gauss_intp(c["nae"], False), "nodes": lambda: L.gauss_intp(c["nae"], True),
          "all": lambda: L.all_sites_intp(c["nae"])}[c["rows"]]()
    m = _slab(c["pair"], c["cells"], c["nae"], c["layers"], ip, 31, 0.02 if lj else 0.05)
    kw = dict(units="lj" if lj else "metal", pair=c["pair"], skin=c.get("skin", 7.5),
              every=1, delay=0, check=True, dt=0.005 if lj else 0.001)
    if lj:
        kw["lj"] = (1.0, 1.0, c["rc"])
    else:
        kw["eam_file"] = C.EAM_FILE
    o = oracle_lib.Oracle(m, **kw)
    o.setup()
    o.atom_list()
    fr = o.atom_forces()
    o.elem_lists()
    nr = o.elem_forces()
    s = cacg_lib.System(0)
    try:
        s.command(f"units {kw['units']}")
        s.command("boundary f p p")
        s.load_model(m)
        if lj:
            s.command(f"pair_style lj/cut {c['rc']!r}")
            s.command("pair_coeff 1 1 1.0 1.0")
        else:
            s.command("pair_style eam")
            s.command(f"pair_coeff 1 1 {C.EAM_FILE}")
        s.command(f"neighbor {kw['skin']!r} bin")
        s.command("fix 1 all nve")
        s.set_precision(cacg_lib.FP64_EXACT if mode == "exact" else cacg_lib.FP64)
        s.init()
        s.setup()
        s.neighbor_build()
        s.neighbor_ebuild()
        s.neighbor_nbuild()
        s.pair_compute()
        s.pair_ecompute()
        f, nf = s.atoms()["f"], s.elements()["nodef"]
    finally:
        s.close()
    for got, ref in ((f, fr), (nf, nr)):
        if mode == "exact":
            assert np.array_equal(got.view(np.int64), np.ascontiguousarray(ref).view(np.int64))
        else:
            assert np.abs(got - ref).max() <= FP64_TOL * np.abs(ref).max()


@pytest.mark.parametrize("nae,skin", [(8, 2.0 * C.A_LJ), (6, 1.5 ** 0.5 * 2.0 * C.A_LJ), (4, 2.8)])
def test_lists_on_a_perfect_lattice(cacg_lib, oracle_lib, nae, skin):
    """List radii at (and off) a shell of the undisplaced lattice: pairs whose
    FP32 distance cannot tell on which side of the radius they lie, own and
    other elements' sites among them, entry for entry."""
    m = _slab("lj/cut", (3, 2 * nae, 2 * nae), nae, 2, L.gauss_intp(nae, False), 5, 0.0)
    o = oracle_lib.Oracle(m, units="lj", pair="lj/cut", skin=skin, lj=(1.0, 1.0, 2.5), dt=0.005)
    o.setup()
    want = tuple(o.atom_list()) + tuple(o.elem_lists())
    s = cacg_lib.System(0)
    try:
        s.command("units lj")
        s.command("boundary f p p")
        s.load_model(m)
        s.command("pair_style lj/cut 2.5")
        s.command("pair_coeff 1 1 1.0 1.0")
        s.command(f"neighbor {skin!r} bin")
        s.init()
        s.setup()
        s.neighbor_build()
        s.neighbor_ebuild()
        s.neighbor_nbuild()
        got = tuple(s.atom_list()) + tuple(s.elem_lists())
    finally:
        s.close()
    for g, w in zip(got, want):
        assert np.array_equal(g, w)
