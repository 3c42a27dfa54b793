"""FP64 products and sums by the integer units (soft_fp64.cuh) against the host's
FP64, and the passes that use them against the oracle, bit for bit."""
import os
import subprocess

import numpy as np
import pytest

import cac_code_gb300
import cases as C
from cac_code_gb300 import lattice as L

HARNESS = r"""
#include "soft_fp64.cuh"
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
using namespace cacg::soft;
static double of(uint64_t u) { double d; memcpy(&d, &u, 8); return d; }
static uint64_t to(double d) { uint64_t u; memcpy(&u, &d, 8); return u; }
static Op op(double d) { return op_of((uint32_t) (to(d) >> 32), (uint32_t) to(d)); }
int main(int argc, char **argv) {
  const int mode = atoi(argv[1]);
  std::mt19937_64 g(mode + 1);
  auto draw = [&](int m) {
    uint64_t r = g(), f = r & 0xFFFFFFFFFFFFFull, e = 1023, s = r >> 63;
    if (m == 0) e = 1020 + g() % 7;                         // ordinary
    if (m == 1) e = 1023 - DOT_RANGE + g() % (2 * DOT_RANGE + 1);  // the whole range
    if (m == 2) e = 963 + g() % 121, f &= ~0ull << (g() % 53);    // short: exact, ties
    if (m == 3) { if (g() % 3 == 0) return 0.0; e = 1023 + g() % 5; f &= 0xFFF0000000000ull; }
    if (m == 4) e = 1023 + g() % 3, f = g() % 2 ? 0xFFFFFFFFFFFFFull - g() % 3 : g() % 3;
    return of(s << 63 | e << 52 | f);
  };
  long bad = 0;
  for (long it = 0; it < 400000; it++) {
    double w[8], x[8];
    for (int k = 0; k < 8; k++) w[k] = draw(mode), x[k] = draw((mode + it) % 5);
    if (it % 4 == 0)  // cancellation, to the last bit or altogether
      for (int k = 1; k < 8; k += 2) w[k] = w[k - 1], x[k] = -x[k - 1] * (1 + it % 3 * 0x1p-53);
    volatile double a = w[0] * x[0];
    Acc s = mul(op(w[0]), op(x[0]));
    for (int k = 1; k < 8; k++) {
      volatile double p = w[k] * x[k];
      a = a + p;
      s = add(s, mul(op(w[k]), op(x[k])));
      bad += of(bits(s)) != a;
    }
    const double q = it % 7 ? std::ldexp((double) (g() >> (11 + g() % 50)), -53) : 1.0;
    volatile double h = w[0] * q;  // Horner steps
    Acc t = mul(op(w[0]), op(q));
    for (int k = 1; k < 4; k++) {
      h = h + w[k];
      t = add(t, acc_of(op(w[k])));
      bad += of(bits(t)) != h;
      if (k < 3) h = h * q, t = mul(op_of(t), op(q));
    }
  }
  printf("%ld\n", bad);
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    d = tmp_path_factory.mktemp("soft")
    (d / "h.cpp").write_text(HARNESS)
    inc = os.path.join(os.path.dirname(cac_code_gb300.__file__), "csrc")
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-I", inc, "-o", str(d / "h"), str(d / "h.cpp")],
                   check=True)
    return str(d / "h")


@pytest.mark.parametrize("mode", range(5))
def test_soft_sums_are_the_hosts(harness, mode):
    assert subprocess.run([harness, str(mode)], capture_output=True, check=True).stdout.strip() == b"0"


@pytest.mark.gpu
@pytest.mark.parametrize("layers,tiny", [(4, False), (8, False), (20, False), (20, True)])
def test_exact_forces(cacg_lib, oracle_lib, layers, tiny):
    """64 elements and at most 1,216 atoms (a cluster of blocks each), 128 (a block of 256
    threads) and 320 (positions from the integer units); with ``tiny`` some nodes have
    coordinates outside their range, and those elements' positions come from the FP64
    unit."""
    rng = np.random.default_rng(8)
    m = L.make_slab_model(C.A_CU, L.AnalyticEAM().mass, (2, 22, 22), 11, layers,
                          L.gauss_intp(11, True))
    if layers == 4:  # a few atoms of the slab
        m.atom_x, m.atom_v = m.atom_x[:1200], m.atom_v[:1200]
    m.atom_x = m.atom_x + rng.normal(0.0, 0.05, m.atom_x.shape)
    m.nodex = m.nodex + rng.normal(0.0, 0.05, m.nodex.shape)
    L.remap_into_box(m)
    if tiny:
        x = m.nodex.reshape(-1, 3)
        near = np.flatnonzero(np.abs(x[:, 1]) < 0.2)
        assert len(near) > 3
        x[near[::3], 1] = 1e-300
        x[near[1::3], 1] = 0.0
        m.nodex = x.reshape(m.nodex.shape)
    kw = dict(units="metal", pair="eam", skin=7.5, every=1, delay=0, check=True, dt=0.001,
              eam_file=C.EAM_FILE)
    o = oracle_lib.Oracle(m, **kw)
    o.setup()
    o.atom_list()
    fr = o.atom_forces()
    o.elem_lists()
    nr = o.elem_forces()
    s = cacg_lib.System(0)
    try:
        s.command("units metal")
        s.command("boundary f p p")
        s.load_model(m)
        s.command("pair_style eam")
        s.command(f"pair_coeff 1 1 {C.EAM_FILE}")
        s.command("neighbor 7.5 bin")
        s.command("fix 1 all nve")
        s.set_precision(cacg_lib.FP64_EXACT)
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
    assert m.nelements == 16 * layers
    for got, ref in ((f, fr), (nf, nr)):
        assert np.array_equal(got.view(np.int64), np.ascontiguousarray(ref).view(np.int64))
