"""FP64 EAM forces on a device without room for the pairs' distances."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
#include <stdlib.h>
#define REAL(name) dlsym(dlopen("libcudart.so.13", RTLD_LAZY), name)
int cudaMalloc(void **p, size_t n) {
  if (n >= strtoull(getenv("LARGEST_BLOCK"), 0, 10)) return 2;  /* out of memory */
  return ((int (*)(void **, size_t)) REAL("cudaMalloc"))(p, n);
}
"""

SCRIPT = r"""
import hashlib, sys
import numpy as np
from cac_code_gb300 import cacg, workloads as W

m, cfg = W.c2_sample()
for mode in (cacg.FP64_EXACT, cacg.FP64):
    s = cacg.System(0)
    W.configure_system(s, m, cfg, W.write_eam(sys.argv[1]))
    s.set_precision(mode)
    s.init()
    s.run(12)
    a, e = s.atoms(), s.elements()
    h = hashlib.sha256()
    for q in (a["x"], a["v"], a["f"], e["nodex"], e["nodef"]):
        h.update(np.ascontiguousarray(q).tobytes())
    print(h.hexdigest(), s.counts()["graph_steps"] > 0)
    s.close()
"""


def test_distances_formed_again_give_the_same_bits(cacg_lib, tmp_path):
    """9,680 atoms: lists of at most 9 MB, distances of 12 to 37 MB, which a preloaded library
    refuses.  Twelve steps with a rebuild decision and captured steps, both FP64 modes."""
    src, so = tmp_path / "one.c", tmp_path / "one.so"
    src.write_text(SHIM)
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-w", str(src), "-o", str(so), "-ldl"], check=True)
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    out = []
    for mb in (100000, 11):
        p = subprocess.run([sys.executable, "-c", SCRIPT, str(tmp_path / "Cu.eam")], cwd=root,
                           capture_output=True, text=True, timeout=120,
                           env=dict(os.environ, LD_PRELOAD=str(so), LARGEST_BLOCK=str(mb << 20)))
        assert p.returncode == 0, p.stderr[-800:]
        out.append(p.stdout.split())
    assert out[0] == out[1] and out[0][1] == out[0][3] == "True", out
