"""`tune fused_variant` picks the arrangement of the mixed element passes at any number of
elements.  All give the same bits, so the kernels launched are taken down by a preloaded
library that sits before the runtime's launches."""
import os
import re
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
#include <stdio.h>
typedef struct { unsigned x, y, z; } dim3;
static struct { const void *f, *k; const char *name; } fn[1024];
static int nfn;
#define REAL(name) dlsym(dlopen("libcudart.so.13", RTLD_LAZY), name)
void __cudaRegisterFunction(void **h, const char *f, char *d, const char *name, int lim, void *t,
                            void *b, void *bd, void *gd, int *w) {
  if (nfn < 1024) fn[nfn].f = f, fn[nfn++].name = name;
  ((void (*)(void **, const char *, char *, const char *, int, void *, void *, void *, void *, int *))
       REAL("__cudaRegisterFunction"))(h, f, d, name, lim, t, b, bd, gd, w);
}
int __cudaGetKernel(void **k, const void *f) {
  int rc = ((int (*)(void **, const void *)) REAL("__cudaGetKernel"))(k, f);
  for (int i = 0; i < nfn; i++)
    if (fn[i].f == f) fn[i].k = *k;
  return rc;
}
int __cudaLaunchKernel(void *k, dim3 g, dim3 b, void **args, size_t smem, void *s) {
  for (int i = 0; i < nfn; i++)
    if (fn[i].k == k) fprintf(stderr, "launch %s\n", fn[i].name);
  return ((int (*)(void *, dim3, dim3, void **, size_t, void *)) REAL("__cudaLaunchKernel"))(
      k, g, b, args, smem, s);
}
"""

SCRIPT = r"""
import sys
import numpy as np
from cac_code_gb300 import cacg, workloads as W

m, cfg = W.c2_eam(cells=(4, 22, 22), layers=int(sys.argv[1]), seed=13)
s = cacg.System(0)
W.configure_system(s, m, cfg, W.write_eam(sys.argv[2], 2000))
s.set_precision(cacg.MIXED)
s.init()
s.run(0)
s.pair_ecompute()
out = []
for v in (0, 1, 2):
    s.command(f"tune fused_variant {v}")
    print("variant", v, file=sys.stderr, flush=True)
    s.pair_ecompute()
    print("done", file=sys.stderr, flush=True)
    out.append(s.elements()["nodef"].copy())
assert all(np.array_equal(o.view(np.int64), out[0].view(np.int64)) for o in out)
"""


@pytest.mark.parametrize("layers", [10, 100])
def test_each_variant_runs_and_gives_the_same_bits(cacg_lib, tmp_path, layers):
    """160 and 1,600 elements (1 and 11 a multiprocessor)."""
    src, so = tmp_path / "log.c", tmp_path / "log.so"
    src.write_text(SHIM)
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-w", str(src), "-o", str(so), "-ldl"], check=True)
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    p = subprocess.run([sys.executable, "-c", SCRIPT, str(layers), str(tmp_path / "Cu.eam")], cwd=root,
                       capture_output=True, text=True, timeout=120,
                       env=dict(os.environ, LD_PRELOAD=str(so)))
    assert p.returncode == 0, p.stderr[-800:]
    parts = re.findall(r"variant (\d)\n(.*?)done", p.stderr, re.S)
    assert [v for v, _ in parts] == ["0", "1", "2"]
    for v, log in parts:
        rho = re.findall(r"k_elem_rho_fusedILi(\d)", log)
        force = re.findall(r"k_elem_force_fusedILb1ELi(\d)", log)
        assert rho and force and set(rho + force) == {v}, (v, rho, force)
