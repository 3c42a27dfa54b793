"""A surrogate call that fails leaves no copy from the caller's memory in flight."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
static int copies, full;
int in_flight(void) { return copies; }
void no_memory(int on) { full = on; }
#define REAL(name) dlsym(dlopen("libcudart.so.13", RTLD_LAZY), name)
int cudaMalloc(void **p, size_t n) {
  /* after the data set has been copied in, none is left for the step's arrays */
  if (full && copies) return 2;
  return ((int (*)(void **, size_t)) REAL("cudaMalloc"))(p, n);
}
int cudaMemcpyAsync(void *d, const void *s, size_t n, int kind, void *st) {
  copies++;
  return ((int (*)(void *, const void *, size_t, int, void *)) REAL("cudaMemcpyAsync"))(d, s, n, kind, st);
}
int cudaStreamSynchronize(void *st) {
  copies = 0;
  return ((int (*)(void *)) REAL("cudaStreamSynchronize"))(st);
}
"""

SCRIPT = r"""
import ctypes, sys
import numpy as np
from cac_code_gb300 import cacg

shim = ctypes.CDLL(sys.argv[1])
rng = np.random.default_rng(1)
x = rng.normal(size=(512, 32)).astype(np.float32)
t = rng.normal(size=(512, 24)).astype(np.float32)
m = cacg.Mlp(0, members=1, seed=2)
m.set_normalization(np.zeros(32), np.ones(32), np.zeros(24), np.ones(24), 1.0)
for call in (lambda: m.train(x, t, epochs=1, batch=512), lambda: m.loss_grad(0, x, t),
             lambda: m.predict(x)):
    shim.no_memory(1)
    try:
        call()
        print("ran")
    except cacg.CacgError:
        print("error", shim.in_flight())
    shim.no_memory(0)
    call()
print("done")
"""


def test_an_error_waits_for_the_copies(cacg_lib, tmp_path):
    """Device memory runs out behind the copies of the data set; afterwards the call runs."""
    src, so = tmp_path / "copies.c", tmp_path / "copies.so"
    src.write_text(SHIM)
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-w", str(src), "-o", str(so), "-ldl"], check=True)
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    p = subprocess.run([sys.executable, "-c", SCRIPT, str(so)], cwd=root, capture_output=True, text=True,
                       timeout=120, env=dict(os.environ, LD_PRELOAD=str(so)))
    assert p.returncode == 0, p.stderr[-800:]
    lines = p.stdout.split("\n")
    assert lines[0] == "error 0" and "done" in lines, lines
    assert all(s in ("error 0", "ran", "done", "") for s in lines), lines
