"""The surrogate's kernels on more than one device of a process.

The limit of dynamic shared memory belongs to a device.  A second one is stood in for by a
preloaded library that counts two devices, maps both to device 0 and refuses a launch of
more than 48 KB whose limit was not raised on its device, as the runtime does.
"""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
typedef struct { unsigned x, y, z; } dim3;
static int dev;
static struct { const void *f, *k; int limit[2]; } fn[512];
static int nfn;
static int find(const void *f) {
  for (int i = 0; i < nfn; i++)
    if (fn[i].f == f) return i;
  fn[nfn].f = f;
  return nfn++;
}
#define REAL(name) dlsym(dlopen("libcudart.so.13", RTLD_LAZY), name)
int cudaGetDeviceCount(int *n) { *n = 2; return 0; }
int cudaSetDevice(int d) { dev = d; return ((int (*)(int)) REAL("cudaSetDevice"))(0); }
int cudaGetDevice(int *d) { *d = dev; return 0; }
int cudaDeviceGetAttribute(int *v, int a, int d) {
  return ((int (*)(int *, int, int)) REAL("cudaDeviceGetAttribute"))(v, a, 0);
}
int cudaFuncSetAttribute(const void *f, int a, int v) {
  if (a == 8) fn[find(f)].limit[dev] = v;  /* MaxDynamicSharedMemorySize */
  return ((int (*)(const void *, int, int)) REAL("cudaFuncSetAttribute"))(f, a, v);
}
int __cudaGetKernel(void **k, const void *f) {
  int rc = ((int (*)(void **, const void *)) REAL("__cudaGetKernel"))(k, f);
  fn[find(f)].k = *k;
  return rc;
}
int __cudaLaunchKernel(void *k, dim3 g, dim3 b, void **args, size_t smem, void *s) {
  if (smem > 48 * 1024)
    for (int i = 0; i < nfn; i++)
      if (fn[i].k == k && fn[i].limit[dev] < (int) smem) return 1;  /* invalid value */
  return ((int (*)(void *, dim3, dim3, void **, size_t, void *)) REAL("__cudaLaunchKernel"))(
      k, g, b, args, smem, s);
}
"""

SCRIPT = r"""
import numpy as np
from cac_code_gb300 import cacg

rng = np.random.default_rng(1)
x = rng.normal(size=(256, 32)).astype(np.float32)
t = rng.normal(size=(256, 24)).astype(np.float32)

def once(device):
    m = cacg.Mlp(device, members=2, seed=2)
    m.fit_normalization(x, t)
    m.train(x, t, epochs=1, batch=128, lr=1e-3, seed=3)
    out = [m.params(0), m.params(1), *m.predict(x)]
    out.append(m.loss_grad(0, x, t)[1])
    m.close()
    return out

assert all(np.array_equal(p, q) for p, q in zip(once(0), once(1)))
print("same")
"""


def test_a_second_device_gets_its_own_limits(cacg_lib, tmp_path):
    """A net on the second device trains and predicts as the first one's."""
    src, so = tmp_path / "two.c", tmp_path / "two.so"
    src.write_text(SHIM)
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-w", str(src), "-o", str(so), "-ldl"], check=True)
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    p = subprocess.run([sys.executable, "-c", SCRIPT], cwd=root, capture_output=True, text=True,
                       timeout=120, env=dict(os.environ, LD_PRELOAD=str(so)))
    assert p.returncode == 0 and p.stdout.strip() == "same", p.stderr[-800:]
