"""Training batches whose arrays do not fit the device for all members at a time."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stdlib.h>
static struct { void *p; size_t n; } blk[4096];
static size_t total;
#define REAL(name) dlsym(dlopen("libcudart.so.13", RTLD_LAZY), name)
int cudaMalloc(void **p, size_t n) {
  if (total + n > strtoull(getenv("DEVICE_BYTES"), 0, 10)) return 2;  /* out of memory */
  int rc = ((int (*)(void **, size_t)) REAL("cudaMalloc"))(p, n);
  for (int i = 0; rc == 0 && i < 4096; i++)
    if (!blk[i].p) {
      blk[i].p = *p, blk[i].n = n, total += n;
      break;
    }
  return rc;
}
int cudaFree(void *p) {
  for (int i = 0; p && i < 4096; i++)
    if (blk[i].p == p) blk[i].p = 0, total -= blk[i].n;
  return ((int (*)(void *)) REAL("cudaFree"))(p);
}
"""

SCRIPT = r"""
import hashlib
import numpy as np
from cac_code_gb300 import cacg

rng = np.random.default_rng(1)
x = rng.normal(size=(40000, 32)).astype(np.float32)
t = rng.normal(size=(40000, 24)).astype(np.float32)
m = cacg.Mlp(0, members=3, seed=2)
m.fit_normalization(x, t)
loss = m.train(x, t, epochs=2, batch=16384, lr=1e-3, seed=3)
h = hashlib.sha256(np.concatenate([m.params(k) for k in range(3)] + list(m.predict(x[:500]))[:1],
                                  axis=None).tobytes())
m.close()
print(loss, h.hexdigest())
"""


def test_fewer_members_at_a_time_give_the_same_bits(cacg_lib, tmp_path):
    """Batches of 16,384 rows: 160 to 240 MB of arrays a member.  A preloaded library plays a
    device of 350 MB, which has room for one member's, or for two at most."""
    src, so = tmp_path / "mem.c", tmp_path / "mem.so"
    src.write_text(SHIM)
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-w", str(src), "-o", str(so), "-ldl"], check=True)
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    out = []
    for mb in (100000, 350):
        p = subprocess.run([sys.executable, "-c", SCRIPT], cwd=root, capture_output=True, text=True,
                           timeout=120, env=dict(os.environ, LD_PRELOAD=str(so),
                                                 DEVICE_BYTES=str(mb << 20)))
        assert p.returncode == 0, p.stderr[-800:]
        out.append(p.stdout)
    assert out[0] == out[1]
