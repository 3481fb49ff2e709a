"""A line pass asks the runtime for a kernel's attributes and occupancy once per
host thread, not on every launch.  A shim in front of the CUDA runtime (compiled
here, preloaded into a child process) counts the calls over operators that have
run before: cubic and mixed axis lengths, whose passes alternate kernels."""
import os
import shutil
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
static int calls = 0;
int runtime_queries(void) { return calls; }
#define NEXT(name) dlsym(RTLD_NEXT, name)
int cudaFuncSetAttribute(const void* f, int a, int v) {
  ++calls;
  return ((int (*)(const void*, int, int))NEXT("cudaFuncSetAttribute"))(f, a, v);
}
int cudaDeviceGetAttribute(int* v, int a, int d) {
  ++calls;
  return ((int (*)(int*, int, int))NEXT("cudaDeviceGetAttribute"))(v, a, d);
}
int cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* f, int b, size_t m, unsigned g) {
  ++calls;
  return ((int (*)(int*, const void*, int, size_t, unsigned))NEXT(
      "cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags"))(n, f, b, m, g);
}
int cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void* f, int b, size_t m) {
  ++calls;
  return ((int (*)(int*, const void*, int, size_t))NEXT("cudaOccupancyMaxActiveBlocksPerMultiprocessor"))(n, f, b, m);
}
"""

CHILD = r"""
import ctypes, sys
import numpy as np, torch
sys.path.insert(0, sys.argv[1])
import monalisa_b200 as mb
shim = ctypes.CDLL(None)
for N, n, nCh in (([64, 64], [32, 32], 6), ([64, 64, 64], [32, 32, 32], 8), ([48, 40, 64], [24, 20, 32], 3)):
    rng = np.random.default_rng(nCh)
    t = (rng.random((len(N), 500)) - 0.5) * (np.array(N)[:, None] - 4)
    Gu, Gut = mb.bmTraj2SparseMat(t, np.ones(500), N, [1] * len(N))
    nu = int(np.prod(n))
    rec = mb.SensaRecon(Gu, Gut, np.ones((nu, nCh), np.complex64), n)
    x = torch.ones(nu, dtype=torch.complex64, device="cuda")
    y = torch.ones((500, nCh), dtype=torch.complex64, device="cuda")
    def pair():
        rec.plan.shanna(x)
        rec.plan.nakatsha(y)
    pair()
    before = shim.runtime_queries()
    assert before > 0
    for _ in range(5):
        pair()
    print("QUERIES", shim.runtime_queries() - before)
    torch.cuda.synchronize()
"""


def test_repeated_passes_query_nothing(tmp_path):
    cc = shutil.which("gcc")
    if cc is None:
        pytest.skip("no C compiler")
    src, so = tmp_path / "count.c", tmp_path / "count.so"
    src.write_text(SHIM)
    subprocess.run([cc, "-shared", "-fPIC", "-o", str(so), str(src), "-ldl"], check=True)
    env = dict(os.environ, LD_PRELOAD=str(so))
    r = subprocess.run([sys.executable, "-c", CHILD, ROOT], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert [v for v in r.stdout.splitlines() if v.startswith("QUERIES")] == ["QUERIES 0"] * 3, r.stdout
