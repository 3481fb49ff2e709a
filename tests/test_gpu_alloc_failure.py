"""A plan whose creation fails for want of device memory leaves the caller's
matrices usable: the next plan on them gives what a plan on untouched matrices
gives.  A shim in front of the CUDA runtime (compiled here, preloaded into a
child process) refuses the k-th device allocation made while a plan is created,
for every k until creation succeeds; the GPU's memory is not filled."""
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
static int left = -1;  /* allocations until the refused one; < 0: none refused */
void refuse_allocation(int k) { left = k; }
static int refuse(void) { return left >= 0 && left-- == 0; }
#define NEXT(name) dlsym(RTLD_NEXT, name)
int cudaMalloc(void** p, size_t n) {
  if (refuse()) return *p = NULL, 2; /* cudaErrorMemoryAllocation */
  return ((int (*)(void**, size_t))NEXT("cudaMalloc"))(p, n);
}
int cudaMallocAsync(void** p, size_t n, void* s) {
  if (refuse()) return *p = NULL, 2;
  return ((int (*)(void**, size_t, void*))NEXT("cudaMallocAsync"))(p, n, s);
}
"""

CHILD = r"""
import ctypes, sys
import numpy as np, torch
sys.path.insert(0, sys.argv[1])
import monalisa_b200 as mb
shim = ctypes.CDLL(None)
for nCh in (4, 3):
    rng = np.random.default_rng(nCh)
    # a cell of 1500 samples: rows of one heavy unit and of several
    t = np.concatenate([rng.uniform(-14, 14, (2, 900)), rng.uniform(-0.3, 0.3, (2, 1500)),
                        5.0 + rng.uniform(-0.2, 0.2, (2, 100))], 1)
    C = (rng.standard_normal((256, nCh)) + 1j * rng.standard_normal((256, nCh))).astype(np.complex64)
    y = torch.from_numpy((rng.standard_normal((2500, nCh)) + 1j).astype(np.complex64)).cuda()
    make = lambda: mb.bmTraj2SparseMat(t, np.ones(t.shape[1]), [32, 32], [1, 1])
    ref = mb.SensaRecon(*make(), C, [16, 16])
    want = ref.plan.nakatsha(y).cpu()
    assert float(want.abs().max()) > 0
    torch.cuda.synchronize()
    refused, k = 0, 0
    while True:
        mats = make()
        shim.refuse_allocation(k)
        try:
            rec, failed = mb.SensaRecon(*mats, C, [16, 16]), False
        except mb.MonalisaError:
            failed = True
        shim.refuse_allocation(-1)
        if failed:
            refused += 1
            rec = mb.SensaRecon(*mats, C, [16, 16])
        assert torch.equal(torch.view_as_real(rec.plan.nakatsha(y).cpu()), torch.view_as_real(want)), k
        rec.plan.close()
        if not failed:
            break
        k += 1
    print("REFUSED", nCh, refused)
"""


def test_matrices_survive_a_refused_allocation(tmp_path):
    cc = shutil.which("gcc")
    if cc is None:
        pytest.skip("no C compiler")
    src, so = tmp_path / "refuse.c", tmp_path / "refuse.so"
    src.write_text(SHIM)
    subprocess.run([cc, "-shared", "-fPIC", "-o", str(so), str(src), "-ldl"], check=True)
    env = dict(os.environ, LD_PRELOAD=str(so))
    r = subprocess.run([sys.executable, "-c", CHILD, ROOT], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    counts = [int(v.split()[2]) for v in r.stdout.splitlines() if v.startswith("REFUSED")]
    assert len(counts) == 2 and min(counts) >= 15, r.stdout  # the tables and buffers of a plan
