"""The register line-FFT passes (the default) against the shared-memory passes
(variant pass_buffers = 2: TMA / cp.async / direct-DFT kernels), which the
oracle pins: every axis length that has register passes in 2-D (both column
widths of the y pass: few and many columns), anisotropic 3-D grids, even, odd
and large coil counts, oversampling 2 (the kernels specialised for it) and
others, every adjoint strategy and per-coil images.  (The FP16 intermediates of
mixed precision run through them by default in test_gpu_mixed.py.)

Tolerance: both sides are FP32 transforms of at most 3 axes x 10 radix-2
stages; rounding grows like sqrt(30) * 6e-8 = 3.3e-7 per side, 2e-6 bounds
their difference with a factor 3."""
import os
import re

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LENGTHS = sorted(int(m) for m in re.findall(r"X\((\d+), \d+, \d+, \w+\)", open(
    os.path.join(ROOT, "monalisa_b200", "csrc", "mlg_fft_reg_lengths.h")).read()))
TOL = 2e-6


def rel(a, b):
    a, b = np.ravel(a).astype(np.complex128), np.ravel(b).astype(np.complex128)
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def _recon(N, n, nCh, seed, nPt=3000, precision="fp32"):
    import monalisa_b200 as mb

    rng = np.random.default_rng(seed)
    t = (rng.random((len(N), nPt)) - 0.5) * (np.array(N)[:, None] - 4)
    Gu, Gut = mb.bmTraj2SparseMat(t, np.ones(nPt), N, [1] * len(N))
    C = (rng.standard_normal((int(np.prod(n)), nCh)) + 1j * rng.standard_normal((int(np.prod(n)), nCh)))
    return mb.SensaRecon(Gu, Gut, C.astype(np.complex64), n, precision=precision), rng


def _cplx(rng, *shape):
    import torch

    return torch.from_numpy((rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)).cuda()


def _both(plan, rng, modes):
    """Forward and adjoints by the register passes and by the others."""
    nu = int(np.prod(plan.n_u))
    x, xc, y = _cplx(rng, nu), _cplx(rng, nu, plan.nCh), _cplx(rng, plan.nPt, plan.nCh)
    out = []
    for v in ({"register_passes": 1}, {"pass_buffers": 2}):
        plan.variant = v
        assert plan.variant["register_passes"] == (1 if "register_passes" in v else 0)
        o = [plan.shanna(x), plan.shanna(xc, per_coil=True)]
        for m in modes:
            plan.adjoint_mode = m
            o.append(plan.nakatsha(y, scale=2.0))
        out.append([v.cpu().numpy() for v in o])
    plan.status()
    for a, b in zip(*out):
        assert np.isfinite(a).all()
        assert rel(a, b) <= TOL, rel(a, b)


@pytest.mark.parametrize("N", LENGTHS)
def test_every_length_2d(N):
    over = 2.0 if (N // 4) % 2 == 0 else 1.6
    n = int(N / over) // 2 * 2
    for nCh in (1, 2) if N > 600 else (1, 6):
        rec, rng = _recon([N, N], [n, n], nCh, N + nCh)
        _both(rec.plan, rng, ["full_grid"] + (["masked"] if nCh % 2 == 0 else []))
        rec.plan.close()


@pytest.mark.parametrize("N,n,nCh", [
    ([64, 64, 64], [32, 32, 32], 16),    # 32-column bundles, specialised for oversampling 2
    ([96, 80, 64], [60, 50, 40], 12),    # three lengths, oversampling 1.6, two lines share a bundle
    ([64, 96, 112], [32, 48, 56], 5),    # odd coils: a cell's coils straddle bundles
    ([48, 60, 72], [24, 30, 36], 20),    # lengths without specialised kernels
    ([40, 40, 160], [20, 20, 80], 34),   # more coils than one warp, x passes with the large CTA
    ([128, 20, 24], [64, 12, 12], 3),    # a length without register passes between others
    ([256, 32, 32], [128, 16, 16], 8),
])
def test_3d(N, n, nCh):
    rec, rng = _recon(N, n, nCh, 7 * nCh)
    modes = ["full_grid", "fused"] + (["masked"] if nCh % 2 == 0 else [])
    _both(rec.plan, rng, modes)
    rec.plan.close()


def test_solver_partial_sums():
    """CG-SENSE takes its norms from the inverse x pass's partial sums."""
    rec, rng = _recon([64, 64, 48], [32, 32, 24], 6, 3)
    y = _cplx(rng, rec.nPt, 6).cpu().numpy() * 30
    out = []
    for v in ({"register_passes": 1}, {"pass_buffers": 2}):
        rec.plan.variant = v
        out.append(rec.run_host(y, np.ones(rec.nPt), nIter=1, nCGD=6, ve_max=1.0))
    assert rel(out[0], out[1]) <= 1e-5  # six steps of a few 1e-6 each at most
    rec.plan.close()


@pytest.mark.parametrize("nCh", [1, 2, 3, 12, 16, 33])
def test_gut_rows_of_every_length(nCh):
    """The adjoint product over rows of 1 to several thousand entries: inline
    records, loops with every remainder, rows of one heavy unit, rows of several
    (the last unit to finish adds them; twice, so that the counters are seen
    reset), against the product of every row (variant full_grid, no records).
    Rows of n entries summed in another order: 6e-8 sqrt(n), n <= 4096 -> 4e-6."""
    import torch

    import monalisa_b200 as mb

    rng = np.random.default_rng(nCh)
    N = 32
    # clusters of samples at one grid point: their 9 cells get rows of that many entries
    sizes = list(range(1, 14)) + [16, 17, 63, 64, 65, 66, 255, 256, 257, 300, 513, 1500, 4000]
    t = np.concatenate([np.repeat(np.array([[(3 * (i % 10)) - 14.0], [(3 * (i // 10)) - 14.0]]), n, 1)
                        for i, n in enumerate(sizes)], 1) + rng.uniform(-0.2, 0.2, (2, sum(sizes)))
    Gu, Gut = mb.bmTraj2SparseMat(t, np.ones(t.shape[1]), [N, N], [1, 1])
    C = (rng.standard_normal((256, nCh)) + 1j * rng.standard_normal((256, nCh))).astype(np.complex64)
    rec = mb.SensaRecon(Gu, Gut, C, [16, 16])
    y = _cplx(rng, rec.nPt, nCh)
    HY = torch.from_numpy(rng.random(rec.nPt).astype(np.float32)).cuda()
    first = rec.plan.nakatsha(y, HY=HY, scale=3.0).cpu().numpy()
    again = rec.plan.nakatsha(y, HY=HY, scale=3.0).cpu().numpy()
    assert np.array_equal(first, again)
    rec.plan.variant = {"pass_buffers": 0}
    rec.plan.adjoint_mode = "full_grid"
    ref = rec.plan.nakatsha(y, HY=HY, scale=3.0).cpu().numpy()
    assert rel(first, ref) <= 4e-6, rel(first, ref)
    rec.plan.close()


@pytest.mark.parametrize("nCh", [1, 4])
@pytest.mark.parametrize("nPt", [1, 300])
def test_products_without_rows(nCh, nPt):
    """All samples far outside the grid: Gu's rows and Gut's list of non-empty
    rows are empty, both operators give zeros."""
    import torch

    import monalisa_b200 as mb

    Gu, Gut = mb.bmTraj2SparseMat(np.full((2, nPt), 500.0), np.ones(nPt), [32, 32], [1, 1])
    rng = np.random.default_rng(0)
    C = (rng.standard_normal((256, nCh)) + 1j * rng.standard_normal((256, nCh))).astype(np.complex64)
    rec = mb.SensaRecon(Gu, Gut, C, [16, 16])
    y = torch.ones((rec.nPt, nCh), dtype=torch.complex64, device="cuda")
    for mode in ("full_grid", "masked"):
        try:
            rec.plan.adjoint_mode = mode
        except (mb.MonalisaError, ValueError):  # not offered for this coil count
            continue
        assert float(rec.plan.nakatsha(y).abs().max()) == 0
    x = torch.ones(256, dtype=torch.complex64, device="cuda")
    assert rec.plan.shanna(x).shape == (rec.nPt, nCh) and float(rec.plan.shanna(x).abs().max()) == 0
    rec.plan.close()
