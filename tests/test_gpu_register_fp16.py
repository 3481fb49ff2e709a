"""The register line passes on FP16 intermediates (mixed precision), on grids
that reach their two-column kernels (32-column bundles, with and without exact
twofold oversampling) and the one-column ones, and FP16 matrix values at odd coil
counts.

A mixed solve of two CG steps rounds five arrays to FP16 (B and the grid in two
forward operators, B in one adjoint), each value by at most 2^-11 of itself.
The second step's direction is formed from a residual that the first reduced
by a factor of about two while its rounding is that of the first step's vectors:
5 * 2^-11 * 2 = 4.9e-3 bounds the image's distance from the FP32 solve, and
twice that two FP16 solves' distance from each other."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 5 * 2.0 ** -11 * 2


def rel(a, b):
    a, b = np.ravel(a).astype(np.complex128), np.ravel(b).astype(np.complex128)
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def _recon(N, n, nCh, nPt, precision):
    import monalisa_b200 as mb

    rng = np.random.default_rng(nCh)
    t = (rng.random((len(N), nPt)) - 0.5) * (np.array(N)[:, None] - 4)
    nu = int(np.prod(n))
    C = (rng.standard_normal((nu, nCh)) + 1j * rng.standard_normal((nu, nCh))).astype(np.complex64)
    Gu, Gut = mb.bmTraj2SparseMat(t, np.ones(nPt), N, [1] * len(N))
    x = (rng.standard_normal(nu) + 1j * rng.standard_normal(nu)).astype(np.complex64)
    return mb.SensaRecon(Gu, Gut, C, n, precision=precision), x


@pytest.mark.parametrize("N,n,nCh", [
    ([64, 64, 64], [32, 32, 32], 16),     # two columns per thread, exact halves
    ([64, 64, 64], [40, 40, 40], 16),     # two columns per thread, other ranges
    ([96, 96, 64], [60, 60, 40], 12),     # two lines in a bundle
    ([32, 32, 32], [16, 16, 16], 4),      # one column per thread, four-column bundles
])
def test_mixed_solve(N, n, nCh):
    import torch

    out = {}
    for precision in ("fp32", "mixed"):
        rec, x = _recon(N, n, nCh, 8 * int(np.prod(n)) // nCh, precision)
        if precision == "fp32":
            y = rec.plan.shanna(torch.from_numpy(x).cuda()).cpu().numpy()
        for reg in (1, 0):
            rec.plan.variant = {"pass_buffers": 2, "register_passes": reg}
            assert rec.plan.half_intermediate == rec.plan.half_grid == (precision == "mixed")
            out[precision, reg] = rec.run_host(y, np.ones(rec.nPt), nIter=1, nCGD=2, ve_max=1.0)
        rec.plan.close()
    assert rel(out["fp32", 1], out["fp32", 0]) <= 1e-5
    e = rel(out["mixed", 1], out["fp32", 1])
    assert 1e-6 < e <= TOL, e  # FP16 ran
    assert rel(out["mixed", 1], out["mixed", 0]) <= 2 * TOL


@pytest.mark.parametrize("nCh", [1, 3, 5])
def test_fp16_values_of_odd_coil_counts(nCh):
    """The operators of nCh coils and those of nCh + 1, the last one's map zero:
    the same FP16 values and entry order, FP32 sums and transforms."""
    import torch

    import monalisa_b200 as mb

    N, n, nu = [48, 40], [24, 20], 480
    rng = np.random.default_rng(nCh)
    t = (rng.random((2, 4000)) - 0.5) * (np.array(N)[:, None] - 4)
    t[:, :300] = 3.2 + 0.1 * rng.random((2, 300))  # rows above 64 and above 256 entries
    Gu, Gut = mb.bmTraj2SparseMat(t, np.ones(4000), N, [1, 1])
    C = (rng.standard_normal((nu, nCh)) + 1j * rng.standard_normal((nu, nCh))).astype(np.complex64)
    x = (rng.standard_normal(nu) + 1j * rng.standard_normal(nu)).astype(np.complex64)
    C1 = np.concatenate([C, np.zeros_like(C[:, :1])], 1)
    plans = [mb.SensaRecon(Gu, Gut, c, n, precision=p).plan
             for c, p in ((C, "fp16_values"), (C1, "fp16_values"), (C, "fp32"))]
    xd = torch.from_numpy(x).cuda()
    torch.manual_seed(nCh)
    y = torch.randn((4000, nCh + 1), dtype=torch.complex64, device="cuda")
    yo = y[:, :nCh].contiguous()
    f = [p.shanna(xd).cpu().numpy() for p in plans]
    a = [p.nakatsha(v, scale=2.0).cpu().numpy() for p, v in zip(plans, (yo, y, yo))]
    assert rel(f[0], f[1][:, :nCh]) <= 2e-6 and rel(a[0], a[1]) <= 4e-6
    # FP16 values ran: rounded by up to 2^-11 each
    assert 1e-6 < rel(f[0], f[2]) <= 2.0 ** -11 * 2 and 1e-6 < rel(a[0], a[2]) <= 2.0 ** -11 * 2
