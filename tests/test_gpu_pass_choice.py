"""Plans at their defaults on grids where some of the passes run on the
shared-memory kernels and the others on the register ones (96- to 192-point axes
of many lines, 8 to 32 coils), against the shared-memory kernels alone and against
a plan of the same problem split into single coils, which runs the register
passes throughout.

Tolerance: FP32 transforms of 3 axes x at most 8 radix-2 stages on both sides:
3e-7 each by sqrt(24) * 6e-8, 2e-6 with a factor 3; the coils' sum in another
order adds less."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 2e-6


def rel(a, b):
    a, b = np.ravel(a).astype(np.complex128), np.ravel(b).astype(np.complex128)
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("N,n,nCh", [
    ([96, 96, 96], [60, 60, 60], 32),     # x, y and z, forward and back
    ([96, 96, 96], [48, 48, 48], 32),     # exact halves: the inverse masked pass stays
    ([128, 96, 64], [80, 60, 40], 16),    # x back by the pipelined kernel; z too short
    ([96, 128, 96], [58, 80, 60], 24),    # x and y at 24 coils
    ([96, 192, 96], [48, 96, 48], 12),    # y of 192 points, 24-column bundles
])
def test_default_plan(N, n, nCh):
    import torch

    import monalisa_b200 as mb

    rng = np.random.default_rng(nCh)
    nu, nPt = int(np.prod(n)), 3000
    t = (rng.random((3, nPt)) - 0.5) * (np.array(N)[:, None] - 4)
    Gu, Gut = mb.bmTraj2SparseMat(t, np.ones(nPt), N, [1, 1, 1])
    C = (rng.standard_normal((nu, nCh)) + 1j * rng.standard_normal((nu, nCh))).astype(np.complex64)
    cplx = lambda *s: torch.from_numpy(
        (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)).cuda()
    x, y = cplx(nu), cplx(nPt, nCh)
    rec = mb.SensaRecon(Gu, Gut, C, n)
    assert rec.plan.variant["register_passes"] == 1
    f, a = rec.plan.shanna(x).cpu().numpy(), rec.plan.nakatsha(y, scale=2.0).cpu().numpy()
    again = rec.plan.nakatsha(y, scale=2.0).cpu().numpy()
    assert np.array_equal(a, again)
    rec.plan.variant = {"pass_buffers": 2}
    assert rel(f, rec.plan.shanna(x).cpu().numpy()) <= TOL
    assert rel(a, rec.plan.nakatsha(y, scale=2.0).cpu().numpy()) <= TOL
    rec.plan.close()
    total = 0
    for c in range(nCh):
        one = mb.SensaRecon(Gu, Gut, C[:, c:c + 1], n)
        if c in (0, nCh - 1):
            assert rel(f[:, c], one.plan.shanna(x).cpu().numpy()) <= TOL
        total = total + one.plan.nakatsha(y[:, c:c + 1].contiguous(), scale=2.0).cpu().numpy().astype(np.complex128)
        one.plan.close()
    assert rel(a, total) <= TOL
