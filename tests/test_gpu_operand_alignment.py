"""Device operands at an odd offset into a larger buffer (8-byte aligned): the
products and operators give the bits that aligned operands give, for even coil
counts (whose kernels move coil pairs, 16 bytes at a time) and odd ones, and
write nothing beside a result."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _shifted(v):
    """A copy of v one complex value into a buffer of its own."""
    import torch

    buf = torch.full((v.numel() + 2,), 7.0, dtype=v.dtype, device=v.device)
    out = buf[1:1 + v.numel()].view(v.shape)
    out.copy_(v)
    assert out.data_ptr() % 16 == 8
    return out, buf


def _same(got, buf, want):
    import torch

    assert torch.equal(torch.view_as_real(got), torch.view_as_real(want))
    assert buf[0] == 7 and buf[-1] == 7


# register passes, and a length of the direct-DFT passes
@pytest.mark.parametrize("N,n", [([32, 32], [16, 16]), ([22, 24], [12, 12]), ([24, 20, 16], [12, 10, 8])])
@pytest.mark.parametrize("nCh", [2, 3, 6])
def test_operands_at_odd_offsets(N, n, nCh):
    import torch

    import monalisa_b200 as mb

    rng = np.random.default_rng(nCh)
    dim, nu = len(N), int(np.prod(n))
    t = (rng.random((dim, 700)) - 0.5) * (np.array(N)[:, None] - 4)
    Gu, Gut = mb.bmTraj2SparseMat(t, np.ones(700), N, [1] * dim)
    C = (rng.standard_normal((nu, nCh)) + 1j * rng.standard_normal((nu, nCh))).astype(np.complex64)
    rec = mb.SensaRecon(Gu, Gut, C, n)
    plan = rec.plan
    cplx = lambda *s: torch.randn(*s, dtype=torch.complex64, device="cuda")
    x, xc, y, v = cplx(nu), cplx(nu, nCh), cplx(plan.nPt, nCh), cplx(int(np.prod(N)), nCh)
    for a, per_coil in ((x, False), (xc, True)):
        want = plan.shanna(a, per_coil=per_coil)
        out, buf = _shifted(torch.zeros_like(want))
        plan.shanna(_shifted(a)[0], out=out, per_coil=per_coil)
        _same(out, buf, want)
    modes = ["full_grid", "fused"] + (["masked"] if nCh % 2 == 0 else [])
    for mode in modes:
        plan.adjoint_mode = mode
        want = plan.nakatsha(y, scale=2.0)
        out, buf = _shifted(torch.zeros_like(want))
        plan.nakatsha(_shifted(y)[0], scale=2.0, out=out)
        _same(out, buf, want)
    want = Gu.spmm(v)
    out, buf = _shifted(torch.zeros_like(want))
    Gu.spmm(_shifted(v)[0], out=out)
    _same(out, buf, want)
    rec.plan.close()
