"""What the captured solver steps depend on beside the buffers: a plan or chain
whose variant, strategy, precision or grid scale changed between two solves gives
the bits of one that had the setting from the start.  And values that are not
finite through the masked passes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N, n, nu = [32, 32, 32], [16, 16, 16], 4096
DK = np.array([0.7, 1.3, 0.9])


def _data(nCh, bins):
    import monalisa_b200 as mb

    rng = np.random.default_rng(10 * nCh + bins)
    mats, rows = [], []
    for b in range(bins):
        m = 3000 + 500 * b
        t = (rng.random((3, m)) - 0.5) * 28
        t[:, :400] = 0.3 * rng.random((3, 400))
        mats.append(mb.bmTraj2SparseMat(t, np.ones(m), N, [1, 1, 1]))
        rows.append(m)
    cplx = lambda *s: (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)
    return mats, sum(rows), cplx(nu, nCh), cplx(sum(rows), nCh)


def _set_dk(plan):
    from monalisa_b200 import _native

    _native.call("mlg_plan_set_dk", plan.handle, _native.dptr(DK.copy()))


def _attr(name, value):
    return lambda plan: setattr(plan, name, value)


CHANGES = {
    "dk": _set_dk,
    "variant": _attr("variant", {"pass_buffers": 0}),
    "register off": _attr("variant", {"register_passes": 0}),
    "records": _attr("variant", {"gut_records": 0}),
    "full grid": _attr("adjoint_mode", "full_grid"),
    "fused": _attr("adjoint_mode", "fused"),
    "mixed": _attr("precision", "mixed"),
    "fp16 values": _attr("precision", "fp16_values"),
}


@pytest.mark.parametrize("change", list(CHANGES))
@pytest.mark.parametrize("nCh", [3, 4])
def test_sensa_after_a_change(nCh, change):
    import torch

    import monalisa_b200 as mb

    mats, rows, C, y = _data(nCh, 1)
    yd, ve = torch.from_numpy(y).cuda(), torch.ones(rows, device="cuda")

    def solve(rec):
        x = torch.zeros(nu, dtype=torch.complex64, device="cuda")
        return torch.view_as_real(rec.run_dev(yd, ve, x, nIter=1, nCGD=4, ve_max=1.0)).cpu()

    used, fresh = mb.SensaRecon(*mats[0], C, n), mb.SensaRecon(*mats[0], C, n)
    first = solve(used)
    CHANGES[change](used.plan)
    CHANGES[change](fresh.plan)
    assert torch.equal(solve(used), solve(fresh))
    assert torch.equal(solve(used), solve(fresh))  # replayed
    assert torch.isfinite(first).all() and float(first.abs().max()) > 0


@pytest.mark.parametrize("change", ["variant", "register off", "records", "full grid", "fused", "fp16 values"])
@pytest.mark.parametrize("frame", [0, 1])
def test_chain_after_a_change(change, frame):
    import torch

    import monalisa_b200 as mb

    mats, rows, C, y = _data(4, 2)
    yd, ve = torch.from_numpy(y).cuda(), torch.ones(rows, device="cuda")

    def solve(chain):
        x, z, u = (torch.zeros((2, nu), dtype=torch.complex64, device="cuda") for _ in range(3))
        chain.run_dev(yd, ve, x, z, u, 0.01, 0.1, 2, 3, 1.0)
        return torch.view_as_real(x).cpu()

    make = lambda: mb.TevaMorphosiaChain([m[0] for m in mats], [m[1] for m in mats], C, n)
    used, fresh = make(), make()
    first = solve(used)
    for c in (used, fresh):
        CHANGES[change](c.plans[frame])
    assert torch.equal(solve(used), solve(fresh))
    assert torch.equal(solve(used), solve(fresh))
    assert torch.isfinite(first).all() and float(first.abs().max()) > 0


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("nCh", [3, 4])
def test_values_that_are_not_finite(nCh, bad):
    """One sample of one coil: its cells spread over every pixel of the adjoint, in
    every strategy; one pixel spreads over every sample of the forward.  The finite
    call after it is not touched by what the grid still holds."""
    import torch

    import monalisa_b200 as mb

    mats, rows, C, y = _data(nCh, 1)
    plan = mb.SensaRecon(*mats[0], C, n).plan
    good = torch.from_numpy(y).cuda()
    evil = good.clone()
    evil[1000, 1] = bad
    x = torch.ones(nu, dtype=torch.complex64, device="cuda")
    xe = x.clone()
    xe[77] = bad
    for mode in ("masked", "full_grid", "fused"):
        plan.adjoint_mode = mode
        want, fwd = plan.nakatsha(good), plan.shanna(x)
        assert torch.isfinite(torch.view_as_real(want)).all()
        out = plan.nakatsha(evil)
        assert not torch.isfinite(out.real + out.imag).any(), mode
        assert torch.equal(torch.view_as_real(plan.nakatsha(good)), torch.view_as_real(want)), mode
        y1 = plan.shanna(xe)
        assert not torch.isfinite(y1.real + y1.imag).any(), mode
        assert torch.equal(torch.view_as_real(plan.shanna(x)), torch.view_as_real(fwd)), mode
        assert torch.equal(torch.view_as_real(plan.nakatsha(good)), torch.view_as_real(want)), mode
