"""Adjoint strategies of odd coil counts: the strategy that is set is the one
that runs and that the plan reports, the masked one (the default) exists while
the register passes are on and the first pass's axis has one, and the autotuner
times each."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,n,masked", [([32, 40], [16, 20], True), ([24, 20, 32], [12, 10, 16], True),
                                        ([24, 32, 20], [12, 16, 10], False)])
def test_strategies_of_odd_counts(N, n, masked):
    import torch

    import monalisa_b200 as mb

    rng = np.random.default_rng(1)
    nu, dim = int(np.prod(n)), len(N)
    t = (rng.random((dim, 900)) - 0.5) * (np.array(N)[:, None] - 4)  # no row above 256 entries
    Gu, Gut = mb.bmTraj2SparseMat(t, np.ones(900), N, [1] * dim)
    C = (rng.standard_normal((nu, 3)) + 1j * rng.standard_normal((nu, 3))).astype(np.complex64)
    plan = mb.SensaRecon(Gu, Gut, C, n).plan
    y = torch.from_numpy((rng.standard_normal((900, 3)) + 1j * rng.standard_normal((900, 3))).astype(np.complex64)).cuda()

    def adjoint():
        before = mb.launch_count()
        x = plan.nakatsha(y, scale=2.0).cpu().numpy()
        return x, mb.launch_count() - before

    if not masked:  # an axis of 20 points
        assert plan.adjoint_mode == "fused" and adjoint()[1] == dim
        with pytest.raises(mb.MonalisaError):
            plan.adjoint_mode = "masked"
        assert set(plan.autotune(2, variants=False)) == {"full_grid", "fused"}
        plan.close()
        return
    assert plan.adjoint_mode == "masked"
    ref, launches = adjoint()
    assert launches == dim + 1  # the product of the non-empty rows, a pass per axis
    for mode, count in (("fused", dim), ("full_grid", dim + 1), ("masked", dim + 1)):
        plan.adjoint_mode = mode
        assert plan.adjoint_mode == mode
        x, launches = adjoint()
        assert launches == count, mode
        # FP32 transforms and rows of a few dozen entries in one order or another
        assert np.linalg.norm(x - ref) <= 2e-6 * np.linalg.norm(ref), mode
    times = plan.autotune(2, variants=False)
    assert set(times) == {"full_grid", "fused", "masked"} and plan.adjoint_mode in times
    plan.adjoint_mode = "masked"
    plan.variant = {"pass_buffers": 2}  # without register passes: as before they existed
    assert plan.adjoint_mode == "fused" and adjoint()[1] == dim
    with pytest.raises(mb.MonalisaError):
        plan.adjoint_mode = "masked"
    plan.precision = "fp16_values"
    assert plan.adjoint_mode == "full_grid" and adjoint()[1] == dim + 1
    plan.variant = {"register_passes": 1}
    assert plan.adjoint_mode == "masked"
    plan.close()
