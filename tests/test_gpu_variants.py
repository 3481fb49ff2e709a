"""mlg_plan_set_variant beside the register passes, as a C caller uses it: the
values that mlg_plan_get_variant gave change nothing, another pass_buffers turns the
register passes off and the earlier one brings them back, unless they were turned
off by name; the tuner reports their time with the others'."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_variant_values_restore_the_plan():
    import torch

    import monalisa_b200 as mb
    from monalisa_b200 import _native as N

    rng = np.random.default_rng(0)
    n, Ng, nCh = [16, 16, 16], [32, 32, 32], 4
    t = (rng.random((3, 2000)) - 0.5) * 28
    Gu, Gut = mb.bmTraj2SparseMat(t, np.ones(2000), Ng, [1, 1, 1])
    C = (rng.standard_normal((4096, nCh)) + 1j * rng.standard_normal((4096, nCh))).astype(np.complex64)
    plan = mb.SensaRecon(Gu, Gut, C, n).plan
    x = torch.from_numpy((rng.standard_normal(4096) + 1j * rng.standard_normal(4096)).astype(np.complex64)).cuda()

    def get():
        v = [ctypes.c_int() for _ in range(3)]
        N.call("mlg_plan_get_variant", plan.handle, *[ctypes.byref(c) for c in v])
        return [c.value for c in v]

    def register():
        v = ctypes.c_int()
        N.call("mlg_plan_get_register_passes", plan.handle, ctypes.byref(v))
        return v.value

    def put(v):
        N.call("mlg_plan_set_variant", plan.handle, *v)

    home = get()
    want = plan.shanna(x)
    assert register() == 1
    put(home)
    assert register() == 1 and get() == home
    put([home[0], 1 - home[1], home[2]])  # Gut's rows alone
    assert register() == 1
    put(home)
    put([0, home[1], home[2]])
    assert register() == 0 and get()[0] == 0
    put([3, home[1], home[2]])
    assert register() == 0
    put(home)
    assert register() == 1 and get() == home
    assert torch.equal(torch.view_as_real(plan.shanna(x)), torch.view_as_real(want))
    N.call("mlg_plan_set_register_passes", plan.handle, 0)
    put([0, home[1], home[2]])
    put(home)
    assert register() == 0  # turned off by name
    times = plan.autotune(2)
    assert times["passes_register"] > 0
    passes = [k for k in ("passes_register", "passes_tma_2buf", "passes_tma_3buf", "passes_cp_async") if k in times]
    assert len(passes) == 4
    assert register() == (1 if times["passes_register"] < min(
        [times[k] for k in passes[1:]] + [times.get("fwd_full_store", 1e9)]) else 0)
    plan.close()
