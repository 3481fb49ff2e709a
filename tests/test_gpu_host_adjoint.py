"""The host-array adjoint (bmNakatsha) makes a plan for one call: at odd coil
counts it builds none of the tables that only repeated adjoints earn back (fewer
launches than the even count beside it, whose products need them), and gives what
a kept plan gives.  Two orders of summation over rows of up to 600 entries and
FP32 transforms: 6e-8 * sqrt(600) + 2e-6 = 3.5e-6."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,n", [([40, 32], [20, 16]), ([32, 24, 16], [16, 12, 8])])
def test_one_call(N, n):
    import torch

    import monalisa_b200 as mb

    rng = np.random.default_rng(len(N))
    nu = int(np.prod(n))
    t = (rng.random((len(N), 2500)) - 0.5) * (np.array(N)[:, None] - 4)
    t[:, :600] = 1.5 + 0.2 * rng.random((len(N), 600))
    Gu, Gut = mb.bmTraj2SparseMat(t, np.ones(2500), N, [1] * len(N))
    host = Gut.download()
    launches = {}
    for nCh in (3, 4):
        C = (rng.standard_normal((nu, nCh)) + 1j * rng.standard_normal((nu, nCh))).astype(np.complex64)
        y = (rng.standard_normal((2500, nCh)) + 1j * rng.standard_normal((2500, nCh))).astype(np.complex64)
        plan = mb.NufftPlan(N, n, nCh, Gu, Gut, C, np.conj(C))
        want = plan.nakatsha(torch.from_numpy(y).cuda()).cpu().numpy()
        before = mb.launch_count()
        x = mb.bmNakatsha(y, host, np.conj(C), True, n).ravel()
        launches[nCh] = mb.launch_count() - before
        assert np.linalg.norm(x - want) <= 3.5e-6 * np.linalg.norm(want)
        plan.close()
    assert launches[3] < launches[4], launches
