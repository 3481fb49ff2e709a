"""CG-SENSE's captured step: its scalars summed in the updates (few partial sums)
or in kernels of their own (over 1024), and the solution's address, which the step
reads from device memory."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(N, n, nCh, spokes, seed):
    import monalisa_b200 as mb

    rng = np.random.default_rng(seed)
    dim = len(N)
    e = rng.standard_normal((dim, spokes))
    e /= np.linalg.norm(e, axis=0)
    r = (np.arange(N[0]) - N[0] // 2) * 0.97
    t = (e[:, :, None] * r[None, None, :]).reshape(dim, -1)
    ve = (np.abs(np.tile(r, spokes)) + 0.3).astype(np.float64) / N[0]
    nu = int(np.prod(n))
    C = (rng.standard_normal((nu, nCh)) + 1j * rng.standard_normal((nu, nCh))).astype(np.complex64)
    Gu, Gut = mb.bmTraj2SparseMat(t, ve, N, [1] * dim)
    y = (rng.standard_normal((t.shape[1], nCh)) + 1j * rng.standard_normal((t.shape[1], nCh))).astype(np.complex64)
    return mb.SensaRecon(Gu, Gut, C, n), y, ve


# few partial sums; thousands (Gu: 400 000 rows x 8 coils); the smallest
@pytest.mark.parametrize("N,n,nCh,spokes", [([64, 64], [32, 32], 3, 40), ([64, 64, 64], [32, 32, 32], 8, 6250),
                                            ([20, 18], [10, 8], 1, 11)])
def test_steps_replay_for_every_solution_buffer(N, n, nCh, spokes):
    """Calls with alternating solution buffers, all kept alive, give the same
    bits, and those of two runs of fewer steps joined: nIter = 2 restarts."""
    import torch

    rec, y, ve = _case(N, n, nCh, spokes, 5)
    nu = int(np.prod(n))
    yd, vd = torch.from_numpy(y).cuda(), torch.from_numpy(ve.astype(np.float32)).cuda()
    xs = [torch.zeros(nu, dtype=torch.complex64, device="cuda") for _ in range(3)]
    for x in xs:
        rec.run_dev(yd, vd, x, nIter=2, nCGD=4, ve_max=1.0)
    two = torch.zeros(nu, dtype=torch.complex64, device="cuda")
    for _ in range(2):
        rec.run_dev(yd, vd, two, nIter=1, nCGD=4, ve_max=1.0)
    torch.cuda.synchronize()
    for x in xs + [two]:
        assert torch.equal(torch.view_as_real(x), torch.view_as_real(xs[0]))
    assert float(xs[0].abs().max()) > 0
    rec.plan.close()


def test_chain_step_replays_for_every_solution_buffer():
    """The temporal chain's captured step, called with alternating x, z, u."""
    import torch

    import monalisa_b200 as mb

    rng = np.random.default_rng(3)
    N, n, nCh = [48, 40], [24, 20], 3
    t = [(rng.random((2, m)) - 0.5) * 36 for m in (700, 911)]
    mats = [mb.bmTraj2SparseMat(v, np.ones(v.shape[1]), N, [1, 1]) for v in t]
    nu, rows = 480, 1611
    C = (rng.standard_normal((nu, nCh)) + 1j * rng.standard_normal((nu, nCh))).astype(np.complex64)
    chain = mb.TevaMorphosiaChain([m[0] for m in mats], [m[1] for m in mats], C, n)
    y = torch.from_numpy((rng.standard_normal((rows, nCh)) + 1j * rng.standard_normal((rows, nCh))).astype(np.complex64)).cuda()
    ve = torch.ones(rows, device="cuda")
    bufs = [[torch.zeros((2, nu), dtype=torch.complex64, device="cuda") for _ in range(3)] for _ in range(3)]
    for x, z, u in bufs:
        chain.run_dev(y, ve, x, z, u, 0.01, 0.1, 2, 4, 1.0)
    torch.cuda.synchronize()
    for b in bufs[1:]:
        for v, w in zip(b, bufs[0]):
            assert torch.equal(torch.view_as_real(v), torch.view_as_real(w))
    assert float(bufs[0][0].abs().max()) > 0
