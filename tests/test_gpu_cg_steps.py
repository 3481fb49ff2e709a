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
