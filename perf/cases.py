"""Performance cases of monalisa_b200: what a reconstruction program has the
library do, through its public entry points, at the sizes of real protocols.

Operations (``op``):
  forward / adjoint / pair   NufftPlan.shanna and .nakatsha (pair: both), the
                             step of every iterative reconstruction
  sensa                      SensaRecon.run_dev, one CG-SENSE reconstruction
  chain                      TevaMorphosiaChain.run_dev, temporal-TV ADMM over
                             frame bins
  grid                       the leight adjoint gridder on device buffers
                             (mlg_gridder_n2u_leight_dev)
  mathilda                   bmMathilda, the gridded reconstruction from host
                             arrays to a host image

Trajectories are radial (2-D golden angle, 3-D koosh ball), rotated by the
seed; k-space is the analytic transform of Gaussian blobs seen by smooth
coils, plus noise; volume elements are the radial ones.  ``exact`` restates
every operation in 64 bits with torch alone.
"""
from __future__ import annotations

import math

import numpy as np
import torch

SIGMA, K_MAX = 0.61, 10.0            # Gaussian window
TAU, ALPHA, KB_MAX = 1.95, 10.0, 10.0  # Kaiser-Bessel window
VE_MAX = 10.0
EPS32 = 10 * float(np.finfo(np.float32).eps)


def _case(op, N, n, coils, spokes, reads, kernel="gauss", precision="fp32", steps=0, bins=1, name=None):
    c = dict(op=op, dim=len(N), coils=coils, spokes=spokes, reads=reads, kernel=kernel, precision=precision,
             steps=steps, bins=bins)
    for k, (a, b) in enumerate(zip(N, n)):
        c["N%d" % k], c["n%d" % k] = a, b
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # one operator application of a full-size 3-D acquisition (4096 spokes,
        # 16 coils), each direction: the largest single calls
        _case("forward", [256] * 3, [128] * 3, 16, 4096, 256, name="forward_3d_128_c16"),
        _case("adjoint", [256] * 3, [128] * 3, 16, 4096, 256, name="adjoint_3d_128_c16"),
        # one frame bin of a motion-resolved acquisition (12 coils)
        _case("pair", [192] * 3, [96] * 3, 12, 850, 256, name="pair_3d_96_c12"),
        # a slab whose grid lengths (160, 120) are neither 2^k nor 3 * 2^k
        _case("pair", [160, 160, 120], [80, 80, 60], 8, 1000, 160, name="pair_3d_80_c8"),
        # a 2-D slice with a usual coil array
        _case("pair", [512, 512], [256, 256], 12, 256, 512, name="pair_2d_256_c12"),
        # a 2-D slice at oversampling 1.6 with an odd coil count, Kaiser-Bessel window
        _case("pair", [384, 384], [240, 240], 5, 201, 384, kernel="kaiser", name="pair_2d_240_c5"),
        # a whole small reconstruction: 2-D, coil-combined data
        _case("sensa", [512, 512], [256, 256], 1, 256, 512, kernel="kaiser", steps=20, name="sensa_2d_256_c1"),
        # a whole full-size reconstruction
        _case("sensa", [256] * 3, [128] * 3, 16, 4096, 256, steps=12, name="sensa_3d_128_c16"),
        # a reconstruction in reduced precision
        _case("sensa", [192] * 3, [96] * 3, 12, 1024, 256, precision="mixed", steps=10,
              name="sensa_3d_96_c12_mixed"),
        # two ADMM iterations over frame bins of unequal size
        _case("chain", [192] * 3, [96] * 3, 12, 600, 256, steps=4, bins=5, name="chain_3d_96_c12"),
        # gridding of a full-size acquisition onto its grid, device buffers
        _case("grid", [256] * 3, [128] * 3, 16, 4096, 256, name="grid_3d_256_c16"),
        # a gridded preview reconstruction, host arrays in, host image out
        _case("mathilda", [128] * 3, [64] * 3, 8, 512, 128, name="mathilda_3d_64_c8"),
    ]


def _smooth(v):
    for p in (2, 3, 5, 7):
        while v % p == 0:
            v //= p
    return v == 1


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _axis(rng, lo, hi):
    """A grid length: a multiple of 4, prime factors up to 7 with a split into
    two factors of at most 32, and an image length at oversampling 2 or 1.6."""
    ok = [v for v in range(lo, hi + 1, 4)
          if _smooth(v) and any(v % a == 0 and v // a <= 32 for a in range(1, 33))]
    x = rng.uniform(math.log(lo), math.log(hi))
    N = min(ok, key=lambda v: abs(math.log(v) - x) + 0.05 * rng.random())
    n = N // 2 if rng.random() < 0.7 else int(N / 1.6)
    return N, n - n % 2


def draw(rng):
    op = rng.choice(["forward", "adjoint", "pair", "pair", "sensa", "chain", "grid", "mathilda"])
    dim = 3 if op == "chain" or rng.random() < 0.6 else 2
    coils = rng.choice([1, 2, 3, 4, 5, 6, 8, 8, 10, 12, 12, 16])
    kernel = rng.choice(["gauss", "gauss", "kaiser"])
    if op in ("grid", "mathilda"):
        kernel = "gauss"
    if dim == 3:
        hi = {"mathilda": 128, "chain": 160}.get(op, 224)
        Nx, nx = _axis(rng, 48, hi)
        Nz, nz = (Nx, nx) if rng.random() < 0.5 else _axis(rng, 40, Nx)
        N, n = [Nx, Nx, Nz], [nx, nx, nz]
        spokes = _log(rng, 100, 2500 if op not in ("mathilda", "chain") else 500)
    else:
        Nx, nx = _axis(rng, 96, 768)
        N, n = [Nx, Nx], [nx, nx]
        spokes = _log(rng, 24, 600)
    reads = N[0] if rng.random() < 0.6 else 2 * _log(rng, N[0] // 4, N[0] // 2)
    steps = rng.randint(3, 10) if op == "sensa" else (rng.randint(2, 4) if op == "chain" else 0)
    precision = "mixed" if op == "sensa" and rng.random() < 0.3 else "fp32"
    bins = rng.randint(2, 4) if op == "chain" else 1
    return _case(op, N, n, coils, spokes, reads, kernel, precision, steps, bins)


# ---- inputs -------------------------------------------------------------------

def _dims(c):
    return [c["N%d" % k] for k in range(c["dim"])], [c["n%d" % k] for k in range(c["dim"])]


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _kp(c):
    return [SIGMA, K_MAX] if c["kernel"] == "gauss" else [TAU, ALPHA, KB_MAX]


def _traj(c, rs, spokes):
    """Radial lines through the centre: t [dim, spokes * reads] in grid units
    (sample fastest along a line) and the volume elements."""
    N, _ = _dims(c)
    R = c["reads"]
    r = (np.arange(R) - R // 2) / R
    gold = (1 + 5 ** 0.5) / 2
    k = np.arange(spokes)
    if c["dim"] == 2:
        phi = k * math.pi / gold + rs.uniform(0, 2 * math.pi)
        e = np.stack([np.cos(phi), np.sin(phi)])
    else:
        z = (k + rs.uniform(0.2, 0.8)) / spokes
        phi = k * (2 * math.pi / gold) + rs.uniform(0, 2 * math.pi)
        s = np.sqrt(1 - z * z)
        e = np.stack([s * np.cos(phi), s * np.sin(phi), z])
    t = np.stack([(e[d][:, None] * r[None, :] * N[d]).ravel() for d in range(c["dim"])])
    dr, vol = 1.0 / R, math.prod(N)
    if c["dim"] == 2:
        w = np.abs(r) * dr * math.pi / spokes
        w[R // 2] = math.pi * (dr / 2) ** 2 / spokes
    else:
        w = r * r * dr * 2 * math.pi / spokes
        w[R // 2] = 4 / 3 * math.pi * (dr / 2) ** 3 / spokes
    return t, np.tile(w * vol, spokes)


def _coils(c, g, dev):
    """Smooth complex sensitivities [prod(n), coils], x fastest: order-2
    polynomials of the position with random complex coefficients."""
    _, n = _dims(c)
    ax = [torch.linspace(-1, 1, v, device=dev) for v in n]
    pos = torch.meshgrid(*ax[::-1], indexing="ij")[::-1]
    basis = [torch.ones(tuple(n[::-1]), device=dev)] + list(pos) + [p * p - 1 / 3 for p in pos]
    basis = torch.stack([b.reshape(-1) for b in basis], 1)
    co = torch.randn(basis.shape[1], c["coils"], 2, generator=g, dtype=torch.float32) * 0.35
    co[0] += torch.randn(c["coils"], 2, generator=g)
    co = co.to(dev)
    return torch.complex(basis @ co[..., 0], basis @ co[..., 1])


def _blobs(c, g, t, dev, amp=1.0):
    """k-space [nPt, coils] complex64 of Gaussian blobs, plus noise."""
    N, n = _dims(c)
    m = 9
    cen = (torch.rand(m, c["dim"], generator=g) - 0.5) * 0.7
    width = 0.02 + 0.08 * torch.rand(m, generator=g)
    a = amp * (0.5 + torch.rand(m, 1, 1, generator=g)) * torch.randn(m, c["coils"], 2, generator=g)
    tt = torch.from_numpy(np.ascontiguousarray(t)).to(dev)  # [dim, nPt]
    y = torch.zeros(tt.shape[1], c["coils"], dtype=torch.complex64, device=dev)
    for b in range(m):
        ph, q, vol = 0.0, 0.0, 1.0
        for d in range(c["dim"]):
            f = tt[d] / N[d]
            ph = ph + f * float(cen[b, d] * n[d])
            q = q + (f * float(width[b]) * n[d]) ** 2
            vol *= float(width[b]) * n[d] * math.sqrt(2 * math.pi) / N[d]
        s = torch.polar(vol * torch.exp(-2 * math.pi ** 2 * q), -2 * math.pi * ph).to(torch.complex64)
        y += s[:, None] * torch.complex(a[b, :, 0], a[b, :, 1]).to(dev)[None, :]
    gd = torch.Generator(device=dev)
    gd.manual_seed(int(torch.randint(1 << 30, (1,), generator=g)))
    y += 1e-4 * amp * torch.randn(y.shape, generator=gd, dtype=torch.complex64, device=dev)
    return y


def _inputs(c, seed):
    """Everything that run() and exact() start from, from the seed alone."""
    dev = _dev()
    rs = np.random.RandomState(seed % (1 << 31))
    g = torch.Generator()
    g.manual_seed(seed)
    _, n = _dims(c)
    nu = math.prod(n)
    s = {"traj": [], "amp": 30.0}
    for b in range(c["bins"]):
        spokes = c["spokes"] if c["bins"] == 1 else int(c["spokes"] * rs.uniform(0.5, 1.5))
        s["traj"].append(_traj(c, rs, spokes))
    if c["op"] != "grid":
        s["C"] = _coils(c, g, dev)
    if c["op"] in ("forward", "pair"):
        gd = torch.Generator(device=dev)
        gd.manual_seed(seed + 77)
        s["x"] = torch.randn(nu, generator=gd, dtype=torch.complex64, device=dev)
    if c["op"] != "forward":
        s["y"] = [_blobs(c, g, t, dev, s["amp"]) for t, _ in s["traj"]]
        s["ve"] = [torch.from_numpy(v.astype(np.float32)).to(dev) for _, v in s["traj"]]
    return s


def _grid_units(c, t):
    """Single-precision grid coordinates (1-based) and the samples inside the
    grid box, as the gridder takes them."""
    N, _ = _dims(c)
    tg = np.asarray(t, np.float32) + np.array([N[d] // 2 + 1 for d in range(c["dim"])], np.float32)[:, None]
    keep = np.ones(tg.shape[1], bool)
    for d in range(c["dim"]):
        keep &= (tg[d] >= 1) & (tg[d] <= N[d])
    return tg, keep


def prepare(case, seed):
    import monalisa_b200 as mb

    c = case
    N, n = _dims(c)
    s = _inputs(c, seed)
    st = {"op": c["op"], "case": c}
    if c["op"] == "grid":
        (t, _), y, ve = s["traj"][0], s["y"][0], s["ve"][0]
        tg, keep = _grid_units(c, t)
        k = torch.from_numpy(keep).to(y.device)
        st["t"] = [torch.from_numpy(np.ascontiguousarray(tg[d][keep])).to(y.device) for d in range(c["dim"])]
        st["re"], st["im"] = y.real[k].contiguous(), y.imag[k].contiguous()
        st["ve"] = ve[k].contiguous()
        return st
    if c["op"] == "mathilda":
        st["y"] = s["y"][0].cpu().numpy()
        st["t"], st["v"] = s["traj"][0]
        st["C"] = s["C"].cpu().numpy()
        return st
    C = s["C"].cpu().numpy()
    mats = [mb.bmTraj2SparseMat(t, v, N, [1] * c["dim"], c["kernel"], 3, _kp(c)) for t, v in s["traj"]]
    if c["op"] == "chain":
        st["chain"] = mb.TevaMorphosiaChain([m[0] for m in mats], [m[1] for m in mats], C, n)
        st["y"], st["ve"] = torch.cat(s["y"]), torch.cat(s["ve"])
        return st
    st["rec"] = mb.SensaRecon(*mats[0], C, n, precision=c["precision"])
    for k in ("x", "y", "ve"):
        if k in s:
            st[k] = s[k][0] if isinstance(s[k], list) else s[k]
    if "ve" in st and c["op"] != "sensa":
        st["HY"] = st["ve"].clamp(max=VE_MAX)
    return st


# ---- one pass -----------------------------------------------------------------

def run(state):
    st, c = state, state["case"]
    N, n = _dims(c)
    op = st["op"]
    scale = float(math.prod(N))
    if op == "forward":
        return st["rec"].plan.shanna(st["x"])
    if op == "adjoint":
        return st["rec"].plan.nakatsha(st["y"], HY=st["HY"], scale=scale)
    if op == "pair":
        return {"y": st["rec"].plan.shanna(st["x"]), "x": st["rec"].plan.nakatsha(st["y"], HY=st["HY"], scale=scale)}
    if op == "sensa":
        x = torch.zeros(math.prod(n), dtype=torch.complex64, device=st["y"].device)
        return st["rec"].run_dev(st["y"], st["ve"], x, nIter=1, nCGD=c["steps"], ve_max=VE_MAX)
    if op == "chain":
        x = torch.zeros((c["bins"], math.prod(n)), dtype=torch.complex64, device=st["y"].device)
        z, u = torch.empty_like(x), torch.empty_like(x)
        st["chain"].run_dev(st["y"], st["ve"], x, z, u, 0.01, 0.1, 2, c["steps"], VE_MAX)
        return {"x": x, "z": z, "u": u}
    if op == "grid":
        from monalisa_b200 import _native as L

        t = st["t"] + [None] * (3 - c["dim"])
        M = N + [1] * (3 - c["dim"])
        bR = torch.empty((math.prod(N), c["coils"]), dtype=torch.float32, device=st["re"].device)
        bI = torch.empty_like(bR)
        L.call("mlg_gridder_n2u_leight_dev", c["dim"], L.tptr(st["re"]), L.tptr(st["im"]), L.tptr(t[0]), L.tptr(t[1]),
               L.tptr(t[2]), L.tptr(st["ve"]), c["coils"], st["re"].shape[0], M[0], M[1], M[2], 3, SIGMA, K_MAX,
               L.tptr(bR), L.tptr(bI), L.stream_ptr())
        return {"re": bR, "im": bI}
    import monalisa_b200 as mb

    return mb.bmMathilda(st["y"], st["t"], st["v"], st["C"], N, n, [1] * c["dim"], "gauss", 3, [SIGMA, K_MAX])


# ---- what a pass cannot do without ----------------------------------------------

def _op_work(c, nPt, forward):
    """One operator application: the image, coil maps and matrix entries
    (column and value) read, the k-space or image side written; the transform
    and the products' multiply-adds."""
    N, n = _dims(c)
    C, nu, Nu = c["coils"], math.prod(n), math.prod(N)
    nnz = nPt * 3 ** c["dim"]
    b = nu * 8 + nu * C * 8 + nnz * 8 + nPt * C * 8 + (0 if forward else nPt * 4)
    return b, 5.0 * Nu * math.log2(Nu) * C + 4.0 * nnz * C + 8.0 * nu * C


def work(case):
    c = case
    N, n = _dims(c)
    C, nu, Nu, nPt = c["coils"], math.prod(n), math.prod(N), c["spokes"] * c["reads"]
    f, a = _op_work(c, nPt, True), _op_work(c, nPt, False)
    if c["op"] in ("grid", "mathilda"):
        b = nPt * (4 * c["dim"] + 4) + nPt * C * 8
        fl = nPt * 3 ** c["dim"] * (4.0 * C + 10)
        if c["op"] == "grid":
            return {"bytes": b + Nu * C * 8, "flops": fl}
        return {"bytes": b + nu * C * 8 + nu * 8, "flops": fl + 5.0 * Nu * math.log2(Nu) * C}
    count = {"forward": (1, 0), "adjoint": (0, 1), "pair": (1, 1), "sensa": (c["steps"] + 2, c["steps"]),
             "chain": (c["bins"] * 2 * (c["steps"] + 1), c["bins"] * 2 * c["steps"])}[c["op"]]
    return {"bytes": count[0] * f[0] + count[1] * a[0], "flops": count[0] * f[1] + count[1] * a[1]}


# ---- the same in 64 bits ----------------------------------------------------------

def _weight(c, d):
    if c["kernel"] == "gauss":
        s = float(np.float32(SIGMA))
        return torch.exp(-0.5 * (d / s) ** 2) / (math.sqrt(2 * math.pi) * s)
    tau, al = float(np.float32(TAU)), float(np.float32(ALPHA))
    u = (1 - (d / tau) ** 2).clamp(min=0)
    return torch.special.i0(al * torch.sqrt(u)) / torch.special.i0(torch.tensor(al, dtype=torch.float64, device=d.device))


def _offsets(dim):
    r = (-1, 0, 1)
    return [(x, y, z)[:dim] for z in (r if dim > 2 else (0,)) for y in (r if dim > 1 else (0,)) for x in r]


class _Exact:
    """Gu, KFC and KFC_conj of one trajectory as 64-bit torch tensors."""

    def __init__(self, c, t, C):
        dev = C.device
        self.c = c
        self.N, self.n = _dims(c)
        N, dim = self.N, c["dim"]
        tg = torch.from_numpy(np.ascontiguousarray(t)).to(dev)
        tg = torch.stack([tg[d] + (N[d] // 2 + 1) for d in range(dim)])
        self.keep = torch.ones(tg.shape[1], dtype=torch.bool, device=dev)
        for d in range(dim):
            self.keep &= (tg[d] >= 1) & (tg[d] <= N[d])
        node = torch.floor(tg + 0.5)
        rest = tg - node
        self.idx, self.w = [], []
        for o in _offsets(dim):
            d2, lin, stride = 0.0, 0, 1
            for d in range(dim):
                d2 = d2 + (rest[d] - o[d]) ** 2
                lin = lin + torch.remainder(node[d].to(torch.int64) + o[d] - 1, N[d]) * stride
                stride *= N[d]
            self.idx.append(lin)
            self.w.append(_weight(c, torch.sqrt(d2)) * self.keep)
        tot = sum(self.w)
        tot = torch.where(tot > 0, tot, torch.ones_like(tot))
        self.w = [v / tot for v in self.w]
        K = _crop(_deapod(c, dev), N, self.n).reshape(-1, 1)
        self.KFC = K * C.to(torch.complex128) / math.prod(N)
        self.KFCc = K * C.to(torch.complex128).conj()

    def forward(self, x):
        out = []
        ax = tuple(range(self.c["dim"]))
        for k in range(self.c["coils"]):
            v = _pad((x * self.KFC[:, k]).reshape(self.n[::-1]), self.N, self.n)
            v = torch.fft.fftshift(torch.fft.fftn(torch.fft.ifftshift(v), dim=ax)).reshape(-1)
            y = 0
            for i, w in zip(self.idx, self.w):
                y = y + v[i] * w
            out.append(y)
        return torch.stack(out, 1)

    def adjoint(self, y):
        x = 0
        ax = tuple(range(self.c["dim"]))
        Nu = math.prod(self.N)
        for k in range(self.c["coils"]):
            v = torch.zeros(Nu, 2, dtype=torch.float64, device=y.device)
            yk = torch.view_as_real(y[:, k].contiguous())
            for i, w in zip(self.idx, self.w):
                v.index_add_(0, i, yk * w[:, None])
            v = torch.view_as_complex(v).reshape(self.N[::-1])
            v = torch.fft.fftshift(torch.fft.ifftn(torch.fft.ifftshift(v), dim=ax))
            x = x + _crop(v, self.N, self.n).reshape(-1) * self.KFCc[:, k]
        return x


def _slices(N, n):
    return tuple(slice(a // 2 - b // 2, a // 2 - b // 2 + b) for a, b in zip(N[::-1], n[::-1]))


def _pad(v, N, n):
    out = torch.zeros(N[::-1], dtype=v.dtype, device=v.device)
    out[_slices(N, n)] = v
    return out


def _crop(v, N, n):
    return v[_slices(N, n)]


def _deapod(c, dev):
    """The deapodisation on the grid [N_z][N_y][N_x]: the reciprocal of the
    window's transform (sampled at half cells), clipped."""
    N, _ = _dims(c)
    if c["dim"] == 1:
        raise ValueError("2-D and 3-D cases only")
    m = torch.arange(-2, 3, dtype=torch.float64, device=dev)
    g = torch.meshgrid(*([m / 2] * c["dim"]), indexing="ij")
    v = _weight(c, torch.sqrt(sum(a * a for a in g)))
    for d in range(c["dim"]):  # contracts the leading window axis, appends the frequency axis
        f = torch.arange(N[d], dtype=torch.float64, device=dev) - N[d] // 2
        cs = torch.cos(2 * math.pi * f[:, None] * m[None, :] / (2 * N[d]))
        v = torch.tensordot(v, cs, dims=([0], [1]))
    v = v.abs() / v.abs().max()
    kmax = float(np.float32(K_MAX if c["kernel"] == "gauss" else KB_MAX))
    v = torch.clamp(1 / v, max=kmax)
    return v.permute(*range(c["dim"] - 1, -1, -1)).contiguous()


def _dot(v, h=None):
    q = torch.view_as_real(v) ** 2
    return float((q.sum(-1) * h).sum()) if h is not None else float(q.sum())


def _sensa(c, e, y, ve):
    HX = float(np.prod(np.float32(1) / np.array(e.N, np.float32)))
    HY = ve.double().clamp(max=VE_MAX)[:, None]
    back = lambda r: e.adjoint(HY * r) / HX
    x = torch.zeros(math.prod(e.n), dtype=torch.complex128, device=y.device)
    res = y - e.forward(x)
    d = back(res)
    sq, p = HX * _dot(d), d
    for i in range(c["steps"]):
        if sq < EPS32:
            break
        Mp = e.forward(p)
        a = sq / _dot(Mp, HY)
        x = x + a * p
        if i == c["steps"] - 1:
            break
        res = res - a * Mp
        d = back(res)
        nxt = HX * _dot(d)
        p = d + (nxt / sq) * p
        sq = nxt
    return x


def _chain(c, es, ys, ves):
    F = c["bins"]
    HX = float(np.float32(np.prod(np.float32(1) / np.array(es[0].N, np.float32))))
    HY = [v.double().clamp(max=VE_MAX)[:, None] for v in ves]
    delta, rho = float(np.float32(0.01)), float(np.float32(0.1))
    M = lambda v: [e.forward(q) for e, q in zip(es, v)]
    D = lambda v: [v[i] - v[i - 1] for i in range(F)]
    back = lambda ry, rz: [es[i].adjoint(HY[i] * ry[i]) / HX + rho * (rz[i] - rz[(i + 1) % F]) for i in range(F)]
    sqn = lambda v, h=None: sum(_dot(q, None if h is None else h[i]) for i, q in enumerate(v))
    x = [torch.zeros(math.prod(es[0].n), dtype=torch.complex128, device=ys[0].device) for _ in range(F)]
    z, u = D(x), [torch.zeros_like(q) for q in x]
    for _ in range(2):
        ry = [a - b for a, b in zip(ys, M(x))]
        rz = [a - b - q for a, b, q in zip(z, u, D(x))]
        dA = back(ry, rz)
        p, sq = dA, HX * sqn(dA)
        for j in range(c["steps"]):
            if sq < EPS32:
                break
            Mp, Fp = M(p), D(p)
            a = sq / (sqn(Mp, HY) + rho * HX * sqn(Fp))
            x = [q + a * v for q, v in zip(x, p)]
            if j == c["steps"] - 1:
                break
            ry = [q - a * v for q, v in zip(ry, Mp)]
            rz = [q - a * v for q, v in zip(rz, Fp)]
            dA = back(ry, rz)
            nxt = HX * sqn(dA)
            p = [q + (nxt / sq) * v for q, v in zip(dA, p)]
            sq = nxt
        w = [a + b for a, b in zip(u, D(x))]
        soft = lambda v: torch.sign(v) * (v.abs() - delta / rho).clamp(min=0)
        z = [torch.complex(soft(q.real), soft(q.imag)) for q in w]
        u = [a - b for a, b in zip(w, z)]
    return {"x": torch.stack(x), "z": torch.stack(z), "u": torch.stack(u)}


def _leight(c, tg, y, dn):
    """The clipped-window gridding with per-cell normalisation: tg [dim][m]
    float32 grid coordinates (1-based), y [m, coils], dn [m] ->
    [prod(N), coils] complex128."""
    N, dim = _dims(c)[0], c["dim"]
    dev = y.device
    sg = float(np.float32(SIGMA))
    node = [torch.trunc(t + 0.5).double() for t in tg]
    Nu = math.prod(N)
    out = torch.zeros(Nu, 2 * c["coils"], dtype=torch.float64, device=dev)
    tot = torch.zeros(Nu, dtype=torch.float64, device=dev)
    yr = torch.view_as_real(y.to(torch.complex128)).reshape(y.shape[0], -1)
    g1 = 1 / (math.sqrt(2 * 3.141592) * sg)
    for o in _offsets(dim):
        d2, lin, stride = 0.0, 0, 1
        ok = torch.ones(y.shape[0], dtype=torch.bool, device=dev)
        for d in range(dim):
            d2 = d2 + (tg[d].double() - node[d] - o[d]) ** 2
            cell = node[d].to(torch.int64) - 1 + o[d]
            ok &= (cell >= 0) & (cell < N[d])
            lin = lin + cell * stride
            stride *= N[d]
        w = (g1 * torch.exp(-d2 / (2 * sg * sg)) * dn.double())[ok]
        out.index_add_(0, lin[ok], w[:, None] * yr[ok])
        tot.index_add_(0, lin[ok], w)
    out /= torch.where(tot < 1e-5, torch.ones_like(tot), tot)[:, None]
    return torch.view_as_complex(out.reshape(Nu, c["coils"], 2))


def exact(case, seed):
    c = case
    N, n = _dims(c)
    s = _inputs(c, seed)
    scale = float(math.prod(N))
    if c["op"] in ("grid", "mathilda"):
        (t, v), y = s["traj"][0], s["y"][0]
        tg, keep = _grid_units(c, t)
        k = torch.from_numpy(keep).to(y.device)
        tt = [torch.from_numpy(np.ascontiguousarray(tg[d][keep])).to(y.device) for d in range(c["dim"])]
        gr = _leight(c, tt, y[k], s["ve"][0][k])
        if c["op"] == "grid":
            return {"re": gr.real.contiguous(), "im": gr.imag.contiguous()}
        K = _deapod(c, y.device)
        num, den = 0, 0
        for i in range(c["coils"]):
            q = gr[:, i].reshape(N[::-1])
            q = torch.fft.fftshift(torch.fft.ifftn(torch.fft.ifftshift(q))) * scale * K
            q = _crop(q, N, n).reshape(-1)
            ci = s["C"][:, i].to(torch.complex128)
            num, den = num + ci.conj() * q, den + torch.view_as_real(ci).square().sum(-1)
        return (num / den).cpu().numpy()
    es = [_Exact(c, t, s["C"]) for t, _ in s["traj"]]
    if c["op"] == "forward":
        return es[0].forward(s["x"].to(torch.complex128))
    y = [q.to(torch.complex128) for q in s["y"]]
    if c["op"] == "sensa":
        return _sensa(c, es[0], y[0], s["ve"][0])
    if c["op"] == "chain":
        return _chain(c, es, y, s["ve"])
    x = es[0].adjoint(y[0] * s["ve"][0].double().clamp(max=VE_MAX)[:, None]) * scale
    return x if c["op"] == "adjoint" else {"y": es[0].forward(s["x"].to(torch.complex128)), "x": x}
