"""Performance cases: the work a user of this framework has it do.

Every case goes through a public entry point -- ``tomocam.MBIR`` on host
arrays, or the device-level ``Plan`` / ``mbir_batched`` / ``autograd`` calls
on CUDA tensors.  ``listed`` gives the fixed cases, ``draw`` one more from
the same ranges, ``prepare`` what a program has in hand before the call,
``run`` one pass, ``work`` the bytes and operations the pass cannot do
without, and ``exact`` the same outputs computed in 64 bits with plain torch.

Inputs are seeded: volumes of random ellipsoids of density 0.1 .. 1 with a
N(0, 0.01) texture, their parallel-beam projections in closed form with 1 %
noise, and A^T y = H x of such a volume.
"""
import math

import numpy as np
import torch

import tomocam
from tomocam_b200 import autograd as tad
from tomocam_b200.plan import BatchScan, Plan, mbir_batched

SIGMA = 100.0  # 1 / the default smoothness 0.01
P_SHAPE = 1.2
MRF_C = float(np.float32(0.001))


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # tomocam.MBIR on one 256-pixel slice, the reference's plain call:
        # every launch is small, set-up and latency count
        {"name": "mbir_host_1x256", "op": "mbir_host", "slices": 1, "n": 256, "nproj": 180,
         "iters": 20, "smoothness": 0.05, "shift": 0},
        # tomocam.MBIR on a stack of a 2048-pixel detector, off-centre axis:
        # the whole call with its copies, on the padded 2908^2 grid
        {"name": "mbir_host_16x2048", "op": "mbir_host", "slices": 16, "n": 2048, "nproj": 1969,
         "iters": 30, "smoothness": 0.01, "shift": 3},
        # the full-volume iteration on the device (a slab of the 256 slices)
        {"name": "solve_96x2048", "op": "solve", "slices": 96, "n": 2048, "nproj": 1969, "iters": 4},
        # an ordinary reconstruction with an odd width and an odd slice count
        {"name": "solve_5x767", "op": "solve", "slices": 5, "n": 767, "nproj": 601, "iters": 20},
        # the operator pair of the throughput workload (1500 angles, 1536^2)
        {"name": "radon_16x1536", "op": "radon", "slices": 16, "n": 1536, "nproj": 1500},
        {"name": "iradon_16x1536", "op": "iradon", "slices": 16, "n": 1536, "nproj": 1500, "ramp": False},
        # filtered back-projection of a few odd-sized slices
        {"name": "fbp_5x1001", "op": "iradon", "slices": 5, "n": 1001, "nproj": 721, "ramp": True},
        # one small projection: the latency of a single operator call
        {"name": "radon_1x256", "op": "radon", "slices": 1, "n": 256, "nproj": 180},
        # the data gradient on the grid MBIR pads a 2048-pixel detector to,
        # and of one small slice (a caller's own optimiser, one step at a time)
        {"name": "toeplitz_6x2908", "op": "toeplitz", "slices": 6, "n": 2908, "nproj": 1969},
        {"name": "toeplitz_1x200", "op": "toeplitz", "slices": 1, "n": 200, "nproj": 180},
        # independent scans of uneven size solved together
        {"name": "batched_24", "op": "batched", "scans": 24, "nmin": 256, "nmax": 1024, "layout": 4,
         "iters": 10},
        # training through an unrolled, checkpointed reconstruction
        {"name": "unrolled_32x768", "op": "unrolled", "slices": 32, "n": 768, "nproj": 720, "iters": 10},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ones' ranges; sizes spread over their logarithm."""
    op = rng.choice(["mbir_host", "solve", "solve", "radon", "radon", "iradon", "iradon",
                     "toeplitz", "toeplitz", "batched", "unrolled"])
    if op == "batched":
        return {"op": op, "scans": _log(rng, 3, 24), "nmin": 128, "nmax": 1024,
                "layout": rng.randrange(1 << 30), "iters": rng.randint(4, 10)}
    top = {"mbir_host": 2048, "unrolled": 768}.get(op, 2908)
    n = _log(rng, 128, top)
    # as many slices as the largest listed case's pixels allow, at most 64
    area = {"mbir_host": 8 * 2048 ** 2, "unrolled": 32 * 768 ** 2, "solve": 64 * 2048 ** 2}.get(op, 12 * 1536 ** 2)
    slices = _log(rng, 1, max(1, min(64, area // n ** 2)))
    case = {"op": op, "slices": slices, "n": n, "nproj": max(30, min(1969, int(n * rng.uniform(0.6, 1.2))))}
    if op == "mbir_host":
        case.update(iters=rng.randint(5, 30), smoothness=rng.choice([0.01, 0.02, 0.05]), shift=rng.randint(-4, 4))
    elif op == "solve":
        case.update(iters=rng.randint(2, 6))
    elif op == "unrolled":
        case.update(iters=rng.randint(2, 8))
    elif op == "iradon":
        case.update(ramp=rng.random() < 0.5)
    return case


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _angles(nproj):
    return (np.arange(nproj) * (np.pi / nproj)).astype(np.float32)


def _gen(seed):
    return torch.Generator("cuda").manual_seed(seed)


def _ellipsoids(slices, seed, count=16):
    """Per slice and ellipsoid: centre, half-axes (in units of n/2), angle, density."""
    r = np.random.default_rng(seed)
    cx, cy = r.uniform(-0.4, 0.4, (2, count))
    ax, ay = r.uniform(0.06, 0.35, (2, count))
    th, rho = r.uniform(0, np.pi, count), r.uniform(0.1, 1.0, count)
    cz, az = r.uniform(0, slices, count), r.uniform(0.4, 1.2, count) * (slices + 1)
    z = np.arange(slices)[:, None] + 0.5
    cut = np.sqrt(np.clip(1.0 - ((z - cz) / az) ** 2, 0.0, None))  # the slice's section of each ellipsoid
    return [[(cx[k], cy[k], ax[k] * cut[s, k], ay[k] * cut[s, k], th[k], rho[k])
             for k in range(count) if cut[s, k] > 0.05] for s in range(slices)]


def _volume(slices, n, seed):
    """float32 [slices, n, n]: ellipsoids with a N(0, 0.01) texture."""
    vol = 0.01 * torch.randn((slices, n, n), device="cuda", generator=_gen(seed))
    c = (torch.arange(n, device="cuda", dtype=torch.float32) - (n - 1) / 2) / (n / 2)
    for s, parts in enumerate(_ellipsoids(slices, seed)):
        for cx, cy, ax, ay, th, rho in parts:
            xr = (c - cx)[None, :] * math.cos(th) + (c - cy)[:, None] * math.sin(th)
            yr = (c - cy)[:, None] * math.cos(th) - (c - cx)[None, :] * math.sin(th)
            vol[s] += rho * (((xr / ax) ** 2 + (yr / ay) ** 2) <= 1.0)
    return vol


def _sinogram(slices, n, nproj, seed, shift=0):
    """float32 [slices, nproj, n]: line integrals of the ellipsoids in pixels, 1 % noise."""
    th = torch.as_tensor(_angles(nproj), device="cuda", dtype=torch.float64)[:, None]
    t = (torch.arange(n, device="cuda", dtype=torch.float64) - n // 2 - shift) / (n / 2)
    out = torch.zeros((slices, nproj, n), device="cuda", dtype=torch.float32)
    for s, parts in enumerate(_ellipsoids(slices, seed)):
        for cx, cy, ax, ay, rot, rho in parts:
            a2 = (ax * torch.cos(th - rot)) ** 2 + (ay * torch.sin(th - rot)) ** 2
            d = t[None, :] - (cx * torch.cos(th) + cy * torch.sin(th))
            out[s] += (rho * ax * ay * n * torch.sqrt((a2 - d * d).clamp(min=0.0)) / a2).float()
    noise = torch.randn(out.shape, device="cuda", generator=_gen(seed + 1))
    return (out + 0.01 * out.max() * noise).clamp_(min=0.0)


def _psf(n, nproj):
    """The point-spread function in 64 bits, [n, 2n-1] (its rows dy = 0 .. n-1;
    it is even): sum over angles and radii r_j = 2 pi (j - n//2) / (n - 1) of
    cos(r_j t), t = dx cos + dy sin, which sums in closed form over j."""
    dx = torch.arange(-(n - 1), n, device="cuda", dtype=torch.float64)
    dy = torch.arange(n, device="cuda", dtype=torch.float64)[:, None]
    a = _angles(nproj).astype(np.float64)
    out = torch.zeros((n, 2 * n - 1), device="cuda", dtype=torch.float64)
    for k in range(nproj):
        h = dx * (math.cos(a[k]) * math.pi / (n - 1)) + dy * (math.sin(a[k]) * math.pi / (n - 1))
        h = torch.remainder(h + math.pi / 2, math.pi) - math.pi / 2  # the sum's period
        # radii centred on 0 (odd n) or on half a step below it (even n)
        den = torch.sin(h) if n % 2 else torch.tan(h)
        near = den.abs() < 1e-12
        v = torch.where(near, float(n), torch.sin(n * h) / torch.where(near, 1.0, den))
        out += v
    return out


class _Toeplitz:
    """H x = (psf * x) / n^3 (linear convolution, cropped), plain torch FFTs."""

    def __init__(self, n, nproj, dtype):
        self.n, self.dtype = n, dtype
        self.m = m = next(k for k in range(2 * n - 1, 4 * n) if not _rough(k))
        half = _psf(n, nproj)
        grid = torch.zeros((m, m), device="cuda", dtype=torch.float64)
        cols = torch.arange(-(n - 1), n, device="cuda") % m
        grid[:n, cols] = half
        grid[(-torch.arange(1, n, device="cuda") % m)[:, None], cols] = half[1:].flip(1)
        self.spec = torch.fft.rfft2(grid).real.to(dtype).clone()

    def __call__(self, x):
        out = torch.empty(x.shape, device="cuda", dtype=self.dtype)
        for s in range(x.shape[0]):
            f = torch.fft.rfft2(x[s].to(self.dtype), s=(self.m, self.m))
            out[s] = torch.fft.irfft2(f * self.spec, s=(self.m, self.m))[:self.n, :self.n]
        return out / float(self.n) ** 3


def _rough(m):
    for p in (2, 3, 5, 7):
        while m % p == 0:
            m //= p
    return m != 1


def _scan(slices, n, nproj, seed):
    """A^T y, ||y||^2 and an initial guess of one scan: y = A x of a seeded
    volume (A^T y = H x, ||y||^2 = x.Hx and a little noise), the guess that
    volume blurred, at 0.9 of its density."""
    x = _volume(slices, n, seed)
    aty = _Toeplitz(n, nproj, torch.float32)(x)
    sino_sq = 1.001 * float((x.double() * aty).sum())
    x0 = 0.45 * (x + torch.roll(x, 1, 2))
    x0 += 0.02 * torch.randn(x.shape, device="cuda", generator=_gen(seed + 2))
    return aty, sino_sq, x0


def _batch(case):
    """(n, nproj, beta) of each scan of a batched case."""
    r = np.random.default_rng(case["layout"])
    if case["nmin"] == 256:  # the uneven-batch workload's own sizes
        ns = r.choice([256, 384, 512, 768, 1024], case["scans"])
        ps = r.choice([180, 360, 720, 1024, 1500], case["scans"])
    else:
        ns = np.exp(r.uniform(np.log(case["nmin"]), np.log(case["nmax"]), case["scans"])).astype(int)
        ps = (ns * r.uniform(0.6, 1.2, case["scans"])).astype(int)
    return [(int(n), int(p), float(b)) for n, p, b in zip(ns, ps, r.uniform(0.1, 2.0, case["scans"]))]


def _inputs(case, seed):
    op = case["op"]
    if op == "batched":
        return [_scan(1, n, p, seed + 10 * i) for i, (n, p, _) in enumerate(_batch(case))]
    S, n, P = case["slices"], case["n"], case["nproj"]
    if op == "mbir_host":
        return _sinogram(S, n, P, seed, case["shift"]).cpu().numpy()
    if op == "radon":
        return _volume(S, n, seed)
    if op == "iradon":
        return _sinogram(S, n, P, seed)
    if op == "toeplitz":  # a gradient in the middle of a descent: A^T y beside H x, not equal to it
        return _volume(S, n, seed), 0.3 * _volume(S, n, seed + 5) * P / n
    if op == "solve":
        return _scan(S, n, P, seed)
    aty, _, x0 = _scan(S, n, P, seed)
    return aty, x0, _volume(S, n, seed)


def _center(case):
    return case["n"] / 2.0 + case["shift"]


def prepare(case, seed):
    data = _inputs(case, seed)
    st = {"case": case, "data": data}
    if case["op"] == "mbir_host":
        st["angles"] = _angles(case["nproj"])
    elif case["op"] == "batched":
        st["plans"] = [Plan(n, _angles(p), pow2_toeplitz=True) for n, p, _ in _batch(case)]
    else:
        need_psf = case["op"] not in ("radon", "iradon")
        st["plan"] = Plan(case["n"], _angles(case["nproj"]), psf=need_psf)
        if case["op"] == "unrolled":
            st["step"] = 0.5 / st["plan"].info["lipschitz"]
    torch.cuda.synchronize()
    return st


def run(state):
    case, data = state["case"], state["data"]
    op = case["op"]
    if op == "mbir_host":
        return tomocam.MBIR(data, state["angles"], _center(case), case["iters"], case["smoothness"])
    if op == "batched":
        xs = [x0.clone() for _, _, x0 in data]
        scans = [BatchScan(pl, aty, sq, x, SIGMA, P_SHAPE, beta)
                 for pl, (aty, sq, _), x, (_, _, beta) in zip(state["plans"], data, xs, _batch(case))]
        hist = mbir_batched(scans, case["iters"])
        return xs, hist
    plan = state["plan"]
    if op == "radon":
        return plan.radon(data)
    if op == "iradon":
        return plan.iradon(data, ramp=case["ramp"])
    if op == "toeplitz":
        return plan.toeplitz_grad(data[0], data[1])
    if op == "solve":
        return plan.mbir_solve(data[0], data[1], data[2], case["iters"], SIGMA, P_SHAPE)
    aty, x0, target = data
    x0 = x0.detach().requires_grad_(True)
    beta = torch.tensor(0.5, dtype=torch.float64, requires_grad=True)
    sigma = torch.tensor(SIGMA, dtype=torch.float64, requires_grad=True)
    xk = tad.unrolled_mbir(x0, plan, aty, case["iters"], state["step"], beta, sigma)
    (0.5 * ((xk - target) ** 2).sum()).backward()
    return xk.detach(), x0.grad, beta.grad, sigma.grad


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
def _toeplitz_flops(n):
    """Two real transforms of one n^2 slice padded to 2n: its n rows, then the columns, there and back."""
    m = 2 * n
    return 5.0 * n * m * math.log2(m) + 5.0 * m * m * math.log2(m)


def _nufft_flops(n, nproj):
    """One real 2-D transform padded to 2n, a 7 x 7 kernel at every point, the detector's transforms."""
    return 0.5 * _toeplitz_flops(n) + nproj * n * (4.0 * 49 + 2.5 * math.log2(n))


PRIOR_FLOPS = 13 * 20.0  # per voxel: 13 edges


def work(case):
    op = case["op"]
    if op == "batched":
        lay = _batch(case)
        return {"bytes": sum(12.0 * n * n for n, _, _ in lay),
                "flops": sum(case["iters"] * (_toeplitz_flops(n) + PRIOR_FLOPS * n * n) for n, _, _ in lay)}
    S, n, P = case["slices"], case["n"], case["nproj"]
    image, sino = 4.0 * S * n * n, 4.0 * S * P * n
    if op in ("radon", "iradon"):
        return {"bytes": image + sino, "flops": S * _nufft_flops(n, P)}
    if op == "toeplitz":
        return {"bytes": 3 * image, "flops": S * _toeplitz_flops(n)}
    if op == "solve":
        return {"bytes": 3 * image, "flops": S * case["iters"] * (_toeplitz_flops(n) + PRIOR_FLOPS * n * n)}
    if op == "unrolled":  # forward, and one Hessian product per iteration back
        return {"bytes": 5 * image, "flops": 2.0 * S * case["iters"] * (_toeplitz_flops(n) + PRIOR_FLOPS * n * n)}
    g = n + 2 * (int(0.42 * n) // 2)  # the grid MBIR pads the detector to
    return {"bytes": image + sino,
            "flops": S * (case["iters"] * (_toeplitz_flops(g) + PRIOR_FLOPS * g * g)
                          + _nufft_flops(n, P) + _nufft_flops(g, P))}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
def _radii(n):
    """Non-negative radii r_j and how often each counts in the sum over all
    of them (a real image's spectrum is Hermitian; for even n the radius
    -n/2 stands alone, and its real part counts like +n/2's)."""
    k = torch.arange(0, n // 2 + 1, device="cuda", dtype=torch.float64)
    twice = torch.full_like(k, 2.0)
    twice[0] = 1.0
    if n % 2 == 0:
        twice[-1] = 1.0
    return 2.0 * math.pi / (n - 1) * k, k, twice


def _waves(r, n, c):
    """exp(i r c m) for m = -n//2 .., [radii, n]."""
    m = torch.arange(n, device="cuda", dtype=torch.float64) - n // 2
    ph = (r * c)[:, None] * m[None, :]
    return torch.cos(ph), torch.sin(ph)


def _exact_radon(x, nproj):
    S, n, _ = x.shape
    r, k, twice = _radii(n)
    d = torch.arange(n, device="cuda", dtype=torch.float64) - n // 2
    ph = 2.0 * math.pi / n * torch.remainder(k[:, None] * d[None, :], n)
    back_c, back_s = torch.cos(ph) * twice[:, None], torch.sin(ph) * twice[:, None]
    xm = x.double().reshape(S * n, n).T.contiguous()
    out = torch.empty((S, nproj, n), device="cuda", dtype=torch.float64)
    for p, a in enumerate(_angles(nproj).astype(np.float64)):
        cx, sx = _waves(r, n, math.cos(a))
        cy, sy = _waves(r, n, math.sin(a))
        tc = (cx @ xm).reshape(-1, S, n)
        ts = (sx @ xm).reshape(-1, S, n)
        # spectrum: sum_y exp(-i r y sin) sum_x exp(-i r x cos) x
        re = (tc * cy[:, None] - ts * sy[:, None]).sum(2)
        im = -(ts * cy[:, None] + tc * sy[:, None]).sum(2)
        out[:, p] = (re.T @ back_c - im.T @ back_s) / (n * n)
    return out


def _exact_iradon(y, ramp):
    S, P, n = y.shape
    r, k, twice = _radii(n)
    d = torch.arange(n, device="cuda", dtype=torch.float64) - n // 2
    ph = 2.0 * math.pi / n * torch.remainder(k[:, None] * d[None, :], n)
    w = twice * (k / n) if ramp else twice
    fc, fs = torch.cos(ph) * w[:, None], torch.sin(ph) * w[:, None]
    out = torch.zeros((S * n, n), device="cuda", dtype=torch.float64)
    for p, a in enumerate(_angles(P).astype(np.float64)):
        yp = y[:, p].double()
        re, im = yp @ fc.T, -(yp @ fs.T)                       # [S, radii]
        cx, sx = _waves(r, n, math.cos(a))
        cy, sy = _waves(r, n, math.sin(a))
        # Re c exp(i r (x cos + y sin))
        gr = (re[:, None] * cy.T[None] - im[:, None] * sy.T[None]).reshape(S * n, -1)
        gi = (re[:, None] * sy.T[None] + im[:, None] * cy.T[None]).reshape(S * n, -1)
        out.addmm_(gr, cx)
        out.addmm_(gi, sx, alpha=-1.0)
    return out.reshape(S, n, n) / (n * n)


_W = {1: float(np.float32(0.0523)), 2: float(np.float32(0.0370)), 3: float(np.float32(0.0302))}


def _edges(vols, body):
    """Calls body(slab, weight, differences) for the 26 clamped neighbours, the
    differences v - v_neighbour of each volume, a few planes at a time."""
    S, n, _ = vols[0].shape
    pz, pn = (torch.arange(-1, k + 1, device="cuda").clamp(0, k - 1) for k in (S, n))
    step = max(1, (1 << 26) // (n * n))
    for z in range(0, S, step):
        e = min(S, z + step)
        for dz in (-1, 0, 1):
            pad = [v[pz[z + 1 + dz:e + 1 + dz]][:, pn][:, :, pn] for v in vols]
            for dy in (-1, 0, 1):
                for dx in (-1, 0, 1):
                    o = abs(dz) + abs(dy) + abs(dx)
                    if o:
                        body(slice(z, e), _W[o], [v[z:e] - q[:, 1 + dy:1 + dy + n, 1 + dx:1 + dx + n]
                                                  for v, q in zip(vols, pad)])


def _rho(d, sigma, p=P_SHAPE):
    """t = (|d|/sigma)^(2-p) and rho'(d)."""
    t = (d.abs() / sigma) ** (2.0 - p)
    c = MRF_C + t
    return t, c, d / (c * sigma ** 2) * (2.0 - (2.0 - p) * t / c)


def _prior_grad(x, sigma):
    g = torch.zeros_like(x)

    def body(sl, w, d):
        g[sl] += w * _rho(d[0], sigma)[2]

    _edges([x], body)
    return g


def _prior_hvp(x, v, sigma, p=P_SHAPE):
    """Hess U v, v.grad U, v.dgrad U/dsigma."""
    hv = torch.zeros_like(x)
    dots = [0.0, 0.0]

    def body(sl, w, diffs):
        d, dv = diffs
        t, c, d1 = _rho(d, sigma, p)
        d2 = ((2.0 * MRF_C + p * t) / c ** 2 + (2.0 - p) * t * ((p - 4.0) * MRF_C - p * t) / c ** 3) / sigma ** 2
        hv[sl] += w * d2 * dv
        dots[0] += w * float((v[sl] * d1).sum())
        dots[1] -= w * float((v[sl] * (d * d2 + d1)).sum()) / sigma

    _edges([x, v], body)
    return hv, dots[0], dots[1]


def _exact_solve(H, aty, sino_sq, x0, iters, sigma, beta_prior=1.0):
    """Optimizer::run2: Nesterov steps with backtracking, x = sol after an
    accepted step; H of an extrapolated point follows from linearity."""
    n = x0.shape[1]
    step0 = step = min(1.0 / float(H(torch.ones((1, n, n), device="cuda", dtype=torch.float64)).max()), 1.0)
    aty = aty.double()
    sol = x0.double()
    x, hsol = sol, H(sol)
    hx = hsol
    t = tnew = 1.0
    hist = np.zeros((iters, 3))

    def objective(v, hv):
        return math.sqrt(float((v * hv).sum()) - 2.0 * float((v * aty).sum()) + sino_sq)

    for it in range(iters):
        while True:
            hist[it, 2] += 1
            b = tnew * (1.0 / t - 1.0)
            tnew = 0.5 * (math.sqrt(t ** 4 + 4.0 * t * t) - t * t)
            if sol is x:
                y, hy = sol, hsol
            else:
                y, hy = sol + (sol - x) * b, hsol + (hsol - hx) * b
            g = _prior_grad(y, sigma).mul_(beta_prior).add_(hy).sub_(aty)
            sol = y - step * g
            hsol = H(sol)
            fx, fy = objective(sol, hsol), objective(y, hy)
            if fx > fy + 0.5 * step * float((g * g).sum()):
                step *= 0.9
            else:
                break
        step, t = step0, tnew
        hist[it, 0], hist[it, 1] = fx, math.sqrt(float(((sol - x) ** 2).sum()))
        x, hx = sol, hsol
    return sol, hist


def _exact_unrolled(H, aty, x0, target, iters, step, beta, sigma):
    aty = aty.double()
    xs = [x0.double()]
    for _ in range(iters):
        s = xs[-1]
        xs.append(s - step * (H(s) - aty + beta * _prior_grad(s, sigma)))
    v = xs[-1] - target.double()
    gb = gs = 0.0
    for s in reversed(xs[:-1]):
        hp, vg, vgs = _prior_hvp(s, v, sigma)
        gb -= step * vg
        gs -= step * beta * vgs
        v = v - step * (H(v) + beta * hp)
    return xs[-1], v, torch.tensor(gb, dtype=torch.float64), torch.tensor(gs, dtype=torch.float64)


def _exact_mbir_host(sino, center, iters, sigma):
    y = torch.as_tensor(sino, device="cuda").double()
    y = y / y.max()
    S, P, D = y.shape
    x0 = _exact_iradon(y, True)
    off = (D + 1) // 2 - math.floor(center + 0.5)
    npad = max(int(0.42 * D) // 2, abs(off))
    n = D + 2 * npad
    yp = torch.zeros((S, P, n), device="cuda", dtype=torch.float64)
    yp[:, :, npad:npad + D] = y
    yp = torch.roll(yp, -off, 2)
    g = torch.zeros((S, n, n), device="cuda", dtype=torch.float64)
    g[:, npad:npad + D, npad:npad + D] = x0
    H = _Toeplitz(n, P, torch.float64)
    sol, _ = _exact_solve(H, _exact_iradon(yp, False), float((yp * yp).sum()), g, iters, sigma)
    return sol[:, npad:npad + D, npad:npad + D]


def exact(case, seed):
    """What run returns, in 64 bits; None where that would take too long."""
    op = case["op"]
    if op == "batched":
        xs, hists = [], []
        for (n, P, beta), (aty, sq, x0) in zip(_batch(case), _inputs(case, seed)):
            x, h = _exact_solve(_Toeplitz(n, P, torch.float64), aty, sq, x0, case["iters"], SIGMA, beta)
            xs.append(x)
            hists.append(h)
        return xs, np.stack(hists)
    S, n, P = case["slices"], case["n"], case["nproj"]
    transform = 2.0 * S * P * float(n) ** 3
    if op == "mbir_host":
        if 4.0 * transform > 2e13:
            return None
        return _exact_mbir_host(_inputs(case, seed), _center(case), case["iters"], 1.0 / case["smoothness"])
    if op in ("radon", "iradon"):
        if transform > 2e14:
            return None
        data = _inputs(case, seed)
        return _exact_radon(data, P) if op == "radon" else _exact_iradon(data, case["ramp"])
    data = _inputs(case, seed)
    H = _Toeplitz(n, P, torch.float64)
    if op == "toeplitz":
        return H(data[0]) - data[1].double()
    if op == "solve":
        return _exact_solve(H, data[0], data[1], data[2], case["iters"], SIGMA)
    lipschitz = float(H(torch.ones((1, n, n), device="cuda", dtype=torch.float64)).max())
    return _exact_unrolled(H, data[0], data[1], data[2], case["iters"], 0.5 / lipschitz, 0.5, SIGMA)
