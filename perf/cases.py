"""The work that a user of this framework has it do, as cases to measure: the
projectors, the solvers built on them, the filtered back projection, the
warm-start network's inference and gradient, and the alignment's shift search
and Fourier shift, each through the package's public entry points.

A case is a dict of plain values; `prepare` makes a program's state for it,
`run` does one pass, `work` says what the pass cannot do without and `exact`
gives the outputs in 64 bits from plain torch.
"""
import math
import os
import re

import numpy as np
import torch

import arec3d_gb300 as gb
from arec3d_gb300 import warmstart

WEIGHTINGS = {"lin": gb.LIN, "kb": gb.KB, "sq": gb.SQ}


def listed():
    return [
        # a small region or a test volume: a few slices, where launches and latency count
        dict(name="cgls_sq_65x90x12", kind="cgls", weighting="sq", nx=65, na=90, ny=12, iters=4),
        # an odd detector width and slice count with the Kaiser-Bessel weighting
        dict(name="cgls_kb_401x300x75", kind="cgls", weighting="kb", nx=401, na=300, ny=75,
             iters=4),
        # the plain SIRT benchmark: 256 x 256 x 64 slices, 180 angles, 50 iterations
        dict(name="sirt_sq_256x180x64", kind="sirt", weighting="sq", nx=256, na=180, ny=64,
             iters=50),
        # the linear weighting, the default projector of the reference's parameter file
        dict(name="sirt_lin_256x180x64", kind="sirt", weighting="lin", nx=256, na=180, ny=64,
             iters=10),
        # the first reconstruction of the warm start at the training data's size
        dict(name="fbp_sq_512x360x128", kind="fbp", weighting="sq", nx=512, na=360, ny=128),
        # the projector pair at the headline benchmark's size, one direction each
        dict(name="project_sq_1024x1200x512", kind="project", weighting="sq", nx=1024, na=1200,
             ny=512),
        dict(name="backproject_sq_1024x1200x512", kind="backproject", weighting="sq", nx=1024,
             na=1200, ny=512),
        # the warm start's network on one batch of slices of the headline benchmark
        dict(name="unet_forward_1024x16", kind="unet", size=1024, batch=16),
        # one training batch of the network: output and parameter gradient
        dict(name="unet_gradient_256x16", kind="unet_grad", size=256, batch=16),
        # the alignment benchmark's shift search, a part of its 720 pairs
        dict(name="shifts_2048x2048x48", kind="shifts", ny=2048, nx=2048, nz=48),
        # binned detector images whose sides are not powers of two
        dict(name="shifts_750x1000x30", kind="shifts", ny=750, nx=1000, nz=30),
        # shifting a projection stack by the shifts found
        dict(name="fshift_512x512x180", kind="fshift", ny=512, nx=512, nz=180),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _smooth(n):
    """The largest length <= n with prime factors 2, 3, 5 and 7 only."""
    while True:
        m = n
        for p in (2, 3, 5, 7):
            while m % p == 0:
                m //= p
        if m == 1:
            return n
        n -= 1


def draw(rng):
    kind = rng.choice(["cgls", "cgls", "sirt", "fbp", "project", "project", "backproject",
                       "backproject", "unet", "unet_grad", "shifts", "shifts", "fshift"])
    if kind in ("project", "backproject"):
        nx, na, ny = _log_int(rng, 64, 1024), _log_int(rng, 24, 1200), _log_int(rng, 1, 512)
        return dict(kind=kind, weighting=rng.choice(["sq", "sq", "kb"]), nx=nx, na=na, ny=ny)
    if kind == "cgls":
        return dict(kind=kind, weighting=rng.choice(["sq", "sq", "kb"]), nx=_log_int(rng, 64, 512),
                    na=_log_int(rng, 36, 360), ny=_log_int(rng, 4, 128), iters=rng.randint(2, 4))
    if kind == "sirt":
        return dict(kind=kind, weighting=rng.choice(["sq", "kb", "lin"]),
                    nx=_log_int(rng, 64, 256), na=_log_int(rng, 36, 180), ny=_log_int(rng, 4, 64),
                    iters=rng.randint(3, 10))
    if kind == "fbp":
        return dict(kind=kind, weighting="sq", nx=_log_int(rng, 96, 768), na=_log_int(rng, 60, 500),
                    ny=_log_int(rng, 4, 200))
    if kind == "unet":
        return dict(kind=kind, size=8 * _log_int(rng, 16, 128), batch=_log_int(rng, 1, 16))
    if kind == "unet_grad":
        return dict(kind=kind, size=8 * _log_int(rng, 8, 32), batch=_log_int(rng, 1, 16))
    if kind == "shifts":
        return dict(kind=kind, ny=_smooth(_log_int(rng, 96, 2048)),
                    nx=_smooth(_log_int(rng, 96, 2048)), nz=_log_int(rng, 1, 48))
    return dict(kind=kind, ny=_smooth(_log_int(rng, 96, 1024)),
                nx=_smooth(_log_int(rng, 96, 1024)), nz=_log_int(rng, 1, 180))


# ------------------------------------------------------------------------------------------
# inputs


def _angles(na):
    return (np.arange(na) * (math.pi / na)).astype(np.float32)


def _spheres(case, seed, n=24):
    """Random spheres in a cylinder: rows of (cx, cz, cy, radius, attenuation)."""
    rng = np.random.default_rng(seed)
    nx, ny = case["nx"], case["ny"]
    R = 0.47 * nx
    rad = rng.uniform(0.01, 0.16, n) * nx
    rr, th = (R - rad) * np.sqrt(rng.uniform(0, 1, n)), rng.uniform(0, 2 * math.pi, n)
    return np.stack([rr * np.cos(th), rr * np.sin(th), rng.uniform(0, ny, n), rad,
                     rng.uniform(0, 0.02, n)], 1)


def _volume(case, seed, plan):
    """The spheres' attenuation at the pixel centres, [nrays][ys], with a little texture."""
    xs, zs = _pixels(0.5 * (case["nx"] - 1))
    px = torch.tensor(xs, device="cuda", dtype=torch.float32)[:, None]
    pz = torch.tensor(zs, device="cuda", dtype=torch.float32)[:, None]
    y = torch.arange(case["ny"], device="cuda", dtype=torch.float32)[None, :]
    x = torch.zeros(plan.nrays, plan.ys, device="cuda")
    v = x[:, :case["ny"]]
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    v += 1e-3 + 2e-4 * torch.randn(v.shape, generator=g, device="cuda")
    for cx, cz, cy, r, mu in _spheres(case, seed):
        inside = (px - cx) ** 2 + (pz - cz) ** 2 + (y - cy) ** 2 <= r * r
        v += float(mu) * inside
    return x


def _sinogram(case, seed, plan, photons=1e4):
    """The spheres' measured line integrals with Poisson noise, [na][nx][ys]."""
    ang = torch.tensor(_angles(case["na"]), device="cuda")
    u = torch.arange(case["nx"], device="cuda", dtype=torch.float32) - 0.5 * (case["nx"] - 1)
    y = torch.arange(case["ny"], device="cuda", dtype=torch.float32)
    b = torch.zeros(case["na"], case["nx"], plan.ys, device="cuda")
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    sph = _spheres(case, seed)
    for a0 in range(0, case["na"], 64):  # in blocks: the temporaries stay small
        p = b[a0:a0 + 64, :, :case["ny"]]
        c, s = torch.cos(ang[a0:a0 + 64]), torch.sin(ang[a0:a0 + 64])
        for cx, cz, cy, r, mu in sph:
            d = u[None, :] - (float(cx) * c + float(cz) * s)[:, None]
            h = (float(r) ** 2 - d * d)[:, :, None] - ((y - float(cy)) ** 2)[None, None, :]
            p += 2 * float(mu) * h.clamp_(min=0).sqrt_()
        n = torch.poisson(photons * torch.exp(-p), generator=g).clamp_(min=1)
        p.copy_(-torch.log(n / photons))
    return b


def _smooth_noise(nz, ny, nx, g):
    """Band-limited random images, about unit variance."""
    f = torch.fft.rfft2(torch.randn(nz, ny, nx, generator=g, device="cuda"))
    ky = torch.fft.fftfreq(ny, device="cuda")[:, None]
    kx = torch.fft.rfftfreq(nx, device="cuda")[None, :]
    f *= torch.exp(-(kx * kx + ky * ky) / (2 * 0.08 ** 2))
    im = torch.fft.irfft2(f, s=(ny, nx))
    return im / im.std()


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("project", "backproject", "cgls", "sirt", "fbp"):
        plan = gb.Plan(WEIGHTINGS[case["weighting"]], 0.5 * (case["nx"] - 1), case["ny"],
                       _angles(case["na"]))
        st = dict(case=case, plan=plan)
        if kind == "project":
            st["x"] = _volume(case, seed, plan)
            st["q"] = torch.zeros(plan.sino_shape, device="cuda")
            return st
        st["b"] = _sinogram(case, seed, plan)
        st["x"] = torch.zeros(plan.vol_shape, device="cuda")
        if kind == "fbp":
            st["work"] = torch.zeros_like(st["b"])
            st["n2"] = torch.zeros(1, dtype=torch.float64, device="cuda")
        return st
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    if kind in ("unet", "unet_grad"):
        n, size = case["batch"], case["size"]
        if kind == "unet":
            net, _ = warmstart.load(gb, warmstart.DEFAULT_WEIGHTS, size, n)
        else:
            net = gb.UNet(size, n, train=True)
            net.set_params(_params())
        # a normalised first reconstruction: smooth structure and noise
        x = _smooth_noise(n, size, size, g)
        x += 0.5 * torch.randn(x.shape, generator=g, device="cuda")
        st = dict(case=case, net=net, x=x, y=torch.empty_like(x))
        if kind == "unet_grad":
            st["dout"] = torch.randn(x.shape, generator=g, device="cuda") / x.numel()
            st["grads"] = torch.zeros(net.nparams, device="cuda")
        return st
    nz, ny, nx = case["nz"], case["ny"], case["nx"]
    a = _smooth_noise(nz, ny, nx, g)
    if kind == "fshift":
        return dict(case=case, a=a, out=torch.empty_like(a),
                    sx=40 * torch.rand(nz, generator=g, device="cuda") - 20,
                    sy=40 * torch.rand(nz, generator=g, device="cuda") - 20)
    # the same images moved by whole pixels and a fraction, each with its own noise
    rng = np.random.default_rng(seed)
    lim = min(20, min(ny, nx) // 4)
    b = torch.empty_like(a)
    ky = torch.fft.fftfreq(ny, device="cuda")[:, None]
    kx = torch.fft.rfftfreq(nx, device="cuda")[None, :]
    for z in range(nz):
        dy, dx = rng.integers(-lim, lim + 1, 2) + rng.uniform(-0.4, 0.4, 2)
        ph = torch.exp(-2j * math.pi * (float(dy) * ky + float(dx) * kx))
        b[z] = torch.fft.irfft2(torch.fft.rfft2(a[z]) * ph, s=(ny, nx))
    a += 0.02 * torch.randn(a.shape, generator=g, device="cuda")
    b += 0.02 * torch.randn(b.shape, generator=g, device="cuda")
    f = dict(device="cuda", dtype=torch.float32)
    return dict(case=case, a=a, b=b, sx=torch.empty(nz, **f), sy=torch.empty(nz, **f),
                ix=torch.empty(nz, device="cuda", dtype=torch.int32),
                iy=torch.empty(nz, device="cuda", dtype=torch.int32))


def _params():
    """The committed network's parameters, float32 on the device."""
    bits = np.load(warmstart.DEFAULT_WEIGHTS)["params_bf16"].astype(np.uint32) << 16
    return torch.from_numpy(bits.view(np.float32).copy()).cuda()


# ------------------------------------------------------------------------------------------
# one pass


def _step(case):
    return 1.0 / (case["na"] * case["nx"])


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "project":
        st["plan"].project(st["x"], st["q"])
        return st["q"]
    if kind == "backproject":
        st["plan"].backproject(st["b"], st["x"])
        return st["x"]
    if kind == "cgls":
        rel, info = st["plan"].cgls(st["b"], st["x"], case["iters"], 0.0)
        return st["x"], rel.astype(np.float32), info.iterations
    if kind == "sirt":
        rel, info = st["plan"].sirt(st["b"], st["x"], _step(case), case["iters"], 0.0)
        return st["x"], rel.astype(np.float32), info.iterations
    if kind == "fbp":
        st["plan"].fbp(st["b"], st["x"], st["work"], atb_norm2=st["n2"])
        return st["x"], st["work"], st["n2"].float()
    if kind == "unet":
        st["net"].forward(st["x"], st["y"])
        return st["y"]
    if kind == "unet_grad":
        st["net"].forward(st["x"], st["y"])
        st["net"].backward(st["dout"], st["grads"])
        return st["y"], st["grads"]
    if kind == "shifts":
        gb.cc_shifts(st["a"], st["b"], st["sx"], st["sy"], st["ix"], st["iy"])
        return st["sx"], st["sy"], st["ix"], st["iy"]
    gb.fshift2d_device(st["a"], st["out"], st["sx"], st["sy"])
    return st["out"]


# ------------------------------------------------------------------------------------------
# what a pass cannot do without

_CONV = [(1, 32, 1), (32, 32, 1), (32, 64, 4), (64, 64, 4), (64, 128, 16), (128, 128, 16),
         (128, 256, 64), (256, 256, 64), (256, 128, 16), (256, 128, 16), (128, 128, 16),
         (128, 64, 4), (128, 64, 4), (64, 64, 4), (64, 32, 1), (64, 32, 1), (32, 32, 1)]


def work(case):
    kind = case["kind"]
    if "na" in case:
        xs, _ = _pixels(0.5 * (case["nx"] - 1))
        vol, sino = xs.size * case["ny"], case["na"] * case["nx"] * case["ny"]
        proj = (4 if case["weighting"] == "lin" else 6) * xs.size * case["na"] * case["ny"]
        passes = {"project": 1, "backproject": 1, "fbp": 2, "cgls": 2 * case.get("iters", 0) + 1,
                  "sirt": 2 * case.get("iters", 0) - 1}[kind]
        flops = passes * proj
        if kind == "fbp":
            flops += case["nx"] * sino  # half of the taps are zero
        out = {"fbp": vol + sino}.get(kind, sino if kind == "project" else vol)
        return {"bytes": 4 * (out + (vol if kind == "project" else sino)), "flops": flops}
    if kind in ("unet", "unet_grad"):
        px = case["batch"] * case["size"] ** 2
        flops = px * (sum(2 * 9 * i * o / d for i, o, d in _CONV) + 2 * 32)
        params = sum(9 * i * o for i, o, _ in _CONV)
        if kind == "unet":
            return {"bytes": 8 * px + 2 * params, "flops": flops}
        return {"bytes": 12 * px + 8 * params, "flops": 3 * flops}
    n = case["ny"] * case["nx"]
    fft = 5 * n * math.log2(n)
    if kind == "shifts":  # two real forward transforms and one real inverse
        return {"bytes": 8 * case["nz"] * n, "flops": case["nz"] * (1.5 * fft + 6 * n)}
    return {"bytes": 8 * case["nz"] * n, "flops": case["nz"] * (2 * fft + 8 * n)}


# ------------------------------------------------------------------------------------------
# the same in 64 bits, plain torch


def _mask(r):
    nx = int(round(2 * r + 1))
    i = np.arange(nx)
    t = np.trunc(i - r).astype(np.int64) ** 2
    return t[:, None] + t[None, :] <= int(r * r)  # [iz][ix]


def _pixels(r):
    """Pixel-centre offsets (x, z) of the cylinder's rays, row by row."""
    iz, ix = np.nonzero(_mask(r))
    return ix - r, iz - r


class _Exact:
    """The projector pair of a case in 64 bits, by gathers over ray and bin indices."""

    def __init__(self, case):
        self.w, self.nx, self.na = case["weighting"], case["nx"], case["na"]
        r = 0.5 * (self.nx - 1)
        if self.w == "lin":
            # the reference's shifted reads of its coordinate table (two past the end are zero)
            iz, ix = np.nonzero(_mask(r))
            cord = np.concatenate([np.stack([ix, iz], 1).ravel(), np.zeros(4, np.int64)])
            k = 2 * np.arange(ix.size)
            self.r = int(r) + 1
            xs, zs = cord[k + 3] - self.r, cord[k + 4] - self.r
        else:
            self.r = r
            xs, zs = _pixels(r)
        self.xs = torch.tensor(xs, dtype=torch.float64, device="cuda")
        self.zs = torch.tensor(zs, dtype=torch.float64, device="cuda")
        self.ang = _angles(self.na)
        if self.w == "kb":
            path = os.path.join(os.path.dirname(gb.__file__), "csrc", "kb_lut_table.inc")
            with open(path) as f:
                text = re.sub(r"/\*.*?\*/", "", f.read(), flags=re.S)
            lut = [float.fromhex(v.strip().rstrip("f")) for v in text.split(",") if v.strip()]
            self.lut = torch.tensor(lut, dtype=torch.float64, device="cuda")
        self.j = torch.arange(3, device="cuda")
        step = max(1, int(3e7 / (3 * self.xs.numel())))
        self.chunks = [(a, min(self.na, a + step)) for a in range(0, self.na, step)]

    def taps(self, a):
        """(first bin, its weight and the next two) of every ray at angle a."""
        phi = self.ang[a]
        c, s = float(np.cos(phi)), float(np.sin(phi))  # float32 cosines, as the reference's
        xb = self.xs * c + self.zs * s + self.r
        if self.w == "lin":
            xb = xb.float().double()
            fl = torch.floor(xb)
            d = xb - fl
            return fl.long() - 1, torch.stack([1 - d, d, torch.zeros_like(d)], 1)
        iq = torch.round(xb)
        if self.w == "kb":
            t = (xb - iq)[:, None] - (self.j - 1)
            t = t.abs() / float(np.float32(3.0 / 999))
            i = t.long().clamp(max=510)
            t = t - i
            return iq.long() - 1, self.lut[i] * (1 - t) + self.lut[i + 1] * t
        cd, sd = math.cos(float(phi)), math.sin(float(phi))
        p, q = abs(0.5 * (cd - sd)), abs(0.5 * (cd + sd))
        lo, hi = min(p, q), max(p, q) + 1e-6
        top = 1 / ((hi - lo) + 2 * lo)

        def cdf(x):
            lin = top * x + 0.5 * top * (hi + lo)
            k = 0.5 * top / (hi - lo)
            v = torch.where(x > 0, 1 - k * (hi - x) ** 2, k * (x + hi) ** 2)
            v = torch.where(x.abs() < lo + 1e-3, lin, v)
            return torch.where(x > hi, torch.ones_like(x),
                               torch.where(x < -hi, torch.zeros_like(x), v))

        xv = iq - xb
        f1, f2 = cdf(xv - 0.5), cdf(xv + 0.5)
        return iq.long() - 1, torch.stack([f1, f2 - f1, 1 - f2], 1)

    def entries(self, a0, a1):
        """Flat bin index (angle after a0, bin) and weight of every ray's taps; bins off the
        detector have weight zero."""
        bins, ws = [], []
        for a in range(a0, a1):
            b, w = self.taps(a)
            b = b[:, None] + self.j
            on = (b >= 0) & (b < self.nx)
            ws.append(torch.where(on, w, torch.zeros_like(w)))
            bins.append(torch.where(on, b, torch.zeros_like(b)) + (a - a0) * self.nx)
        return torch.stack(bins, 1), torch.stack(ws, 1)  # [nrays][angles][3]

    def project(self, x):
        out = []
        n = self.xs.numel()
        ray = torch.arange(n, device="cuda")[:, None, None]
        for a0, a1 in self.chunks:
            b, w = self.entries(a0, a1)
            flat, order = torch.sort(b.reshape(-1))
            rays = ray.expand(b.shape).reshape(-1)[order]
            off = torch.searchsorted(flat, torch.arange((a1 - a0) * self.nx, device="cuda"))
            out.append(torch.nn.functional.embedding_bag(rays, x, off, mode="sum",
                                                         per_sample_weights=w.reshape(-1)[order]))
        return torch.cat(out).view(self.na, self.nx, -1)

    def back(self, s):
        g = torch.zeros(self.xs.numel(), s.shape[2], dtype=torch.float64, device="cuda")
        for a0, a1 in self.chunks:
            b, w = self.entries(a0, a1)
            n = b.shape[0]
            g += torch.nn.functional.embedding_bag(
                b.view(n, -1), s[a0:a1].reshape(-1, s.shape[2]), mode="sum",
                per_sample_weights=w.view(n, -1))
        return g


def _exact_cgls(P, b, iters):
    s, x = b.clone(), None
    g = P.back(s)
    gamma = gamma0 = r0 = None
    rel, best, xbest, ibest = [], None, None, iters - 1
    gamma = float(g.square().sum())
    r0 = best = math.sqrt(gamma)
    x = torch.zeros_like(g)
    p = torch.zeros_like(g)
    for it in range(1, iters + 1):
        p = g + (0.0 if it == 1 else gamma / gamma0) * p
        q = P.project(p)
        alpha = gamma / float(q.square().sum())
        x = x + alpha * p
        s = s - alpha * q
        g = P.back(s)
        gamma0, gamma = gamma, float(g.square().sum())
        rel.append(math.sqrt(gamma) / r0)
        if math.sqrt(gamma) < best:
            best, xbest, ibest = math.sqrt(gamma), x, it
    if ibest < iters - 1:  # the reference gives the best iterate back
        x = xbest
    return x, np.array(rel)


def _exact_sirt(P, b, lam, iters):
    atb = P.back(b)
    norm = math.sqrt(float(atb.square().sum()))
    lam = float(np.float32(lam))
    x = torch.zeros_like(atb)
    rel = []
    for it in range(iters):
        grad = atb if it == 0 else atb - P.back(P.project(x))
        rel.append(math.sqrt(float(grad.square().sum())) / norm)
        x = x + lam * grad
    return x, np.array(rel)


def _exact_fbp(P, b):
    nx, na = P.nx, P.na
    d = torch.arange(nx, device="cuda", dtype=torch.float64)
    h = torch.where(d % 2 == 1, -1 / (math.pi * d.clamp(min=1)) ** 2, torch.zeros_like(d))
    h[0] = 0.25
    i = torch.arange(nx, device="cuda")
    H = h[(i[:, None] - i[None, :]).abs()] * (math.pi / na)
    f = torch.matmul(H, b)
    return P.back(f), f, P.back(b).square().sum().reshape(1)


def _exact_unet(case, x, dout=None):
    F = torch.nn.functional
    p = _params().double()
    ws, at = [], 0
    for ci, co, _ in _CONV:
        w = p[at:at + 9 * ci * co].view(co, 3, 3, ci).permute(0, 3, 1, 2).contiguous()
        at += 9 * ci * co
        ws.append((w, p[at:at + co].clone()))
        at += (co + 7) // 8 * 8
    w, at = p[at:at + 32].clone().view(1, 32, 1, 1), at + 32
    ws.append((w, p[at:at + 1].clone()))
    if dout is not None:
        for w, b in ws:
            w.requires_grad_()
            b.requires_grad_()

    def conv(l, t):
        return F.relu(F.conv2d(t, ws[l][0], ws[l][1], padding=1))

    def up(t):
        return F.interpolate(t, scale_factor=2, mode="nearest")

    t = x.double()[:, None]
    e1 = conv(1, conv(0, t))
    e2 = conv(3, conv(2, F.max_pool2d(e1, 2)))
    e3 = conv(5, conv(4, F.max_pool2d(e2, 2)))
    e4 = conv(7, conv(6, F.max_pool2d(e3, 2)))
    g3 = conv(10, conv(9, torch.cat([conv(8, up(e4)), e3], 1)))
    g2 = conv(13, conv(12, torch.cat([conv(11, up(g3)), e2], 1)))
    g1 = conv(16, conv(15, torch.cat([conv(14, up(g2)), e1], 1)))
    y = (F.conv2d(g1, ws[17][0], ws[17][1]) + t)[:, 0]
    if dout is None:
        return y
    y.backward(dout.double())
    flat = []
    for w, b in ws:
        flat.append(w.grad.permute(0, 2, 3, 1).reshape(-1))
        flat.append(F.pad(b.grad, (0, -b.numel() % 8)))
    return y.detach(), torch.cat(flat)


def _exact_shift(a, b):
    """Sub-pixel position of the correlation's peak: whole pixel, 3 x 3 paraboloid, wrapped."""
    ny, nx = a.shape
    c = torch.fft.ifft2(torch.fft.fft2(a.double()).conj() * torch.fft.fft2(b.double())).real
    iy, ix = divmod(int(c.abs().argmax()), nx)
    z = c[[(iy - 1) % ny, iy, (iy + 1) % ny]][:, [(ix - 1) % nx, ix, (ix + 1) % nx]].cpu().numpy()
    gy, gx = np.mgrid[-1:2, -1:2]
    A = np.stack([np.ones(9), gx.ravel(), gy.ravel(), (gx * gx).ravel(), (gx * gy).ravel(),
                  (gy * gy).ravel()], 1)
    _, bx, by, xx, xy, yy = np.linalg.lstsq(A, z.ravel(), rcond=None)[0]
    dx, dy = np.linalg.solve([[2 * xx, xy], [xy, 2 * yy]], [-bx, -by])
    sx, sy = ix + min(1, max(-1, dx)), iy + min(1, max(-1, dy))
    return sx - nx * (sx > nx // 2), sy - ny * (sy > ny // 2)


def exact(case, seed):
    kind = case["kind"]
    if kind == "unet" and case["batch"] * case["size"] ** 2 > 1 << 21:
        return None  # too long in 64 bits
    st = prepare(case, seed)
    if kind in ("unet", "unet_grad"):
        return _exact_unet(case, st["x"], st.get("dout"))
    if kind == "shifts":
        s = [_exact_shift(a, b) for a, b in zip(st["a"], st["b"])]
        return np.array([v[0] for v in s]), np.array([v[1] for v in s]), None, None
    if kind == "fshift":
        ny, nx = case["ny"], case["nx"]
        ky = torch.fft.fftfreq(ny, device="cuda", dtype=torch.float64)[:, None]
        kx = torch.fft.fftfreq(nx, device="cuda", dtype=torch.float64)[None, :]
        out = torch.empty(st["a"].shape, dtype=torch.float64, device="cuda")
        for z in range(case["nz"]):
            ph = -2 * math.pi * (float(st["sx"][z]) * kx + float(st["sy"][z]) * ky)
            f = torch.fft.fft2(st["a"][z].double()) * torch.polar(torch.ones_like(ph), ph)
            out[z] = torch.fft.ifft2(f).real
        return out
    P = _Exact(case)
    if kind == "project":
        return P.project(st["x"].double())
    b = st["b"].double()
    if kind == "backproject":
        return P.back(b)
    if kind == "fbp":
        return _exact_fbp(P, b)
    if kind == "cgls":
        x, rel = _exact_cgls(P, b, case["iters"])
    else:
        x, rel = _exact_sirt(P, b, _step(case), case["iters"])
    return x, rel, None
