"""Performance cases: the calls that users of deepmr_b200 make, over the range of sizes they make them at.

A case is a dict of plain values. ``op`` names the call:

  fwd      ``apply_nufft(image, plan)``: simulation, the data-consistency residual
  adj      ``apply_nufft_adj(kspace, plan, weight=dcf)``: gridding reconstruction
  adj_det  the same with bitwise reproducible gridding
  lowrank  ``apply_nufft_adj(kspace, plan, basis=...)``: subspace coefficients of a
           time series
  selfadj  ``apply_nufft_selfadj(image, toeplitz_kernel)``: the normal operator of
           an iterative reconstruction
  cg       ``cg_sense(...)`` with the plan and the Toeplitz kernel in hand: one
           whole reconstruction
  grad     one training step on an image and a trajectory: loss ``|A x - y|^2``
           and both gradients; the plan is made in the step, since the
           trajectory moves

``exact`` restates the same transforms (float32 rescaled coordinates, the
Kaiser-Bessel weights, apodisation, FFT) in 64 bits with plain torch.
"""

import math

import numpy as np
import torch

import deepmr_b200.fft as F
from deepmr_b200 import recon

GOLDEN = math.pi * (math.sqrt(5.0) - 1.0) / 2.0


def listed():
    return [
        # a navigator or preview frame: one coil, one small slice, latency only
        dict(name="fwd2d_64_1coil", op="fwd", ndim=2, n=64, coils=1, views=48, samples=128, width=4, os=1.25, frames=1),
        # one 2D golden-angle slice, the 2D workload of the benchmark (width 3, oversampling 2)
        dict(name="adj2d_128_8coil", op="adj", ndim=2, n=128, coils=8, views=256, samples=256, width=3, os=2.0, frames=1),
        # 500 spiral frames of uneven length (dynamic imaging), both directions
        dict(name="fwd2d_224_500frames", op="fwd", ndim=2, n=224, coils=16, views=1, samples=1000, width=4, os=1.25,
             frames=500),
        dict(name="adj2d_224_500frames", op="adj", ndim=2, n=224, coils=16, views=1, samples=1000, width=4, os=1.25,
             frames=500),
        # subspace reconstruction of a time series (fingerprinting, T2 mapping)
        dict(name="lowrank2d_192_120frames", op="lowrank", ndim=2, n=192, coils=8, views=4, samples=384, width=4, os=1.25,
             frames=120, ncoeff=5),
        # learned sampling: loss and gradients with respect to image and trajectory
        dict(name="grad2d_256_12coil", op="grad", ndim=2, n=256, coils=12, views=402, samples=512, width=4, os=1.25,
             frames=1),
        # one request of the reconstruction server
        dict(name="cg2d_256_16coil", op="cg", ndim=2, n=256, coils=16, views=256, samples=512, width=4, os=1.25, frames=1,
             iters=20),
        # 3D kooshball, 32 coils: the headline workload, both directions
        dict(name="fwd3d_192_32coil", op="fwd", ndim=3, n=192, coils=32, views=50000, samples=384, width=4, os=1.25,
             frames=1),
        dict(name="adj3d_192_32coil", op="adj", ndim=3, n=192, coils=32, views=50000, samples=384, width=4, os=1.25,
             frames=1),
        # 3D with an odd matrix and few (compressed) coils, forward
        dict(name="fwd3d_101_5coil", op="fwd", ndim=3, n=101, coils=5, views=9001, samples=211, width=5, os=1.5, frames=1),
        # reproducible gridding of a mid-size acquisition
        dict(name="adjdet3d_128_12coil", op="adj_det", ndim=3, n=128, coils=12, views=16001, samples=256, width=4, os=1.25,
             frames=1),
        # 3D iterative reconstruction: the Toeplitz normal operator
        dict(name="selfadj3d_144_8coil", op="selfadj", ndim=3, n=144, coils=8, views=6000, samples=288, width=4, os=1.25,
             frames=1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["fwd", "fwd", "adj", "adj", "adj_det", "lowrank", "selfadj", "cg", "grad"])
    kind = rng.choice(["2d", "frames", "3d", "3d"]) if op in ("fwd", "adj") else op
    width, os = rng.choice([(4, 1.25), (4, 1.25), (3, 2.0), (5, 1.5)])
    if kind == "2d":
        n = _log(rng, 48, 384)
        return dict(op=op, ndim=2, n=n, coils=_log(rng, 1, 32), views=_log(rng, max(8, n // 4), 2 * n),
                    samples=n + rng.randrange(n + 1), width=width, os=os, frames=1)
    if kind == "frames":
        n = _log(rng, 96, 224)
        return dict(op=op, ndim=2, n=n, coils=_log(rng, 2, 16), views=rng.choice([1, 1, 3]),
                    samples=rng.randrange(400, 1400), width=4, os=1.25, frames=_log(rng, 20, 400))
    if kind in ("3d", "adj_det"):
        n = _log(rng, 48, 176)
        coils = _log(rng, 1, 32)
        return dict(op=op, ndim=3, n=n, coils=coils, views=_log(rng, n * n // 3, n * n), samples=n + rng.randrange(n),
                    width=width, os=os if n <= 144 else 1.25, frames=1)
    if kind == "lowrank":
        n = _log(rng, 96, 224)
        return dict(op=op, ndim=2, n=n, coils=_log(rng, 2, 12), views=rng.randrange(1, 6), samples=2 * n, width=4, os=1.25,
                    frames=_log(rng, 24, 160), ncoeff=rng.randrange(3, 9))
    if kind == "selfadj":
        n = _log(rng, 48, 160)
        return dict(op=op, ndim=3, n=n, coils=_log(rng, 1, 16), views=_log(rng, n * n // 12, n * n // 3), samples=2 * n,
                    width=4, os=1.25, frames=1)
    if kind == "cg":
        n = rng.choice([128, 192, 256, 320, _log(rng, 96, 320)])
        return dict(op=op, ndim=2, n=n, coils=rng.choice([8, 12, 16, 32]), views=_log(rng, n // 2, 2 * n), samples=2 * n,
                    width=4, os=1.25, frames=1, iters=20)
    n = _log(rng, 64, 288)
    return dict(op="grad", ndim=2, n=n, coils=_log(rng, 2, 16), views=_log(rng, n // 2, 2 * n), samples=2 * n, width=4,
                os=1.25, frames=1)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _trajectory(c, seed):
    """Golden-angle radial (2D), golden-means kooshball (3D) or one rotated
    spiral set per frame, coordinates (views, samples, ndim) in grid units; a
    list of uneven frames when there are several single-shot frames."""
    dev = torch.device("cuda")
    f64 = dict(dtype=torch.float64, device=dev)
    n, rot = c["n"], 0.1 + 0.37 * (seed % 997)
    if c["frames"] > 1:
        g = torch.Generator().manual_seed(c["frames"])
        out = []
        for f in range(c["frames"]):
            m = c["samples"]
            if c["views"] == 1:  # lengths within 20 % of the nominal, the same for every seed
                m = int(m * (0.8 + 0.4 * torch.rand(1, generator=g).item()))
            t = torch.arange(m, dtype=torch.float64) / m
            v = torch.arange(c["views"], dtype=torch.float64)[:, None]
            r = 0.4999 * t**1.5
            phi = 2 * math.pi * (n / 8) * t + rot + (f + 2 * math.pi * v / c["views"]) * GOLDEN
            out.append((torch.stack([r * torch.cos(phi), r * torch.sin(phi)], -1) * n).float())
        if c["views"] == 1:
            return [o[0].to(dev) for o in out]
        return torch.stack(out).to(dev)
    i = torch.arange(c["views"], **f64)
    r = torch.arange(c["samples"], **f64) / c["samples"] - 0.5
    if c["ndim"] == 2:
        phi = rot + i * GOLDEN
        d = torch.stack([torch.cos(phi), torch.sin(phi)], -1)
    else:
        cz = torch.remainder(rot + i * 0.4656, 1.0)
        az = 2 * math.pi * torch.remainder(i * 0.6823 + rot, 1.0)
        sz = torch.sqrt(1 - cz * cz)
        d = torch.stack([sz * torch.cos(az), sz * torch.sin(az), cz], -1)
    return (d[:, None, :] * r[None, :, None] * n).float()


def _flat(coord):
    """Samples (total, ndim) and the first sample of each frame."""
    if isinstance(coord, list):
        offs = np.cumsum([0] + [p.shape[0] for p in coord])
        return torch.cat(coord, 0), offs
    if coord.dim() == 4:
        per = coord.shape[1] * coord.shape[2]
        return coord.reshape(-1, coord.shape[-1]), np.arange(coord.shape[0] + 1) * per
    return coord.reshape(-1, coord.shape[-1]), np.asarray([0, coord.shape[0] * coord.shape[1]])


def _noise(shape, gen):
    return torch.view_as_complex(torch.randn(tuple(shape) + (2,), generator=gen, device="cuda") * 0.5**0.5)


def _image(c, gen, lead):
    """Coil images: an object that fills the field of view and falls off towards its edge, with random texture."""
    n, ndim = c["n"], c["ndim"]
    x = torch.linspace(-1, 1, n, device="cuda")
    r2 = sum(((x * x) / 0.8).reshape([-1 if b == a else 1 for b in range(ndim)]) for a in range(ndim))
    img = _noise(tuple(lead) + (n,) * ndim, gen)
    return img.mul_(torch.exp(-r2 * r2) + 0.02)


def _kspace(c, gen, flat, batch):
    """Samples whose magnitude falls with the distance from the centre, over a noise floor."""
    r = flat.norm(dim=-1) / c["n"]
    env = 1.0 / (1.0 + (12.0 * r) ** 2) + 0.01
    k = _noise((batch, flat.shape[0]), gen)
    return k.mul_(env)


def _dcf(flat):
    r = flat.norm(dim=-1)
    return r / r.max() + 1e-3


def _maps(c, gen):
    """Smooth coil sensitivities with unit root sum of squares."""
    n, k = c["n"], c["coils"]
    x = torch.linspace(-1, 1, n, device="cuda")
    p = torch.rand(k, 6, generator=gen, device="cuda")
    ang = torch.arange(k, device="cuda") * (2 * math.pi / k) + p[:, 0]
    cx, cy = 1.1 * torch.cos(ang), 1.1 * torch.sin(ang)
    r2 = (x[None, None, :] - cx[:, None, None]) ** 2 + (x[None, :, None] - cy[:, None, None]) ** 2
    ph = 2 * p[:, 1, None, None] * x[None, None, :] + 2 * p[:, 2, None, None] * x[None, :, None] + 6 * p[:, 3, None, None]
    m = torch.polar(torch.exp(-r2 / 1.5), ph)
    return m / torch.sqrt((m.abs() ** 2).sum(0, keepdim=True))


def _inputs(c, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    coord = _trajectory(c, seed)
    flat, offs = _flat(coord)
    op, k = c["op"], c["coils"]
    kshape = (k,) + (tuple(coord.shape[:-1]) if not isinstance(coord, list) else (flat.shape[0],))
    d = dict(coord=coord, flat=flat, offs=offs)
    if op in ("fwd", "selfadj"):
        d["x"] = _image(c, gen, (k,) if c["frames"] == 1 else (k, c["frames"]))
    if op in ("adj", "adj_det", "lowrank", "cg"):
        d["y"] = _kspace(c, gen, flat, k).reshape(kshape)
        d["dcf"] = _dcf(flat).reshape(kshape[1:])
    if op == "lowrank":
        t = torch.linspace(0.05, 1, c["frames"], device="cuda")
        rates = torch.linspace(0.5, 8, 3 * c["ncoeff"], device="cuda") + torch.rand(1, generator=gen, device="cuda")
        u = torch.linalg.svd(torch.exp(-t[:, None] * rates[None]))[0][:, :c["ncoeff"]]
        d["basis"] = u.t().contiguous().to(torch.complex64)  # (ncoeff, frames)
    if op == "cg":
        d["maps"] = _maps(c, gen)
        d["y"] = _image_kspace(c, d, gen)
    if op == "selfadj":
        d["dcf"] = _dcf(flat).reshape(coord.shape[:-1])
    if op == "grad":
        d["x"] = _image(c, gen, (k,))
        d["y"] = _kspace(c, gen, flat, k).reshape(kshape)
    return d


def _image_kspace(c, d, gen):
    """Coil k-space for a reconstruction: separable direct transform of a few point-like and box-like parts, plus noise."""
    n = c["n"]
    kx, ky = d["flat"][:, 0].double() / n, d["flat"][:, 1].double() / n
    y = torch.zeros(d["flat"].shape[0], dtype=torch.complex128, device="cuda")
    for a, (w, h, x0, y0) in enumerate(((0.62, 0.78, 0.0, 0.02), (0.2, 0.12, 0.13, -0.1), (0.08, 0.2, -0.2, 0.1))):
        box = torch.sinc(kx * w * n) * torch.sinc(ky * h * n) * (w * h) * (1.0, 0.6, -0.5)[a]
        y += torch.polar(box, -2 * math.pi * (kx * x0 * n + ky * y0 * n))
    # smooth coil weighting changes k-space locally; a per-coil gain and phase stands for it
    g = torch.polar(0.5 + torch.rand(c["coils"], generator=gen, device="cuda"),
                    6.28 * torch.rand(c["coils"], generator=gen, device="cuda"))
    out = (g[:, None].to(torch.complex128) * y * n).to(torch.complex64)
    out += 1e-3 * n * _noise(out.shape, gen)
    return out.reshape(d["y"].shape)


def prepare(case, seed):
    c, d = case, _inputs(case, seed)
    s = dict(case=c)
    if c["op"] != "grad":
        s["plan"] = None if c["op"] == "selfadj" else F.plan_nufft(d["coord"], c["n"], c["width"], c["os"], device="cuda")
    if c["op"] in ("selfadj", "cg"):
        s["gram"] = F.plan_toeplitz_nufft(d["coord"].cpu(), c["n"], dcf=d["dcf"], width=6 if c["op"] == "cg" else 4, device="cuda")
    for k in ("x", "y", "dcf", "basis", "maps"):
        if k in d:
            s[k] = d[k]
    if c["op"] in ("grad", "cg"):
        s["coord"] = d["coord"]
    return s


def run(state):
    s, c = state, state["case"]
    op = c["op"]
    if op == "fwd":
        return F.apply_nufft(s["x"], s["plan"])
    if op == "adj":
        return F.apply_nufft_adj(s["y"], s["plan"], weight=s["dcf"])
    if op == "adj_det":
        old = F.set_deterministic_gridding(True)
        try:
            return F.apply_nufft_adj(s["y"], s["plan"], weight=s["dcf"])
        finally:
            F.set_deterministic_gridding(old)
    if op == "lowrank":
        return F.apply_nufft_adj(s["y"], s["plan"], basis=s["basis"], weight=s["dcf"])
    if op == "selfadj":
        return F.apply_nufft_selfadj(s["x"], s["gram"])
    if op == "cg":
        return recon.cg_sense(s["y"], s["coord"], (c["n"], c["n"]), s["maps"], dcf=s["dcf"], niter=c["iters"], lamda=0.01,
                              plan=s["plan"], gram=s["gram"])
    x = s["x"].detach().clone().requires_grad_(True)
    k = s["coord"].detach().clone().requires_grad_(True)
    r = F.nufft(x, k, width=c["width"], oversamp=c["os"], device="cuda") - s["y"]
    loss = (r.real**2 + r.imag**2).sum()
    loss.backward()
    return loss.detach(), x.grad, k.grad


def _total(c):
    return c["frames"] * c["views"] * c["samples"]


def work(case):
    """Compulsory bytes (inputs, coordinates and outputs once) and operations (taps, FFTs of the oversampled grid)."""
    c = case
    m, k, d, fr = _total(c), c["coils"], c["ndim"], c["frames"]
    img, grid = c["n"] ** d, math.ceil(c["os"] * c["n"]) ** d
    taps = 4.0 * m * k * c["width"] ** d  # real weight times complex value, multiply and add
    fft = lambda pts, num: 5.0 * pts * math.log2(max(2, pts)) * num
    if c["op"] in ("fwd", "adj", "adj_det"):
        by = 8.0 * k * fr * img + 8.0 * k * m + 4.0 * d * m + (4.0 * m if c["op"] != "fwd" else 0)
        return dict(bytes=by, flops=taps + fft(grid, k * fr))
    if c["op"] == "lowrank":
        by = 8.0 * k * c["ncoeff"] * img + 8.0 * k * m + 4.0 * (d + 1) * m
        return dict(bytes=by, flops=taps + fft(grid, k * c["ncoeff"]) + 8.0 * k * fr * grid * c["ncoeff"])
    full = (2 * c["n"]) ** d
    if c["op"] == "selfadj":
        return dict(bytes=16.0 * k * img + 8.0 * full, flops=2 * fft(full, k) + 8.0 * full * k)
    if c["op"] == "cg":
        ah = 8.0 * k * m + 4.0 * (d + 1) * m
        it = 8.0 * full + 8.0 * k * img + 10 * 8.0 * img
        return dict(bytes=ah + c["iters"] * it, flops=taps + fft(grid, k) + c["iters"] * (2 * fft(full, k) + 8.0 * full * k))
    by = 3 * 8.0 * k * m + 2 * 8.0 * k * img + 2 * 4.0 * d * m
    return dict(bytes=by, flops=(2 + 1 + d) * taps + 2 * fft(grid, k))


# ---------------------------------------------------------------------------
# 64-bit restatement
# ---------------------------------------------------------------------------
def _kb(u, beta):
    """I0(beta sqrt(1 - u^2)) by Abramowitz & Stegun 9.8.1 / 9.8.2, zero outside |u| <= 1."""
    a2 = beta * beta * (1 - u * u)
    t2 = a2 / 3.75**2
    small = 1 + t2 * (3.5156229 + t2 * (3.0899424 + t2 * (1.2067492 + t2 * (0.2659732 + t2 * (0.0360768 + t2 * 0.0045813)))))
    a = torch.sqrt(a2.clamp_min(3.75**2))
    v = 3.75 / a
    p = 0.00392377
    for q in (-0.01647633, 0.02635537, -0.02057706, 0.00916281, -0.00157565, 0.00225319, 0.01328592, 0.39894228):
        p = q + v * p
    large = p * torch.exp(a) / torch.sqrt(a)
    return torch.where(u.abs() > 1, torch.zeros_like(u), torch.where(a2 < 3.75**2, small, large))


class _Exact:
    """Taps, apodisation and grid of a transform, in 64 bits (coordinates rescaled in float32)."""

    def __init__(self, flat, offs, n, ndim, width, os):
        self.nd, self.n, self.W = ndim, n, width
        os32 = np.float32(os)
        self.G = int(math.ceil(np.float32(os32 * np.float32(n))))
        self.beta = float(np.float32(math.pi * (((width / os32) * (os32 - np.float32(0.5))) ** 2 - np.float32(0.8)) ** 0.5))
        self.resc = float(np.float32(np.float32(self.G) / np.float32(n)))
        k = flat * torch.tensor(self.resc, dtype=torch.float32, device=flat.device)
        self.k = (k + float(self.G // 2)).double()
        self.x0 = torch.ceil(self.k - 0.5 * width).long()
        self.offs = offs
        h = np.ceil(-width / 2) + np.arange(width)
        self.scale = float(_kb(torch.tensor(h / (width / 2)), self.beta).sum()) ** ndim
        i = torch.arange(n, dtype=torch.float64, device=flat.device) - n // 2
        a = torch.sqrt((self.beta**2 - (math.pi * width * i / self.G) ** 2).to(torch.complex128))
        a = (a / torch.sinh(a)).real
        self.apod = a / a[n // 2]
        self.frames = len(offs) - 1
        self.pts = self.G**ndim
        f = torch.bucketize(torch.arange(flat.shape[0], device=flat.device),
                            torch.as_tensor(np.asarray(offs[1:]), device=flat.device), right=True)
        self.fbase = f * self.pts

    def taps(self, lo, hi, k=None):
        """(index, weight) of each tap of samples lo..hi."""
        kk = (self.k if k is None else k)[lo:hi]
        ax = []
        for a in range(self.nd):  # x, y[, z]
            ax.append([])
            for t in range(self.W):
                x = self.x0[lo:hi, a] + t
                w = _kb((x.double() - kk[:, a]) / (self.W / 2), self.beta)
                ax[a].append((torch.remainder(x - self.G // 2, self.G), w))
        for t in np.ndindex(*([self.W] * self.nd)):
            idx, w = self.fbase[lo:hi], 1.0
            stride = 1
            for a in range(self.nd):
                i, wa = ax[a][t[a]]
                idx = idx + i * stride
                stride *= self.G
                w = w * wa
            yield idx, w

    def pos(self):
        return torch.remainder(torch.arange(self.n, device="cuda") - self.n // 2, self.G)

    def apodise(self, img):
        for a in range(self.nd):
            img = img * self.apod.reshape([-1] + [1] * a)
        return img

    def to_grid(self, img):
        """Grid (frames * points, batch) of images (batch, frames, *n)."""
        b = img.shape[0]
        g = torch.zeros((b, self.frames) + (self.G,) * self.nd, dtype=torch.complex128, device="cuda")
        p = self.pos()
        sel = torch.meshgrid(*([p] * self.nd), indexing="ij")
        g[(slice(None), slice(None)) + tuple(sel)] = self.apodise(img.to(torch.complex128))
        g = torch.fft.fftn(g, dim=tuple(range(2, 2 + self.nd)))
        return g.reshape(b, -1).t().contiguous()

    def interp(self, grid, k=None):
        m, b = self.k.shape[0], grid.shape[1]
        out = torch.zeros((m, b), dtype=torch.complex128, device="cuda")
        step = max(1, (1 << 28) // (16 * b))
        for lo in range(0, m, step):
            hi = min(m, lo + step)
            acc = 0.0
            for idx, w in self.taps(lo, hi, k):
                acc = acc + grid[idx] * w[:, None]
            out[lo:hi] = acc
        return out / self.scale

    def grid(self, y):
        """Grid (frames * points, batch) of samples (total, batch)."""
        m, b = y.shape
        g = torch.zeros((self.frames * self.pts, 2 * b), dtype=torch.float64, device="cuda")
        yr = torch.view_as_real(y.contiguous()).reshape(m, 2 * b)
        step = max(1, (1 << 28) // (16 * b))
        for lo in range(0, m, step):
            hi = min(m, lo + step)
            for idx, w in self.taps(lo, hi):
                g.index_add_(0, idx, yr[lo:hi] * w[:, None])
        return torch.view_as_complex(g.reshape(-1, b, 2)) / self.scale

    def from_grid(self, g):
        """Images (batch, frames, *n) of a grid (frames * points, batch)."""
        b = g.shape[1]
        g = g.t().reshape((b, -1) + (self.G,) * self.nd)
        p = self.pos()
        sel = torch.meshgrid(*([p] * self.nd), indexing="ij")
        g = torch.fft.ifftn(g, dim=tuple(range(2, 2 + self.nd)))
        return self.apodise(g[(slice(None), slice(None)) + tuple(sel)])


def _exact_gram(d, n, ndim, width):
    """Toeplitz kernel: normalised transform of the point spread function on the doubled grid."""
    e = _Exact((d["flat"].double() * 2).float(), d["offs"], 2 * n, ndim, width, 1.25)
    psf = e.from_grid(e.grid(d["dcf"].reshape(-1, 1).to(torch.complex128)))[0, 0]
    dims = tuple(range(ndim))
    k = torch.fft.fftn(torch.fft.ifftshift(psf, dim=dims), dim=dims, norm="ortho")
    return k / k.abs()[k != 0].mean()


def _exact_selfadj(x, kern, ndim):
    n, big = x.shape[-1], kern.shape[-1]
    o = big // 2 - n // 2
    dims = tuple(range(-ndim, 0))
    sl = (Ellipsis,) + (slice(o, o + n),) * ndim
    g = torch.zeros(x.shape[:-ndim] + kern.shape, dtype=torch.complex128, device="cuda")
    g[sl] = x
    return torch.fft.ifftn(torch.fft.fftn(g, dim=dims) * kern, dim=dims)[sl]


def exact(case, seed):
    c, d = case, _inputs(case, seed)
    n, nd, op = c["n"], c["ndim"], c["op"]
    if op == "selfadj":
        kern = _exact_gram(d, n, nd, 4)
        return torch.stack([_exact_selfadj(x.to(torch.complex128), kern, nd) for x in d["x"]])
    e = _Exact(d["flat"], d["offs"], n, nd, c["width"], c["os"])
    if op == "fwd":
        x = d["x"] if c["frames"] > 1 else d["x"][:, None]
        y = e.interp(e.to_grid(x)).t()
        shape = (c["coils"], y.shape[1]) if isinstance(d["coord"], list) else (c["coils"],) + tuple(d["coord"].shape[:-1])
        return y.reshape(shape).contiguous()
    if op in ("adj", "adj_det", "lowrank", "cg"):
        w = d["dcf"].reshape(-1).double()
        g = e.grid((d["y"].reshape(c["coils"], -1).to(torch.complex128) * w).t())
        if op == "lowrank":
            g = torch.einsum("cf,fpb->cpb", d["basis"].to(torch.complex128), g.reshape(e.frames, e.pts, -1))
            return e.from_grid(g.reshape(-1, g.shape[-1]))
        x = e.from_grid(g)
        if op != "cg":
            return x if c["frames"] > 1 else x[:, 0]
        kern = _exact_gram(d, n, nd, 6)
        maps = d["maps"].to(torch.complex128)
        aha = lambda v: (maps.conj() * _exact_selfadj(maps * v, kern, nd)).sum(0) + 0.01 * v
        r = (maps.conj() * x[:, 0]).sum(0)
        sol, p, rs = torch.zeros_like(r), r.clone(), (r.abs() ** 2).sum()
        for _ in range(c["iters"]):
            q = aha(p)
            alpha = rs / (p.conj() * q).sum()
            sol, r = sol + alpha * p, r - alpha * q
            new = (r.abs() ** 2).sum()
            p, rs = r + (new / rs) * p, new
        return sol
    k = e.k.clone().requires_grad_(True)
    grid = e.to_grid(d["x"][:, None])
    y = d["y"].reshape(c["coils"], -1).t().to(torch.complex128)
    r = e.interp(grid, k) - y
    loss = (r.real**2 + r.imag**2).sum()
    gk = torch.autograd.grad(loss, k)[0] * e.resc
    gx = e.from_grid(e.grid(2 * r.detach()))[:, 0]
    return loss.detach(), gx, gk.reshape(d["coord"].shape)
