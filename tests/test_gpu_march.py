"""GPU parity of the 3D kernels on coil-interleaved grids (interpolation,
gridding, deterministic gridding) at the sizes where their tiles, lane groups
and chunks have remainders: widths 2..6, coil counts around each lane-group
boundary and across a 32-coil chunk, grids that are no multiple of a tile, that
wrap, and that are smaller than a tile's region, compiled FFT lengths and cuFFT
ones, frames, real k-space with per-coil weights, and planar C-ABI grids.

Tolerance: relative L2 error <= 1e-5 in float32, as in the other parity tests
(weights, sums and FFT in float32 stay near 1e-6).
"""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

TOL = 1e-5


def rel(a, b):
    a = np.asarray(torch.as_tensor(a).detach().cpu(), dtype=np.complex128).ravel()
    b = np.asarray(torch.as_tensor(b).detach().cpu(), dtype=np.complex128).ravel()
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def _coord(shape, nsamples, seed, lead=()):
    """Random samples over the whole band, a dense cluster at the centre (split
    work units) and samples on the band's edges (taps that wrap)."""
    rng = np.random.default_rng(seed)
    n = np.asarray(shape[::-1], dtype=np.float64)
    c = rng.uniform(-0.5, 0.5, lead + (nsamples, 3)) * n
    c[..., : nsamples // 2, :] *= 0.02
    c[..., -8:, :] = np.sign(c[..., -8:, :]) * n * 0.4999
    return c[..., None, :, :].astype(np.float32) if lead else c[None].astype(np.float32)


CASES = [
    # shape, width, oversampling, coils
    ((16, 12, 20), 4, 1.25, (1, 2, 3, 4, 5, 8, 9, 16, 17, 33)),
    ((13, 9, 11), 3, 2.0, (1, 3, 4, 10, 11, 17)),
    ((10, 14, 9), 5, 1.5, (1, 2, 3, 4, 6, 7, 13)),
    ((12, 10, 8), 2, 2.0, (1, 8, 9, 20)),
    ((9, 11, 10), 6, 2.0, (1, 5, 6, 18)),
    ((5, 4, 6), 4, 1.25, (1, 6, 20)),  # grid (7, 5, 8): smaller than a tile's region
]


@pytest.mark.parametrize("shape,width,os,coils", CASES, ids=[f"w{c[1]}-{'x'.join(map(str, c[0]))}" for c in CASES])
def test_march_vs_oracle(shape, width, os, coils):
    import deepmr_b200.fft as F
    from deepmr_b200 import synth
    from oracle import nufft_ref as R

    c = torch.as_tensor(_coord(shape, 1500, seed=width))
    plan = F.plan_nufft(c, shape, width, os, device="cuda")
    oplan = R.plan_nufft(c, shape, width, os)
    most = max(coils)
    img = synth.complex_gaussian((most,) + shape, seed=1)
    ksp = synth.complex_gaussian((most,) + tuple(c.shape[:-1]), seed=2)
    w = torch.rand(tuple(c.shape[:-1]), generator=torch.Generator().manual_seed(3))
    y_ref = R.apply_nufft(img, oplan)
    x_ref = R.apply_nufft_adj(ksp, oplan, weight=w)
    for k in coils:
        assert rel(F.apply_nufft(img[:k].cuda(), plan), y_ref[:k]) < TOL, k
        assert rel(F.apply_nufft_adj(ksp[:k].cuda(), plan, weight=w.cuda()), x_ref[:k]) < TOL, k
        old = F.set_deterministic_gridding(True)
        try:
            x = F.apply_nufft_adj(ksp[:k].cuda(), plan, weight=w.cuda())
            x2 = F.apply_nufft_adj(ksp[:k].cuda(), plan, weight=w.cuda())
        finally:
            F.set_deterministic_gridding(old)
        assert rel(x, x_ref[:k]) < TOL, k
        assert torch.equal(x, x2), k


@pytest.mark.parametrize("det", [False, True], ids=["atomic", "deterministic"])
def test_march_frames_real_weights_and_planar(det):
    """Frames, real k-space and per-coil weights through the public call, and
    the planar C-ABI gridding and interpolation of the same plan."""
    import deepmr_b200.fft as F
    from deepmr_b200 import _lib
    from oracle import nufft_ref as R

    shape, nf, k = (11, 12, 13), 3, 6
    c = torch.as_tensor(_coord(shape, 600, seed=4, lead=(nf,)))
    g = torch.Generator().manual_seed(5)
    y = torch.randn((k, nf) + tuple(c.shape[1:-1]), generator=g)
    w = torch.rand(y.shape, generator=g)
    plan = F.plan_nufft(c, shape, 4, 1.25, device="cuda")
    oplan = R.plan_nufft(c, shape, 4, 1.25)
    old = F.set_deterministic_gridding(det)
    try:
        x = F.apply_nufft_adj(y.cuda(), plan, weight=w.cuda())
    finally:
        F.set_deterministic_gridding(old)
    assert rel(x, R.apply_nufft_adj(y * w, oplan)) < TOL
    ip, L = plan.interpolator, _lib.lib()
    st = _lib.stream_ptr(torch.device("cuda", torch.cuda.current_device()))
    yd, wd = y.cuda(), w.cuda()
    grid = torch.full((k, nf) + tuple(ip.dshape), float("nan"), dtype=torch.complex64, device="cuda")
    _lib.check(L.dmr_grid(ip.handle, _lib.ptr(yd), 1, _lib.ptr(grid), k, _lib.ptr(wd), 1, int(det), st))
    back = torch.empty(y.shape, dtype=torch.complex64, device="cuda")
    _lib.check(L.dmr_interp(ip.handle, _lib.ptr(grid), _lib.ptr(back), k, None, 0, st))
    # <interp(grid(y w)), y w> = |grid(y w)|^2: the two kernels are each other's transpose
    lhs = torch.sum(back.to(torch.complex128) * (yd * wd).to(torch.float64))
    rhs = torch.sum(grid.to(torch.complex128).abs() ** 2)
    assert abs(lhs - rhs) / abs(rhs) < 1e-5


def test_march_nan_stays_in_its_taps():
    """A sample that is not finite reaches the W^3 grid points of its taps and
    no others, for every lane layout."""
    import deepmr_b200.fft as F
    from deepmr_b200 import _lib

    shape = (16, 16, 16)  # grid 20^3
    c = torch.as_tensor(_coord(shape, 400, seed=6))
    c[0, 100] = torch.tensor([0.3, -2.2, 4.1])
    plan = F.plan_nufft(c, shape, 4, 1.25, device="cuda")
    ip, L = plan.interpolator, _lib.lib()
    st = _lib.stream_ptr(torch.device("cuda", torch.cuda.current_device()))
    for k in (1, 5, 12, 20):
        y = torch.ones((k, 400), dtype=torch.complex64, device="cuda")
        y[0, 100] = float("nan")
        for det in (0, 1):
            grid = torch.empty((k,) + tuple(ip.dshape), dtype=torch.complex64, device="cuda")
            _lib.check(L.dmr_grid(ip.handle, _lib.ptr(y), 0, _lib.ptr(grid), k, None, 0, det, st))
            bad = torch.isnan(grid.real)
            assert int(bad[0].sum()) == 64 and int(bad[1:].sum()) == 0, (k, det)


@pytest.mark.parametrize("shape,width,os", [((18, 23), 4, 1.25), ((17, 12), 3, 2.0), ((9, 14), 5, 1.5), ((10, 8), 2, 2.0),
                                            ((11, 9), 6, 2.0), ((32, 32), 4, 1.25), ((4, 5), 4, 1.25)])
@pytest.mark.parametrize("nsamples", [40, 1200], ids=["sparse", "dense"])
def test_2d_vs_oracle(shape, width, os, nsamples):
    """2D: direct interpolation, direct (sparse) and tiled (dense) gridding, both
    modes, around the coil-lane boundaries; samples on the band's edges wrap."""
    import deepmr_b200.fft as F
    from deepmr_b200 import synth
    from oracle import nufft_ref as R

    rng = np.random.default_rng(width)
    n = np.asarray(shape[::-1], dtype=np.float64)
    c = rng.uniform(-0.5, 0.5, (1, nsamples, 2)) * n
    c[:, : nsamples // 2] *= 0.05
    c[:, -8:] = np.sign(c[:, -8:]) * n * 0.4999
    c = torch.as_tensor(c.astype(np.float32))
    plan = F.plan_nufft(c, shape, width, os, device="cuda")
    oplan = R.plan_nufft(c, shape, width, os)
    img = synth.complex_gaussian((34,) + shape, seed=1)
    ksp = synth.complex_gaussian((34,) + tuple(c.shape[:-1]), seed=2)
    w = torch.rand(tuple(c.shape[:-1]), generator=torch.Generator().manual_seed(3))
    y_ref = R.apply_nufft(img, oplan)
    x_ref = R.apply_nufft_adj(ksp, oplan, weight=w)
    for k in (1, 2, 3, 5, 8, 9, 17, 32, 34):
        assert rel(F.apply_nufft(img[:k].cuda(), plan), y_ref[:k]) < TOL, k
        for det in (False, True):
            old = F.set_deterministic_gridding(det)
            try:
                x = F.apply_nufft_adj(ksp[:k].cuda(), plan, weight=w.cuda())
                x2 = F.apply_nufft_adj(ksp[:k].cuda(), plan, weight=w.cuda())
            finally:
                F.set_deterministic_gridding(old)
            assert rel(x, x_ref[:k]) < TOL, (k, det)
            assert not det or torch.equal(x, x2), k


@pytest.mark.parametrize("width,os,shape,coils", [(4, 1.25, (24, 32), (1, 5, 12, 35)), (3, 2.0, (16, 20), (2, 17)),
                                                  (6, 2.0, (11, 13), (1, 34)), (2, 1.5, (18, 9), (3, 33))])
def test_2d_trajectory_gradient_frames_weights(width, os, shape, coils):
    """The 2D gradient kernel around its lane groups and coil chunks, on fused
    FFT lengths (interleaved grids) and cuFFT ones (a planar chunk at a time),
    against central differences of the float64 operator.

    Tolerance 2e-5 of the gradient's norm: the rescaled coordinate is a float32
    up to 48 (rounding 2e-6, times the second derivative, about the first's
    size) and the differences add 1e-8 (step squared) + 1e-9 (1e-13 / step)."""
    import deepmr_b200.fft as F
    from oracle import nufft_ref as R

    nf, npts, most, eps = 2, 30, max(coils), 1e-4
    rng = np.random.default_rng(7)
    n = np.asarray(shape[::-1], dtype=np.float64)
    grid = np.ceil(os * n)
    # samples off the points where the tap set changes
    t = rng.integers(1, grid - 2, (nf, npts, 2)) + (0.5 if width % 2 else 0.0) + rng.uniform(0.05, 0.95, (nf, npts, 2))
    c = ((t - grid // 2) * n / grid).astype(np.float32)
    plan = F.plan_nufft(torch.as_tensor(c[:, None]), shape, width, os, device="cuda")
    gen = torch.Generator().manual_seed(8)
    cplx = lambda *s: torch.complex(torch.randn(s, generator=gen), torch.randn(s, generator=gen))  # noqa: E731
    img, v, w = cplx(most, nf, *shape), cplx(most, nf, 1, npts), torch.rand(nf, 1, npts, generator=gen)
    per_coil = np.zeros((most, nf, npts, 2))  # Re(conj(v) w dy/dc)
    for f in range(nf):
        f64 = R.Forward64(img[:, f].numpy(), c[f][None], shape, width, os)
        for p in range(npts):
            for a in range(2):
                d = np.zeros(2)
                d[a] = eps
                x = c[f, p].astype(np.float64)
                dy = (f64.sample(x + d) - f64.sample(x - d)) / (2 * eps)
                per_coil[:, f, p, a] = np.real(np.conj(v[:, f, 0, p].numpy()) * dy) * float(w[f, 0, p])
    for k in coils:
        got = F.traj_grad(plan, img[:k].cuda(), v[:k].cuda(), weight=w.cuda(), post_scale=0.5)
        assert rel(got.reshape(nf, npts, 2), 0.5 * per_coil[:k].sum(0)) < 2e-5, k


@pytest.mark.parametrize("ndim,shape,nf,ncoeff,coils", [(2, (24, 32), 40, 9, 5), (2, (24, 32), 3, 7, 33),
                                                        (3, (16, 12, 20), 5, 17, 2), (2, (16, 16), 950, 20, 1)])
def test_lowrank_coefficient_counts(ndim, shape, nf, ncoeff, coils):
    """The projection's rounded coefficient counts (4, 8, 16, 32), more
    coefficients than frames, two coil chunks, and a basis that is larger than
    shared memory (950 frames of 20 coefficients), on interleaved grids."""
    import deepmr_b200.fft as F
    from deepmr_b200 import synth
    from oracle import nufft_ref as R

    rng = np.random.default_rng(9)
    c = torch.as_tensor((rng.uniform(-0.49, 0.49, (nf, 1, 60, ndim)) * np.asarray(shape[::-1])).astype(np.float32))
    gen = torch.Generator().manual_seed(10)
    basis = torch.complex(torch.randn(ncoeff, nf, generator=gen), torch.randn(ncoeff, nf, generator=gen))
    img = synth.complex_gaussian((coils, ncoeff) + shape, seed=1)
    ksp = synth.complex_gaussian((coils, nf, 1, 60), seed=2)
    plan = F.plan_nufft(c, shape, 4, 1.25, device="cuda")
    oplan = R.plan_nufft(c, shape, 4, 1.25)
    y = F.apply_nufft(img.cuda(), plan, basis_adjoint=basis.conj().t())
    assert rel(y, R.apply_nufft_lowrank(img, oplan, basis.conj().t())) < TOL
    x = F.apply_nufft_adj(ksp.cuda(), plan, basis=basis)
    assert rel(x, R.apply_nufft_adj_lowrank(ksp, oplan, basis)) < TOL
