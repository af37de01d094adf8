"""Calls at the limits of the interleaved kernels: what they do not take runs on
the other kernels with the same results, and what a plan asks of its caller does
not depend on which calls it has seen.

Tolerance: relative L2 error <= 1e-5 in float32 against float64 sums or the
oracle, as in the other parity tests.
"""

import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

TOL = 1e-5


def rel(a, b):
    a = np.asarray(torch.as_tensor(a).detach().cpu(), dtype=np.complex128).ravel()
    b = np.asarray(torch.as_tensor(b).detach().cpu(), dtype=np.complex128).ravel()
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


class CPlan:
    """A plan through the C ABI with grid extents of its own (the public call keeps
    extents in 16 bits), no oversampling: sample k sits at grid position k + G // 2."""

    def __init__(self, grid, width, coord):
        from deepmr_b200 import _lib

        self.L, self.lib = _lib.lib(), _lib
        self.grid, self.width, self.n, nd = grid, width, len(coord), len(grid)
        self.beta = 2.34 * width
        self.coord = torch.as_tensor(coord).cuda()
        self.handle = ctypes.c_void_p()
        shape, ones = _lib.i32_array(grid), _lib.f32_array([1.0] * nd)
        _lib.check(self.L.dmr_plan_create(
            nd, shape, shape, _lib.i32_array([width] * nd), _lib.f32_array([self.beta] * nd), ones, _lib.ptr(self.coord),
            (ctypes.c_int64 * 2)(0, self.n), 1, None, self.stream(), ctypes.byref(self.handle)))
        # taps of every sample: FFT-order positions and weights, float64 from the float32 coordinate
        idx, w = np.zeros(self.n, dtype=np.int64)[:, None], np.ones((self.n, 1))
        for a in reversed(range(nd)):  # z first: row-major
            G = grid[nd - 1 - a]
            k = (coord[:, a] + np.float32(G // 2)).astype(np.float64)
            x = np.ceil(k - width / 2)[:, None] + np.arange(width)
            u = (x - k[:, None]) / (width / 2)
            wa = np.where(np.abs(u) <= 1, np.i0(self.beta * np.sqrt(np.maximum(1 - u * u, 0))), 0)
            idx = (idx[:, :, None] * G + ((x.astype(np.int64) - G // 2) % G)[:, None, :]).reshape(self.n, -1)
            w = (w[:, :, None] * wa[:, None, :]).reshape(self.n, -1)
        scale = ctypes.c_double()
        _lib.check(self.L.dmr_plan_scale(self.handle, ctypes.byref(scale)))
        self.idx, self.w = idx, w / scale.value

    def stream(self):
        return self.lib.stream_ptr(torch.device("cuda", torch.cuda.current_device()))

    def interp(self, g):
        y = torch.full((g.shape[0], self.n), float("nan"), dtype=torch.complex64, device="cuda")
        self.lib.check(self.L.dmr_interp(self.handle, self.lib.ptr(g), self.lib.ptr(y), len(g), None, 0, self.stream()))
        return y

    def gridding(self, y, det):
        g = torch.full((y.shape[0],) + tuple(self.grid), float("nan"), dtype=torch.complex64, device="cuda")
        self.lib.check(self.L.dmr_grid(self.handle, self.lib.ptr(y), 0, self.lib.ptr(g), len(y), None, 0, int(det),
                                       self.stream()))
        return g

    def exact_interp(self, g):
        g = g.cpu().numpy().astype(np.complex128).reshape(g.shape[0], -1)
        return np.stack([(c[self.idx] * self.w).sum(1) for c in g])

    def exact_gridding(self, y):
        n = int(np.prod(self.grid))
        out = []
        for c in y.cpu().numpy().astype(np.complex128):
            v, i = (c[:, None] * self.w).ravel(), self.idx.ravel()
            out.append(np.bincount(i, v.real, n) + 1j * np.bincount(i, v.imag, n))
        return np.stack(out)

    def close(self):
        self.lib.check(self.L.dmr_plan_destroy(self.handle))


def _samples(grid, n, seed):
    """All over the grid and its last cells on each side."""
    rng = np.random.default_rng(seed)
    ext = np.asarray(grid[::-1], dtype=np.float64)
    c = rng.uniform(-0.5, 0.5, (n, len(grid))) * (ext - 1)
    c[-16:] = np.sign(c[-16:]) * (ext / 2 - rng.uniform(0.5, 3.0, (16, len(grid))))
    return c.astype(np.float32)


@pytest.mark.parametrize("grid", [(8, 65536), (8, 65537), (32768, 8), (32769, 8)], ids=lambda g: f"{g[0]}x{g[1]}")
@pytest.mark.parametrize("nsamples", [300, 140000], ids=["sparse", "dense"])
def test_long_2d_grids(grid, nsamples):
    """The longest grids whose positions fit a 2D record (65,536 x, 32,768 y) and
    the next ones, below and above the density that tiles are used from."""
    from deepmr_b200 import synth

    p = CPlan(grid, 4, _samples(grid, nsamples, 1))
    for k in (1, 3):
        g = synth.complex_gaussian((k,) + grid, seed=1).cuda()
        y = synth.complex_gaussian((k, nsamples), seed=2).cuda()
        assert rel(p.interp(g), p.exact_interp(g)) < TOL, k
        assert rel(p.gridding(y, False), p.exact_gridding(y)) < TOL, k
    p.close()


def test_failed_plan_creation_leaves_nothing_in_flight():
    """Whatever allocation fails while a plan is being made, the call returns only
    when the work on the plan's buffers is done (they are freed on another
    stream), and the next plan is made as ever."""
    import deepmr_b200.fft as F
    from deepmr_b200 import _lib, synth
    from oracle import nufft_ref as R

    c3 = torch.as_tensor(synth.kooshball_3d(60, 32, 16).astype(np.float32))
    c2 = torch.as_tensor(synth.radial_2d(24, 32, 16).astype(np.float32))
    s = torch.cuda.Stream()
    failed = 0
    with torch.cuda.stream(s):
        for c, shape in ((c3, (16, 16, 16)), (c2, (16, 16))):
            args = _plan_args(c, shape)
            for n in range(1, 200):
                torch.cuda._sleep(10_000_000)  # some milliseconds of other work first
                _lib.lib().dmr_plan_test_alloc(n)
                try:
                    h = args()
                except _lib.DmrError as e:
                    assert e.code == -3 and s.query(), n
                    failed += 1
                    continue
                finally:
                    _lib.lib().dmr_plan_test_alloc(0)
                _lib.check(_lib.lib().dmr_plan_destroy(h))
                break
            else:
                pytest.fail("no plan was made")
    assert failed > 20
    img = synth.complex_gaussian((3, 16, 16, 16), seed=1)
    plan = F.plan_nufft(c3, 16, 4, 1.25, device="cuda")
    assert rel(F.apply_nufft(img.cuda(), plan), R.apply_nufft(img, R.plan_nufft(c3, 16, 4, 1.25))) < TOL


def _plan_args(coord, shape):
    """A call that makes a plan of width 4 and oversampling 1.25 on the current
    stream and returns its handle (no other allocations in between)."""
    from deepmr_b200 import _lib

    nd = len(shape)
    flat = coord.reshape(-1, nd).cuda().contiguous()
    torch.cuda.synchronize()

    def make():
        h = ctypes.c_void_p()
        _lib.check(_lib.lib().dmr_plan_create(
            nd, _lib.i32_array(shape), _lib.i32_array([-(-5 * s // 4) for s in shape]), _lib.i32_array([4] * nd),
            _lib.f32_array([7.2] * nd), _lib.f32_array([1.25] * nd), _lib.ptr(flat), (ctypes.c_int64 * 2)(0, len(flat)), 1,
            None, _lib.stream_ptr(flat.device), ctypes.byref(h)))
        return h

    return make


def _problem3(n=24, views=160, samples=64, coils=9):
    """A 3D plan of width 4 whose bin structures are not built, images, k-space."""
    import deepmr_b200.fft as F
    from deepmr_b200 import synth

    c = torch.as_tensor(synth.kooshball_3d(views, samples, n).astype(np.float32))
    plan = F.plan_nufft(c, n, 4, 1.25, device="cuda")
    img = synth.complex_gaussian((coils, n, n, n), seed=1).cuda()
    ksp = synth.complex_gaussian((coils,) + tuple(c.shape[:-1]), seed=2).cuda()
    return plan, img, ksp


def test_bins_build_that_fails_leaves_the_plan_as_it_was():
    """Bin structures that could not be allocated are given back, and the next
    call builds them: any number of failures costs no memory (4 x 80 MB each
    here, were they kept)."""
    import deepmr_b200.fft as F
    from deepmr_b200 import _lib

    rng = np.random.default_rng(3)
    c = torch.as_tensor((rng.uniform(-0.5, 0.5, (1, 20_000_000, 3)) * 64).astype(np.float32))
    plan = F.plan_nufft(c, 64, 4, 1.25, device="cuda")
    img = torch.ones((1, 64, 64, 64), dtype=torch.complex64, device="cuda")
    v = torch.ones((1,) + tuple(c.shape[:-1]), dtype=torch.complex64, device="cuda")
    free = []
    for n in (10,) * 12:  # after the sorted coordinates and indices
        _lib.lib().dmr_plan_test_alloc(n)
        try:
            with pytest.raises(_lib.DmrError) as e:
                F.traj_grad(plan, img, v)
        finally:
            _lib.lib().dmr_plan_test_alloc(0)
        assert e.value.code == -3
        torch.cuda.synchronize()
        free.append(torch.cuda.mem_get_info()[0])
    assert free[1] - free[-1] < 400 << 20, [f >> 20 for f in free]
    g = F.traj_grad(plan, img, v)
    assert torch.isfinite(g).all() and float(g.abs().max()) > 0


def test_threads_on_a_plan_without_bins():
    """Several threads' calls on one plan while one of them builds its bin
    structures: every result is that of a thread alone."""
    import threading

    import deepmr_b200.fft as F

    plan, img, ksp = _problem3()
    adj = F.apply_nufft_adj(ksp, plan)
    fwd = F.apply_nufft(img, plan)
    ref = F.traj_grad(_problem3()[0], img, ksp)
    errors, out = [], {}
    start = threading.Barrier(6)

    def work(i):
        try:
            torch.cuda.set_device(0)
            with torch.cuda.stream(torch.cuda.Stream()):
                start.wait()
                for _ in range(5):
                    out[i] = (F.traj_grad(plan, img, ksp) if i < 2 else
                              F.apply_nufft_adj(ksp, plan) if i < 4 else F.apply_nufft(img, plan))
                torch.cuda.current_stream().synchronize()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(6)]
    torch.cuda.synchronize()
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for i in range(6):
        assert rel(out[i], (ref, ref, adj, adj, fwd, fwd)[i]) < 1e-6, i


@pytest.mark.parametrize("width,os", [(4, 1.25), (6, 1.25)])
def test_workspace_does_not_grow(width, os):
    """A workspace sized before the plan's bin structures were built serves the
    calls after it, all that a plan can make: dense samples (register tiles split
    over blocks), 8 coils and more."""
    import deepmr_b200.fft as F
    from deepmr_b200 import _lib

    L, n, total, k = _lib.lib(), 32, 1_000_000, 8
    rng = np.random.default_rng(4)
    c = torch.as_tensor((rng.uniform(-0.5, 0.5, (1, total, 3)) * n).astype(np.float32))
    plan = F.plan_nufft(c, n, width, os, device="cuda")
    ip = plan.interpolator
    ws, wl = ip.workspace(k), ip.workspace_lowrank(k, 1)
    ksp = torch.ones((k,) + tuple(c.shape[:-1]), dtype=torch.complex64, device="cuda")
    img = torch.ones((k, n, n, n), dtype=torch.complex64, device="cuda")
    one = torch.ones((1, 1), dtype=torch.complex64, device="cuda")
    st = _lib.stream_ptr(ip.device)

    def adjoint(w, det):
        out = torch.empty_like(img)
        _lib.check(L.dmr_nufft_adjoint(ip.handle, _lib.ptr(ksp), 0, _lib.ptr(out), k, None, 0, det, _lib.ptr(w), w.numel(), st))
        return out

    def lowrank(w, det):
        out = torch.empty_like(img)
        _lib.check(L.dmr_nufft_adjoint_lowrank(ip.handle, _lib.ptr(ksp), 0, 1, _lib.ptr(one), _lib.ptr(out), k, None, 0, det,
                                               _lib.ptr(w), w.numel(), st))
        return out

    before = [adjoint(ws, d) for d in (0, 1)] + [lowrank(wl, d) for d in (0, 1)]
    F.traj_grad(plan, img, ksp)  # builds the bins
    assert (ip.workspace(k).numel(), ip.workspace_lowrank(k, 1).numel()) == (ws.numel(), wl.numel())
    after = [adjoint(ws, d) for d in (0, 1)] + [lowrank(wl, d) for d in (0, 1)]
    assert torch.equal(before[1], after[1]) and torch.equal(before[3], after[3])
    old = F.set_deterministic_scratch_limit(1)  # register tiles
    try:
        assert all(torch.isfinite(t).all() for t in after + [adjoint(ws, 1), lowrank(wl, 1)])
    finally:
        F.set_deterministic_scratch_limit(old)


@pytest.mark.parametrize("grid,width,nsamples", [((8, 7264), 4, 20000), ((8, 7265), 4, 20000), ((8, 6400), 6, 24000),
                                                 ((32768, 8), 4, 140000), ((8, 8, 7300), 4, 5000)],
                         ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else str(v))
def test_deterministic_on_wide_grids(grid, width, nsamples):
    """Deterministic gridding on the widest grid that the planes' gather holds in
    shared memory and on wider ones, which the other deterministic kernels take."""
    from deepmr_b200 import synth

    p = CPlan(grid, width, _samples(grid, nsamples, 5))
    for k in (1, 3):
        y = synth.complex_gaussian((k, nsamples), seed=2).cuda()
        g = p.gridding(y, True)
        assert rel(g, p.exact_gridding(y)) < TOL, k
        assert torch.equal(g, p.gridding(y, True)), k
    p.close()


def test_a_reported_error_is_not_reported_again():
    """After an allocation has failed, the next call works (its launches do not
    find the earlier error)."""
    from deepmr_b200 import _lib, synth

    make = _plan_args(torch.as_tensor(synth.kooshball_3d(60, 32, 16).astype(np.float32)), (16, 16, 16))
    _lib.lib().dmr_plan_test_alloc(8)
    try:
        with pytest.raises(_lib.DmrError) as e:
            make()
    finally:
        _lib.lib().dmr_plan_test_alloc(0)
    assert e.value.code == -3
    _lib.check(_lib.lib().dmr_plan_destroy(make()))


@pytest.mark.parametrize("call", ["gradient 3D", "deterministic sparse 2D", "over the scratch limit", "over the limit, 3 coils"])
def test_first_call_that_needs_bins_is_captured(call):
    """A plan's first call that needs its bin structures builds them while it is
    being captured, and the replays give what the call gives by itself."""
    import gc

    import deepmr_b200.fft as F
    from deepmr_b200 import synth

    if call == "deterministic sparse 2D":
        c = torch.as_tensor(synth.radial_2d(6, 64, 32).astype(np.float32))
        make = lambda: F.plan_nufft(c, 32, 4, 1.25, device="cuda")  # noqa: E731
        ksp = synth.complex_gaussian((3,) + tuple(c.shape[:-1]), seed=2).cuda()
    else:
        make = lambda: _problem3()[0]  # noqa: E731
        _, img, ksp = _problem3()
        if call.endswith("3 coils"):
            ksp = ksp[:3].contiguous()
    run = (lambda p: F.traj_grad(p, img, ksp)) if call == "gradient 3D" else (lambda p: F.apply_nufft_adj(ksp, p))
    old = F.set_deterministic_gridding(True), F.set_deterministic_scratch_limit(1 if "limit" in call else 0)
    try:
        ref = run(make())  # (another plan: kernels and tables are loaded)
        plan = make()
        gc.collect()  # (a plan that is destroyed synchronises the device, which a capture forbids)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = run(plan)
        for _ in range(2):
            out.zero_()
            graph.replay()
            assert torch.equal(out, ref)
        assert torch.equal(run(plan), ref)
    finally:
        F.set_deterministic_gridding(old[0])
        F.set_deterministic_scratch_limit(old[1])


@pytest.mark.parametrize("warm,shape", [(None, (187, 209)), ("forward", (221, 143)), ("adjoint", (165, 253))],
                         ids=["cold", "forward warmed", "adjoint warmed"])
def test_captures_of_calls_that_have_not_run(warm, shape):
    """Both directions captured when neither or only the other has run, at
    transform lengths that nothing else here uses (twiddle tables)."""
    import gc

    import deepmr_b200.fft as F
    from deepmr_b200 import synth
    from oracle import nufft_ref as R

    c = torch.as_tensor(synth.radial_2d(30, 64, 64).astype(np.float32))
    plan = F.plan_nufft(c, shape, 4, 2.0, device="cuda")
    img = synth.complex_gaussian((3,) + shape, seed=1)
    ksp = synth.complex_gaussian((3,) + tuple(c.shape[:-1]), seed=2)
    x, y = img.cuda(), ksp.cuda()
    calls = {"forward": lambda: F.apply_nufft(x, plan), "adjoint": lambda: F.apply_nufft_adj(y, plan)}
    if warm:
        calls[warm]()
    gc.collect()
    torch.cuda.synchronize()
    out = {}
    for name, call in calls.items():
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            out[name] = call()
        g.replay()
    torch.cuda.synchronize()
    oplan = R.plan_nufft(c, shape, 4, 2.0)
    assert rel(out["forward"], R.apply_nufft(img, oplan)) < TOL
    assert rel(out["adjoint"], R.apply_nufft_adj(ksp, oplan)) < TOL


@pytest.mark.parametrize("width,n,calls", [(4, 64, (("adj", 17), ("adj", 19))),
                                           (6, 48, (("adj", 18), ("adj", 32), ("adj_det", 3), ("adj_det", 12)))])
def test_rounding_by_coils_and_mode(width, n, calls):
    """Adjoints of samples crowded at the centre (n^2 views, oversampling 1.25): 17 to
    19 coils, and at width 6 any number and either mode, are no further from 64 bits
    than 12 coils are, which are gridded in units of 64 samples. (Units of 512 are
    1.3 to 1.6 times as far off; 1.15 leaves room for the order of the additions,
    3 % from seed to seed.)"""
    from perf import cases

    def err(op, coils):
        c = dict(op=op, ndim=3, n=n, coils=coils, views=n * n, samples=2 * n, width=width, os=1.25, frames=1)
        return rel(cases.run(cases.prepare(c, 3)), cases.exact(c, 3))

    ref = err("adj", 12)
    for call in calls:
        assert err(*call) < 1.15 * ref, call


@pytest.mark.parametrize("width,coils", [(2, (1, 2, 3, 4, 5)), (3, (1, 2, 3, 4, 5)), (4, (1, 2)), (5, (1, 2)),
                                         (6, (1, 2, 3, 10, 11, 20, 21, 31))])
@pytest.mark.parametrize("nsamples", [3000, 24000])
def test_forward_lane_layouts(width, coils, nsamples):
    """Interpolation around the coil counts where its lanes change, items with
    hundreds of samples (parts, more samples than threads), with few and with
    none, and regions that wrap."""
    import deepmr_b200.fft as F
    from deepmr_b200 import synth
    from oracle import nufft_ref as R

    shape = (13, 9, 21)
    rng = np.random.default_rng(width)
    c = rng.uniform(-0.5, 0.5, (1, nsamples, 3)) * np.asarray(shape[::-1])
    c[:, :2000] *= 0.02
    c[:, -8:] = np.sign(c[:, -8:]) * np.asarray(shape[::-1]) * 0.4999
    c = torch.as_tensor(c.astype(np.float32))
    plan, oplan = F.plan_nufft(c, shape, width, 2.0, device="cuda"), R.plan_nufft(c, shape, width, 2.0)
    img = synth.complex_gaussian((max(coils),) + shape, seed=1)
    ref = R.apply_nufft(img, oplan)
    for k in coils:
        assert rel(F.apply_nufft(img[:k].cuda(), plan), ref[:k]) < TOL, k


def test_arguments_that_outlive_their_transform():
    """A weight that leaked from a function transform is taken, and what function
    transforms and tracing compute are the values that ``apply`` computes."""
    import deepmr_b200.fft as F

    c = torch.as_tensor(np.random.default_rng(0).uniform(-8, 8, (1, 40, 2)).astype(np.float32))
    plan = F.plan_nufft(c, (16, 16), 4, 1.25, device="cuda")
    g = torch.Generator().manual_seed(1)
    y = torch.complex(torch.randn(2, 1, 40, generator=g), torch.randn(2, 1, 40, generator=g)).cuda()
    w = torch.rand(1, 40, generator=g).cuda()
    leaked = []

    def leak(t):
        leaked.append(t)
        return (t * t).sum()

    torch.func.grad(leak)(w)
    ref = F.apply_nufft_adj(y, plan, weight=w)
    assert rel(F.apply_nufft_adj(y, plan, weight=leaked[0]), ref) < 1e-6

    x = ref.clone()
    N = __import__("importlib").import_module("deepmr_b200.fft.nufft")
    runs = {
        "vmap": lambda f: torch.func.vmap(f)(x),
        "grad": lambda f: torch.func.grad(lambda t: (f(t).abs() ** 2).sum())(x),
        "trace": lambda f: torch.jit.trace(f, (x,), check_trace=False)(x),
    }
    for name, run in runs.items():
        res = []
        for f in ((lambda t: N.apply_nufft(t, plan)), (lambda t: N.ApplyNUFFT.apply(t, plan, None, None, None, 128))):
            try:
                res.append(run(f))
            except Exception as e:  # noqa: BLE001
                res.append(type(e))
        if isinstance(res[1], torch.Tensor):
            assert rel(res[0].detach(), res[1].detach()) < 1e-6, name
        else:
            assert res[0] is res[1], name


def test_tensor_core_gridding_of_a_plan_that_exists():
    """dmr_tc_min_coils moves the calls of a plan made before it was set (the
    kernel's test stall, which only it obeys, shows that it ran), captured as well,
    and back."""
    import gc

    import deepmr_b200.fft as F
    from deepmr_b200 import _lib
    from oracle import nufft_ref as R
    from deepmr_b200 import synth

    L = _lib.lib()
    plan, _, ksp = _problem3()
    c = torch.as_tensor(synth.kooshball_3d(160, 64, 24).astype(np.float32))
    ref = R.apply_nufft_adj(ksp.cpu(), R.plan_nufft(c, 24, 4, 1.25))

    def ran_on_tensor_cores():
        L.dmr_tc_test_stall(1)
        try:
            F.apply_nufft_adj(ksp, plan)
            plan.interpolator.check_status()
        except _lib.DmrError as e:
            assert e.code == -8
            return True
        finally:
            L.dmr_tc_test_stall(0)
        return False

    assert not ran_on_tensor_cores()
    old = L.dmr_tc_min_coils(9)
    try:
        gc.collect()
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            x = F.apply_nufft_adj(ksp, plan)
        g.replay()
        assert rel(x, ref) < TOL and rel(F.apply_nufft_adj(ksp, plan), ref) < TOL
        assert ran_on_tensor_cores()
        L.dmr_tc_min_coils(10)
        assert not ran_on_tensor_cores()
    finally:
        L.dmr_tc_min_coils(old)
    assert rel(F.apply_nufft_adj(ksp, plan), ref) < TOL
    g = None
    n = ctypes.c_int64()
    _lib.check(L.dmr_tc_timeouts(ctypes.byref(n), 1))


def test_release_gives_back_the_memory_of_destroyed_plans():
    """After a plan of several hundred MB is gone, releasing the library's pools
    leaves the device with the memory it had before."""
    import gc

    import deepmr_b200.fft as F

    gc.collect()
    torch.cuda.synchronize()
    F.release_scratch()
    torch.cuda.empty_cache()
    before = torch.cuda.mem_get_info()[0]
    c = torch.rand((1, 4_000_000, 3)) * 60 - 30
    plan = F.plan_nufft(c, 64, 4, 1.25, device="cuda")
    during = torch.cuda.mem_get_info()[0]
    del plan
    gc.collect()
    F.release_scratch()
    torch.cuda.empty_cache()
    assert before - during > 300 << 20  # (the plan is larger than what the pool keeps)
    assert before - torch.cuda.mem_get_info()[0] < 32 << 20


@pytest.mark.parametrize("shape,os,grid", [((17, 30, 19), (2.0, 1.5, 2.0), (34, 45, 38)),
                                           ((22, 17, 26), (1.5, 2.0, 1.5), (33, 34, 39))])
@pytest.mark.parametrize("width", [3, 4])
def test_run_time_lengths_3d(shape, os, grid, width):
    """Run-time FFT lengths on all axes of a 3D grid, planar (1 coil) and interleaved
    (3 and 9), both directions and modes, real images, and the 3D Toeplitz pass."""
    import deepmr_b200.fft as F
    from deepmr_b200 import _lib, synth
    from oracle import nufft_ref as R

    rng = np.random.default_rng(width)
    c = torch.as_tensor((rng.uniform(-0.5, 0.5, (3, 60, 3)) * np.asarray(shape[::-1])).astype(np.float32))
    plan, oplan = F.plan_nufft(c, shape, width, os, device="cuda"), R.plan_nufft(c, shape, width, os)
    assert _lib.lib().dmr_fft3_fused(plan.interpolator.handle) == 1
    assert tuple(int(g) for g in oplan.os_shape) == grid
    img = synth.complex_gaussian((9,) + shape, seed=1)
    ksp = synth.complex_gaussian((9, 3, 60), seed=2)
    y, x = R.apply_nufft(img, oplan), R.apply_nufft_adj(ksp, oplan)
    for k in (1, 3, 9):
        assert rel(F.apply_nufft(img[:k].cuda(), plan), y[:k]) < TOL, k
        for det in (False, True):
            old = F.set_deterministic_gridding(det)
            try:
                assert rel(F.apply_nufft_adj(ksp[:k].cuda(), plan), x[:k]) < TOL, (k, det)
            finally:
                F.set_deterministic_gridding(old)
    assert rel(F.apply_nufft(img.real.contiguous().cuda(), plan), R.apply_nufft(img.real, oplan)) < TOL
    dcf = torch.as_tensor(rng.uniform(0.5, 1.5, (3, 60)).astype(np.float32))
    T = F.plan_toeplitz_nufft(c, shape, dcf=dcf, device="cuda")
    ref = R.apply_selfadj(img, R.plan_toeplitz(c, shape, dcf=dcf))
    for k in (1, 9):
        assert rel(F.apply_nufft_selfadj(img[:k].cuda(), T), ref[:k]) < TOL, k


def test_calibration_repeats():
    """Calibrating twice gives the same maps, bit for bit (2D radial, ESPIRiT)."""
    from deepmr_b200 import calib

    d = np.load(__file__.replace("test_gpu_routes.py", "golden/calib2d.npz"))
    a = [torch.as_tensor(d[k]).cuda() for k in ("kspace", "coord", "dcf")]
    maps = [calib.espirit_cal(a[0], coord=a[1], dcf=a[2], shape=int(d["shape"]))[0] for _ in range(20)]
    assert all(torch.equal(m, maps[0]) for m in maps[1:])
