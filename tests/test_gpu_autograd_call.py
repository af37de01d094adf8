"""The public transforms enter their autograd functions without the signature
lookup of ``Function.apply``; everything that looks at an autograd function
still sees it (gradients, saved-tensor hooks, function transforms, forward mode,
tracing), exactly as through ``apply``."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def problem():
    import importlib

    import deepmr_b200.fft as F

    N = importlib.import_module("deepmr_b200.fft.nufft")  # the package's attribute of that name is a function
    rng = np.random.default_rng(0)
    c = torch.as_tensor(rng.uniform(-8, 8, (1, 40, 2)).astype(np.float32))
    plan = F.plan_nufft(c, (16, 16), 4, 1.25, device="cuda")
    g = torch.Generator().manual_seed(1)
    x = torch.complex(torch.randn(2, 16, 16, generator=g), torch.randn(2, 16, 16, generator=g)).cuda()
    return N, plan, x


def test_gradient(problem):
    N, plan, x = problem
    grads = []
    for f in ((lambda t: N.apply_nufft(t, plan)), (lambda t: N.ApplyNUFFT.apply(t, plan, None, None, None, 128))):
        t = x.clone().requires_grad_(True)
        y = f(t)
        assert "ApplyNUFFT" in type(y.grad_fn).__name__
        (y.abs() ** 2).sum().backward()
        grads.append(t.grad)
    assert torch.allclose(grads[0], grads[1], rtol=1e-4, atol=1e-4 * float(grads[1].abs().max()))


@pytest.mark.parametrize("transform", ["grad", "vmap", "forward_mode", "trace"])
def test_transforms_as_through_apply(problem, transform):
    """What ``apply`` computes is computed, what it refuses is refused."""
    N, plan, x = problem

    def run(f):
        if transform == "grad":
            return torch.func.grad(lambda t: (f(t).abs() ** 2).sum())(x)
        if transform == "vmap":
            return torch.func.vmap(f)(x)
        if transform == "trace":
            return torch.jit.trace(f, (x,), check_trace=False)(x)
        import torch.autograd.forward_ad as fa

        with fa.dual_level():
            return f(fa.make_dual(x, torch.ones_like(x)))

    res = []
    for f in ((lambda t: N.apply_nufft(t, plan)), (lambda t: N.ApplyNUFFT.apply(t, plan, None, None, None, 128))):
        try:
            res.append(("value", tuple(run(f).shape)))
        except Exception as e:  # noqa: BLE001
            res.append(("raised", type(e)))
    assert res[0] == res[1], res
