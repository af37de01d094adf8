"""The transform lengths of the fused FFT passes (every compiled one; of the
others each radix 2..20, odd lengths, the first and last), along x and along y:
padding and cropping rows, columns, planar grids (1 coil), coil-interleaved ones
(3 coils: the lines of a block cross rows and the last block is partial), real
images, and the fused Toeplitz pass, against the oracle.

Tolerance: relative L2 error <= 1e-5 in float32, as in the other parity tests
(a float32 transform of 640 points is within 1e-6).
"""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

TOL = 1e-5
COMPILED = (32, 40, 48, 56, 64, 80, 96, 112, 120, 128, 140, 144, 160, 168, 192, 200, 224, 240, 256, 280, 288, 320, 336, 384,
            400, 480, 512, 640)
OTHERS = (33, 34, 35, 38, 42, 45, 49, 51, 55, 57, 63, 65, 76, 77, 81, 85, 91, 95, 99, 104, 117, 119, 121, 126, 143, 152, 169,
          171, 182, 187, 195, 209, 221, 225, 234, 247, 252, 255, 266, 270, 285, 289, 300, 304, 323, 340, 342, 360, 361, 380,
          115, 175, 198, 231, 253, 286, 483, 494, 529, 546, 575, 600, 625, 676)


def rel(a, b):
    a = np.asarray(torch.as_tensor(a).detach().cpu(), dtype=np.complex128).ravel()
    b = np.asarray(torch.as_tensor(b).detach().cpu(), dtype=np.complex128).ravel()
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("length", COMPILED + OTHERS)
@pytest.mark.parametrize("axis", ["x", "y"])
def test_length(length, axis):
    import deepmr_b200.fft as F
    from deepmr_b200 import _lib, synth
    from oracle import nufft_ref as R

    n = (length + 1) // 2  # oversampling that gives `length` points
    shape, os = ((16, n), (2.0, length / n)) if axis == "x" else ((n, 16), (length / n, 2.0))
    rng = np.random.default_rng(length)
    c = torch.as_tensor((rng.uniform(-0.5, 0.5, (3, 50, 2)) * np.asarray(shape[::-1])).astype(np.float32))
    plan = F.plan_nufft(c, shape, 3, os, device="cuda")
    assert _lib.lib().dmr_fft3_fused(plan.interpolator.handle) == 1
    oplan = R.plan_nufft(c, shape, 3, os)
    assert int(oplan.os_shape[axis == "x"]) == length
    img = synth.complex_gaussian((3,) + shape, seed=1)
    ksp = synth.complex_gaussian((3, 3, 50), seed=2)
    y, x = R.apply_nufft(img, oplan), R.apply_nufft_adj(ksp, oplan)
    for k in (1, 3):
        assert rel(F.apply_nufft(img[:k].cuda(), plan), y[:k]) < TOL, k
        assert rel(F.apply_nufft_adj(ksp[:k].cuda(), plan), x[:k]) < TOL, k
    assert rel(F.apply_nufft(img.real.contiguous().cuda(), plan), R.apply_nufft(img.real, oplan)) < TOL
    dcf = torch.as_tensor(rng.uniform(0.5, 1.5, (3, 50)).astype(np.float32))
    T = F.plan_toeplitz_nufft(c, shape, dcf=dcf, device="cuda")
    assert rel(F.apply_nufft_selfadj(img.cuda(), T), R.apply_selfadj(img, R.plan_toeplitz(c, shape, dcf=dcf))) < TOL
