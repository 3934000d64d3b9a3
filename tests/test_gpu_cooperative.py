"""The 64- and 128-point 2-D transforms on the GPU where their launches branch: bin-major spectra (a block per tile,
except for the 128-point inverse) and plane-major ones (persistent blocks), more tiles than blocks are resident,
planes with so few rows that warps take half tasks (up to 16 rows at 64 points), odd extents, offsets.
Yardstick: the fp64 DFT, at 5e-6 of the largest value, as for the other stand-alone transforms."""
import ctypes

import numpy as np
import pytest
import torch

import oracle
from fbcunn_b200 import SpatialConvolutionFBFFT, capi
from oracle import spectral

pytestmark = pytest.mark.gpu
TOL = 5e-6

# d1, d2, h, w, offset up, offset left
SHAPES = [(1, 1, 1, 1, 0, 0), (3, 5, 9, 9, 0, 0), (2, 6, 16, 15, 1, 2), (3, 4, 17, 18, 0, 1), (4, 9, 61, 45, 2, 1),
          (13, 100, 64, 64, 0, 0)]


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("plane_major", [0, 1])
@pytest.mark.parametrize("shape", SHAPES, ids=str)
@pytest.mark.parametrize("n", [64, 128])
def test_forward_and_inverse(n, shape, plane_major):
    d1, d2, h, w, oy, ox = shape
    half, kc = n // 2 + 1, d2 if plane_major else (d2 + 3) // 4 * 4
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    x = np.random.default_rng(n + h).standard_normal((d1, d2, h, w)).astype(np.float32)
    real = torch.from_numpy(x).cuda()
    spec = torch.full((half * n * d1 * kc, 2), float("nan"), device="cuda")
    capi.check(capi.lib().fbfftconv_fft2d(_ptr(real), _ptr(spec), d1, d2, h, w, n, oy, ox, 2 * plane_major, stream))
    ref = spectral.rfft2_padded(x, n, n, oy, ox)                                   # d1, d2, ky, kx
    got = spec.cpu().numpy().astype(np.float64)
    got = got[:, 0] + 1j * got[:, 1]
    if plane_major:
        got = got.reshape(d1, d2, n, half)
    else:
        got = got.reshape(n, half, d1, kc).transpose(2, 3, 0, 1)
        assert np.all(got[:, d2:] == 0)                                            # padding planes
        got = got[:, :d2]
    assert np.abs(got - ref).max() <= TOL * np.abs(ref).max()
    back = torch.full_like(real, float("nan"))
    bias = torch.randn(d2, device="cuda")
    capi.check(capi.lib().fbfftconv_ifft2d(_ptr(spec), _ptr(back), _ptr(bias), d1, d2, h, w, n, oy, ox, 0, plane_major,
                                           stream))
    want = n * n * x.astype(np.float64) + bias.cpu().numpy()[None, :, None, None]
    assert np.abs(back.cpu().numpy() - want).max() <= TOL * np.abs(want).max()


# Layers with one transform that keeps the GPU busy by itself beside small ones: beyond 24 tiles per SM at 64 points, 16
# at 128 points plane-major, 4 bin-major.
@pytest.mark.parametrize("s", [oracle.Shape(1800, 5, 1, 33, 34, 3, 3), oracle.Shape(810, 3, 1, 66, 65, 3, 2, 1, 0),
                               oracle.Shape(100, 6, 1, 66, 70, 2, 3)], ids=lambda s: "x".join(map(str, (s.B, s.P, s.iH))))
def test_large_and_small_operands(s):
    def rel(a, ref):
        return float(np.abs(a.cpu().numpy() - ref).max() / np.abs(ref).max())

    rng = np.random.default_rng(s.B)
    x = rng.standard_normal((s.B, s.P, s.iH, s.iW)).astype(np.float32)
    go = rng.standard_normal((s.B, s.F, s.oH, s.oW)).astype(np.float32)
    m = SpatialConvolutionFBFFT(s.P, s.F, s.kW, s.kH, 1, 1, s.padW, s.padH)
    w, b = m.weight.cpu().numpy(), m.bias.cpu().numpy()
    dx, dgo = torch.from_numpy(x).cuda(), torch.from_numpy(go).cuda()
    before = capi.kernel_launches()
    assert rel(m.forward(dx), oracle.update_output(s, x, w, b)) <= 1e-4
    assert capi.kernel_launches() - before == 4  # the large transform has a launch of its own
    assert rel(m.backward(dx, dgo), oracle.update_grad_input(s, go, w)) <= 1e-4
    assert rel(m.gradWeight, oracle.acc_grad_weight(s, x, go, 1.0)) <= 1e-4
    assert rel(m.gradBias, oracle.acc_grad_bias(s, go, 1.0)) <= 1e-4
