"""nn.Module:backward as one native call: gradOutput is transformed once for both passes, the transforms of a
small layer run in one launch, and so do the two inverse transforms with the bias gradient.  Against the fp64
oracle at the passes' bound, max|x - ref| <= 1e-4 * max|ref|."""
import numpy as np
import pytest
import torch

import oracle
from fbcunn_b200 import SpatialConvolutionFBFFT, capi

pytestmark = pytest.mark.gpu
PASS_TOL = 1e-4

SHAPES = [
    oracle.Shape(1, 1, 1, 5, 4, 2, 2, 1, 1),         # 8 points, one plane of each kind
    oracle.Shape(3, 7, 21, 13, 15, 3, 3, 1, 0),      # 16 points
    oracle.Shape(5, 9, 12, 30, 27, 5, 4, 2, 1),      # 32 points
    oracle.Shape(2, 6, 5, 50, 61, 5, 6),             # 64 points, too few tiles to fill the GPU: merged
    oracle.Shape(2, 3, 7, 100, 90, 7, 5, 1, 2),      # 128 points, plane-major
    oracle.Shape(2, 5, 3, 70, 65, 3, 3),             # 128 points, bin-major
    oracle.Shape(600, 4, 9, 6, 6, 3, 3, 1, 1),       # long rows of the bias gradient
    oracle.Shape(512, 20, 9, 20, 20, 3, 3),          # input spectrum above the size that gets a buffer of its own
]


def _rel(a, ref):
    return float(np.abs(np.asarray(a, np.float64) - ref).max() / max(np.abs(ref).max(), 1e-30))


@pytest.mark.parametrize("reuse", ["none", "all"])
@pytest.mark.parametrize("s", SHAPES, ids=lambda s: "x".join(str(v) for v in (s.B, s.P, s.F, s.iH, s.iW, s.kH, s.kW)))
def test_backward_matches_the_oracle(s, reuse):
    rng = np.random.default_rng(s.B * 31 + s.iH)
    x = rng.standard_normal((s.B, s.P, s.iH, s.iW)).astype(np.float32)
    bound = 1.0 / np.sqrt(s.kH * s.kW * s.P)
    w = rng.uniform(-bound, bound, (s.F, s.P, s.kH, s.kW)).astype(np.float32)
    go = rng.standard_normal((s.B, s.F, s.oH, s.oW)).astype(np.float32)
    m = SpatialConvolutionFBFFT(s.P, s.F, s.kW, s.kH, 1, 1, s.padW, s.padH, reuse, accumulate=True)
    m.weight.copy_(torch.from_numpy(w))
    dx, dgo = torch.from_numpy(x).cuda(), torch.from_numpy(go).cuda()
    gw, gb, gi = oracle.acc_grad_weight(s, x, go, 1.0), oracle.acc_grad_bias(s, go, 1.0), oracle.update_grad_input(s, go, w)
    total = 0.0
    for step, scale in enumerate((0.7, 1.0)):  # the second step adds to the gradients of the first
        out = m.updateOutput(dx)
        got = m.backward(dx, dgo, scale)
        total += scale
        assert _rel(out.cpu().numpy(), oracle.update_output(s, x, w, m.bias.cpu().numpy())) <= PASS_TOL
        assert _rel(got.cpu().numpy(), gi) <= PASS_TOL
        assert _rel(m.gradWeight.cpu().numpy(), total * gw) <= PASS_TOL
        assert _rel(m.gradBias.cpu().numpy(), total * gb) <= PASS_TOL
    assert m.timeSteps == {"updateOutput": 2, "updateGradInput": 2, "accGradParameters": 2}
    # without an updateOutput before it, and the two passes called one by one, the same comes out
    m2 = SpatialConvolutionFBFFT(s.P, s.F, s.kW, s.kH, 1, 1, s.padW, s.padH, reuse)
    m2.weight.copy_(m.weight)
    a = m2.backward(dx, dgo).clone(), m2.gradWeight.clone(), m2.gradBias.clone()
    b = m2.updateGradInput(dx, dgo), (m2.accGradParameters(dx, dgo), m2.gradWeight)[1], m2.gradBias
    for p, q in zip(a, b):
        assert float((p - q).abs().max()) <= 2e-6 * float(q.abs().max())


@pytest.mark.parametrize("spare", [False, True])
def test_backward_in_a_block_of_the_callers(spare):
    """The scratch block handed in, with and without room for the gradInput spectrum's own buffer: nothing is written
    behind it and the same gradients come out."""
    s = SHAPES[2]
    rng = np.random.default_rng(3)
    x = rng.standard_normal((s.B, s.P, s.iH, s.iW)).astype(np.float32)
    go = rng.standard_normal((s.B, s.F, s.oH, s.oW)).astype(np.float32)
    m = SpatialConvolutionFBFFT(s.P, s.F, s.kW, s.kH, 1, 1, s.padW, s.padH)
    least = SpatialConvolutionFBFFT(s.P, s.F, s.kW, s.kH, 1, 1, s.padW, s.padH, min_workspace=True)
    dx, dgo = torch.from_numpy(x).cuda(), torch.from_numpy(go).cuda()
    lib = capi.lib()
    full, need = (lib.fbfftconv_workspace_bytes(layer._prepare(dx)) for layer in (m, least))
    assert need < full
    size = full if spare else full - 1
    block = torch.full((full + 512,), 77, dtype=torch.uint8, device="cuda")
    first = -block.data_ptr() % 256
    capi.check(lib.fbfftconv_set_workspace(m._handle, block.data_ptr() + first, size))
    got = m.backward(dx, dgo)
    assert _rel(got.cpu().numpy(), oracle.update_grad_input(s, go, m.weight.cpu().numpy())) <= PASS_TOL
    assert _rel(m.gradWeight.cpu().numpy(), oracle.acc_grad_weight(s, x, go, 1.0)) <= PASS_TOL
    assert _rel(m.gradBias.cpu().numpy(), oracle.acc_grad_bias(s, go, 1.0)) <= PASS_TOL
    assert bool((block[first + (full if spare else need):] == 77).all())
    m.cleanupBuffers()
