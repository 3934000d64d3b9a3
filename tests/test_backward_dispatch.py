"""nn.Module:backward is updateGradInput followed by accGradParameters (fbcunn/SpatialConvolutionFFT.lua:405-416).
The one native call that stands for both is taken only where the two passes are the module's own, and it takes
what they take (no bias gradient).  Without a GPU: the passes, or the library, are stand-ins."""
import types

import pytest
import torch

from fbcunn_b200 import SpatialConvolution, SpatialConvolutionFBFFT, SpatialConvolutionFFTTiled, capi, module

X, GO = torch.zeros(1, 2, 6, 6), torch.zeros(1, 3, 4, 4)


def _layer(cls=SpatialConvolutionFBFFT):
    m = cls(2, 3, 3, 3, device="cpu")
    m.gradInput = torch.zeros_like(X)
    return m


def _recorder(calls):
    return (lambda *a: calls.append(("gradInput", a[-2:])), lambda *a: calls.append(("gradParameters", a[-3:])))


EXPECTED = [("gradInput", (X, GO)), ("gradParameters", (X, GO, 0.5))]


@pytest.mark.parametrize("cls", [SpatialConvolutionFBFFT, SpatialConvolutionFFTTiled, SpatialConvolution])
@pytest.mark.parametrize("where", ["object", "subclass", "class"])
def test_replaced_passes_are_called(cls, where, monkeypatch):
    calls = []
    grad_input, grad_parameters = _recorder(calls)
    if where == "subclass":
        cls = type("Own", (cls,), {"updateGradInput": grad_input, "accGradParameters": grad_parameters})
    m = _layer(cls)
    target = m if where == "object" else cls
    if where != "subclass":
        monkeypatch.setattr(target, "updateGradInput", grad_input)
        monkeypatch.setattr(target, "accGradParameters", grad_parameters)
    assert m.backward(X, GO, 0.5) is m.gradInput
    assert calls == EXPECTED


def test_one_replaced_pass_is_enough(monkeypatch):
    calls = []
    m = _layer()
    m.updateGradInput = lambda *a: calls.append("gradInput")
    monkeypatch.setattr(SpatialConvolutionFBFFT, "accGradParameters", lambda *a: calls.append("gradParameters"))
    m.backward(X, GO)
    assert calls == ["gradInput", "gradParameters"]


def test_backward_without_a_bias_gradient(monkeypatch):
    m = _layer()
    m.gradBias = None  # as accGradParameters takes it
    seen = []
    monkeypatch.setattr(capi, "lib", lambda: types.SimpleNamespace(fbfftconv_backward=lambda *a: seen.append(a) or 0))
    monkeypatch.setattr(module, "_stream", lambda device: 0)
    for check in ("_check_input", "_check_grad_output"):
        monkeypatch.setattr(m, check, lambda *a: None)
    monkeypatch.setattr(m, "_prepare", lambda *a: 1)
    assert m.backward(X, GO) is m.gradInput
    assert seen[0][6:8] == (None, 1.0) and len(seen) == 1
