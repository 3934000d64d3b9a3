"""The work whose speed is measured: the convolution layers and stand-alone transforms that users of this
package run, called through its modules as a training or serving program calls them.

A case is a dict of plain values.  `op` says which module it goes through:

    "conv"   SpatialConvolutionFBFFT: the three passes of a training step, or updateOutput alone
    "tiled"  SpatialConvolutionFFTTiled: the same for images cut into tiles
    "fft2d"  FFTWrapper: a forward and an inverse 2-D transform in the reference's tensor layout
    "fft1d"  FFTWrapper: the same in one dimension

Layer sizes are those of the benchmark's six layers, of the parity tests and of the autotuning
wrapper's candidates; inputs and gradients are N(0, 1), weights U(+-1/sqrt(fan_in)), as the benchmark draws them.
"""
import math

import torch

from fbcunn_b200 import FFTWrapper, SpatialConvolutionFBFFT, SpatialConvolutionFFTTiled


def _conv(name, B, P, F, iH, iW, kH, kW, padH=0, padW=0, step=True, reuse="none", accumulate=False, tile=0):
    case = dict(op="tiled" if tile else "conv", B=B, P=P, F=F, iH=iH, iW=iW, kH=kH, kW=kW, padH=padH, padW=padW,
                step=step, reuse=reuse, accumulate=accumulate, tile=tile)
    return dict(case, name=name) if name else case


def _fft(name, op, planes, batch_dims, N):
    case = dict(op=op, planes=planes, batch_dims=batch_dims, N=N)
    return dict(case, name=name) if name else case


def listed():
    return [
        # one image through a small layer when serving: four tiny launches and the call itself
        _conv("serve one image", 1, 16, 16, 32, 32, 5, 5, step=False),
        # the benchmark's smallest layer, a training step
        _conv("small layer step", 16, 16, 16, 32, 32, 5, 5),
        # first layer of an image network: three colour planes, the largest transform size
        _conv("first layer step", 128, 3, 96, 128, 128, 11, 11),
        # the benchmark's middle layers: 64-, 32- and 16-point transforms at a full batch
        _conv("64-pixel layer step", 128, 64, 128, 64, 64, 9, 9),
        _conv("32-pixel layer step", 128, 128, 128, 32, 32, 9, 9),
        _conv("16-pixel layer step", 128, 128, 128, 16, 16, 7, 7),
        # the wide late layer, padded, odd image size; and the same as one rank of eight sees it
        _conv("wide layer step", 128, 384, 384, 13, 13, 3, 3, 1, 1),
        _conv("wide layer shard step", 16, 384, 384, 13, 13, 3, 3, 1, 1),
        # nothing divides anything: ragged batch, planes, image and kernel; spectra shared between the passes
        # of the step and gradients accumulated over micro-batches
        _conv("ragged layer step", 50, 70, 130, 27, 23, 5, 4, 2, 1, reuse="all", accumulate=True),
        # an image beyond the untiled limit, small kernel
        _conv("tiled 224 step", 32, 64, 64, 224, 224, 3, 3, 1, 1, tile=32),
        # the stand-alone transforms, two batch dimensions and one
        _fft("2-D transforms", "fft2d", 8192, 2, 32),
        _fft("1-D transforms", "fft1d", 1 << 18, 1, 256),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    most = max(_spectra(c) for c in listed()) / 2
    while True:
        kind = rng.random()
        if kind < 0.1:
            N = 2 ** rng.randint(3, 8)
            return _fft(None, "fft1d", _log_int(rng, 64, (1 << 26) // N), 1, N)
        if kind < 0.2:
            N = 2 ** rng.randint(3, 7)
            return _fft(None, "fft2d", _log_int(rng, 16, min(60000, (1 << 26) // (N * N))), 1, N)
        P = 3 if rng.random() < 0.15 else _log_int(rng, 4, 384)
        shape = dict(B=_log_int(rng, 1, 128), P=P, F=_log_int(rng, 8, 384))
        tiled = kind < 0.3
        iH = _log_int(rng, 130, 260) if tiled else _log_int(rng, 7, 128)
        iW = iH if rng.random() < 0.5 else max(3, min(260 if tiled else 128, int(iH * rng.uniform(0.6, 1.4))))
        kH = rng.randint(1, min(5 if tiled else 11, iH))
        kW = kH if rng.random() < 0.7 and kH <= iW else rng.randint(1, min(5 if tiled else 11, iW))
        padH, padW = (rng.randint(0, (k - 1) // 2) for k in (kH, kW))
        if not tiled and max(iH + 2 * padH, iW + 2 * padW) > 128:
            continue
        case = _conv(None, shape["B"], shape["P"], shape["F"], iH, iW, kH, kW, padH, padW, step=rng.random() < 0.75,
                     reuse=rng.choice(["none", "none", "all"]), accumulate=rng.random() < 0.3,
                     tile=rng.choice([16, 32]) if tiled else 0)
        if _spectra(case) <= most and case["B"] * _tiles(case)[0] <= 60000:
            return case


# -- sizes -------------------------------------------------------------------------------------------
def _out(c):
    return c["iH"] + 2 * c["padH"] - c["kH"] + 1, c["iW"] + 2 * c["padW"] - c["kW"] + 1


def _tiles(c):
    """(tiles per image, transform size) of a layer; an untiled one is a single tile."""
    h, w = c["iH"] + 2 * c["padH"], c["iW"] + 2 * c["padW"]
    if c["tile"]:
        h, w = min(h, c["tile"]), min(w, c["tile"])
    oH, oW = _out(c)
    tiles = -(-oH // (h - c["kH"] + 1)) * -(-oW // (w - c["kW"] + 1))
    N = 8
    while N < max(h, w, c["kH"], c["kW"]):
        N *= 2
    return tiles, N


def _spectra(c):
    """Complex values and products of a case, in units of about one byte moved: what bounds a drawn case."""
    if c["op"].startswith("fft"):
        return 16.0 * c["planes"] * c["N"] ** (2 if c["op"] == "fft2d" else 1)
    tiles, N = _tiles(c)
    B, bins = c["B"] * tiles, N * (N // 2 + 1)
    one = 8.0 * bins * (2 * (B * c["P"] + B * c["F"]) + 2 * c["F"] * c["P"]) + 8.0 * bins * B * c["P"] * c["F"] / 30
    return one * (3 if c["step"] else 1)


# -- a case ------------------------------------------------------------------------------------------
def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape):
        return torch.empty(shape, device="cuda").normal_(generator=g)

    if case["op"] == "fft2d":
        n, d = case["N"], case["planes"]
        batch = (d // 16, 16) if case["batch_dims"] == 2 else (d,)
        time = normal(*batch, n, n)
        return dict(case=case, wrapper=FFTWrapper("fbfft", 0, 0), time=time, back=torch.empty_like(time),
                    freq=torch.empty(batch + (n // 2 + 1, n, 2), device="cuda"))
    if case["op"] == "fft1d":
        n, d = case["N"], case["planes"]
        time = normal(d, n)
        return dict(case=case, wrapper=FFTWrapper("fbfft", 0, 0), time=time, back=torch.empty_like(time),
                    freq=torch.empty((d, n // 2 + 1, 2), device="cuda"))
    args = (case["P"], case["F"], case["kW"], case["kH"], 1, 1, case["padW"], case["padH"])
    if case["op"] == "tiled":
        m = SpatialConvolutionFFTTiled(*args, case["tile"], case["tile"], case["reuse"], accumulate=case["accumulate"])
    else:
        m = SpatialConvolutionFBFFT(*args, case["reuse"], accumulate=case["accumulate"])
    bound = 1.0 / math.sqrt(case["kH"] * case["kW"] * case["P"])
    m.weight.uniform_(-bound, bound, generator=g)
    m.bias.uniform_(-0.01, 0.01, generator=g)
    state = dict(case=case, module=m, input=normal(case["B"], case["P"], case["iH"], case["iW"]))
    if case["step"]:
        state["gradOutput"] = normal(case["B"], case["F"], *_out(case))
    return state


def run(state):
    case = state["case"]
    if case["op"].startswith("fft"):
        w = state["wrapper"]
        w.fft_reference_layout(state["time"], state["freq"], case["batch_dims"])
        w.ffti_reference_layout(state["back"], state["freq"], case["batch_dims"])
        return state["freq"], state["back"]
    m = state["module"]
    output = m.forward(state["input"])
    if not case["step"]:
        return output
    gradInput = m.backward(state["input"], state["gradOutput"])
    return output, gradInput, m.gradWeight, m.gradBias


def work(case):
    """Bytes: the real tensors (and the caller's spectra) of each call, read or written once.  Operations: the
    transforms and the products per frequency of each call."""
    if case["op"].startswith("fft"):
        d, n = case["planes"], case["N"]
        points, freqs = (n * n, n * (n // 2 + 1)) if case["op"] == "fft2d" else (n, n // 2 + 1)
        return {"bytes": 2.0 * d * (4 * points + 8 * freqs), "flops": 2.0 * d * 2.5 * points * math.log2(points)}
    B, P, F = case["B"], case["P"], case["F"]
    oH, oW = _out(case)
    n_in, n_out, n_w = B * P * case["iH"] * case["iW"], B * F * oH * oW, F * P * case["kH"] * case["kW"]
    tiles, N = _tiles(case)
    planes = B * tiles * (P + F) + F * P
    flops = 8.0 * N * (N // 2 + 1) * B * tiles * P * F + planes * 2.5 * N * N * math.log2(N * N)
    calls = 3 if case["step"] else 1
    return {"bytes": 4.0 * calls * (n_in + n_out + n_w), "flops": calls * flops}


def tolerance(case):
    # 32-bit sums throughout (the tensor-core products carry a 3xTF32 split, good to fp32 level)
    return {"rel": 1e-5}
