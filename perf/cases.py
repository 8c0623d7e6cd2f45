"""Performance cases of the WTConv layers.

Each case is one pass through the public modules ``WTConv2d`` / ``WTConv1d``: the inference forward of a
layer, or its training step (forward, backward to the input and to every parameter, optimizer update).  The
listed cases are the shapes of the repository's own configurations and tests -- the WTConvNeXt-T layer set,
the segmentation and time-series layers, the small default layer -- plus the odd, strided and default-layout
uses around them; ``draw`` gives more cases of the same ranges.
"""
from __future__ import annotations

import math

import torch

from wtconv_b200 import WTConv1d, WTConv2d

_DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
_LR = 1e-5


def _case2d(mode, dtype, layout, B, C, H, W, L, K=5, stride=1):
    return {"ndim": 2, "mode": mode, "dtype": dtype, "layout": layout, "B": B, "C": C, "H": H, "W": W, "L": L,
            "K": K, "stride": stride}


def _case1d(mode, dtype, B, C, N, L, K=5, stride=1):
    return {"ndim": 1, "mode": mode, "dtype": dtype, "layout": "nchw", "B": B, "C": C, "H": 1, "W": N, "L": L,
            "K": K, "stride": stride}


def listed():
    def named(name, case):
        return dict(case, name=name)
    return [
        # one image through a stage-3 layer: interactive serving, where latency and launches count
        named("infer_one_image", _case2d("infer", "bf16", "cl", 1, 384, 14, 14, 3)),
        # the small default layer (fp32, PyTorch's default layout)
        named("infer_small_nchw_f32", _case2d("infer", "f32", "nchw", 8, 32, 56, 56, 3)),
        # WTConvNeXt-T layers at batch 128: the largest and the most frequent stage (9 of its 18 layers)
        named("infer_stage1", _case2d("infer", "bf16", "cl", 128, 96, 56, 56, 5)),
        named("infer_stage3", _case2d("infer", "bf16", "cl", 128, 384, 14, 14, 3)),
        # segmentation backbone layer at high resolution: the largest planes
        named("infer_segmentation_512", _case2d("infer", "bf16", "cl", 2, 256, 512, 512, 5)),
        # a ragged image crop in half precision with a larger kernel
        named("infer_crop_f16_k7", _case2d("infer", "f16", "cl", 6, 72, 61, 83, 4, K=7)),
        # a down-sampling layer of a network in the default layout
        named("infer_stride2_nchw", _case2d("infer", "bf16", "nchw", 64, 128, 28, 28, 3, stride=2)),
        # training: the first and the last stage of WTConvNeXt-T with mixed precision, and a small
        # fp32 network in the default layout with 3 x 3 kernels
        named("train_stage1", _case2d("train", "bf16", "cl", 64, 96, 56, 56, 5)),
        named("train_stage4", _case2d("train", "bf16", "cl", 64, 768, 7, 7, 2)),
        named("train_small_nchw_f32", _case2d("train", "f32", "nchw", 32, 64, 32, 32, 3, K=3)),
        # time series: the inference layer at an even length, a training step at an odd one
        named("infer_signal_4096", _case1d("infer", "f32", 512, 64, 4096, 4)),
        named("train_signal_4097", _case1d("train", "f32", 64, 64, 4097, 4)),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Another layer and tensor of the ranges above: 7 to 512 pixels per side (square in half of the cases),
    16 to 768 channels (mostly multiples of eight), signals of 128 to 65536 samples, batches of 1 to 512, one
    to five levels, kernel 5 in most cases, now and then a stride, the three data types, both layouts."""
    mode = rng.choices(("infer", "train"), (6, 4))[0]
    dtype = rng.choices(("bf16", "f32", "f16"), (5, 4, 1))[0]
    K = rng.choices((5, 3, 7), (6, 2, 2))[0]
    if rng.random() < 0.2:
        N = _log(rng, 128, 65536)
        case = _case1d(mode, dtype, _log(rng, 1, 512), _log(rng, 4, 256), N, rng.randint(1, 5), K,
                       rng.choices((1, 2), (9, 1))[0])
    else:
        H = _log(rng, 7, 512)
        W = H if rng.random() < 0.5 else max(7, min(512, round(H * rng.uniform(0.6, 1.6))))
        C = _log(rng, 16, 768)
        if rng.random() < 0.85:
            C = max(16, C // 8 * 8)
        L = rng.randint(1, min(5, max(2, math.ceil(math.log2(min(H, W))) - 1)))
        case = _case2d(mode, dtype, rng.choices(("cl", "nchw"), (6, 4))[0], _log(rng, 1, 128), C, H, W, L, K,
                       rng.choices((1, 2), (9, 1))[0])
    # no more work than the largest listed case
    most = work(listed()[4])
    while case["B"] > 1 and any(work(case)[k] > most[k] for k in most):
        case["B"] = case["B"] * 3 // 4
    while any(work(case)[k] > most[k] for k in most):
        case["C"] = max(4, case["C"] * 3 // 4)
    return case


def prepare(case, seed):
    """The layer with seeded parameters (as nn.Conv initialises them, wavelet_scale in 0.05..0.2) and its input
    on the GPU; for a training step also the gradient of the loss and the optimizer.  Inference keeps the
    parameters in the activations' type, training keeps them in fp32 (mixed precision)."""
    dev = torch.device("cuda")
    dtype = _DTYPES[case["dtype"]]
    train = case["mode"] == "train"
    C, K, L, stride, nd = case["C"], case["K"], case["L"], case["stride"], case["ndim"]
    with torch.device(dev):
        m = (WTConv2d if nd == 2 else WTConv1d)(C, C, kernel_size=K, stride=stride, bias=True, wt_levels=L)
    g = torch.Generator(device=dev).manual_seed(int(seed))
    bound = 1.0 / math.sqrt(K ** nd)
    with torch.no_grad():
        for name, p in m.named_parameters():
            if name.startswith("wavelet_scale"):
                p.uniform_(0.05, 0.2, generator=g)
            elif name.startswith(("base_conv", "wavelet_convs")):
                p.uniform_(-bound, bound, generator=g)
    m = m.to(torch.float32 if train else dtype).train(train)
    if nd == 1:
        shape, oshape = (case["B"], C, case["W"]), (case["B"], C, case["W"] // stride)
    else:
        shape = (case["B"], C, case["H"], case["W"])
        oshape = shape[:2] + (-(-case["H"] // stride), -(-case["W"] // stride))

    def tensor(s, std):
        t = torch.randn(s, device=dev, generator=g).mul_(std).to(dtype)
        return t.contiguous(memory_format=torch.channels_last) if case["layout"] == "cl" else t

    state = {"m": m, "x": tensor(shape, 1.0)}
    if train:
        state["x"].requires_grad_()
        state["gy"] = tensor(oshape, 1e-2)
        state["params"] = [p for p in m.parameters() if p.requires_grad]
        state["opt"] = torch.optim.SGD(state["params"], lr=_LR, fused=True)
    return state


def run(state):
    m, x = state["m"], state["x"]
    if "opt" not in state:
        with torch.no_grad():
            return m(x)
    state["opt"].zero_grad(set_to_none=True)
    x.grad = None
    y = m(x)
    y.backward(state["gy"])
    state["opt"].step()
    return {"y": y.detach(), "gx": x.grad, "grads": [p.grad for p in state["params"]],
            "params": [p.detach() for p in state["params"]]}


def work(case):
    """Bytes: input and output (training: also the output gradient and the input gradient) and the parameters,
    each once.  Operations: two per tap and output of the base and of every sub-band convolution and the Haar
    steps; training adds the same again for the input gradient and for the parameter gradients."""
    nd, K, L, s = case["ndim"], case["K"], case["L"], case["stride"]
    elem = 4 if case["dtype"] == "f32" else 2
    train = case["mode"] == "train"
    planes = case["B"] * case["C"]
    h, w = case["H"], case["W"]
    n_in = h * w
    n_out = (-(-h // s)) * (-(-w // s)) if nd == 2 else w // s
    taps, sub = K ** nd, 2 ** nd
    macs, haar = taps * n_in, 0
    for _ in range(L):
        h, w = (-(-h // 2) if nd == 2 else h), -(-w // 2)
        macs += sub * taps * h * w
        haar += 2 * sub * nd * h * w
    params = case["C"] * (taps + 2 + L * sub * (taps + 1))
    nbytes = planes * (n_in + n_out) * elem * (2 if train else 1) + params * (12 if train else elem)
    return {"bytes": nbytes, "flops": planes * (2 * macs + haar) * (3 if train else 1)}


def tolerance(case):
    """32-bit sums of a few hundred terms (parameter gradients: of up to millions, in any order); results that
    are rounded to 16 bits, with 16-bit planes between the levels as the reference layer keeps them."""
    if case["dtype"] == "f32":
        return {"rel": 3e-5} if case["mode"] == "train" else {"rel": 1e-5}
    return {"rel": 1e-2} if case["dtype"] == "bf16" else {"rel": 2e-3}
