"""The work that a user of this package has it do, as cases to be timed.

A case is one pass of a layer (`deconver_b200.Deconv`) or of a network block (instance norm,
1x1 projections, `Deconv`, MLP) at one stage geometry: forward only, as in inference, or forward
and backward, as in a training step.  Sizes are the stage geometries of the repository's 2-D and
3-D networks (widths 32..512 at 256^2..16^2, 64..512 at 64^3..8^3, 128^3 inference), its layer
benchmarks and ragged sizes between them.

Keys of a case: `part` (layer / block), `train` (forward and backward, or forward only), `batch`,
`channels`, `size` ("HxW" or "DxHxW"), `kernel` (taps along every axis), `groups` (-1: one per
channel), `ratio` (source channels per channel), `iters` (multiplicative updates), `dtype`.
"""

import math

import torch
import torch.nn.functional as F
from torch import nn

import deconver_b200

_DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16}
_MLP_RATIO = 4


def _case(batch, channels, size, kernel, train, dtype, part="layer", groups=-1, ratio=4, iters=1, name=None):
    case = {} if name is None else {"name": name}
    case.update(part=part, train=train, batch=batch, channels=channels, size=size, kernel=kernel,
                groups=groups, ratio=ratio, iters=iters, dtype=dtype)
    return case


def listed():
    return [
        # the deepest stage of the 2-D network on one image: launches and host work
        _case(1, 512, "16x16", 5, False, "f32", name="image_deep_fwd_f32"),
        # one 2-D layer on one image, the CPU-comparable benchmark
        _case(1, 32, "256x256", 5, False, "f32", name="image_one_fwd_f32"),
        # second stage of the 2-D network, inference on a batch of 16 images
        _case(16, 64, "128x128", 5, False, "bf16", name="image_batch_fwd_bf16"),
        # first stage of the 2-D network, training on a batch of 16 images
        _case(16, 32, "256x256", 5, True, "f32", name="image_batch_train_f32"),
        # images as a crop leaves them, 3x3 filters, three updates
        _case(5, 24, "203x171", 3, True, "f32", iters=3, name="image_ragged_train_f32"),
        # deepest stage of the 3-D network at the per-GPU batch of an 8-GPU training step
        _case(2, 512, "8x8x8", 3, True, "bf16", name="volume_deep_train_bf16"),
        # its second stage at the same batch
        _case(2, 128, "32x32x32", 3, True, "bf16", name="volume_mid_train_bf16"),
        # one 3-D layer forward and backward, the headline benchmark
        _case(2, 64, "64x64x64", 3, True, "f32", name="volume_train_f32"),
        # a volume cropped to its foreground: no extent a multiple of anything
        _case(2, 48, "37x53x45", 3, True, "f32", name="volume_ragged_train_f32"),
        # first stage of the large 3-D inference, per-GPU batch of an 8-GPU run
        _case(4, 64, "128x128x128", 3, False, "bf16", name="volume_large_fwd_bf16"),
        # a whole block of the 3-D network's first stage in a training step
        _case(2, 64, "64x64x64", 3, True, "bf16", part="block", name="block_train_bf16"),
        # filters shared by groups of four channels, two sources per channel
        _case(2, 32, "32x32x32", 3, True, "f32", groups=8, ratio=2, name="grouped_train_f32"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _around(rng, extent):
    """An extent near `extent`: as it is, or cropped to anything above two thirds of it."""
    return extent if rng.random() < 0.4 else rng.randint(max(5, 2 * extent // 3), extent)


def draw(rng):
    """One more case.  A stage has as many voxels and channels as one of the networks' stages can
    have; `budget` (multiply-adds of the update, as forward passes) keeps it below the largest
    listed case."""
    while True:
        kind = rng.choice(["image", "image", "volume", "volume", "block", "general"])
        train = rng.random() < 0.6
        dtype = rng.choice(["f32", "bf16"])
        if kind == "image" or (kind == "general" and rng.random() < 0.5):
            kernel = rng.choice([5, 5, 3])
            edge = _log(rng, 14, 300)
            dims = (_around(rng, edge), _around(rng, edge))
            batch = _log(rng, 1, 20)
        else:
            kernel = 3
            edge = _log(rng, 7, 128)
            dims = tuple(_around(rng, edge) for _ in range(3))
            batch = _log(rng, 1, 8)
        channels = 8 * _log(rng, 2, 64)
        case = _case(batch, channels, "x".join(str(d) for d in dims), kernel, train, dtype)
        budget = 3.5e10
        if kind == "block":
            case["part"], budget = "block", 1.5e10
        elif kind == "general":
            # any grouping and ratio that the layer's constructor takes, up to 16 channels a group
            m = rng.choice([1, 2, 4])
            case["groups"], case["ratio"], case["channels"] = channels // m, rng.choice([1, 2, 4]), channels
            budget = 4e8
        elif rng.random() < 0.2:
            case["iters"] = rng.choice([2, 3])
        fma = _update_fma(case) * (11.0 / 3.0 if train else 1.0)
        if 2e6 <= fma <= budget:
            return case


def _dims(case):
    return [int(v) for v in case["size"].split("x")]


def _voxels(case):
    return case["batch"] * math.prod(_dims(case))


def _sources(case):
    """Source channels of the layer, all groups together."""
    groups = case["channels"] if case["groups"] == -1 else case["groups"]
    return groups * round(case["channels"] * case["ratio"] / groups)


def _update_fma(case):
    """Multiply-adds of the forward updates: K, and A twice, over every (channel, source) pair of
    a group; the backward has 8/3 as many."""
    groups = case["channels"] if case["groups"] == -1 else case["groups"]
    m = case["channels"] // groups
    taps = case["kernel"] ** len(_dims(case))
    return 3.0 * m * _sources(case) * taps * _voxels(case) * case["iters"]


class _Mixer(nn.Module):
    """in_proj, ReLU, Deconv, out_proj, as a network's block has them."""

    def __init__(self, channels, layer):
        super().__init__()
        self.in_proj = deconver_b200.Linear(channels, channels)
        self.deconv = layer
        self.out_proj = deconver_b200.Linear(4 * channels, channels)

    def forward(self, x):
        return self.out_proj(self.deconv(F.relu(self.in_proj(x))))


class _Block(nn.Module):
    def __init__(self, channels, layer, norm):
        super().__init__()
        self.norm1, self.mixer = norm(channels), _Mixer(channels, layer)
        self.norm2, self.mlp = norm(channels), deconver_b200.MLP(channels, ratio=_MLP_RATIO)

    def forward(self, x):
        x = x + self.mixer(self.norm1(x))
        return x + self.mlp(self.norm2(x))


def prepare(case, seed):
    dims, dtype, dev = _dims(case), _DTYPES[case["dtype"]], torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev).manual_seed(seed)
    channels, kernel = case["channels"], (case["kernel"],) * len(dims)
    layer = deconver_b200.Deconv(channels, kernel_size=kernel, ratio=case["ratio"], groups=case["groups"],
                                 num_iters=case["iters"])
    net = layer
    if case["part"] == "block":
        norm = deconver_b200.InstanceNorm3d if len(dims) == 3 else deconver_b200.InstanceNorm2d
        net = _Block(channels, layer, norm)
    net = net.to(dev)
    with torch.no_grad():
        for p in net.parameters():   # 1x1 weights and biases as nn.Conv1d starts them
            bound = 1.0 / math.sqrt(p.shape[1] if p.dim() > 1 else channels)
            p.copy_((2.0 * torch.rand(p.shape, device=dev, generator=gen) - 1.0) * bound)
        # filters |N(0, 1)| over the taps, and a source that is mostly positive, as in the
        # repository's layer benchmarks and whole-layer comparisons
        h0 = layer.init.h0
        h0.copy_(torch.randn(h0.shape, device=dev, generator=gen).abs() / math.prod(kernel))
        layer.init.linear.linear.bias.add_(1.0)
    net = net.to(dtype)
    shape = (case["batch"], channels, *dims)
    if case["part"] == "block":   # a block's input is the residual stream, the layer's is non-negative
        x = torch.randn(shape, device=dev, generator=gen).to(dtype)
    else:
        x = torch.rand(shape, device=dev, generator=gen).to(dtype)
    state = {"net": net, "x": x, "train": case["train"]}
    if case["train"]:
        out_channels = channels if case["part"] == "block" else _sources(case)
        state["gout"] = torch.randn((case["batch"], out_channels, *dims), device=dev, generator=gen).to(dtype)
        state["params"] = list(net.parameters())
        x.requires_grad_(True)
    return state


def run(state):
    if not state["train"]:
        with torch.no_grad():
            return state["net"](state["x"])
    x, params = state["x"], state["params"]
    x.grad = None
    for p in params:
        p.grad = None
    out = state["net"](x)
    out.backward(state["gout"])
    return [out.detach(), x.grad] + [p.grad for p in params]


def work(case):
    e = 2 if case["dtype"] == "bf16" else 4
    voxels, c, s = _voxels(case), case["channels"], _sources(case)
    taps = case["kernel"] ** len(_dims(case))
    weights = c * s + s + (c // (c if case["groups"] == -1 else case["groups"])) * s * taps
    gemm = voxels * c * s
    out = s
    if case["part"] == "block":
        hidden = _MLP_RATIO * c
        weights += c * c + c + s * c + c + 2 * c * hidden + hidden + c
        gemm += voxels * (c * c + s * c + 2 * c * hidden)
        out = c
    # forward: x, the parameters and the output; backward adds the upstream gradient, the
    # input's gradient and the parameters' gradients
    nbytes = e * (voxels * (c + out) + weights)
    fma = gemm + _update_fma(case)
    if case["train"]:
        nbytes += e * (voxels * (c + out) + weights)
        fma = 3.0 * gemm + _update_fma(case) * 11.0 / 3.0
    return {"bytes": nbytes, "flops": 2.0 * fma}


def tolerance(case):
    """bfloat16: tensors and gradients are rounded to eight bits between the operators.  float32:
    1x1 projections are library products in TF32 (the library's default for convolutions; four of
    them in a row in a block), the update itself is float32."""
    if case["dtype"] == "bf16":
        return {"rel": 1.5e-2, "max": 0.5}
    return {"rel": 3e-3 if case["part"] == "block" else 1e-3, "max": 0.05}
