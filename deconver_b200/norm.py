"""Instance normalisation on the library's own CUDA kernels.

`InstanceNorm1d/2d/3d` take the constructor arguments of `torch.nn.InstanceNorm{1,2,3}d` and can
be handed to the reference's network wherever it takes a `norm` class (`DeconverBlock`,
`deconver/deconver.py:52-65`; the published configurations pass `torch.nn.InstanceNorm3d`).
torch's kernel works with one block per (sample, channel) slab; at the small per-GPU batches of a
batch-sharded training step that is fewer blocks than the GPU has multiprocessors.  The kernels
behind this module split every slab over enough blocks to fill the device
(`csrc/ndc_inorm.cu`; the autograd node is in `csrc/ndc_torch.cpp`).

CUDA tensors, float32 or bfloat16 (statistics always in float32); no running statistics.
"""

from typing import Optional

import torch
from torch import Tensor, nn

from .functional import native

__all__ = ["InstanceNorm1d", "InstanceNorm2d", "InstanceNorm3d", "instance_norm"]

_DTYPES = (torch.float32, torch.bfloat16)


def instance_norm(x: Tensor, weight: Optional[Tensor] = None, bias: Optional[Tensor] = None,
                  eps: float = 1e-5) -> Tensor:
    """``(x - mean) / sqrt(var + eps) [* weight + bias]`` per (sample, channel), biased variance."""
    if not x.is_cuda:
        raise RuntimeError(f"deconver_b200: instance norm input is on {x.device}; CUDA only")
    if x.dtype not in _DTYPES:
        raise NotImplementedError(f"deconver_b200: instance norm of {x.dtype} is not supported")
    if x.dim() < 3:
        raise ValueError("instance norm expects (batch, channels, spatial...)")
    return native("instance_norm", (x, weight, bias), float(eps))


class _InstanceNorm(nn.Module):
    _rank = 0

    def __init__(self, num_features: int, eps: float = 1e-5, momentum: Optional[float] = 0.1,
                 affine: bool = False, track_running_stats: bool = False, device=None,
                 dtype=None) -> None:
        super().__init__()
        if track_running_stats:
            raise NotImplementedError("deconver_b200: running statistics are not supported")
        self.num_features, self.eps, self.momentum, self.affine = num_features, eps, momentum, affine
        self.track_running_stats = False
        if affine:
            kw = dict(device=device, dtype=dtype)
            self.weight = nn.Parameter(torch.ones(num_features, **kw))
            self.bias = nn.Parameter(torch.zeros(num_features, **kw))
        else:
            self.register_parameter("weight", None)
            self.register_parameter("bias", None)

    def forward(self, x: Tensor) -> Tensor:
        if x.dim() != self._rank + 2:
            raise ValueError(f"expected a {self._rank + 2}-D input (got {x.dim()}-D)")
        if x.shape[1] != self.num_features:
            raise ValueError(f"expected {self.num_features} channels (got {x.shape[1]})")
        return instance_norm(x, self.weight, self.bias, self.eps)

    def extra_repr(self) -> str:
        return f"{self.num_features}, eps={self.eps}, affine={self.affine}"


class InstanceNorm1d(_InstanceNorm):
    _rank = 1


class InstanceNorm2d(_InstanceNorm):
    _rank = 2


class InstanceNorm3d(_InstanceNorm):
    _rank = 3
