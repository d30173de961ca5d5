"""Channels-first linear layer.

Mirrors `deconver/layers/linear.py:7-58` of the reference: a 1x1 `nn.Conv1d` over the flattened
spatial axes, so the parameters are named `linear.weight` / `linear.bias` and checkpoints move
both ways.  On CUDA the whole layer is one native autograd node (`csrc/ndc_torch.cpp`): the product
and the input gradient are library GEMMs over the tensors as they lie (the convolution route
converts to channels-last and back for some shapes: 256 -> 64 channels over 4 x 128^3 positions take
4.49 ms against 0.98 ms), the bias is added and its gradient reduced by this library's own kernels
(`csrc/ndc_bias.cu`: the library's broadcast add is not vectorised and its reduction uses one block
per output channel, which shows at the small per-GPU batches of a batch-sharded training step), and
the weight gradient is that of the `Deconv` layer's projection.  CPU tensors, other dtypes and
float32 without a bias take the plain `nn.Conv1d`.
"""

from typing import Optional

import torch
from torch import nn

from .functional import native

_DTYPES = (torch.float32, torch.bfloat16)


def native_operands(x: torch.Tensor, weight: torch.Tensor):
    """``(x, weight)`` in the type the product runs in, or None where the native node does not take
    them.  Under autocast that is its type, as for a convolution."""
    if not x.is_cuda or not weight.is_cuda or x.dim() < 3:
        return None
    if torch.is_autocast_enabled("cuda"):
        dtype = torch.get_autocast_dtype("cuda")
        x, weight = x.to(dtype), weight.to(dtype)
    return (x, weight) if x.dtype in _DTYPES and x.dtype == weight.dtype else None


class Linear(nn.Module):
    def __init__(self, in_channels: int, out_channels: int, bias: bool = True,
                 device: Optional[torch.device] = None, dtype: Optional[torch.dtype] = None):
        super().__init__()
        self.flatten = nn.Flatten(start_dim=2)
        self.linear = nn.Conv1d(in_channels, out_channels, kernel_size=1, bias=bias,
                                device=device, dtype=dtype)

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        bias = self.linear.bias
        operands = native_operands(x, self.linear.weight)
        if operands is not None and (bias is not None or operands[0].dtype == torch.bfloat16):
            return native("linear", (*operands, bias))
        shape = x.shape
        return self.linear(self.flatten(x)).view(shape[0], -1, *shape[2:])
