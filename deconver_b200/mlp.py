"""Channels-first MLP with the first projection's bias fused into the GELU.

Mirrors `deconver/layers/mlp.py:9-62` of the reference: `block = Sequential(Linear, GELU,
Dropout, Linear, Dropout)`, the same constructor and the same parameter names
(`block.0.linear.weight`, ...), so checkpoints move both ways.  On CUDA (float32 / bfloat16) the
first projection runs without its bias and one kernel of this library (`csrc/ndc_bias.cu`)
computes ``gelu(h + bias)`` in a single pass over the hidden tensor, the largest of the block;
the backward computes ``ga * gelu'(h + bias)`` and the bias gradient in one pass.  The library
sequence is a broadcast add, a GELU pass, and on the way back a GELU-gradient pass plus a
reduction: two extra trips over the hidden tensor.  CPU tensors and other dtypes run the plain
sequence.
"""

from typing import Optional

import torch
from torch import nn
from torch.nn.modules.utils import _pair

from .functional import native
from .linear import _DTYPES, Linear, native_operands


def bias_gelu(h: torch.Tensor, bias: Optional[torch.Tensor]) -> torch.Tensor:
    """``gelu(h + bias)`` over the channel axis (dim 1) of a CUDA float32 / bfloat16 tensor."""
    if not h.is_cuda or h.dtype not in _DTYPES:
        raise RuntimeError("bias_gelu runs on CUDA float32 / bfloat16 tensors only")
    return native("bias_gelu", (h, bias))


class MLP(nn.Module):
    def __init__(self, in_channels: int, out_channels: Optional[int] = None,
                 hidden_channels: Optional[int] = None, ratio: float = 4.0,
                 dropout=0.0, **kwargs):
        super().__init__()
        out_channels = out_channels or in_channels
        hidden_channels = hidden_channels or int(ratio * in_channels)
        dropout = _pair(dropout)
        self.block = nn.Sequential(
            Linear(in_channels, hidden_channels, **kwargs),
            nn.GELU(),
            nn.Dropout(dropout[0]),
            Linear(hidden_channels, out_channels, **kwargs),
            nn.Dropout(dropout[1]),
        )

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        first, act, drop1, second, drop2 = self.block
        operands = native_operands(x, first.linear.weight) if type(first) is Linear else None
        if operands is None or not isinstance(act, nn.GELU) or act.approximate != "none":
            return self.block(x)
        a = native("bias_gelu", (native("linear", (*operands, None)), first.linear.bias))
        return drop2(second(drop1(a)))
