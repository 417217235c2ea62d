"""Packed SAGE linear module with the reference's constructor and buffer names.

Mirrors `SAGELinear` (weight_vq/inference/linear.py:274-309 in the reference): buffers
`packed_codes`, `radius_codes`, `radius_grid`, `codebook`, `permutation`, `bias` are
registered under those names, so a reference state_dict loads with no missing or
unexpected keys; `out_features` excludes tile padding; `in_features` comes from the code
tensor's group count.  Unlike the reference, the input-channel gather is never hoisted
out of the operator: the kernels fold it into their activation loads for every shape.
"""

from __future__ import annotations

import torch
from torch import nn

from . import _lib
from .ops import sage, sage_dequantize


def _sage_module(*args):
    """The native call; the first one puts it in this name's place (a look-up per call is host time of a small call)."""
    global _sage_module
    _sage_module = _lib.native_module().sage_module
    return _sage_module(*args)


class SAGELinear(nn.Module):
    """SAGE 64/4, 128/3 or 256/2 packed linear."""

    permutation: torch.Tensor

    def __init__(
        self, packed: dict[str, torch.Tensor], out_features: int, bias: torch.Tensor | None = None
    ):
        super().__init__()
        self.out_features = out_features
        self.in_features = packed["packed_codes"].shape[1] * 128
        for name in ("packed_codes", "radius_codes", "radius_grid", "codebook", "permutation"):
            self.register_buffer(name, packed[name])
        self.register_buffer("bias", bias)

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        b = self._buffers  # (nn.Module attribute access is a Python-level search, per buffer and call)
        if torch.compiler.is_compiling():  # the same as the native call below, in operators that can be traced
            output = sage(
                x.to(torch.float16).contiguous(), b["packed_codes"], b["radius_codes"], b["radius_grid"],
                b["codebook"], b["permutation"], self.out_features,
            ).to(x.dtype)
            return output if self.bias is None else output + self.bias
        return _sage_module(
            x, b["packed_codes"], b["radius_codes"], b["radius_grid"], b["codebook"], b["permutation"],
            self.out_features, b["bias"] if "bias" in b else self.bias,
        )

    def dequantize(self) -> torch.Tensor:
        """Dense FP16 weight [out_features, in_features] in original channel order."""
        return sage_dequantize(
            self.packed_codes, self.radius_codes, self.radius_grid, self.codebook,
            self.permutation, self.out_features,
        )

    def extra_repr(self) -> str:
        return (
            f"in_features={self.in_features}, out_features={self.out_features}, "
            f"entries={self.codebook.shape[1]}, permuted={self.permutation.numel() > 0}"
        )
