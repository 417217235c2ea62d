"""SPHQuant 64/4 packed linear: operator and module with the reference's names.

Mirrors the reference's `wvq::sphquant` op and fake (weight_vq/inference/ops.py:21-39), its
native entry point's checks and messages (csrc/sphquant/sph_gemv_cuda.cu:403-446) and
`SPHQuantLinear` (weight_vq/inference/linear.py:252-271: buffers `packed_codes`,
`radius_extra`, `radius_scales`, `radius_mins`, `codebook`, `bias`; out_features and
in_features derived from the code tensor).  The op is registered as `wvq::sphquant` unless the
reference package already owns that name in this process, then as `sage_b200::sphquant`.
"""

from __future__ import annotations

import torch
from torch import nn

from . import _lib


def sph_gemv_forward(
    x: torch.Tensor,
    packed_codes: torch.Tensor,
    radius_extra: torch.Tensor,
    radius_scales: torch.Tensor,
    radius_mins: torch.Tensor,
    codebook: torch.Tensor,
    group_size: int = 128,
) -> torch.Tensor:
    """Python twin of the reference's `sph_gemv_forward_cuda`."""
    if group_size != 128:
        raise RuntimeError("sph_gemv currently requires group_size=128")
    return _lib.native_module().sph_forward(x, packed_codes, radius_extra, radius_scales, radius_mins, codebook)


def _fake(x, packed_codes, radius_extra, radius_scales, radius_mins, codebook):
    return x.new_empty((*x.shape[:-1], packed_codes.shape[0]))


sphquant = _lib.register_operator(
    "sphquant",
    "(Tensor x, Tensor packed_codes, Tensor radius_extra, Tensor radius_scales, Tensor radius_mins, Tensor codebook) "
    "-> Tensor",
    _fake,
)


def _sph_module(*args):
    """The native call; the first one puts it in this name's place (a look-up per call is host time of a small call)."""
    global _sph_module
    _sph_module = _lib.native_module().sph_module
    return _sph_module(*args)


def sph_dequantize(packed_codes, radius_extra, radius_scales, radius_mins, codebook) -> torch.Tensor:
    """Dense FP16 weight [N, K] = fp16(the reference decode's FP32 weight), bit for bit."""
    n, k = packed_codes.shape[0], packed_codes.shape[1] * 8
    weight = torch.empty((n, k), dtype=torch.float16, device=packed_codes.device)
    lib = _lib.load()
    with torch.cuda.device(weight.device):
        _lib.check(lib.sageb200_sph_dequant(
            packed_codes.data_ptr(), radius_extra.data_ptr(), radius_scales.data_ptr(), radius_mins.data_ptr(),
            codebook.data_ptr(), weight.data_ptr(), n, k, torch.cuda.current_stream(weight.device).cuda_stream))
    return weight


class SPHQuantLinear(nn.Module):
    """SPHQuant 64/4 packed linear (row-major codes, no permutation)."""

    def __init__(self, packed: dict[str, torch.Tensor], bias: torch.Tensor | None = None):
        super().__init__()
        self.out_features = packed["packed_codes"].shape[0]
        self.in_features = packed["packed_codes"].shape[1] * 8
        for name in ("packed_codes", "radius_extra", "radius_scales", "radius_mins", "codebook"):
            self.register_buffer(name, packed[name])
        self.register_buffer("bias", bias)

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        b = self._buffers
        if torch.compiler.is_compiling():  # the same as the native call below, in operators that can be traced
            output = sphquant(x.to(torch.float16).contiguous(), b["packed_codes"], b["radius_extra"],
                              b["radius_scales"], b["radius_mins"], b["codebook"]).to(x.dtype)
            return output if self.bias is None else output + self.bias
        return _sph_module(x, b["packed_codes"], b["radius_extra"], b["radius_scales"], b["radius_mins"],
                           b["codebook"], b["bias"] if "bias" in b else self.bias)

    def dequantize(self) -> torch.Tensor:
        return sph_dequantize(self.packed_codes, self.radius_extra, self.radius_scales, self.radius_mins,
                              self.codebook)
