"""Torch operator for the SAGE packed linear, backed by libsage_b200.so.

Mirrors the reference's dispatcher registration (weight_vq/inference/ops.py:42-61):
`sage(x, packed_codes, radius_codes, radius_grid, codebook, permutation, out_features)`
mutates nothing and has a CUDA kernel only (csrc/torch_ops.cpp), plus a fake kernel that
returns `x.new_empty((*x.shape[:-1], out_features))`.  The op is registered as
`wvq::sage`, the reference's name, unless that name is already taken in this process
(the reference package was imported first), in which case it is `sage_b200::sage`.

Argument checks and their messages follow the reference's native entry point
(csrc/bindings.cpp:13-48).
"""

from __future__ import annotations

import ctypes
import threading

import torch

from . import _lib

_WORKSPACES: dict[tuple[int, int], torch.Tensor] = {}
_RETIRED: list[torch.Tensor] = []  # outgrown buffers a captured graph may still point at
# Held from fetching a buffer until the call's launches are enqueued: threads on one stream share its buffer, a call is
# several launches that hand data to one another through it, and ctypes runs it without the interpreter's lock.
_WORKSPACE_LOCK = threading.Lock()


def _workspace(device: torch.device, stream: int, nbytes: int) -> torch.Tensor:
    """Zero-filled scratch, one per (device, stream); the kernels restore the zeros."""
    key = (device.index, stream)
    buffer = _WORKSPACES.get(key)
    if buffer is None or buffer.numel() < nbytes:
        if buffer is not None:
            _RETIRED.append(buffer)
        buffer = torch.zeros(max(nbytes, 1 << 16), dtype=torch.uint8, device=device)
        _WORKSPACES[key] = buffer
    return buffer


def _check_layout(x, codes, radii, grid, book, permutation, out_features):
    if not (x.is_cuda and x.dtype == torch.float16 and x.is_contiguous() and x.dim() >= 1):
        raise RuntimeError("SAGE requires contiguous CUDA FP16 input")
    for tensor in (codes, radii, grid, book, permutation):
        if tensor.device != x.device or not tensor.is_contiguous():
            raise RuntimeError("SAGE buffers must be contiguous and on the input device")
    k = x.shape[-1]
    tiles = (out_features + 15) // 16
    if not (k > 0 and k % 128 == 0 and out_features > 0):
        raise RuntimeError("SAGE requires positive N and K divisible by 128")
    if not (book.dim() == 3 and book.shape[0] == 4 and book.shape[2] == 2 and book.shape[1] in (64, 128, 256)):
        raise RuntimeError("SAGE codebook must have shape [4, 64/128/256, 2]")
    groups = k // 128
    if not (
        codes.dtype == torch.int32
        and tuple(codes.shape) == (tiles, groups, 16, 8)
        and radii.dtype == torch.int32
        and tuple(radii.shape) == (tiles, groups, 16)
        and grid.dtype == torch.float16
        and tuple(grid.shape) == (tiles, groups, 16, 2)
        and book.dtype == torch.float16
        and permutation.dtype == torch.int32
        and permutation.dim() == 1
        and permutation.numel() in (0, k)
    ):
        raise RuntimeError("Invalid SAGE packed layout")
    if (grid.data_ptr() & 3) or (book.data_ptr() & 3):
        raise RuntimeError("SAGE grid and codebook require 4-byte aligned storage")
    return k


def sage_forward(
    x: torch.Tensor,
    packed_codes: torch.Tensor,
    radius_codes: torch.Tensor,
    radius_grid: torch.Tensor,
    codebook: torch.Tensor,
    permutation: torch.Tensor,
    out_features: int,
) -> torch.Tensor:
    """The native entry point's Python twin (reference csrc/bindings.cpp:8-79)."""
    return _lib.native_module().sage_forward(x, packed_codes, radius_codes, radius_grid, codebook, permutation,
                                             out_features, None)


def sage_forward_scratch(
    x: torch.Tensor,
    packed_codes: torch.Tensor,
    radius_codes: torch.Tensor,
    radius_grid: torch.Tensor,
    codebook: torch.Tensor,
    permutation: torch.Tensor,
    out_features: int,
    scratch: torch.Tensor,
) -> torch.Tensor:
    """`sage_forward` with scratch memory the caller owns: a zero-filled uint8 tensor on x's device of
    at least `sageb200_workspace_bytes(rows, out_features, K)` bytes, 256-byte aligned, used by one
    stream at a time (the kernels leave its arrival counters at zero).  A caller that runs many
    linears on a stream of its own - a decode step being captured in a CUDA graph - thereby avoids
    the temporary and its fill kernel that `sage_forward` takes on any stream but the default one."""
    return _lib.native_module().sage_forward(x, packed_codes, radius_codes, radius_grid, codebook, permutation,
                                             out_features, scratch)


def _fake(x, packed_codes, radius_codes, radius_grid, codebook, permutation, out_features):
    return x.new_empty((*x.shape[:-1], out_features))


sage = _lib.register_operator(
    "sage",
    "(Tensor x, Tensor packed_codes, Tensor radius_codes, Tensor radius_grid, Tensor codebook, Tensor permutation, "
    "SymInt out_features) -> Tensor",
    _fake,
)


_lib.register_typed_operator()


def sage_dequantize(
    packed_codes: torch.Tensor,
    radius_codes: torch.Tensor,
    radius_grid: torch.Tensor,
    codebook: torch.Tensor,
    permutation: torch.Tensor,
    out_features: int,
    *,
    original_order: bool = True,
) -> torch.Tensor:
    """Dense FP16 weight [out_features, K], bit-exact with the reference's dequantisation."""
    return _lib.native_module().dequantize(packed_codes, radius_codes, radius_grid, codebook, permutation, out_features,
                                           original_order)


def sage_grouped(problems: list[tuple], out_features: list[int], activation: tuple | None = None,
                 outputs: list[torch.Tensor] | None = None) -> list[torch.Tensor]:
    """Several packed linears (rows <= 16 each) in one launch.

    `outputs` (optional): contiguous FP16 tensors to write into, one per problem, instead of fresh
    ones - e.g. row ranges of one tensor when the problems are row blocks of the same linear.

    `problems[i]` = (x, packed_codes, radius_codes, radius_grid, codebook, permutation).
    `activation` = (kind, eps, a, b, weight, residual_out) fuses the producer of the shared
    input into the launch (kind 1: residual add + RMSNorm, kind 2: SwiGLU; see
    `sageb200_activation` in include/sage_b200.h); `x` then only supplies shape and dtype.
    """
    if len(problems) > _lib.MAX_GROUPED:
        raise RuntimeError("too many problems for one grouped launch")
    lib = _lib.load()
    array = (_lib.Problem * len(problems))()
    given, outputs = outputs, []
    device = problems[0][0].device
    for i, ((x, codes, radii, grid, book, perm), n) in enumerate(zip(problems, out_features)):
        k = _check_layout(x, codes, radii, grid, book, perm, n)
        rows = x.numel() // k
        if given is None:
            y = torch.empty((*x.shape[:-1], n), dtype=x.dtype, device=x.device)
        else:
            y = given[i]
            if not (y.is_contiguous() and y.dtype == x.dtype and y.device == x.device and y.numel() == rows * n):
                raise RuntimeError("SAGE grouped outputs must be contiguous FP16 tensors of rows x out_features")
        outputs.append(y)
        array[i] = _lib.Problem(
            x.data_ptr(), codes.data_ptr(), radii.data_ptr(), grid.data_ptr(), book.data_ptr(),
            perm.data_ptr() if perm.numel() else None, y.data_ptr(), rows, n, k, book.shape[1],
        )
    with torch.cuda.device(device), _WORKSPACE_LOCK:
        stream = torch.cuda.current_stream(device).cuda_stream
        if activation is None:
            total = lib.sageb200_grouped_workspace_bytes(array, len(problems))
            workspace = _workspace(device, stream, total) if total else None
            _lib.check(
                lib.sageb200_linear_grouped(
                    array,
                    len(problems),
                    workspace.data_ptr() if workspace is not None else None,
                    workspace.numel() if workspace is not None else 0,
                    stream,
                )
            )
        else:
            kind, eps, a, b, weight, residual_out = activation
            pointer = lambda t: t.data_ptr() if t is not None else None  # noqa: E731
            act = _lib.Activation(kind, eps, pointer(a), pointer(b), pointer(weight), pointer(residual_out))
            total = lib.sageb200_fused_workspace_bytes(array, len(problems))
            workspace = _workspace(device, stream, total) if total else None
            _lib.check(
                lib.sageb200_linear_grouped_fused(
                    array,
                    len(problems),
                    ctypes.byref(act),
                    workspace.data_ptr() if workspace is not None else None,
                    workspace.numel() if workspace is not None else 0,
                    stream,
                )
            )
    return outputs
