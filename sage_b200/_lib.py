"""ctypes binding of libsage_b200.so (the C ABI declared in include/sage_b200.h), and the C++ side of the
torch operators (`_native.so`).

Neither is touched at import: `load` brings in both the first time one of them is needed, so a tree may be built
after the package was imported, and a process that only builds maps no compiled code of this package.
There is no fallback: if one is missing or a call fails, an exception is raised.
"""

from __future__ import annotations

import ctypes
import importlib
import os
import pathlib
import threading

import torch

PACKAGE = pathlib.Path(__file__).resolve().parent
# SAGEB200_LIBRARY selects another build of the same library (the profiling build that
# `python -m sage_b200.build --trace` writes beside the product one)
LIBRARY = pathlib.Path(os.environ.get("SAGEB200_LIBRARY", PACKAGE / "libsage_b200.so"))

OK = 0
MAX_GROUPED = 16

NATIVE_SYMBOLS = ("sageb200_status_string", "sageb200_workspace_bytes", "sageb200_linear",
                  "sageb200_sph_workspace_bytes", "sageb200_sph_linear_scratch",
                  "sageb200_linear_takes_type", "sageb200_linear_typed",
                  "sageb200_dequant", "sageb200_pack_logits", "sageb200_codebook_logits", "sageb200_invert_permutation")


# every symbol include/sage_b200.h declares
EXPORTED = (
    "sageb200_version",
    "sageb200_status_string",
    "sageb200_gemv_fuses_permutation",
    "sageb200_gemm_splits",
    "sageb200_workspace_bytes",
    "sageb200_linear",
    "sageb200_linear_takes_type",
    "sageb200_linear_typed",
    "sageb200_linear_rows_workspace_bytes",
    "sageb200_linear_rows",
    "sageb200_linear_grouped",
    "sageb200_grouped_workspace_bytes",
    "sageb200_fused_workspace_bytes",
    "sageb200_linear_grouped_fused",
    "sageb200_experts_workspace_bytes",
    "sageb200_experts",
    "sageb200_expert_blocks_workspace_bytes",
    "sageb200_expert_blocks",
    "sageb200_expert_mlp_fits",
    "sageb200_expert_mlp",
    "sageb200_dequant",
    "sageb200_pack_spherical",
    "sageb200_pack_logits",
    "sageb200_codebook_logits",
    "sageb200_invert_permutation",
    "sageb200_host_staging_bytes",
    "sageb200_linear_host",
    "sageb200_set_tuning",
    "sageb200_sph_linear",
    "sageb200_sph_workspace_bytes",
    "sageb200_sph_linear_scratch",
    "sageb200_sph_dequant",
    "sageb200_linear_static",
    "sageb200_clear_status",
    "sageb200_launch_count",
    "sageb200_glue_launch_count",
)

# every symbol include/sage_b200_debug.h declares (tuning and profiling aids)
EXPORTED_DEBUG = (
    "sageb200_debug_plan",
    "sageb200_set_pdl",
    "sageb200_debug_trace",
    "sageb200_debug_gemm_pairs",
    "sageb200_debug_gemm_plan",
)


# every symbol include/sage_b200_decode.h declares
EXPORTED_DECODE = (
    "sageb200_glue_embed",
    "sageb200_glue_add_rmsnorm",
    "sageb200_glue_add_rmsnorm_permuted",
    "sageb200_glue_swiglu_permuted",
    "sageb200_glue_qk_norm_rope_cache",
    "sageb200_glue_attention_scratch_bytes",
    "sageb200_glue_attention_decode",
    "sageb200_glue_attention_step",
    "sageb200_glue_attention_step_permuted",
    "sageb200_glue_prefill_qk_norm_rope_cache",
    "sageb200_glue_prefill_attention",
    "sageb200_glue_lm_head_step_scratch_bytes",
    "sageb200_glue_lm_head_step",
    "sageb200_glue_moe_route",
    "sageb200_glue_moe_mix",
    "sageb200_glue_dispatch_plan",
    "sageb200_glue_dispatch_rows",
    "sageb200_glue_combine_rows",
    "sageb200_glue_combine_mix",
    "sageb200_glue_swiglu",
    "sageb200_glue_lm_head",
    "sageb200_glue_argmax_advance",
    "sageb200_prompt_workspace_bytes",
    "sageb200_prompt_layers",
    "sageb200_mega_workspace_bytes",
    "sageb200_mega_prepare",
    "sageb200_mega_step",
)


# every symbol include/sage_b200_peer.h declares
EXPORTED_PEER = (
    "sageb200_peer_exchange_bytes",
    "sageb200_peer_create",
    "sageb200_peer_open",
    "sageb200_peer_close",
    "sageb200_peer_destroy",
    "sageb200_peer_all_reduce",
)
PEER_MAX_WORLD = 8
PEER_HANDLE_BYTES = 64


class Activation(ctypes.Structure):
    """struct sageb200_activation."""

    _fields_ = [
        ("kind", ctypes.c_int),
        ("eps", ctypes.c_float),
        ("a", ctypes.c_void_p),
        ("b", ctypes.c_void_p),
        ("weight", ctypes.c_void_p),
        ("residual_out", ctypes.c_void_p),
    ]


class ExpertStack(ctypes.Structure):
    """struct sageb200_expert_stack."""

    _fields_ = [
        ("codes", ctypes.c_void_p),
        ("radii", ctypes.c_void_p),
        ("grid", ctypes.c_void_p),
        ("book", ctypes.c_void_p),
        ("perm", ctypes.c_void_p),
        ("experts", ctypes.c_int),
        ("first_expert", ctypes.c_int),
        ("n", ctypes.c_int),
        ("k", ctypes.c_int),
        ("entries", ctypes.c_int),
    ]


class MegaLinear(ctypes.Structure):
    """struct sageb200_mega_linear."""

    _fields_ = [
        ("codes", ctypes.c_void_p),
        ("radii", ctypes.c_void_p),
        ("grid", ctypes.c_void_p),
        ("book", ctypes.c_void_p),
        ("perm", ctypes.c_void_p),
        ("n", ctypes.c_int),
        ("k", ctypes.c_int),
        ("entries", ctypes.c_int),
    ]


class MegaLayer(ctypes.Structure):
    """struct sageb200_mega_layer."""

    _fields_ = [(name, MegaLinear) for name in ("q", "k", "v", "o", "gate", "up", "down")] + [
        (name, ctypes.c_void_p) for name in ("input_norm", "post_norm", "q_norm", "k_norm", "k_cache", "v_cache")
    ]


class MegaModel(ctypes.Structure):
    """struct sageb200_mega_model."""

    _fields_ = [(name, ctypes.c_int) for name in ("layers", "hidden", "heads", "kv_heads", "head_dim",
                                                  "intermediate", "vocab", "max_seq")] + [
        ("eps", ctypes.c_float)] + [
        (name, ctypes.c_void_p) for name in ("embed", "lm_head", "final_norm", "cos_table", "sin_table")]


class Problem(ctypes.Structure):
    """struct sageb200_problem."""

    _fields_ = [
        ("x", ctypes.c_void_p),
        ("codes", ctypes.c_void_p),
        ("radii", ctypes.c_void_p),
        ("grid", ctypes.c_void_p),
        ("book", ctypes.c_void_p),
        ("perm", ctypes.c_void_p),
        ("y", ctypes.c_void_p),
        ("rows", ctypes.c_int),
        ("n", ctypes.c_int),
        ("k", ctypes.c_int),
        ("entries", ctypes.c_int),
    ]


_handle: ctypes.CDLL | None = None
_native = None
_load_lock = threading.RLock()


def native_module():
    """The C++ side of the operators."""
    if _native is None:
        load()
    return _native


def load() -> ctypes.CDLL:
    """Load the shared library and the operators' C++ side once; raise if they have not been built."""
    global _handle, _native
    if _handle is not None:
        return _handle
    with _load_lock:
        if _handle is None:
            if not LIBRARY.exists():
                raise RuntimeError(
                    f"{LIBRARY} is missing: build it with `python -m sage_b200.build` "
                    "(sage_b200 has no CPU or PyTorch fallback)"
                )
            lib, module = _bind_library(), _import_native()
            module.bind({name: ctypes.cast(getattr(lib, name), ctypes.c_void_p).value for name in NATIVE_SYMBOLS})
            while _unregistered:
                module.register_kernels(*_unregistered.pop())
            _native, _handle = module, lib
    return _handle


def _import_native():
    name = f"{__package__}._native"
    importlib.invalidate_caches()  # (the file may be younger than the folder's cached listing)
    try:
        module = importlib.import_module(name)
    except ModuleNotFoundError as error:  # (any other failure to import it is not a missing build, and says what it is)
        if error.name != name:
            raise
        raise RuntimeError("sage_b200/_native.so is missing: build it with `python -m sage_b200.build`") from None
    if module.torch_version != str(torch.__version__):
        raise RuntimeError(f"sage_b200/_native.so was built for torch {module.torch_version} and this is torch "
                           f"{torch.__version__}: build it again with `python -m sage_b200.build`")
    return module


def _bind_library() -> ctypes.CDLL:
    """The shared library with its functions' types."""
    lib = ctypes.CDLL(str(LIBRARY))
    vp, ci, sz = ctypes.c_void_p, ctypes.c_int, ctypes.c_size_t
    lib.sageb200_version.restype = ci
    lib.sageb200_version.argtypes = []
    lib.sageb200_status_string.restype = ctypes.c_char_p
    lib.sageb200_status_string.argtypes = [ci]
    lib.sageb200_gemv_fuses_permutation.restype = ci
    lib.sageb200_gemv_fuses_permutation.argtypes = [ci, ci]
    lib.sageb200_gemm_splits.restype = ci
    lib.sageb200_gemm_splits.argtypes = [ci, ci, ci, ci]
    lib.sageb200_workspace_bytes.restype = sz
    lib.sageb200_workspace_bytes.argtypes = [ci, ci, ci]
    lib.sageb200_linear.restype = ci
    lib.sageb200_linear.argtypes = [vp, vp, vp, vp, vp, vp, vp, vp, sz, ci, ci, ci, ci, vp]
    lib.sageb200_linear_takes_type.restype = ci
    lib.sageb200_linear_takes_type.argtypes = [ci] * 3
    lib.sageb200_linear_typed.restype = ci
    lib.sageb200_linear_typed.argtypes = [vp, ci] + [vp] * 8 + [sz] + [ci] * 4 + [vp]
    lib.sageb200_linear_rows_workspace_bytes.restype = sz
    lib.sageb200_linear_rows_workspace_bytes.argtypes = [ctypes.POINTER(Problem), ci]
    lib.sageb200_linear_rows.restype = ci
    lib.sageb200_linear_rows.argtypes = [ctypes.POINTER(Problem), ci, vp, sz, vp]
    lib.sageb200_grouped_workspace_bytes.restype = sz
    lib.sageb200_grouped_workspace_bytes.argtypes = [ctypes.POINTER(Problem), ci]
    lib.sageb200_fused_workspace_bytes.restype = sz
    lib.sageb200_fused_workspace_bytes.argtypes = [ctypes.POINTER(Problem), ci]
    lib.sageb200_linear_grouped_fused.restype = ci
    lib.sageb200_linear_grouped_fused.argtypes = [ctypes.POINTER(Problem), ci, ctypes.POINTER(Activation), vp, sz, vp]
    lib.sageb200_experts_workspace_bytes.restype = sz
    lib.sageb200_experts_workspace_bytes.argtypes = [ctypes.POINTER(ExpertStack), ci, ci]
    lib.sageb200_experts.restype = ci
    lib.sageb200_experts.argtypes = [vp, ctypes.c_longlong, ctypes.POINTER(ExpertStack), ctypes.POINTER(vp), ci, vp, ci, vp, sz, vp]
    lib.sageb200_linear_grouped.restype = ci
    lib.sageb200_linear_grouped.argtypes = [ctypes.POINTER(Problem), ci, vp, sz, vp]
    lib.sageb200_dequant.restype = ci
    lib.sageb200_dequant.argtypes = [vp, vp, vp, vp, vp, vp, ci, ci, ci, vp]
    lib.sageb200_host_staging_bytes.restype = sz
    lib.sageb200_host_staging_bytes.argtypes = [ci, ci, ci]
    lib.sageb200_linear_host.restype = ci
    lib.sageb200_linear_host.argtypes = [vp, vp, vp, vp, vp, vp, vp, vp, sz, ci, ci, ci, ci, vp]
    lib.sageb200_set_tuning.restype = ci
    lib.sageb200_set_tuning.argtypes = [ci, ci, ci, ci]
    lib.sageb200_linear_static.restype = ci
    lib.sageb200_linear_static.argtypes = [vp, vp, vp, vp, vp, vp, vp, ci, ci, ci, ci, vp]
    lib.sageb200_sph_linear.restype = ci
    lib.sageb200_sph_linear.argtypes = [vp] * 7 + [ci] * 3 + [vp]
    lib.sageb200_sph_workspace_bytes.restype = sz
    lib.sageb200_sph_workspace_bytes.argtypes = [ci, ci, ci]
    lib.sageb200_sph_linear_scratch.restype = ci
    lib.sageb200_sph_linear_scratch.argtypes = [vp] * 8 + [sz] + [ci] * 3 + [vp]
    lib.sageb200_sph_dequant.restype = ci
    lib.sageb200_sph_dequant.argtypes = [vp] * 6 + [ci] * 2 + [vp]
    lib.sageb200_debug_plan.restype = ci
    lib.sageb200_debug_plan.argtypes = [ci] * 5 + [ctypes.POINTER(ci)]
    lib.sageb200_expert_blocks_workspace_bytes.restype = sz
    lib.sageb200_expert_blocks_workspace_bytes.argtypes = [ctypes.POINTER(ExpertStack), ci, ci]
    lib.sageb200_expert_blocks.restype = ci
    lib.sageb200_expert_blocks.argtypes = [vp, ctypes.POINTER(ExpertStack), ctypes.POINTER(vp), ci, vp, ci, ci, vp, sz, vp]
    lib.sageb200_expert_mlp_fits.restype = ci
    lib.sageb200_expert_mlp_fits.argtypes = [ci] * 4
    lib.sageb200_expert_mlp.restype = ci
    lib.sageb200_expert_mlp.argtypes = [vp, ctypes.POINTER(ExpertStack), vp, vp, vp, ci, ci, vp]
    lib.sageb200_pack_spherical.restype = ci
    lib.sageb200_pack_spherical.argtypes = [vp] * 7 + [ci] * 4 + [vp]
    lib.sageb200_pack_logits.restype = ci
    lib.sageb200_pack_logits.argtypes = [vp, vp, ci] + [vp] * 5 + [ci] * 4 + [vp]
    lib.sageb200_codebook_logits.restype = ci
    lib.sageb200_codebook_logits.argtypes = [vp, vp, ci, ctypes.c_float, ctypes.c_float, ci, vp]
    lib.sageb200_invert_permutation.restype = ci
    lib.sageb200_invert_permutation.argtypes = [vp, vp, vp, ci, vp]
    lib.sageb200_clear_status.restype = ci
    lib.sageb200_clear_status.argtypes = []
    lib.sageb200_set_pdl.restype = ci
    lib.sageb200_set_pdl.argtypes = [ci]
    lib.sageb200_debug_trace.restype = ci
    lib.sageb200_debug_trace.argtypes = [vp]
    lib.sageb200_debug_gemm_pairs.restype = ci
    lib.sageb200_debug_gemm_pairs.argtypes = [ci]
    lib.sageb200_debug_gemm_plan.restype = ci
    lib.sageb200_debug_gemm_plan.argtypes = [ci] * 5 + [ctypes.POINTER(ci)]
    lib.sageb200_launch_count.restype = ctypes.c_ulonglong
    lib.sageb200_launch_count.argtypes = []
    lib.sageb200_glue_launch_count.restype = ctypes.c_ulonglong
    lib.sageb200_glue_launch_count.argtypes = []
    # decode glue (include/sage_b200_decode.h)
    fl, ll = ctypes.c_float, ctypes.c_longlong
    lib.sageb200_glue_embed.restype = ci
    lib.sageb200_glue_embed.argtypes = [vp, vp, vp, ci, ci, ci, vp]
    lib.sageb200_glue_add_rmsnorm.restype = ci
    lib.sageb200_glue_add_rmsnorm.argtypes = [vp, vp, vp, vp, ci, ci, fl, vp]
    lib.sageb200_glue_add_rmsnorm_permuted.restype = ci
    lib.sageb200_glue_add_rmsnorm_permuted.argtypes = [vp, vp, vp, vp, ctypes.POINTER(vp), ctypes.POINTER(vp), ci, ci, ci, fl, vp]
    lib.sageb200_glue_swiglu_permuted.restype = ci
    lib.sageb200_glue_swiglu_permuted.argtypes = [vp, vp, vp, vp, ci, ci, ci, vp]
    lib.sageb200_glue_qk_norm_rope_cache.restype = ci
    lib.sageb200_glue_qk_norm_rope_cache.argtypes = [vp] * 10 + [ci] * 5 + [fl, vp]
    lib.sageb200_glue_attention_scratch_bytes.restype = sz
    lib.sageb200_glue_attention_scratch_bytes.argtypes = [ci, ci, ci]
    lib.sageb200_glue_attention_step.restype = ci
    lib.sageb200_glue_attention_step.argtypes = [vp] * 11 + [ci] * 6 + [ctypes.c_float, vp]
    lib.sageb200_glue_attention_step_permuted.restype = ci
    lib.sageb200_glue_attention_step_permuted.argtypes = [vp] * 12 + [ci] * 6 + [ctypes.c_float, vp]
    lib.sageb200_glue_prefill_qk_norm_rope_cache.restype = ci
    lib.sageb200_glue_prefill_qk_norm_rope_cache.argtypes = [vp] * 10 + [ci] * 6 + [ctypes.c_float, vp]
    lib.sageb200_glue_prefill_attention.restype = ci
    lib.sageb200_glue_prefill_attention.argtypes = [vp] * 5 + [ci] * 6 + [vp]
    lib.sageb200_glue_moe_route.restype = ci
    lib.sageb200_glue_moe_route.argtypes = [vp] * 7 + [ci] * 4 + [ctypes.c_float, vp]
    lib.sageb200_glue_dispatch_plan.restype = ci
    lib.sageb200_glue_dispatch_plan.argtypes = [vp, vp, vp, ci, ci, ci, ci, ci, vp]
    lib.sageb200_glue_dispatch_rows.restype = ci
    lib.sageb200_glue_dispatch_rows.argtypes = [vp, vp, vp, ci, ci, ci, ci, vp]
    lib.sageb200_glue_combine_rows.restype = ci
    lib.sageb200_glue_combine_rows.argtypes = [vp, vp, vp, ci, ci, ci, vp]
    lib.sageb200_glue_combine_mix.restype = ci
    lib.sageb200_glue_combine_mix.argtypes = [vp] * 4 + [ci] * 4 + [vp]
    lib.sageb200_glue_moe_mix.restype = ci
    lib.sageb200_glue_moe_mix.argtypes = [vp] * 3 + [ci] * 3 + [vp]
    lib.sageb200_glue_lm_head_step_scratch_bytes.restype = sz
    lib.sageb200_glue_lm_head_step_scratch_bytes.argtypes = [ci, ci]
    lib.sageb200_glue_lm_head_step.restype = ci
    lib.sageb200_glue_lm_head_step.argtypes = [vp] * 11 + [ci] * 3 + [ctypes.c_float, ci, ci, vp]
    lib.sageb200_glue_attention_decode.restype = ci
    lib.sageb200_glue_attention_decode.argtypes = [vp] * 6 + [ci] * 6 + [vp]
    lib.sageb200_glue_swiglu.restype = ci
    lib.sageb200_glue_swiglu.argtypes = [vp, vp, vp, ll, vp]
    lib.sageb200_glue_lm_head.restype = ci
    lib.sageb200_glue_lm_head.argtypes = [vp, vp, vp, ci, ci, ci, ci, vp]
    lib.sageb200_glue_argmax_advance.restype = ci
    lib.sageb200_glue_argmax_advance.argtypes = [vp] * 5 + [ci, ci, ci, vp]
    lib.sageb200_prompt_workspace_bytes.restype = sz
    lib.sageb200_prompt_workspace_bytes.argtypes = [ctypes.POINTER(MegaModel), ctypes.POINTER(MegaLayer), ci]
    lib.sageb200_prompt_layers.restype = ci
    lib.sageb200_prompt_layers.argtypes = [ctypes.POINTER(MegaModel), ctypes.POINTER(MegaLayer), vp, vp, vp, vp, vp, sz,
                                           ci, ci, ci, vp]
    lib.sageb200_mega_workspace_bytes.restype = sz
    lib.sageb200_mega_workspace_bytes.argtypes = [ctypes.POINTER(MegaModel), ci]
    lib.sageb200_mega_prepare.restype = ci
    lib.sageb200_mega_prepare.argtypes = [ctypes.POINTER(MegaModel), ctypes.POINTER(MegaLayer), vp, sz, vp]
    lib.sageb200_mega_step.restype = ci
    lib.sageb200_mega_step.argtypes = [ctypes.POINTER(MegaModel), vp, vp, vp, vp, vp, vp, ci, vp]
    # all-reduce over peer memory (include/sage_b200_peer.h)
    lib.sageb200_peer_exchange_bytes.restype = sz
    lib.sageb200_peer_exchange_bytes.argtypes = [ci, ll]
    lib.sageb200_peer_create.restype = ci
    lib.sageb200_peer_create.argtypes = [ci, ll, ctypes.POINTER(vp), ctypes.POINTER(ctypes.c_ubyte)]
    lib.sageb200_peer_open.restype = ci
    lib.sageb200_peer_open.argtypes = [ctypes.POINTER(ctypes.c_ubyte), ctypes.POINTER(vp)]
    lib.sageb200_peer_close.restype = ci
    lib.sageb200_peer_close.argtypes = [vp]
    lib.sageb200_peer_destroy.restype = ci
    lib.sageb200_peer_destroy.argtypes = [vp]
    lib.sageb200_peer_all_reduce.restype = ci
    lib.sageb200_peer_all_reduce.argtypes = [ctypes.POINTER(vp), ci, ci, ll, vp, ll, vp]
    if "SAGEB200_PDL" in os.environ:  # debug switch: which kernel families launch dependently
        lib.sageb200_set_pdl(int(os.environ["SAGEB200_PDL"]))
    return lib


def register_operator(name: str, schema: str, fake):
    """Define `wvq::<name>` (or `sage_b200::<name>` when the reference package already owns the former in
    this process) with its fake kernel; the CUDA and autograd kernels are the C++ side's."""
    for namespace in ("wvq", "sage_b200"):
        try:
            library = _define(namespace, name, schema)
            break
        except RuntimeError:
            if namespace == "sage_b200":
                raise
    return _set_kernels(library, namespace, name, fake, derivative=True)


def register_typed_operator():
    """`sage_b200::linear`: a packed linear of FP16 or BF16 rows with its bias, the module's whole arithmetic in one
    operator (internal: the modules call it where no derivative is asked for)."""
    library = _define("sage_b200", "linear",
                      "(Tensor x, Tensor packed_codes, Tensor radius_codes, Tensor radius_grid, Tensor codebook, "
                      "Tensor permutation, SymInt out_features, Tensor? bias) -> Tensor")
    _set_kernels(library, "sage_b200", "linear", lambda x, codes, radii, grid, book, perm, n, bias:
                 x.new_empty((*x.shape[:-1], n)), derivative=False)


def _define(namespace: str, name: str, schema: str) -> torch.library.Library:
    library = torch.library.Library(namespace, "FRAGMENT")
    library.define(name + schema, tags=(torch.Tag.pt2_compliant_tag, torch.Tag.needs_fixed_stride_order))
    return library


def _set_kernels(library: torch.library.Library, namespace: str, name: str, fake, *, derivative: bool):
    torch.library.register_fake(f"{namespace}::{name}", fake, lib=library)
    op = getattr(getattr(torch.ops, namespace), name).default

    # The C++ kernels take the CUDA key, and AutogradCUDA where `derivative`, once `load` has registered them.  Until
    # then a call lands on one of these two, which load them and dispatch again; afterwards only what has no kernel
    # still does (theirs are the general keys, which a key's own kernel goes before).
    def autograd(*args):
        if _native is None and LIBRARY.exists():
            load()
            return op(*args)
        with torch._C._AutoDispatchBelowAutograd():
            return op(*args)

    def backend(*args):
        if _native is None:
            load()
            return op(*args)
        raise NotImplementedError(f"Could not run '{namespace}::{name}' on {args[0].device}: it has a CUDA kernel only")

    if derivative:
        library.impl(name, autograd, "Autograd")
    library.impl(name, backend, "CompositeExplicitAutograd")
    _libraries.append(library)
    with _load_lock:
        if _native is None:
            _unregistered.append((name, namespace))
        else:
            _native.register_kernels(name, namespace)
    return op


_unregistered: list = []  # operators whose C++ kernels `load` has still to register
_libraries: list = []  # the registrations live as long as the process


def check(status: int) -> None:
    """Raise RuntimeError (as the reference's TORCH_CHECK does) on a non-zero status."""
    if status != OK:
        text = load().sageb200_status_string(status).decode()
        raise RuntimeError(f"sage_b200: {text} (status {status})")
