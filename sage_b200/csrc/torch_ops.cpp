// The torch side of the packed linears in C++: the `sage` and `sphquant` operators' CUDA and
// autograd kernels, and the functions the Python modules call.
//
// What bounds it: a packed linear of one token runs for 3-10 us on the GPU, and the same call took
// 42-45 us of host time as Python (the custom-operator wrapper, a dozen attribute checks per
// argument, ctypes marshalling), so every small call waited for the host.  Here a call is one
// argument parse, the same checks on TensorImpl fields, one allocation and the C-ABI call.
// Measured on k_proj of the 4B model at one row, calls back to back: 44.8 -> 9.6 us.
//
// The C ABI functions come as addresses from the ctypes binding (`bind`), so that both sides use
// the one loaded library, whichever build of it was selected.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/core/dispatch/Dispatcher.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/library.h>

#include <memory>
#include <mutex>
#include <string>

#include "../../include/sage_b200.h"

namespace {

using at::Tensor;

struct Abi {
  decltype(&sageb200_status_string) status_string = nullptr;
  decltype(&sageb200_workspace_bytes) workspace_bytes = nullptr;
  decltype(&sageb200_linear) linear = nullptr;
  decltype(&sageb200_linear_takes_type) linear_takes_type = nullptr;
  decltype(&sageb200_linear_typed) linear_typed = nullptr;
  decltype(&sageb200_sph_workspace_bytes) sph_workspace_bytes = nullptr;
  decltype(&sageb200_sph_linear_scratch) sph_linear_scratch = nullptr;
  decltype(&sageb200_dequant) dequant = nullptr;
  decltype(&sageb200_pack_logits) pack_logits = nullptr;
  decltype(&sageb200_codebook_logits) codebook_logits = nullptr;
  decltype(&sageb200_invert_permutation) invert_permutation = nullptr;
} abi;

std::string op_namespace[2];  // where `sage` and `sphquant` are registered

void check_status(int status) {
  TORCH_CHECK(status == SAGEB200_OK, "sage_b200: ", abi.status_string(status), " (status ", status, ")");
}

// The first call loads the library (which binds these addresses) or raises that it is missing.
void check_bound() {
  if (abi.linear) return;
  const PyGILState_STATE state = PyGILState_Ensure();
  PyObject *module = PyImport_ImportModule("sage_b200._lib");
  PyObject *result = module ? PyObject_CallMethod(module, "load", nullptr) : nullptr;
  const bool loaded = result != nullptr;
  Py_XDECREF(result);
  Py_XDECREF(module);
  if (!loaded) {
    python_error error;
    error.persist();
    PyGILState_Release(state);
    throw error;
  }
  PyGILState_Release(state);
  TORCH_CHECK(abi.linear, "sage_b200: the C ABI is not bound");
}

constexpr int64_t kCounterRegion = 64 * 1024;  // the front of the scratch that has to be zero
constexpr int kMaxDevices = 64;

// The default stream's scratch: one zero-filled buffer per device for all threads, grown on demand (the kernels leave
// its counters zero).  A call is several launches that hand data to one another through the buffer (gather or staging,
// then the matmul), so it keeps the device's lock until all of them are enqueued: another thread's call then comes
// behind it on the stream and finds the buffer free.  A buffer that was outgrown goes back to the caching allocator,
// which reuses it in stream order, and no captured graph can hold it because the default stream cannot be captured.
struct SharedScratch {
  std::mutex mutex;
  Tensor buffer;
};
SharedScratch &shared_scratch(int device) {
  static auto *all = new SharedScratch[kMaxDevices];  // never destroyed: the allocator may be gone by then
  return all[device];
}

// Scratch of one call; lives until the call's launches are enqueued.
struct Scratch {
  Tensor buffer;                     // undefined for a call that needs none
  std::unique_lock<std::mutex> use;  // held where the buffer is a shared one
  void *data() const { return buffer.defined() ? buffer.data_ptr() : nullptr; }
  size_t bytes() const { return buffer.defined() ? static_cast<size_t>(buffer.numel()) : 0; }
};

// Scratch of a call that brings none.
Scratch scratch_for(const Tensor &x, int64_t bytes, cudaStream_t stream) {
  Scratch scratch;
  if (bytes == 0) return scratch;
  const auto options = x.options().dtype(at::kByte);
  if (stream == nullptr) {
    SharedScratch &shared = shared_scratch(x.get_device());
    scratch.use = std::unique_lock<std::mutex>(shared.mutex);
    if (!shared.buffer.defined() || shared.buffer.numel() < bytes)
      shared.buffer = at::zeros({std::max<int64_t>(bytes, kCounterRegion)}, options);
    scratch.buffer = shared.buffer;
    return scratch;
  }
  // Any other stream may be under capture, or belong to a compiled graph whose memory pool accepts
  // no allocation that outlives the call: a temporary of this call, its counters zeroed.
  scratch.buffer = at::empty({bytes}, options);
  C10_CUDA_CHECK(cudaMemsetAsync(scratch.buffer.data_ptr(), 0, std::min(bytes, kCounterRegion), stream));
  return scratch;
}

bool shape_is(const Tensor &t, std::initializer_list<int64_t> want) {
  const auto sizes = t.sizes();
  return sizes.size() == want.size() && std::equal(sizes.begin(), sizes.end(), want.begin());
}

int64_t check_layout(c10::Device device, int64_t k, const Tensor &codes, const Tensor &radii, const Tensor &grid,
                     const Tensor &book, const Tensor &perm, int64_t n) {
  for (const Tensor *t : {&codes, &radii, &grid, &book, &perm})
    TORCH_CHECK(t->device() == device && t->is_contiguous(), "SAGE buffers must be contiguous and on the input device");
  const int64_t tiles = (n + 15) / 16, groups = k / 128;
  TORCH_CHECK(k > 0 && k % 128 == 0 && n > 0, "SAGE requires positive N and K divisible by 128");
  TORCH_CHECK(book.dim() == 3 && book.size(0) == 4 && book.size(2) == 2 &&
                  (book.size(1) == 64 || book.size(1) == 128 || book.size(1) == 256),
              "SAGE codebook must have shape [4, 64/128/256, 2]");
  TORCH_CHECK(codes.scalar_type() == at::kInt && shape_is(codes, {tiles, groups, 16, 8}) &&
                  radii.scalar_type() == at::kInt && shape_is(radii, {tiles, groups, 16}) &&
                  grid.scalar_type() == at::kHalf && shape_is(grid, {tiles, groups, 16, 2}) &&
                  book.scalar_type() == at::kHalf && perm.scalar_type() == at::kInt && perm.dim() == 1 &&
                  (perm.numel() == 0 || perm.numel() == k),
              "Invalid SAGE packed layout");
  TORCH_CHECK(!(reinterpret_cast<uintptr_t>(grid.data_ptr()) & 3) && !(reinterpret_cast<uintptr_t>(book.data_ptr()) & 3),
              "SAGE grid and codebook require 4-byte aligned storage");
  return k;
}

// Checks and messages of the reference's entry point (csrc/bindings.cpp:13-48).
int64_t check_sage(const Tensor &x, const Tensor &codes, const Tensor &radii, const Tensor &grid, const Tensor &book,
                   const Tensor &perm, int64_t n, at::ScalarType type = at::kHalf) {
  TORCH_CHECK(x.is_cuda() && x.scalar_type() == type && x.is_contiguous() && x.dim() >= 1,
              "SAGE requires contiguous CUDA FP16 input");
  return check_layout(x.device(), x.size(-1), codes, radii, grid, book, perm, n);
}

Tensor empty_output(const Tensor &x, int64_t n) {
  c10::SmallVector<int64_t, 4> shape(x.sizes().begin(), x.sizes().end());
  shape.back() = n;
  return at::empty(shape, x.options());
}

// `scratch` (optional): the caller's own zero-filled scratch.
Tensor sage_run(const Tensor &x, const Tensor &codes, const Tensor &radii, const Tensor &grid, const Tensor &book,
                const Tensor &perm, int64_t n, const Tensor *scratch) {
  check_bound();
  const int64_t k = check_sage(x, codes, radii, grid, book, perm, n);
  const c10::cuda::CUDAGuard guard(x.device());
  Tensor y = empty_output(x, n);
  const int64_t rows = x.numel() / k;
  if (rows == 0) return y;
  TORCH_CHECK(rows <= 65535, "SAGE launch dimensions exceed supported range");
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(x.get_device()).stream();
  const int64_t bytes = static_cast<int64_t>(abi.workspace_bytes(static_cast<int>(rows), static_cast<int>(n), static_cast<int>(k)));
  Scratch workspace;
  if (bytes && scratch) {
    TORCH_CHECK(scratch->device() == x.device() && scratch->scalar_type() == at::kByte && scratch->numel() >= bytes,
                "SAGE scratch must be a uint8 tensor of at least ", bytes, " bytes on the input device");
    workspace.buffer = *scratch;
  } else {
    workspace = scratch_for(x, bytes, stream);
  }
  check_status(abi.linear(x.data_ptr(), codes.data_ptr(), radii.data_ptr(), grid.data_ptr(), book.data_ptr(),
                          perm.numel() ? perm.data_ptr<int32_t>() : nullptr, y.data_ptr(),
                          workspace.data(), workspace.bytes(), static_cast<int>(rows), static_cast<int>(n),
                          static_cast<int>(k), static_cast<int>(book.size(1)), stream));
  return y;
}

// Checks and messages of the reference's native entry point (csrc/sphquant/sph_gemv_cuda.cu:403-446).
Tensor sph_run(const Tensor &x, const Tensor &codes, const Tensor &extra, const Tensor &scales, const Tensor &mins,
               const Tensor &book) {
  check_bound();
  const Tensor *const tensors[] = {&x, &codes, &extra, &scales, &mins, &book};
  for (const Tensor *t : tensors) TORCH_CHECK(t->is_cuda(), "sph_gemv expects CUDA tensors");
  for (const Tensor *t : {&x, &scales, &mins, &book})
    TORCH_CHECK(t->scalar_type() == at::kHalf, "sph_gemv currently supports FP16 tensors only");
  TORCH_CHECK(codes.scalar_type() == at::kShort && extra.scalar_type() == at::kInt, "invalid SPH packed tensor dtypes");
  for (const Tensor *t : tensors) TORCH_CHECK(t->is_contiguous(), "sph_gemv expects contiguous tensors");
  const int64_t k = x.size(-1), n = codes.size(0), groups = k / 128;
  TORCH_CHECK(k % 128 == 0 && groups <= 128 && k != 0, "invalid SPH input dimension");
  TORCH_CHECK(codes.dim() == 2 && codes.size(1) == k / 8, "invalid SPH packed code shape");
  TORCH_CHECK(shape_is(extra, {n, groups}) && shape_is(scales, {n, groups}) && shape_is(mins, {n, groups}),
              "invalid SPH radius metadata shape");
  TORCH_CHECK(shape_is(book, {64, 8}), "SPH codebook must have shape [64, 8]");
  const c10::cuda::CUDAGuard guard(x.device());
  Tensor y = empty_output(x, n);
  const int64_t rows = x.numel() / k;
  if (rows == 0 || n == 0) return y;
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(x.get_device()).stream();
  const Scratch workspace =
      scratch_for(x, static_cast<int64_t>(abi.sph_workspace_bytes(static_cast<int>(rows), static_cast<int>(n), static_cast<int>(k))), stream);
  check_status(abi.sph_linear_scratch(x.data_ptr(), codes.data_ptr(), extra.data_ptr(), scales.data_ptr(), mins.data_ptr(),
                                      book.data_ptr(), y.data_ptr(), workspace.data(), workspace.bytes(), static_cast<int>(rows),
                                      static_cast<int>(n), static_cast<int>(k), stream));
  return y;
}

// Dense FP16 weight [n, k]; `perm` empty: in the quantised channel order.
Tensor dequantize(const Tensor &codes, const Tensor &radii, const Tensor &grid, const Tensor &book, const Tensor &perm,
                  int64_t n, bool original_order) {
  check_bound();
  TORCH_CHECK(codes.is_cuda() && codes.dim() == 4, "Invalid SAGE packed layout");
  const int64_t k = check_layout(codes.device(), codes.size(1) * 128, codes, radii, grid, book, perm, n);
  const c10::cuda::CUDAGuard guard(codes.device());
  Tensor w = at::empty({n, k}, codes.options().dtype(at::kHalf));
  check_status(abi.dequant(codes.data_ptr(), radii.data_ptr(), grid.data_ptr(), book.data_ptr(),
                           original_order && perm.numel() ? perm.data_ptr<int32_t>() : nullptr, w.data_ptr(),
                           static_cast<int>(n), static_cast<int>(k), static_cast<int>(book.size(1)),
                           c10::cuda::getCurrentCUDAStream(codes.get_device()).stream()));
  return w;
}

// ---- the exporter's packing (sage_b200/packing.py)

struct Packed {
  Tensor codes, high, grid, mins, book, permutation;  // permutation: undefined for the identity, or without an order
};

// `order` (int64, optional): the checkpoint's inverse permutation.  Whether it is the identity decides what is
// returned, and one that is no permutation is refused (the kernels index with its inverse unchecked), so the host has
// to know; it is inverted first and the verdict read while the packing runs.
Packed pack_state(const Tensor &signs, const Tensor &indices, const Tensor &radius_logits, const Tensor &angle_logits,
                  const Tensor &order, bool sage, double scale, double offset) {
  check_bound();
  const Tensor *const inputs[] = {&signs, &indices, &radius_logits, &angle_logits};
  for (const Tensor *t : inputs)
    TORCH_CHECK(t->is_cuda() && t->device() == signs.device() && t->is_contiguous(), "packing wants contiguous tensors on one CUDA device");
  TORCH_CHECK(signs.dim() == 2 && signs.scalar_type() == at::kChar &&
                  (indices.scalar_type() == at::kInt || indices.scalar_type() == at::kLong) &&
                  radius_logits.scalar_type() == at::kFloat && angle_logits.scalar_type() == at::kFloat,
              "invalid trained tensor dtypes");
  const int64_t n = signs.size(0), k = signs.size(1), groups = k / 128, entries = angle_logits.size(0);
  TORCH_CHECK(indices.numel() == n * (k / 8) && radius_logits.numel() == n * (k / 8) && angle_logits.numel() == entries * 7,
              "invalid trained tensor shapes");
  const c10::cuda::CUDAGuard guard(signs.device());
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(signs.get_device()).stream();
  const auto options = signs.options();
  Packed out;
  // (one pinned word and event per thread and device, kept: an answer is read before the call returns)
  struct Answer {
    int *verdict = nullptr;
    cudaEvent_t event = nullptr;
  };
  static thread_local Answer answers[kMaxDevices];
  Answer &answer = answers[signs.get_device()];
  Tensor verdict;
  if (order.defined()) {
    TORCH_CHECK(order.device() == signs.device() && order.scalar_type() == at::kLong && order.is_contiguous() && order.numel() == k,
                "invalid channel permutation");
    if (!answer.verdict) {
      C10_CUDA_CHECK(cudaHostAlloc(reinterpret_cast<void **>(&answer.verdict), sizeof(int), cudaHostAllocDefault));
      C10_CUDA_CHECK(cudaEventCreateWithFlags(&answer.event, cudaEventDisableTiming));
    }
    out.permutation = at::empty({k}, options.dtype(at::kInt));
    verdict = at::empty({1}, options.dtype(at::kInt));
    check_status(abi.invert_permutation(order.data_ptr(), out.permutation.data_ptr(), verdict.data_ptr(), static_cast<int>(k), stream));
    C10_CUDA_CHECK(cudaMemcpyAsync(answer.verdict, verdict.data_ptr(), sizeof(int), cudaMemcpyDeviceToHost, stream));
    C10_CUDA_CHECK(cudaEventRecord(answer.event, stream));
  }
  if (sage) {
    const int64_t tiles = (n + 15) / 16;
    out.codes = at::empty({tiles, groups, 16, 8}, options.dtype(at::kInt));
    out.high = at::empty({tiles, groups, 16}, options.dtype(at::kInt));
    out.grid = at::empty({tiles, groups, 16, 2}, options.dtype(at::kHalf));
    out.book = at::empty({4, entries, 2}, options.dtype(at::kHalf));
  } else {
    out.codes = at::empty({n, k / 8}, options.dtype(at::kShort));
    out.high = at::empty({n, groups}, options.dtype(at::kInt));
    out.grid = at::empty({n, groups}, options.dtype(at::kHalf));
    out.mins = at::empty({n, groups}, options.dtype(at::kHalf));
    out.book = at::empty({entries, 8}, options.dtype(at::kHalf));
  }
  check_status(abi.codebook_logits(angle_logits.data_ptr(), out.book.data_ptr(), static_cast<int>(entries),
                                   static_cast<float>(scale), static_cast<float>(offset), sage, stream));
  check_status(abi.pack_logits(signs.data_ptr(), indices.data_ptr(), static_cast<int>(indices.element_size()),
                               radius_logits.data_ptr(), out.codes.data_ptr(), out.high.data_ptr(), out.grid.data_ptr(),
                               out.mins.defined() ? out.mins.data_ptr() : nullptr, static_cast<int>(n),
                               static_cast<int>(k), static_cast<int>(entries), sage, stream));
  if (order.defined()) {
    C10_CUDA_CHECK(cudaEventSynchronize(answer.event));
    TORCH_CHECK_VALUE((*answer.verdict & 2) == 0, "channel_unpermutation is not a permutation of the input channels");
    if (*answer.verdict == 0) out.permutation = Tensor();
  }
  return out;
}

// ---- module forwards: x in any floating type to FP16, the operator, back, plus the bias

Tensor to_half(const Tensor &x) {
  Tensor half = x.scalar_type() == at::kHalf ? x : x.to(at::kHalf);
  return half.is_contiguous() ? half : half.contiguous();
}
Tensor finish(Tensor y, at::ScalarType type, const Tensor &bias) {
  if (y.scalar_type() != type) y = y.to(type);
  return bias.defined() ? y + bias : y;
}

// x FP16 or BF16 with an optional bias of the same type: one GEMM launch does it all where the shape takes it,
// otherwise the conversions and the bias are operations around the FP16 call.
Tensor linear_run(const Tensor &x, const Tensor &codes, const Tensor &radii, const Tensor &grid, const Tensor &book,
                  const Tensor &perm, int64_t n, const Tensor &bias) {
  check_bound();
  const auto type = x.scalar_type();
  const int64_t k = x.dim() ? x.size(-1) : 0;
  const int64_t rows = k ? x.numel() / k : 0;
  if (rows > 0 && rows <= 65535 && (type == at::kHalf || type == at::kBFloat16) && x.is_contiguous() &&
      (!bias.defined() || (bias.scalar_type() == type && bias.dim() == 1 && bias.numel() == n && bias.is_contiguous() &&
                           bias.device() == x.device())) &&
      abi.linear_takes_type(static_cast<int>(rows), static_cast<int>(n), static_cast<int>(k))) {
    check_sage(x, codes, radii, grid, book, perm, n, type);
    const c10::cuda::CUDAGuard guard(x.device());
    Tensor y = empty_output(x, n);
    const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(x.get_device()).stream();
    const Scratch workspace = scratch_for(
        x, static_cast<int64_t>(abi.workspace_bytes(static_cast<int>(rows), static_cast<int>(n), static_cast<int>(k))), stream);
    check_status(abi.linear_typed(x.data_ptr(), type == at::kBFloat16, codes.data_ptr(), radii.data_ptr(), grid.data_ptr(),
                                  book.data_ptr(), perm.numel() ? perm.data_ptr<int32_t>() : nullptr,
                                  bias.defined() ? bias.data_ptr() : nullptr, y.data_ptr(),
                                  workspace.data(), workspace.bytes(), static_cast<int>(rows), static_cast<int>(n),
                                  static_cast<int>(k), static_cast<int>(book.size(1)), stream));
    return y;
  }
  return finish(sage_run(to_half(x), codes, radii, grid, book, perm, n, nullptr), type, bias);
}

// ---- dispatcher kernels

using SageSignature = Tensor(const Tensor &, const Tensor &, const Tensor &, const Tensor &, const Tensor &,
                             const Tensor &, c10::SymInt);
using SphSignature = Tensor(const Tensor &, const Tensor &, const Tensor &, const Tensor &, const Tensor &,
                            const Tensor &);

const c10::TypedOperatorHandle<SageSignature> &sage_op() {
  static const auto op =
      c10::Dispatcher::singleton().findSchemaOrThrow((op_namespace[0] + "::sage").c_str(), "").typed<SageSignature>();
  return op;
}
using LinearSignature = Tensor(const Tensor &, const Tensor &, const Tensor &, const Tensor &, const Tensor &,
                               const Tensor &, c10::SymInt, const std::optional<Tensor> &);
const c10::TypedOperatorHandle<LinearSignature> &linear_op() {
  static const auto op =
      c10::Dispatcher::singleton().findSchemaOrThrow("sage_b200::linear", "").typed<LinearSignature>();
  return op;
}
Tensor linear_cuda(const Tensor &x, const Tensor &codes, const Tensor &radii, const Tensor &grid, const Tensor &book,
                   const Tensor &perm, c10::SymInt n, const std::optional<Tensor> &bias) {
  return linear_run(x, codes, radii, grid, book, perm, n.guard_int(__FILE__, __LINE__), bias.has_value() ? *bias : Tensor());
}
const c10::TypedOperatorHandle<SphSignature> &sph_op() {
  static const auto op =
      c10::Dispatcher::singleton().findSchemaOrThrow((op_namespace[1] + "::sphquant").c_str(), "").typed<SphSignature>();
  return op;
}

Tensor sage_cuda(const Tensor &x, const Tensor &codes, const Tensor &radii, const Tensor &grid, const Tensor &book,
                 const Tensor &perm, c10::SymInt n) {
  return sage_run(x, codes, radii, grid, book, perm, n.guard_int(__FILE__, __LINE__), nullptr);
}

// Neither operator has a derivative: a result computed from an input that requires one carries a
// node that raises when it is differentiated, and every other call goes straight on.
struct NoDerivative : torch::autograd::Function<NoDerivative> {
  static Tensor forward(torch::autograd::AutogradContext *, const Tensor &anchor, const std::function<Tensor()> &call) {
    at::AutoDispatchBelowADInplaceOrView below;
    return call();
  }
  static torch::autograd::variable_list backward(torch::autograd::AutogradContext *, torch::autograd::variable_list) {
    TORCH_CHECK(false, "Trying to backward through a packed linear, which has no autograd formula");
  }
};

template <typename Call>
Tensor without_derivative(std::initializer_list<const Tensor *> inputs, const Call &call) {
  if (at::GradMode::is_enabled())
    for (const Tensor *t : inputs)
      if (t->requires_grad()) return NoDerivative::apply(*t, std::function<Tensor()>(call));
  at::AutoDispatchBelowADInplaceOrView below;
  return call();
}

Tensor sage_autograd(const Tensor &x, const Tensor &codes, const Tensor &radii, const Tensor &grid, const Tensor &book,
                     const Tensor &perm, c10::SymInt n) {
  return without_derivative({&x, &grid, &book}, [&] { return sage_op().call(x, codes, radii, grid, book, perm, n); });
}
Tensor sph_autograd(const Tensor &x, const Tensor &codes, const Tensor &extra, const Tensor &scales,
                    const Tensor &mins, const Tensor &book) {
  return without_derivative({&x, &scales, &mins, &book},
                            [&] { return sph_op().call(x, codes, extra, scales, mins, book); });
}

// ---- Python

struct WithoutGil {
  PyThreadState *state = PyEval_SaveThread();
  ~WithoutGil() { PyEval_RestoreThread(state); }
};

const Tensor &tensor_of(PyObject *object) {
  static const Tensor none;
  if (object == Py_None) return none;
  if (!THPVariable_Check(object)) throw torch::TypeError(std::string("a tensor is wanted, got ") + Py_TYPE(object)->tp_name);
  return THPVariable_Unpack(object);
}

bool argument_count(Py_ssize_t got, Py_ssize_t want) {
  if (got == want) return true;
  PyErr_Format(PyExc_TypeError, "%zd arguments are wanted, got %zd", want, got);
  return false;
}

long long integer_of(PyObject *object) {
  const long long value = PyLong_AsLongLong(object);
  if (value == -1 && PyErr_Occurred()) throw python_error();
  return value;
}

// sage_module(x, codes, radii, grid, book, perm, out_features, bias)
PyObject *py_sage_module(PyObject *, PyObject *const *a, Py_ssize_t count) {
  HANDLE_TH_ERRORS
  if (!argument_count(count, 8)) return nullptr;
  const long long n = integer_of(a[6]);
  const Tensor &x = tensor_of(a[0]), &codes = tensor_of(a[1]), &radii = tensor_of(a[2]), &grid = tensor_of(a[3]),
               &book = tensor_of(a[4]), &perm = tensor_of(a[5]), &bias = tensor_of(a[7]);
  Tensor y;
  {
    WithoutGil unlocked;
    // (the plain operator for FP16 without a bias, and wherever a gradient may flow through the bias or casts)
    const auto type = x.scalar_type();
    const bool gradient = at::GradMode::is_enabled() && (x.requires_grad() || (bias.defined() && bias.requires_grad()));
    if (!gradient && (type == at::kBFloat16 || (type == at::kHalf && bias.defined())) &&
        (!bias.defined() || bias.scalar_type() == type))
      y = linear_op().call(x.is_contiguous() ? x : x.contiguous(), codes, radii, grid, book, perm, n,
                           bias.defined() ? std::optional<Tensor>(bias) : std::nullopt);
    else
      y = finish(sage_op().call(to_half(x), codes, radii, grid, book, perm, n), type, bias);
  }
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

// sage_forward(x, codes, radii, grid, book, perm, out_features, scratch or None): no dispatcher
PyObject *py_sage_forward(PyObject *, PyObject *const *a, Py_ssize_t count) {
  HANDLE_TH_ERRORS
  if (!argument_count(count, 8)) return nullptr;
  const long long n = integer_of(a[6]);
  const Tensor &x = tensor_of(a[0]), &codes = tensor_of(a[1]), &radii = tensor_of(a[2]), &grid = tensor_of(a[3]),
               &book = tensor_of(a[4]), &perm = tensor_of(a[5]), &scratch = tensor_of(a[7]);
  Tensor y;
  {
    WithoutGil unlocked;
    y = sage_run(x, codes, radii, grid, book, perm, n, scratch.defined() ? &scratch : nullptr);
  }
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

// sph_module(x, codes, extra, scales, mins, book, bias)
PyObject *py_sph_module(PyObject *, PyObject *const *a, Py_ssize_t count) {
  HANDLE_TH_ERRORS
  if (!argument_count(count, 7)) return nullptr;
  const Tensor &x = tensor_of(a[0]), &codes = tensor_of(a[1]), &extra = tensor_of(a[2]), &scales = tensor_of(a[3]),
               &mins = tensor_of(a[4]), &book = tensor_of(a[5]), &bias = tensor_of(a[6]);
  Tensor y;
  {
    WithoutGil unlocked;
    y = finish(sph_op().call(to_half(x), codes, extra, scales, mins, book), x.scalar_type(), bias);
  }
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

// sph_forward(x, codes, extra, scales, mins, book): no dispatcher
PyObject *py_sph_forward(PyObject *, PyObject *const *a, Py_ssize_t count) {
  HANDLE_TH_ERRORS
  if (!argument_count(count, 6)) return nullptr;
  const Tensor &x = tensor_of(a[0]), &codes = tensor_of(a[1]), &extra = tensor_of(a[2]), &scales = tensor_of(a[3]),
               &mins = tensor_of(a[4]), &book = tensor_of(a[5]);
  Tensor y;
  {
    WithoutGil unlocked;
    y = sph_run(x, codes, extra, scales, mins, book);
  }
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

// dequantize(codes, radii, grid, book, perm, out_features, original_order)
PyObject *py_dequantize(PyObject *, PyObject *const *a, Py_ssize_t count) {
  HANDLE_TH_ERRORS
  if (!argument_count(count, 7)) return nullptr;
  const long long n = integer_of(a[5]);
  const bool original_order = PyObject_IsTrue(a[6]) == 1;
  const Tensor &codes = tensor_of(a[0]), &radii = tensor_of(a[1]), &grid = tensor_of(a[2]), &book = tensor_of(a[3]),
               &perm = tensor_of(a[4]);
  Tensor w;
  {
    WithoutGil unlocked;
    w = dequantize(codes, radii, grid, book, perm, n, original_order);
  }
  return THPVariable_Wrap(std::move(w));
  END_HANDLE_TH_ERRORS
}

// pack_state(signs, indices, radius_logits, angle_logits, order or None, sage, scale, offset)
//   -> (codes, high, grid or scales, mins or None, codebook, permutation or None)
PyObject *py_pack_state(PyObject *, PyObject *const *a, Py_ssize_t count) {
  HANDLE_TH_ERRORS
  if (!argument_count(count, 8)) return nullptr;
  const bool sage = PyObject_IsTrue(a[5]) == 1;
  const double scale = PyFloat_AsDouble(a[6]), offset = PyFloat_AsDouble(a[7]);
  if (PyErr_Occurred()) throw python_error();
  const Tensor &signs = tensor_of(a[0]), &indices = tensor_of(a[1]), &radius = tensor_of(a[2]), &angle = tensor_of(a[3]),
               &order = tensor_of(a[4]);
  Packed out;
  {
    WithoutGil unlocked;
    out = pack_state(signs, indices, radius, angle, order, sage, scale, offset);
  }
  PyObject *tuple = PyTuple_New(6);
  if (!tuple) throw python_error();
  Tensor *const parts[] = {&out.codes, &out.high, &out.grid, &out.mins, &out.book, &out.permutation};
  for (int i = 0; i < 6; ++i) PyTuple_SET_ITEM(tuple, i, parts[i]->defined() ? THPVariable_Wrap(*parts[i]) : Py_NewRef(Py_None));
  return tuple;
  END_HANDLE_TH_ERRORS
}

// bind({"sageb200_linear": address, ...})
PyObject *py_bind(PyObject *, PyObject *table) {
  HANDLE_TH_ERRORS
  auto address = [&](const char *name) {
    PyObject *value = PyDict_GetItemString(table, name);
    TORCH_CHECK(value, "no address for ", name);
    return static_cast<uintptr_t>(integer_of(value));
  };
#define SAGE_BIND(name) abi.name = reinterpret_cast<decltype(abi.name)>(address("sageb200_" #name))
  SAGE_BIND(status_string);
  SAGE_BIND(workspace_bytes);
  SAGE_BIND(linear_takes_type);
  SAGE_BIND(linear_typed);
  SAGE_BIND(sph_workspace_bytes);
  SAGE_BIND(sph_linear_scratch);
  SAGE_BIND(dequant);
  SAGE_BIND(pack_logits);
  SAGE_BIND(codebook_logits);
  SAGE_BIND(invert_permutation);
  SAGE_BIND(linear);
#undef SAGE_BIND
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

// register_kernels("sage", "wvq"): the CUDA and autograd kernels of an operator whose schema Python defined
PyObject *py_register_kernels(PyObject *, PyObject *const *a, Py_ssize_t count) {
  HANDLE_TH_ERRORS
  if (!argument_count(count, 2)) return nullptr;
  const std::string op = PyUnicode_AsUTF8(a[0]), space = PyUnicode_AsUTF8(a[1]);
  static auto *libraries = new std::vector<std::unique_ptr<torch::Library>>;
  auto library = [&](c10::DispatchKey key) -> torch::Library & {
    libraries->push_back(std::make_unique<torch::Library>(torch::Library::IMPL, space, key, __FILE__, __LINE__));
    return *libraries->back();
  };
  if (op == "linear") {
    library(c10::DispatchKey::CUDA).impl("linear", &linear_cuda);
    Py_RETURN_NONE;
  }
  const bool sage = op == "sage";
  op_namespace[sage ? 0 : 1] = space;
  if (sage) {
    library(c10::DispatchKey::CUDA).impl("sage", &sage_cuda);
    library(c10::DispatchKey::AutogradCUDA).impl("sage", &sage_autograd);
  } else {
    library(c10::DispatchKey::CUDA).impl("sphquant", &sph_run);
    library(c10::DispatchKey::AutogradCUDA).impl("sphquant", &sph_autograd);
  }
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

template <typename Function>
PyCFunction as_method(Function function) {
  return reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(function));
}

PyMethodDef methods[] = {
    {"bind", py_bind, METH_O, nullptr},
    {"register_kernels", as_method(py_register_kernels), METH_FASTCALL, nullptr},
    {"sage_module", as_method(py_sage_module), METH_FASTCALL, nullptr},
    {"sage_forward", as_method(py_sage_forward), METH_FASTCALL, nullptr},
    {"sph_module", as_method(py_sph_module), METH_FASTCALL, nullptr},
    {"dequantize", as_method(py_dequantize), METH_FASTCALL, nullptr},
    {"pack_state", as_method(py_pack_state), METH_FASTCALL, nullptr},
    {"sph_forward", as_method(py_sph_forward), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native() {
  PyObject *module = PyModule_Create(&module_def);
  // (torch's C++ interface has no stable ABI: the loader compares this with the torch it runs under)
  if (module && PyModule_AddStringConstant(module, "torch_version", SAGEB200_TORCH_VERSION) < 0) Py_CLEAR(module);
  return module;
}
