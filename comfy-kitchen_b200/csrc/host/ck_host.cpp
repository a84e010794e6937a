// The wrappers of backends/cuda in native code, for the calls that need nothing special.
//
// A call of the C-ABI library from Python (argument checks, two to four torch.empty, a ctypes call of some 16 arguments) took
// 8 to 13 us of host time, as long as the kernels of a few hundred rows.  Each function here makes the same checks
// on the C++ tensors, allocates the results, calls the library and returns them; it returns None for anything
// else (other types, devices or layouts, somebody who watches operator calls, CK_STRICT=1, an error of the library),
// and the Python wrapper then does the call, or raises what it always raised.  Nothing is kept between calls.
#include <Python.h>

#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/core/DimVector.h>
#include <ATen/core/Tensor.h>
#include <ATen/ops/empty.h>
#include <ATen/record_function.h>
#include <c10/core/GradMode.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdint>
#include <cstdlib>

namespace {

using at::ScalarType;
using at::Tensor;

// ---- the library's entry points (include/ck_b200.h), as backends/cuda loaded them
struct Library {
  int (*quantize_nvfp4)(const void*, int, const float*, void*, void*, int64_t, int64_t, int64_t, int64_t, int, void*);
  int64_t (*quantize_nvfp4_dynamic_scratch_bytes)(int64_t);
  int64_t (*quantize_nvfp4_dynamic_whole_input_bytes)(int64_t);
  int (*quantize_nvfp4_dynamic)(const void*, int, float*, void*, void*, int64_t, int64_t, int64_t, int64_t, int, void*, int64_t, void*);
  int (*quantize_mxfp8)(const void*, int, void*, void*, int64_t, int64_t, int64_t, int64_t, void*);
  int (*dequantize_nvfp4)(const void*, const float*, const void*, void*, int, int64_t, int64_t, int, void*);
  int (*dequantize_mxfp8)(const void*, const void*, void*, int, int64_t, int64_t, void*);
  int64_t (*scaled_mm_workspace_bytes)(int, int64_t, int64_t, int64_t);
  int (*scaled_mm_nvfp4_ws)(const void*, const void*, const void*, const void*, const float*, const float*, const float*, const void*, int, void*,
                            int, int64_t, int64_t, int64_t, void*, int64_t, void*);
  int (*scaled_mm_mxfp8_ws)(const void*, const void*, const void*, const void*, const void*, int, void*, int, int64_t, int64_t, int64_t, void*,
                            int64_t, void*);
  int64_t (*linear_nvfp4_from_float_workspace_bytes)(int64_t, int64_t, int);
  int (*linear_nvfp4_from_float)(const void*, int, const float*, const void*, const void*, const float*, const void*, int, void*, int, int64_t,
                                 int64_t, int64_t, void*, int64_t, void*);
  int64_t (*linear_mxfp8_from_float_workspace_bytes)(int64_t, int64_t);
  int (*linear_mxfp8_from_float)(const void*, int, const void*, const void*, const void*, int, void*, int, int64_t, int64_t, int64_t, void*,
                                 int64_t, void*);
};
Library lib = {};
PyTypeObject* parameter_type = nullptr;

constexpr int64_t kOnChip = 256;  // the workspace size of a GEMM that does not use one

int64_t round_up(int64_t x, int64_t m) { return (x + m - 1) / m * m; }

// dtype codes of the C ABI, -1 for types that no kernel takes as a dense operand
int code_of(ScalarType t) {
  switch (t) {
    case ScalarType::Float: return 0;
    case ScalarType::Half: return 1;
    case ScalarType::BFloat16: return 2;
    default: return -1;
  }
}

// Nobody watches or rewrites operator calls on this thread (profilers and other observers, torch function and dispatch
// modes, functorch, tracing, functionalization), and no check of the device's status word is asked for behind each call.
bool quiet() {
  static const c10::DispatchKeySet usual = c10::DispatchKeySet({c10::DispatchKey::BackendSelect, c10::DispatchKey::ADInplaceOrView}) |
                                           c10::autocast_dispatch_keyset;
  if (!usual.has_all(c10::impl::tls_local_dispatch_key_set().included_)) return false;
  if (c10::impl::TorchDispatchModeTLS::any_modes_set() || at::impl::PythonTorchFunctionTLS::stack_len() != 0 || at::hasCallbacks()) return false;
  const char* strict = std::getenv("CK_STRICT");
  return strict == nullptr || strict[0] != '1' || strict[1] != 0;
}

// What follows refuses a call by a null pointer or false, never by an exception: the Python wrapper, whose call it then is, should not
// pay for having asked (0.2 us; 1.3 to 1.7 with a C++ exception).

// A plain dense CUDA tensor on the current device, of no autograd graph; null for anything else.
const Tensor* plain(PyObject* o, int device) {
  if (Py_TYPE(o) != reinterpret_cast<PyTypeObject*>(THPVariableClass) && Py_TYPE(o) != parameter_type) return nullptr;
  const Tensor& t = THPVariable_Unpack(o);
  static const c10::DispatchKeySet usual = c10::DispatchKeySet(c10::DispatchKey::CUDA) | c10::DispatchKeySet(c10::DispatchKey::AutogradCUDA) |
                                           c10::DispatchKeySet(c10::DispatchKey::ADInplaceOrView) |
                                           c10::DispatchKeySet(c10::DispatchKey::AutocastCUDA);
  const bool ok = usual.has_all(t.key_set()) && t.is_cuda() && t.get_device() == device && t.is_contiguous() &&
                  !(t.requires_grad() && c10::GradMode::is_enabled());
  return ok ? &t : nullptr;
}

const Tensor* matrix(PyObject* o, int device) {
  const Tensor* t = plain(o, device);
  return t != nullptr && t->dim() == 2 && t->size(0) > 0 && t->size(1) > 0 ? t : nullptr;
}

// Rows of any rank from two on.
const Tensor* rows_of(PyObject* o, int device) {
  const Tensor* t = plain(o, device);
  return t != nullptr && t->dim() >= 2 && t->numel() > 0 ? t : nullptr;
}

const Tensor* matrix(PyObject* o, int device, ScalarType type) {
  const Tensor* t = matrix(o, device);
  return t != nullptr && t->scalar_type() == type ? t : nullptr;
}

const float* scalar(PyObject* o, int device) {
  const Tensor* t = plain(o, device);
  return t != nullptr && t->scalar_type() == ScalarType::Float && t->numel() == 1 ? static_cast<const float*>(t->const_data_ptr()) : nullptr;
}

struct Bias {
  const void* ptr = nullptr;
  int code = 0;
};
bool bias_of(PyObject* o, int device, int64_t n, Bias* b) {
  if (o == Py_None) return true;
  const Tensor* t = plain(o, device);
  if (t == nullptr || code_of(t->scalar_type()) < 0 || t->numel() != n) return false;
  b->code = code_of(t->scalar_type());
  b->ptr = t->const_data_ptr();
  return true;
}

bool scales_fit(const Tensor& s, int64_t rows, int64_t columns) { return s.size(0) == round_up(rows, 128) && s.size(1) == round_up(columns, 4); }

// A dense type that the caller names; `*type` stays what it is for None.
bool dtype_of(PyObject* o, ScalarType* type) {
  if (o == Py_None) return true;
  if (!THPDtype_Check(o)) return false;
  *type = reinterpret_cast<THPDtype*>(o)->scalar_type;
  return code_of(*type) >= 0;
}

Tensor result(at::IntArrayRef sizes, ScalarType type, int device) {
  return at::empty(sizes, at::TensorOptions().dtype(type).device(at::Device(at::kCUDA, static_cast<c10::DeviceIndex>(device))));
}

// What passes from one launch of a call to the next: the caching allocator's block of the current stream, which goes back behind
// the kernels that use it (and belongs to the graph in a captured call).
struct Workspace {
  c10::DataPtr block;
  int64_t bytes;
  explicit Workspace(int64_t n) : bytes(n) {
    if (n > 0) block = c10::cuda::CUDACachingAllocator::get()->allocate(static_cast<size_t>(n));
  }
  void* ptr() { return block.get(); }
};

// Rows of `columns` values in the shape of x.
Tensor rows_like(const Tensor& x, int64_t columns, ScalarType type, int device) {
  if (x.dim() == 2) return result({x.size(0), columns}, type, device);
  at::DimVector sizes(x.sizes());
  sizes.back() = columns;
  return result(sizes, type, device);
}

struct Call {
  int device;
  void* stream;
  Call() : device(c10::cuda::current_device()), stream(c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(device)).stream()) {}
};

struct WithoutGil {
  PyThreadState* state = PyEval_SaveThread();
  ~WithoutGil() { PyEval_RestoreThread(state); }
};

// A call of the library without the GIL (its arguments were evaluated with it); false: refused.
template <typename... P, typename... A>
bool launched(int (*fn)(P...), A... args) {
  const WithoutGil released;
  return fn(args...) == 0;
}

PyObject* pair(Tensor a, Tensor b) {
  PyObject* t = PyTuple_New(2);
  if (t == nullptr) return nullptr;
  PyTuple_SET_ITEM(t, 0, THPVariable_Wrap(std::move(a)));
  PyTuple_SET_ITEM(t, 1, THPVariable_Wrap(std::move(b)));
  return t;
}

// What `body` returns; None when that is null (refused) or something goes wrong in it: the call is the Python wrapper's then.
template <typename Body>
PyObject* or_none(PyObject* const* args, Py_ssize_t got, Py_ssize_t wanted, Body&& body) {
  try {
    if (got == wanted && THPVariable_Check(args[0]) && THPVariable_Unpack(args[0]).is_cuda() && quiet()) {
      PyObject* r = body();
      if (r != nullptr || PyErr_Occurred() != nullptr) return r;
    }
  } catch (const std::exception&) {
  }
  Py_RETURN_NONE;
}

using Args = PyObject* const*;

// ---- quantizers -------------------------------------------------------------------------------
PyObject* quantize_nvfp4(PyObject*, Args a, Py_ssize_t n_args) {  // x, per_tensor_scale, pad_16x, hi_first
  return or_none(a, n_args, 4, [&]() -> PyObject* {
    const Call c;
    const Tensor* x = matrix(a[0], c.device);
    const float* scale = scalar(a[1], c.device);
    if (x == nullptr || scale == nullptr || !PyBool_Check(a[2]) || !PyBool_Check(a[3])) return nullptr;
    const int code = code_of(x->scalar_type());
    const bool pad = a[2] == Py_True, hi_first = a[3] == Py_True;
    const int64_t rows = x->size(0), cols = x->size(1), out_rows = pad ? round_up(rows, 16) : rows, out_cols = pad ? round_up(cols, 16) : cols;
    if (code < 0 || out_cols % 16 != 0) return nullptr;
    Tensor q = result({out_rows, out_cols / 2}, ScalarType::Byte, c.device);
    Tensor s = result({round_up(out_rows, 128), round_up(out_cols / 16, 4)}, ScalarType::Float8_e4m3fn, c.device);
    if (!launched(lib.quantize_nvfp4, x->const_data_ptr(), code, scale, q.mutable_data_ptr(), s.mutable_data_ptr(), rows, cols, out_rows, out_cols,
                  hi_first, c.stream)) {
      return nullptr;
    }
    return pair(std::move(q), std::move(s));
  });
}

// `kept_scratch(x)`: a buffer that is kept for the calls that write nothing to it.  Which they are is the library's to say: it is asked for up to
// the size at which not even one row, whose line is the lowest, takes a reduction kernel.
PyObject* quantize_nvfp4_dynamic(PyObject*, Args a, Py_ssize_t n_args) {  // x, pad_16x, hi_first, kept_scratch
  return or_none(a, n_args, 4, [&]() -> PyObject* {
    const Call c;
    const Tensor* x = matrix(a[0], c.device);
    if (x == nullptr || !PyBool_Check(a[1]) || !PyBool_Check(a[2])) return nullptr;
    const int code = code_of(x->scalar_type());
    const bool pad = a[1] == Py_True, hi_first = a[2] == Py_True;
    const int64_t rows = x->size(0), cols = x->size(1), out_rows = pad ? round_up(rows, 16) : rows, out_cols = pad ? round_up(cols, 16) : cols;
    // the streaming quantizer's form; the one-kernel scale's scratch is the Python wrapper's
    if (code < 0 || out_cols != cols || cols % (64 / x->element_size()) != 0 || reinterpret_cast<uintptr_t>(x->const_data_ptr()) % 32 != 0) return nullptr;
    const int64_t need = lib.quantize_nvfp4_dynamic_scratch_bytes(rows * cols);
    void* scratch = nullptr;
    Tensor kept;
    if (x->nbytes() <= static_cast<size_t>(lib.quantize_nvfp4_dynamic_whole_input_bytes(1))) {
      PyObject* of_x = PyObject_CallOneArg(a[3], a[0]);
      if (of_x == nullptr) return nullptr;  // an error, raised
      const Tensor* t = plain(of_x, c.device);
      if (t != nullptr) kept = *t;
      Py_DECREF(of_x);
      if (t == nullptr || kept.scalar_type() != ScalarType::Byte || kept.numel() < need) return nullptr;
      scratch = kept.mutable_data_ptr();
    }
    Workspace ws(scratch == nullptr ? need : 0);
    if (scratch == nullptr) scratch = ws.ptr();
    Tensor q = result({out_rows, out_cols / 2}, ScalarType::Byte, c.device);
    Tensor s = result({round_up(out_rows, 128), round_up(out_cols / 16, 4)}, ScalarType::Float8_e4m3fn, c.device);
    Tensor scale = result({}, ScalarType::Float, c.device);
    if (!launched(lib.quantize_nvfp4_dynamic, x->const_data_ptr(), code, static_cast<float*>(scale.mutable_data_ptr()), q.mutable_data_ptr(),
                  s.mutable_data_ptr(), rows, cols, out_rows, out_cols, hi_first, scratch, need, c.stream)) {
      return nullptr;
    }
    PyObject* t = PyTuple_New(3);
    if (t == nullptr) return nullptr;
    PyTuple_SET_ITEM(t, 0, THPVariable_Wrap(std::move(q)));
    PyTuple_SET_ITEM(t, 1, THPVariable_Wrap(std::move(s)));
    PyTuple_SET_ITEM(t, 2, THPVariable_Wrap(std::move(scale)));
    return t;
  });
}

PyObject* quantize_mxfp8(PyObject*, Args a, Py_ssize_t n_args) {  // x, pad_32x
  return or_none(a, n_args, 2, [&]() -> PyObject* {
    const Call c;
    const Tensor* x = matrix(a[0], c.device);
    if (x == nullptr || !PyBool_Check(a[1])) return nullptr;
    const int code = code_of(x->scalar_type());
    const bool pad = a[1] == Py_True;
    const int64_t rows = x->size(0), cols = x->size(1), out_rows = pad ? round_up(rows, 32) : rows, out_cols = pad ? round_up(cols, 32) : cols;
    if (code < 0 || out_cols % 32 != 0) return nullptr;
    Tensor q = result({out_rows, out_cols}, ScalarType::Float8_e4m3fn, c.device);
    Tensor s = result({round_up(out_rows, 128), round_up(out_cols / 32, 4)}, ScalarType::Float8_e8m0fnu, c.device);
    if (!launched(lib.quantize_mxfp8, x->const_data_ptr(), code, q.mutable_data_ptr(), s.mutable_data_ptr(), rows, cols, out_rows, out_cols, c.stream)) {
      return nullptr;
    }
    return pair(std::move(q), std::move(s));
  });
}

PyObject* dequantize_nvfp4(PyObject*, Args a, Py_ssize_t n_args) {  // qx, per_tensor_scale, block_scales, output_type, hi_first
  return or_none(a, n_args, 5, [&]() -> PyObject* {
    const Call c;
    const Tensor* q = matrix(a[0], c.device, ScalarType::Byte);
    const float* scale = scalar(a[1], c.device);
    const Tensor* s = matrix(a[2], c.device, ScalarType::Float8_e4m3fn);
    ScalarType type = ScalarType::BFloat16;
    if (q == nullptr || scale == nullptr || s == nullptr || a[3] == Py_None || !dtype_of(a[3], &type) || !PyBool_Check(a[4])) return nullptr;
    const bool hi_first = a[4] == Py_True;
    const int64_t rows = q->size(0), cols = 2 * q->size(1);
    if (cols % 16 != 0 || !scales_fit(*s, rows, cols / 16)) return nullptr;
    Tensor out = result({rows, cols}, type, c.device);
    if (!launched(lib.dequantize_nvfp4, q->const_data_ptr(), scale, s->const_data_ptr(), out.mutable_data_ptr(), code_of(type), rows, cols, hi_first,
                  c.stream)) {
      return nullptr;
    }
    return THPVariable_Wrap(std::move(out));
  });
}

PyObject* dequantize_mxfp8(PyObject*, Args a, Py_ssize_t n_args) {  // qx, block_scales, output_type
  return or_none(a, n_args, 3, [&]() -> PyObject* {
    const Call c;
    const Tensor* q = matrix(a[0], c.device, ScalarType::Float8_e4m3fn);
    const Tensor* s = matrix(a[1], c.device, ScalarType::Float8_e8m0fnu);
    ScalarType type = ScalarType::BFloat16;
    if (q == nullptr || s == nullptr || a[2] == Py_None || !dtype_of(a[2], &type)) return nullptr;
    const int64_t rows = q->size(0), cols = q->size(1);
    if (cols % 32 != 0 || !scales_fit(*s, rows, cols / 32)) return nullptr;
    Tensor out = result({rows, cols}, type, c.device);
    if (!launched(lib.dequantize_mxfp8, q->const_data_ptr(), s->const_data_ptr(), out.mutable_data_ptr(), code_of(type), rows, cols, c.stream)) return nullptr;
    return THPVariable_Wrap(std::move(out));
  });
}

// ---- GEMMs ------------------------------------------------------------------------------------
PyObject* scaled_mm_nvfp4(PyObject*, Args a, Py_ssize_t n_args) {  // a, b, scales of tensors and blocks (a, b each), bias, out_dtype, alpha
  return or_none(a, n_args, 9, [&]() -> PyObject* {
    const Call c;
    const Tensor* x = matrix(a[0], c.device, ScalarType::Byte);
    const Tensor* w = matrix(a[1], c.device, ScalarType::Byte);
    const float* tsa = scalar(a[2], c.device);
    const float* tsb = scalar(a[3], c.device);
    const Tensor* sa = matrix(a[4], c.device, ScalarType::Float8_e4m3fn);
    const Tensor* sb = matrix(a[5], c.device, ScalarType::Float8_e4m3fn);
    const float* alpha = a[8] == Py_None ? nullptr : scalar(a[8], c.device);
    if (x == nullptr || w == nullptr || tsa == nullptr || tsb == nullptr || sa == nullptr || sb == nullptr || (alpha == nullptr && a[8] != Py_None)) {
      return nullptr;
    }
    const int64_t m = x->size(0), n = w->size(0), k = 2 * x->size(1);
    Bias bias;
    ScalarType type = ScalarType::BFloat16;
    if (w->size(1) != x->size(1) || k % 32 != 0 || n % 8 != 0 || !scales_fit(*sa, m, k / 16) || !scales_fit(*sb, n, k / 16) ||
        !bias_of(a[6], c.device, n, &bias) || !dtype_of(a[7], &type)) {
      return nullptr;
    }
    Tensor out = result({m, n}, type, c.device);
    const int64_t need = lib.scaled_mm_workspace_bytes(0, m, n, k);
    Workspace ws(need > kOnChip ? need : 0);
    if (!launched(lib.scaled_mm_nvfp4_ws, x->const_data_ptr(), w->const_data_ptr(), sa->const_data_ptr(), sb->const_data_ptr(), tsa, tsb, alpha, bias.ptr,
                  bias.code, out.mutable_data_ptr(), code_of(type), m, n, k, ws.ptr(), ws.bytes, c.stream)) {
      return nullptr;
    }
    return THPVariable_Wrap(std::move(out));
  });
}

PyObject* scaled_mm_mxfp8(PyObject*, Args a, Py_ssize_t n_args) {  // a, b, block scales of a, of b, bias, out_dtype
  return or_none(a, n_args, 6, [&]() -> PyObject* {
    const Call c;
    const Tensor* x = matrix(a[0], c.device, ScalarType::Float8_e4m3fn);
    const Tensor* w = matrix(a[1], c.device, ScalarType::Float8_e4m3fn);
    const Tensor* sa = matrix(a[2], c.device, ScalarType::Float8_e8m0fnu);
    const Tensor* sb = matrix(a[3], c.device, ScalarType::Float8_e8m0fnu);
    if (x == nullptr || w == nullptr || sa == nullptr || sb == nullptr) return nullptr;
    const int64_t m = x->size(0), n = w->size(0), k = x->size(1);
    Bias bias;
    ScalarType type = ScalarType::BFloat16;
    if (w->size(1) != k || k % 32 != 0 || n % 8 != 0 || !scales_fit(*sa, m, k / 32) || !scales_fit(*sb, n, k / 32) ||
        !bias_of(a[4], c.device, n, &bias) || !dtype_of(a[5], &type)) {
      return nullptr;
    }
    Tensor out = result({m, n}, type, c.device);
    const int64_t need = lib.scaled_mm_workspace_bytes(1, m, n, k);
    Workspace ws(need > kOnChip ? need : 0);
    if (!launched(lib.scaled_mm_mxfp8_ws, x->const_data_ptr(), w->const_data_ptr(), sa->const_data_ptr(), sb->const_data_ptr(), bias.ptr, bias.code,
                  out.mutable_data_ptr(), code_of(type), m, n, k, ws.ptr(), ws.bytes, c.stream)) {
      return nullptr;
    }
    return THPVariable_Wrap(std::move(out));
  });
}

// ---- one-call linears -------------------------------------------------------------------------
// The activation has any rank from two on, and the result its shape (the layers' callers pass [batch, tokens, features]).
ScalarType linear_type(ScalarType x) { return x == ScalarType::Half ? x : ScalarType::BFloat16; }  // of a result whose type nobody names

PyObject* linear_nvfp4_from_float(PyObject*, Args a, Py_ssize_t n_args) {  // x, w_codes, w_scale, w_block_scales, bias, x_scale, out_dtype
  return or_none(a, n_args, 7, [&]() -> PyObject* {
    const Call c;
    const Tensor* x = rows_of(a[0], c.device);
    if (x == nullptr || (a[5] == Py_None && reinterpret_cast<uintptr_t>(x->const_data_ptr()) % 32 != 0)) return nullptr;  // the one-kernel scale comes first
    const Tensor* w = matrix(a[1], c.device, ScalarType::Byte);
    const float* w_scale = scalar(a[2], c.device);
    const Tensor* sw = matrix(a[3], c.device, ScalarType::Float8_e4m3fn);
    const float* x_scale = a[5] == Py_None ? nullptr : scalar(a[5], c.device);
    if (w == nullptr || w_scale == nullptr || sw == nullptr || (x_scale == nullptr && a[5] != Py_None)) return nullptr;
    const int code = code_of(x->scalar_type());
    const int64_t k = x->size(-1), m = x->numel() / k, n = w->size(0);
    Bias bias;
    ScalarType type = linear_type(x->scalar_type());
    if (code < 0 || 2 * w->size(1) != k || k % 32 != 0 || n % 8 != 0 || !scales_fit(*sw, n, k / 16) || !bias_of(a[4], c.device, n, &bias) ||
        !dtype_of(a[6], &type)) {
      return nullptr;
    }
    const int64_t need = lib.linear_nvfp4_from_float_workspace_bytes(m, k, x_scale == nullptr);
    if (need <= 0) return nullptr;
    Workspace ws(need);
    Tensor out = rows_like(*x, n, type, c.device);
    if (!launched(lib.linear_nvfp4_from_float, x->const_data_ptr(), code, x_scale, w->const_data_ptr(), sw->const_data_ptr(), w_scale, bias.ptr, bias.code,
                  out.mutable_data_ptr(), code_of(type), m, n, k, ws.ptr(), ws.bytes, c.stream)) {
      return nullptr;
    }
    return THPVariable_Wrap(std::move(out));
  });
}

PyObject* linear_mxfp8_from_float(PyObject*, Args a, Py_ssize_t n_args) {  // x, w_data, w_block_scales, bias, out_dtype
  return or_none(a, n_args, 5, [&]() -> PyObject* {
    const Call c;
    const Tensor* x = rows_of(a[0], c.device);
    const Tensor* w = matrix(a[1], c.device, ScalarType::Float8_e4m3fn);
    const Tensor* sw = matrix(a[2], c.device, ScalarType::Float8_e8m0fnu);
    if (x == nullptr || w == nullptr || sw == nullptr) return nullptr;
    const int code = code_of(x->scalar_type());
    const int64_t k = x->size(-1), m = x->numel() / k, n = w->size(0);
    Bias bias;
    ScalarType type = linear_type(x->scalar_type());
    if (code < 0 || w->size(1) != k || k % 32 != 0 || n % 8 != 0 || !scales_fit(*sw, n, k / 32) || !bias_of(a[3], c.device, n, &bias) ||
        !dtype_of(a[4], &type)) {
      return nullptr;
    }
    const int64_t need = lib.linear_mxfp8_from_float_workspace_bytes(m, k);
    if (need <= 0) return nullptr;
    Workspace ws(need);
    Tensor out = rows_like(*x, n, type, c.device);
    if (!launched(lib.linear_mxfp8_from_float, x->const_data_ptr(), code, w->const_data_ptr(), sw->const_data_ptr(), bias.ptr, bias.code,
                  out.mutable_data_ptr(), code_of(type), m, n, k, ws.ptr(), ws.bytes, c.stream)) {
      return nullptr;
    }
    return THPVariable_Wrap(std::move(out));
  });
}

// ---- set-up -----------------------------------------------------------------------------------
// bind({name: address of ck_<name>}, torch.nn.Parameter)
PyObject* bind(PyObject*, Args a, Py_ssize_t n_args) {
  if (n_args != 2 || !PyDict_Check(a[0]) || !PyType_Check(a[1])) {
    PyErr_SetString(PyExc_TypeError, "bind: a dict of addresses and the Parameter type");
    return nullptr;
  }
  Library got = {};
  bool complete = true;
  auto take = [&](auto& fn, const char* name) {
    PyObject* v = PyDict_GetItemString(a[0], name);
    void* p = v != nullptr ? PyLong_AsVoidPtr(v) : nullptr;
    fn = reinterpret_cast<std::remove_reference_t<decltype(fn)>>(p);
    complete = complete && p != nullptr;
  };
#define CK_TAKE(name) take(got.name, "ck_" #name)
  CK_TAKE(quantize_nvfp4);
  CK_TAKE(quantize_nvfp4_dynamic_scratch_bytes);
  CK_TAKE(quantize_nvfp4_dynamic_whole_input_bytes);
  CK_TAKE(quantize_nvfp4_dynamic);
  CK_TAKE(quantize_mxfp8);
  CK_TAKE(dequantize_nvfp4);
  CK_TAKE(dequantize_mxfp8);
  CK_TAKE(scaled_mm_workspace_bytes);
  CK_TAKE(scaled_mm_nvfp4_ws);
  CK_TAKE(scaled_mm_mxfp8_ws);
  CK_TAKE(linear_nvfp4_from_float_workspace_bytes);
  CK_TAKE(linear_nvfp4_from_float);
  CK_TAKE(linear_mxfp8_from_float_workspace_bytes);
  CK_TAKE(linear_mxfp8_from_float);
#undef CK_TAKE
  if (!complete) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "bind: an entry point is missing");
    return nullptr;
  }
  lib = got;
  Py_INCREF(a[1]);
  parameter_type = reinterpret_cast<PyTypeObject*>(a[1]);
  Py_RETURN_NONE;
}

#define CK_METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {CK_METHOD(bind),
                         CK_METHOD(quantize_nvfp4),
                         CK_METHOD(quantize_nvfp4_dynamic),
                         CK_METHOD(quantize_mxfp8),
                         CK_METHOD(dequantize_nvfp4),
                         CK_METHOD(dequantize_mxfp8),
                         CK_METHOD(scaled_mm_nvfp4),
                         CK_METHOD(scaled_mm_mxfp8),
                         CK_METHOD(linear_nvfp4_from_float),
                         CK_METHOD(linear_mxfp8_from_float),
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_ck_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__ck_host() { return PyModule_Create(&module); }
