// Native host path of the ops: argument checks, output allocation and launch of every op of the registry as one C function
// per op, so that a call from Python costs one function call instead of a dispatch, a predicate and a custom-op wrapper
// written in Python. Measured per op on the host of a B200 box: 50 us through the Python path, about 5 us through this one;
// a one-image layer's kernels take 3 to 15 us, so the Python path bounded every small call.
//
// A function here serves exactly the calls whose outcome it can produce itself: plain CUDA tensors of the op's dtypes,
// layouts and shapes, outside of tracing, tensor subclasses, dispatch modes and autograd recording. For everything else -
// another dtype or layout that the Python implementation converts, a shape it declines, wrong arguments - it returns
// NotImplemented and the caller goes through the registry's general path, which is also what raises errors.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/TracerMode.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/GradMode.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <dlfcn.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <list>
#include <memory>
#include <mutex>
#include <unordered_map>
#include <utility>
#include <vector>

#include "flashim_sm100.h"

namespace {

using at::Tensor;
using c10::ScalarType;

constexpr auto kE4M3 = ScalarType::Float8_e4m3fn;
constexpr auto kE8M0 = ScalarType::Float8_e8m0fnu;
constexpr auto kBF16 = ScalarType::BFloat16;
constexpr auto kF32 = ScalarType::Float;
constexpr auto kI8 = ScalarType::Char;
constexpr auto kU8 = ScalarType::Byte;

// ---- the C ABI, resolved from the library that the Python side loaded ------------------------------------------------

#define FIM_ENTRIES(X)                                                                                                     \
  X(fim_quantize_mxfp8_static) X(fim_quantize_mxfp8_dynamic) X(fim_quantize_int8_static) X(fim_quantize_mxfp8_static_nchw)  \
  X(fim_quantize_int8_static_nchw) X(fim_maxpool2_quantize_int8) X(fim_romav2_refiner_input) X(fim_romav2_refiner_heads)    \
  X(fim_dw5x5_bf16) X(fim_dw5x5_mxfp8) X(fim_dw5x5_relu_int8) X(fim_mxfp8_conv2d) X(fim_mxfp8_conv2d_bf16) X(fim_int8_conv2d) \
  X(fim_mxfp8_gelu_mlp_residual) X(fim_int8_conv2d_maxpool) X(fim_bf16_conv2d) X(fim_gelu_quantize_mxfp8)

struct Abi {
#define FIM_MEMBER(name) decltype(&::name) name = nullptr;
  FIM_ENTRIES(FIM_MEMBER)
#undef FIM_MEMBER
} abi;

// Python objects handed over by bind(): the status word per device, the error check, the per-call check of the status word
// (None unless asked for), the weight-scale swizzle and the container classes.
PyObject *py_status_word, *py_check, *py_check_status, *py_swizzle, *py_quantized_tensor, *py_int8_tensor;
PyObject *name_values, *name_scale, *name_scale_exponent, *name_logical_shape, *empty_tuple;

constexpr int kMaxDevices = 64;
struct Device {
  int state = 0;  // 0: not looked at, 1: compute capability 10.0, -1: another one
  int* status = nullptr;
  PyObject* status_tensor = nullptr;
} devices[kMaxDevices];

struct Failed {};  // a Python error is set
[[noreturn]] void failed() { throw Failed(); }

// ---- arguments -------------------------------------------------------------------------------------------------------

struct Signature {
  int count, required;
  const char* names[20];
  PyObject* interned[20];
};

// Positional and keyword arguments into `out` (nullptr where absent); false when they do not fit the signature.
bool bind_arguments(const Signature& s, PyObject* const* args, Py_ssize_t nargs, PyObject* kwnames, PyObject** out) {
  if (nargs > s.count) return false;
  for (int i = 0; i < s.count; ++i) out[i] = i < nargs ? args[i] : nullptr;
  const Py_ssize_t nkw = kwnames == nullptr ? 0 : PyTuple_GET_SIZE(kwnames);
  for (Py_ssize_t k = 0; k < nkw; ++k) {
    PyObject* name = PyTuple_GET_ITEM(kwnames, k);
    int at = -1;
    for (int i = 0; i < s.count && at < 0; ++i) {
      if (name == s.interned[i] || PyUnicode_Compare(name, s.interned[i]) == 0) at = i;
    }
    if (at < 0 || out[at] != nullptr) return false;
    out[at] = args[nargs + k];
  }
  for (int i = 0; i < s.required; ++i) {
    if (out[i] == nullptr) return false;
  }
  return true;
}

// A plain CUDA tensor (no subclass behaviour, no functorch level, no lazy conjugation) whose use nothing records.
const Tensor* plain_tensor(PyObject* o) {
  if (o == nullptr || !THPVariable_Check(o)) return nullptr;
  static const uint64_t kAllowed =
      c10::DispatchKeySet({c10::DispatchKey::CUDA, c10::DispatchKey::AutogradCUDA, c10::DispatchKey::AutocastCUDA,
                           c10::DispatchKey::ADInplaceOrView}).raw_repr();
  const Tensor& t = THPVariable_Unpack(o);
  if (!t.defined() || !t.is_cuda() || (t.key_set().raw_repr() & ~kAllowed) != 0) return nullptr;
  if (t.requires_grad() && c10::GradMode::is_enabled()) return nullptr;
  return &t;
}

// An optional tensor argument: true with *t == nullptr for None or absent.
bool optional_tensor(PyObject* o, const Tensor** t) {
  *t = nullptr;
  if (o == nullptr || o == Py_None) return true;
  *t = plain_tensor(o);
  return *t != nullptr;
}

bool integer(PyObject* o, int* v) {
  if (o == nullptr || !PyLong_CheckExact(o)) return false;
  const long value = PyLong_AsLong(o);
  if (value == -1 && PyErr_Occurred()) {
    PyErr_Clear();
    return false;
  }
  if (value < INT32_MIN || value > INT32_MAX) return false;
  *v = static_cast<int>(value);
  return true;
}

bool flag(PyObject* o) { return o != nullptr && PyObject_IsTrue(o) == 1; }

bool number(PyObject* o, double* v) {
  *v = o == nullptr ? 0.0 : PyFloat_AsDouble(o);
  if (o == nullptr || (*v == -1.0 && PyErr_Occurred())) {
    PyErr_Clear();
    return false;
  }
  return true;
}

const void* ptr(const Tensor* t) { return t == nullptr ? nullptr : t->data_ptr(); }
bool at16(const Tensor& t) { return (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15u) == 0; }
bool dense16(const Tensor& t) { return t.is_contiguous() && at16(t); }
bool vector_of(const Tensor& t, ScalarType dtype, int64_t n) { return t.scalar_type() == dtype && t.numel() == n && t.is_contiguous(); }
bool bias_ok(const Tensor* t, int64_t n) { return t == nullptr || (vector_of(*t, kBF16, n) && at16(*t)); }
bool scalar_f32(const Tensor& t) { return t.scalar_type() == kF32 && t.numel() == 1; }
bool matrix(const Tensor& t, ScalarType dtype, int64_t rows, int64_t cols) {
  return t.dim() == 2 && t.scalar_type() == dtype && t.size(0) == rows && t.size(1) == cols && dense16(t);
}
// NHWC memory of a logical [B, C, H, W] tensor, read in place
bool channels_last(const Tensor& t) {
  const int64_t c = t.size(1), h = t.size(2), w = t.size(3);
  return t.stride(1) == 1 && t.stride(3) == c && t.stride(2) == w * c && t.stride(0) == h * w * c;
}

int64_t swizzled_bytes(int64_t rows, int64_t groups) { return (rows + 127) / 128 * ((groups + 3) / 4) * 512; }

// ---- one call --------------------------------------------------------------------------------------------------------

// The device of a call (all tensors of one op live on it), its stream and status word; the guard makes it current.
struct Call {
  c10::cuda::OptionalCUDAGuard guard;
  int index;
  void* stream = nullptr;
  int* status = nullptr;

  // false: the general path decides (wrong device, tracing, modes)
  bool begin(const Tensor& t) {
    if (c10::impl::TorchDispatchModeTLS::any_modes_set() || at::tracer::impl::is_dispatch_enabled() ||
        at::impl::torch_function_mode_enabled()) {
      return false;
    }
    index = t.get_device();
    if (index < 0 || index >= kMaxDevices) return false;
    Device& d = devices[index];
    if (d.state == 0) {
      const auto* properties = at::cuda::getDeviceProperties(index);
      d.state = properties->major == 10 && properties->minor == 0 ? 1 : -1;
    }
    if (d.state < 0) return false;
    if (d.status == nullptr) {
      PyObject* word = PyObject_CallFunction(py_status_word, "i", index);
      if (word == nullptr) failed();
      d.status_tensor = word;  // kept for the life of the process, as the Python side keeps it
      d.status = static_cast<int*>(THPVariable_Unpack(word).data_ptr());
    }
    status = d.status;
    if (index != c10::cuda::current_device()) guard.set_index(index);
    stream = at::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(index)).stream();
    return true;
  }

  bool here(const Tensor* t) const { return t == nullptr || t->get_device() == index; }
  template <typename... T>
  bool here(const Tensor* t, T... rest) const {
    return here(t) && here(rest...);
  }

  Tensor empty(at::IntArrayRef sizes, ScalarType dtype) const {
    return at::detail::empty_cuda(sizes, dtype, c10::Device(c10::kCUDA, static_cast<c10::DeviceIndex>(index)), std::nullopt);
  }

  // Swizzled E8M0 bytes; a kernel writes all of them but the padding of ragged sizes, which is zero like the reference's.
  Tensor scales(int64_t rows, int64_t groups, ScalarType dtype = kU8) const {
    Tensor t = empty({swizzled_bytes(rows, groups)}, dtype);
    if (rows % 128 != 0 || groups % 4 != 0) {
      C10_CUDA_CHECK(cudaMemsetAsync(t.data_ptr(), 0, t.numel(), static_cast<cudaStream_t>(stream)));
    }
    return t;
  }

  // Launch through the C ABI without the interpreter lock (a full launch queue blocks), then report.
  template <typename F>
  void launch(const char* what, F&& f) const {
    PyThreadState* saved = PyEval_SaveThread();
    const int code = f();
    PyEval_RestoreThread(saved);
    if (code != 0) {
      PyObject* r = PyObject_CallFunction(py_check, "is", code, what);
      Py_XDECREF(r);
      if (r == nullptr) failed();
    }
    if (py_check_status != Py_None) {
      cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
      cudaStreamIsCapturing(static_cast<cudaStream_t>(stream), &capturing);
      if (capturing == cudaStreamCaptureStatusNone) {
        PyObject* r = PyObject_CallFunction(py_check_status, "s", ("cuda:" + std::to_string(index)).c_str());
        Py_XDECREF(r);
        if (r == nullptr) failed();
      }
    }
  }
};

PyObject* wrap(Tensor t) { return THPVariable_Wrap(std::move(t)); }

PyObject* pair(Tensor a, Tensor b) {
  PyObject *x = wrap(std::move(a)), *y = wrap(std::move(b));
  PyObject* r = PyTuple_New(2);
  PyTuple_SET_ITEM(r, 0, x);
  PyTuple_SET_ITEM(r, 1, y);
  return r;
}

// A container of quant/tensor.py without its __init__: the fields are what its checks demand by construction here.
PyObject* container(PyObject* cls, std::initializer_list<std::pair<PyObject*, PyObject*>> fields) {
  auto* type = reinterpret_cast<PyTypeObject*>(cls);
  PyObject* self = type->tp_new(type, empty_tuple, nullptr);
  PyObject* dict = self == nullptr ? nullptr : PyObject_GenericGetDict(self, nullptr);
  bool ok = dict != nullptr;
  for (auto& [name, value] : fields) {  // the values are owned by this call
    ok = ok && value != nullptr && PyDict_SetItem(dict, name, value) == 0;
    Py_XDECREF(value);
  }
  Py_XDECREF(dict);
  if (!ok) {
    Py_XDECREF(self);
    failed();
  }
  return self;
}

PyObject* new_ref(PyObject* o) {
  Py_INCREF(o);
  return o;
}

PyObject* shape_tuple(const Tensor& t) {
  PyObject* r = PyTuple_New(t.dim());
  for (int64_t i = 0; i < t.dim(); ++i) PyTuple_SET_ITEM(r, i, PyLong_FromLongLong(t.size(i)));
  return r;
}

// ---- swizzled weight scales, once per exponent tensor ----------------------------------------------------------------
// Keyed on the storage; an entry holds its source, so the address cannot be reused while the entry lives, and is valid for
// one shape and version of it. At most 512 entries, the least recently used one goes first. Guarded by the interpreter lock.
//
// A graph under capture reads at its replays, any number of times and long after the call. Scales that it finds here stay for as long
// as it (or an executable made from it) does, whatever becomes of their entry; scales that it has to form are formed by
// every replay, so the call's own result never exists and is not kept here.

//
// Any stream may find an entry. Until its scales are known to be formed (`formed`: an event behind the kernels that form them), each
// call's stream waits for that; and the allocator learns of each stream that reads them beside the one they were allocated on, so that
// their memory is not given to another tensor before those reads are done.

struct Swizzled {
  const void* key;
  Tensor source, packed;
  uint32_t version;
  cudaEvent_t formed = nullptr;
  std::vector<cudaStream_t> readers;  // the first: where the scales were formed
  Swizzled(const void* k, Tensor s, Tensor p, uint32_t v) : key(k), source(std::move(s)), packed(std::move(p)), version(v) {}
  Swizzled(const Swizzled&) = delete;
  ~Swizzled() {
    if (formed != nullptr) cudaEventDestroy(formed);
  }
};
std::list<Swizzled> swizzled;
std::unordered_map<const void*, std::list<Swizzled>::iterator> swizzled_at;
constexpr size_t kSwizzledEntries = 512;

void drop_swizzled(std::unordered_map<const void*, std::list<Swizzled>::iterator>::iterator at) {
  std::list<Swizzled> gone;  // (destroyed last: the tables are whole again by then)
  gone.splice(gone.begin(), swizzled, at->second);
  swizzled_at.erase(at);
}

// Tensors whose last graph has gone. A graph lets go of them on a thread and at a time of the driver's choosing, where no call may be
// made that frees them, so they wait here for the next look-up. (The list is never destroyed: graphs may go while the process ends.)
std::mutex released_mutex;
std::vector<Tensor*>& released = *new std::vector<Tensor*>;
std::atomic<bool> any_released{false};

void release_to_next_call(void* tensor) {
  const std::lock_guard<std::mutex> lock(released_mutex);
  released.push_back(static_cast<Tensor*>(tensor));
  any_released = true;
}

void free_released() {
  if (!any_released) return;
  std::vector<Tensor*> gone;
  {
    const std::lock_guard<std::mutex> lock(released_mutex);
    gone.swap(released);
    any_released = false;
  }
  for (Tensor* t : gone) delete t;
}

// The graph that the current stream of the tensor's device is captured into; nullptr: none.
cudaGraph_t graph_under_capture(const Tensor& t) {
  if (!t.is_cuda()) return nullptr;
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  unsigned long long id = 0;
  cudaGraph_t graph = nullptr;
  const cudaError_t rc = cudaStreamGetCaptureInfo_v2(at::cuda::getCurrentCUDAStream(t.get_device()).stream(), &status, &id, &graph);
  if (rc != cudaSuccess) (void)cudaGetLastError();  // (a legacy stream beside another thread's capture: not captured itself)
  return rc == cudaSuccess && status == cudaStreamCaptureStatusActive ? graph : nullptr;
}

void keep_for_graph(cudaGraph_t graph, const Tensor& packed) {
  auto held = std::make_unique<Tensor>(packed);
  cudaUserObject_t object;
  C10_CUDA_CHECK(cudaUserObjectCreate(&object, held.get(), release_to_next_call, 1, cudaUserObjectNoDestructorSync));
  held.release();
  C10_CUDA_CHECK(cudaGraphRetainUserObject(graph, object, 1, cudaGraphUserObjectMove));
}

// Behind the kernels that formed an entry's scales on the current stream of their device
void mark_formed(Swizzled& e) {
  if (!e.packed.is_cuda()) return;
  const c10::cuda::CUDAGuard guard(e.packed.device());
  const cudaStream_t stream = at::cuda::getCurrentCUDAStream(e.packed.get_device()).stream();
  C10_CUDA_CHECK(cudaEventCreateWithFlags(&e.formed, cudaEventDisableTiming));
  C10_CUDA_CHECK(cudaEventRecord(e.formed, stream));
  e.readers.push_back(stream);
}

// Ahead of a call that reads them on that stream; false: under capture, and they may not be formed yet (a graph cannot wait for that)
bool order_reader(Swizzled& e, bool captured) {
  if (!e.packed.is_cuda()) return true;
  const auto stream = at::cuda::getCurrentCUDAStream(e.packed.get_device());
  if (e.formed != nullptr) {
    // (relaxed: a query counts as unsafe while any thread captures a graph)
    c10::cuda::CUDAStreamCaptureModeGuard mode(cudaStreamCaptureModeRelaxed);
    const cudaError_t rc = cudaEventQuery(e.formed);
    if (rc == cudaSuccess) {
      C10_CUDA_CHECK(cudaEventDestroy(std::exchange(e.formed, nullptr)));
    } else {
      (void)cudaGetLastError();
      if (rc != cudaErrorNotReady) C10_CUDA_CHECK(rc);
      if (captured) return false;
      C10_CUDA_CHECK(cudaStreamWaitEvent(stream.stream(), e.formed, 0));
    }
  }
  if (!captured && std::find(e.readers.begin(), e.readers.end(), stream.stream()) == e.readers.end()) {
    c10::cuda::CUDACachingAllocator::recordStream(e.packed.storage().data_ptr(), stream);
    e.readers.push_back(stream.stream());
  }
  return true;
}

// The packed scales, held by the caller: another thread may take the entry out while this one runs without the interpreter
// lock. Undefined: not for the cache (inference tensors have no version).
Tensor swizzled_scales(const Tensor& exponent) {
  if (exponent.is_inference()) return {};
  free_released();
  cudaGraph_t graph = graph_under_capture(exponent);
  const void* key = exponent.data_ptr();
  auto hit = swizzled_at.find(key);
  if (hit != swizzled_at.end()) {
    Swizzled& e = *hit->second;
    const bool valid = e.version == exponent._version() && e.source.sizes() == exponent.sizes() && e.source.strides() == exponent.strides();
    if (valid && order_reader(e, graph != nullptr)) {
      swizzled.splice(swizzled.begin(), swizzled, hit->second);
      if (graph != nullptr) keep_for_graph(graph, e.packed);
      return e.packed;
    }
    if (!valid) drop_swizzled(hit);
  }
  const auto version = static_cast<uint32_t>(exponent._version());
  PyObject* source = wrap(exponent);
  PyObject* made = PyObject_CallFunctionObjArgs(py_swizzle, source, nullptr);
  Py_DECREF(source);
  if (made == nullptr) failed();
  const Tensor packed = THPVariable_Unpack(made);
  Py_DECREF(made);
  if (graph != nullptr) return packed;
  // (the call may have let another thread in, which may have made the same entry: one per key)
  hit = swizzled_at.find(key);
  if (hit != swizzled_at.end()) drop_swizzled(hit);
  swizzled.emplace_front(key, exponent, packed, version);
  swizzled_at[key] = swizzled.begin();
  mark_formed(swizzled.front());
  if (swizzled.size() > kSwizzledEntries) drop_swizzled(swizzled_at.find(swizzled.back().key));
  return packed;
}

// ---- convs: geometry and epilogue ------------------------------------------------------------------------------------

// kh, kw, sh, sw, ph, pw, dh, dw from eight arguments, for NHWC codes `x` and a dense weight [Cout, kh * kw * Cin]
bool conv_geometry(const Tensor& x, const Tensor& weight, PyObject* const* a, FimConvGeometry* g) {
  if (x.dim() != 4 || !dense16(x) || weight.dim() != 2 || !dense16(weight)) return false;
  if (!integer(a[0], &g->kh) || !integer(a[1], &g->kw) || !integer(a[2], &g->stride_h) || !integer(a[3], &g->stride_w) ||
      !integer(a[4], &g->pad_h) || !integer(a[5], &g->pad_w) || !integer(a[6], &g->dil_h) || !integer(a[7], &g->dil_w)) {
    return false;
  }
  g->batch = x.size(0), g->height = x.size(1), g->width = x.size(2), g->cin = x.size(3), g->cout = weight.size(0);
  return g->stride_h >= 1 && g->stride_h <= 4 && g->stride_w >= 1 && g->stride_w <= 4 && g->cin % 32 == 0 && g->cout % 32 == 0 &&
         g->cin > 0 && g->cout > 0 && x.numel() > 0 && g->kh >= 1 && g->kw >= 1 && g->dil_h >= 1 && g->dil_w >= 1 && g->pad_h >= 0 &&
         g->pad_w >= 0 && weight.size(1) == static_cast<int64_t>(g->kh) * g->kw * g->cin;
}

int out_size(int size, int k, int p, int d, int s) { return (size + 2 * p - d * (k - 1) - 1) / s + 1; }

bool out_sizes(const FimConvGeometry& g, int64_t (&sizes)[4]) {
  if (g.height + 2 * g.pad_h - g.dil_h * (g.kh - 1) < 1 || g.width + 2 * g.pad_w - g.dil_w * (g.kw - 1) < 1) return false;
  sizes[0] = g.batch, sizes[1] = out_size(g.height, g.kh, g.pad_h, g.dil_h, g.stride_h);
  sizes[2] = out_size(g.width, g.kw, g.pad_w, g.dil_w, g.stride_w), sizes[3] = g.cout;
  return true;
}

FimConvGeometry pointwise(int64_t rows, int64_t cin, int64_t cout) {
  return {1, 1, static_cast<int>(rows), static_cast<int>(cin), static_cast<int>(cout), 1, 1, 1, 1, 0, 0, 1, 1};
}
bool rows_fit(int64_t rows) { return rows > 0 && rows < INT32_MAX; }

bool set_residual(const Tensor* residual, const int64_t (&sizes)[4], FimConvEpilogue* ep) {
  if (residual == nullptr) return true;
  if (residual->dim() != 4 || residual->scalar_type() != kBF16 || residual->size(3) > sizes[3]) return false;
  for (int i = 0; i < 4; ++i) ep->res_stride[i] = residual->stride(i);
  ep->residual = residual->data_ptr();
  ep->res_channels = residual->size(3);
  return true;
}

// "none" / "relu" / "gelu" / "relu_early"
bool activation(PyObject* o, int fallback, int* act) {
  *act = fallback;
  if (o == nullptr) return true;
  static const char* kNames[] = {"none", "relu", "gelu", "relu_early"};
  if (!PyUnicode_CheckExact(o)) return false;
  for (int i = 0; i < 4; ++i) {
    if (PyUnicode_CompareWithASCIIString(o, kNames[i]) == 0) {
      *act = i;
      return true;
    }
  }
  return false;
}

ScalarType out_dtype(int mode) {
  switch (mode) {
    case FIM_OUT_BF16: return kBF16;
    case FIM_OUT_F32: return kF32;
    case FIM_OUT_INT8: return kI8;
    default: return kE4M3;
  }
}

// ---- the ops ---------------------------------------------------------------------------------------------------------
// Each returns nullptr for "not served here" (the wrapper turns that into NotImplemented).

using Args = PyObject* const*;

// the channels-last view of an NCHW-contiguous tensor, not itself row-major
bool channels_first_view(const Tensor& v) {
  return v.dim() == 4 && !v.is_contiguous() && v.stride(2) == 1 && v.stride(1) == v.size(2) && v.stride(3) == v.size(1) * v.size(2) &&
         v.stride(0) == v.size(3) * v.size(1) * v.size(2);
}

int float_code(const Tensor& v) { return v.scalar_type() == kF32 ? FIM_DTYPE_F32 : v.scalar_type() == kBF16 ? FIM_DTYPE_BF16 : -1; }

PyObject* quantize_mxfp8(Args a) {  // value, scale_exponent
  const Tensor *v = plain_tensor(a[0]), *e = plain_tensor(a[1]);
  if (v == nullptr || e == nullptr || v->dim() < 2 || v->numel() == 0 || float_code(*v) < 0) return nullptr;
  const int64_t c = v->size(-1), padded = (c + 31) / 32 * 32;
  if (e->dim() != 1 || !vector_of(*e, kI8, padded / 32)) return nullptr;
  const bool first = channels_first_view(*v);
  if (!first && !dense16(*v)) return nullptr;
  Call call;
  if (!call.begin(*v) || !call.here(e)) return nullptr;
  c10::SmallVector<int64_t, 5> sizes(v->sizes().begin(), v->sizes().end());
  sizes.back() = padded;
  Tensor out = call.empty(sizes, kE4M3);
  call.launch("quantize_mxfp8", [&] {
    if (first) {
      return abi.fim_quantize_mxfp8_static_nchw(v->data_ptr(), float_code(*v), static_cast<const int8_t*>(e->data_ptr()), out.data_ptr(),
                                                v->size(0), c, v->size(1) * v->size(2), call.stream);
    }
    return abi.fim_quantize_mxfp8_static(v->data_ptr(), float_code(*v), static_cast<const int8_t*>(e->data_ptr()), out.data_ptr(),
                                         v->numel() / c, c, call.stream);
  });
  return container(py_quantized_tensor, {{name_values, wrap(out)}, {name_scale_exponent, new_ref(a[1])}, {name_logical_shape, shape_tuple(*v)}});
}

PyObject* quantize_int8(Args a) {  // value, scale, channel_scale
  const Tensor *v = plain_tensor(a[0]), *s = plain_tensor(a[1]);
  if (v == nullptr || s == nullptr || (a[2] != nullptr && a[2] != Py_None) || v->numel() == 0 || float_code(*v) < 0) return nullptr;
  if (!scalar_f32(*s) || s->dim() != 0) return nullptr;
  const bool first = channels_first_view(*v);
  if (first ? v->size(3) % 16 != 0 : !dense16(*v)) return nullptr;
  Call call;
  if (!call.begin(*v) || !call.here(s)) return nullptr;
  Tensor out = call.empty(v->sizes(), kI8);
  call.launch("quantize_int8", [&] {
    const float* scale = static_cast<const float*>(s->data_ptr());
    if (first) {
      return abi.fim_quantize_int8_static_nchw(v->data_ptr(), float_code(*v), scale, out.data_ptr(), v->size(0), v->size(3),
                                               v->size(1) * v->size(2), call.stream);
    }
    return abi.fim_quantize_int8_static(v->data_ptr(), float_code(*v), scale, out.data_ptr(), v->numel(), call.stream);
  });
  return container(py_int8_tensor, {{name_values, wrap(out)}, {name_scale, new_ref(a[1])}});
}

PyObject* quantize_mxfp8_dynamic(Args a) {  // value
  const Tensor* v = plain_tensor(a[0]);
  if (v == nullptr || v->dim() < 1 || v->numel() == 0 || float_code(*v) < 0 || !dense16(*v) || v->size(-1) % 32 != 0) return nullptr;
  Call call;
  if (!call.begin(*v)) return nullptr;
  const int64_t c = v->size(-1), rows = v->numel() / c;
  Tensor out = call.empty(v->sizes(), kE4M3), scales = call.scales(rows, c / 32);
  call.launch("quantize_mxfp8_dynamic", [&] {
    return abi.fim_quantize_mxfp8_dynamic(v->data_ptr(), float_code(*v), out.data_ptr(), scales.data_ptr(), 1, rows, c, call.stream);
  });
  return pair(out, scales);
}

PyObject* gelu_quantize(Args a) {  // value, scale_exponent, approximate, input_bias
  const Tensor *v = plain_tensor(a[0]), *e = plain_tensor(a[1]), *bias;
  if (v == nullptr || e == nullptr || !optional_tensor(a[3], &bias)) return nullptr;
  if (a[2] != nullptr && !(PyUnicode_CheckExact(a[2]) && PyUnicode_CompareWithASCIIString(a[2], "none") == 0)) return nullptr;
  if (v->dim() < 2 || v->numel() == 0 || v->scalar_type() != kBF16 || !dense16(*v) || v->size(-1) % 32 != 0) return nullptr;
  const int64_t c = v->size(-1);
  if (e->dim() != 1 || !vector_of(*e, kI8, c / 32) || (bias != nullptr && !vector_of(*bias, kF32, c))) return nullptr;
  Call call;
  if (!call.begin(*v) || !call.here(e, bias)) return nullptr;
  Tensor out = call.empty(v->sizes(), kE4M3);
  call.launch("gelu_quantize", [&] {
    return abi.fim_gelu_quantize_mxfp8(v->data_ptr(), static_cast<const float*>(ptr(bias)), static_cast<const int8_t*>(e->data_ptr()),
                                       out.data_ptr(), v->numel() / c, c, call.stream);
  });
  return container(py_quantized_tensor, {{name_values, wrap(out)}, {name_scale_exponent, new_ref(a[1])}, {name_logical_shape, shape_tuple(*v)}});
}

// The conv of the two MXFP8 conv ops: static exponents (int8 [Cin / 32]) or per-pixel scales (`pixel_scales`).
PyObject* mx_conv(const Tensor& x, const Tensor* exponent, const Tensor* pixel_scales, const Tensor& weight, const Tensor& weight_scales,
                  const Tensor* bias, const FimConvGeometry& g, const Tensor* residual, int act, int mode, const Tensor* out_exponent,
                  Call& call, bool bf16_in = false) {
  int64_t sizes[4];
  FimConvEpilogue ep = {};
  if (!out_sizes(g, sizes) || !set_residual(residual, sizes, &ep)) return nullptr;
  ep.bias = ptr(bias), ep.act = act, ep.out_mode = mode;
  ep.out_exponent = static_cast<const int8_t*>(ptr(out_exponent));
  Tensor out = call.empty(sizes, out_dtype(mode)), scales;
  if (mode == FIM_OUT_E4M3_DYNAMIC) {
    scales = call.scales(sizes[0] * sizes[1] * sizes[2], sizes[3] / 32);
    ep.out_scales = scales.data_ptr();
  }
  call.launch("mxfp8_conv2d", [&] {
    if (bf16_in) {
      return abi.fim_mxfp8_conv2d_bf16(x.data_ptr(), static_cast<const int8_t*>(ptr(exponent)), weight.data_ptr(), weight_scales.data_ptr(),
                                       &g, &ep, out.data_ptr(), call.status, call.stream);
    }
    return abi.fim_mxfp8_conv2d(x.data_ptr(), static_cast<const int8_t*>(ptr(exponent)), ptr(pixel_scales), weight.data_ptr(),
                                weight_scales.data_ptr(), &g, &ep, out.data_ptr(), call.status, call.stream);
  });
  return mode == FIM_OUT_E4M3_DYNAMIC ? pair(out, scales) : wrap(out);
}

bool out_exponent_ok(const Tensor* e, int64_t cout) { return e == nullptr || (e->dim() == 1 && vector_of(*e, kI8, cout / 32)); }

// x, channel_exponent, weight, weight_exponent, bias, kh .. dw (5-12), relu, residual, out_exponent
PyObject* mxfp8_conv2d(Args a) {
  const Tensor *x = plain_tensor(a[0]), *e = plain_tensor(a[1]), *w = plain_tensor(a[2]), *we = plain_tensor(a[3]), *bias, *res, *oe;
  if (x == nullptr || e == nullptr || w == nullptr || we == nullptr) return nullptr;
  if (!optional_tensor(a[4], &bias) || !optional_tensor(a[14], &res) || !optional_tensor(a[15], &oe)) return nullptr;
  FimConvGeometry g;
  if (x->scalar_type() != kE4M3 || w->scalar_type() != kE4M3 || !conv_geometry(*x, *w, a + 5, &g)) return nullptr;
  if (e->dim() != 1 || !vector_of(*e, kI8, g.cin / 32) || we->dim() != 2 || we->scalar_type() != kI8 || we->size(0) != g.cout ||
      we->size(1) != w->size(1) / 32 || !bias_ok(bias, g.cout) || !out_exponent_ok(oe, g.cout)) {
    return nullptr;
  }
  Call call;
  if (!call.begin(*x) || !call.here(e, w, we, bias, res, oe)) return nullptr;
  const Tensor packed = swizzled_scales(*we);
  if (!packed.defined()) return nullptr;
  return mx_conv(*x, e, nullptr, *w, packed, bias, g, res, flag(a[13]) ? FIM_ACT_RELU : FIM_ACT_NONE,
                 oe == nullptr ? FIM_OUT_BF16 : FIM_OUT_E4M3_STATIC, oe, call);
}

// the output format three optional arguments of the fused convs select; false for a contradiction
bool fused_mode(const Tensor* out_exponent, PyObject* dynamic, PyObject* fp32, int* mode) {
  const bool d = flag(dynamic), f = flag(fp32);
  if ((out_exponent != nullptr) + d + f > 1) return false;
  *mode = f ? FIM_OUT_F32 : d ? FIM_OUT_E4M3_DYNAMIC : out_exponent != nullptr ? FIM_OUT_E4M3_STATIC : FIM_OUT_BF16;
  return true;
}

// x, act_scale, weight, weight_scales, bias, kh .. dw (5-12), act, residual, out_exponent, dynamic_out, out_fp32
PyObject* mxfp8_conv2d_fused(Args a) {
  const Tensor *x = plain_tensor(a[0]), *s = plain_tensor(a[1]), *w = plain_tensor(a[2]), *ws = plain_tensor(a[3]), *bias, *res, *oe;
  if (x == nullptr || s == nullptr || w == nullptr || ws == nullptr) return nullptr;
  if (!optional_tensor(a[4], &bias) || !optional_tensor(a[14], &res) || !optional_tensor(a[15], &oe)) return nullptr;
  FimConvGeometry g;
  int act, mode;
  if (x->scalar_type() != kE4M3 || w->scalar_type() != kE4M3 || !conv_geometry(*x, *w, a + 5, &g) || !activation(a[13], 0, &act) ||
      !fused_mode(oe, a[16], a[17], &mode)) {
    return nullptr;
  }
  const bool per_pixel = s->scalar_type() == kU8;
  if (per_pixel) {
    if (g.kh != 1 || g.kw != 1 || g.stride_h != 1 || g.stride_w != 1 || g.pad_h != 0 || g.pad_w != 0 || !dense16(*s) ||
        s->numel() != swizzled_bytes(x->numel() / g.cin, g.cin / 32)) {
      return nullptr;
    }
  } else if (s->dim() != 1 || !vector_of(*s, kI8, g.cin / 32)) {
    return nullptr;
  }
  if (ws->scalar_type() != kU8 || !dense16(*ws) || ws->numel() != swizzled_bytes(g.cout, w->size(1) / 32) || !bias_ok(bias, g.cout) ||
      !out_exponent_ok(oe, g.cout)) {
    return nullptr;
  }
  Call call;
  if (!call.begin(*x) || !call.here(s, w, ws, bias, res, oe)) return nullptr;
  return mx_conv(*x, per_pixel ? nullptr : s, per_pixel ? s : nullptr, *w, *ws, bias, g, res, act, mode, oe, call);
}

// x, act_exponent, weight, weight_scales, bias, act, residual, out_exponent, dynamic_out, out_fp32
PyObject* mxfp8_conv2d_bf16(Args a) {
  const Tensor *x = plain_tensor(a[0]), *w = plain_tensor(a[2]), *ws = plain_tensor(a[3]), *e, *bias, *res, *oe;
  if (x == nullptr || w == nullptr || ws == nullptr || !optional_tensor(a[1], &e) || !optional_tensor(a[4], &bias) ||
      !optional_tensor(a[6], &res) || !optional_tensor(a[7], &oe)) {
    return nullptr;
  }
  int act, mode;
  if (x->scalar_type() != kBF16 || x->dim() != 4 || !dense16(*x) || x->numel() == 0 || x->size(3) % 128 != 0 || w->dim() != 2 ||
      !matrix(*w, kE4M3, w->size(0), x->size(3)) || w->size(0) % 32 != 0 || !activation(a[5], 0, &act) || !fused_mode(oe, a[8], a[9], &mode)) {
    return nullptr;
  }
  FimConvGeometry g = {static_cast<int>(x->size(0)), static_cast<int>(x->size(1)), static_cast<int>(x->size(2)), static_cast<int>(x->size(3)),
                       static_cast<int>(w->size(0)), 1, 1, 1, 1, 0, 0, 1, 1};
  if (ws->scalar_type() != kU8 || !dense16(*ws) || ws->numel() != swizzled_bytes(g.cout, g.cin / 32) || !bias_ok(bias, g.cout) ||
      !out_exponent_ok(oe, g.cout) || (e != nullptr && (e->dim() != 1 || !vector_of(*e, kI8, g.cin / 32)))) {
    return nullptr;
  }
  Call call;
  if (!call.begin(*x) || !call.here(e, w, ws, bias, res, oe)) return nullptr;
  return mx_conv(*x, e, nullptr, *w, *ws, bias, g, res, act, mode, oe, call, true);
}

// x, x_scales, w1, w1_scales, b1, w2, w2_scales, b2, residual
PyObject* mxfp8_gelu_mlp_residual(Args a) {
  const Tensor* t[9];
  for (int i = 0; i < 9; ++i) {
    if ((t[i] = plain_tensor(a[i])) == nullptr) return nullptr;
  }
  const Tensor &x = *t[0], &xs = *t[1], &w1 = *t[2], &s1 = *t[3], &b1 = *t[4], &w2 = *t[5], &s2 = *t[6], &b2 = *t[7], &res = *t[8];
  if (x.dim() < 1 || x.numel() == 0 || x.scalar_type() != kE4M3 || !dense16(x)) return nullptr;
  const int64_t c = x.size(-1), rows = x.numel() / c;
  if ((c != 128 && c != 256) || !matrix(w1, kE4M3, 2 * c, c) || !matrix(w2, kE4M3, c, 2 * c)) return nullptr;
  auto swizzle_ok = [](const Tensor& s, int64_t r, int64_t k) { return s.scalar_type() == kU8 && dense16(s) && s.numel() == swizzled_bytes(r, k / 32); };
  if (!swizzle_ok(xs, rows, c) || !swizzle_ok(s1, 2 * c, c) || !swizzle_ok(s2, c, 2 * c) || !bias_ok(&b1, 2 * c) || !bias_ok(&b2, c) ||
      res.scalar_type() != kBF16 || res.sizes() != x.sizes() || !dense16(res)) {
    return nullptr;
  }
  Call call;
  if (!call.begin(x) || !call.here(t[1], t[2], t[3], t[4], t[5], t[6], t[7], t[8])) return nullptr;
  Tensor out = call.empty(x.sizes(), kBF16);
  call.launch("mxfp8_gelu_mlp_residual", [&] {
    return abi.fim_mxfp8_gelu_mlp_residual(x.data_ptr(), xs.data_ptr(), w1.data_ptr(), s1.data_ptr(), b1.data_ptr(), w2.data_ptr(),
                                           s2.data_ptr(), b2.data_ptr(), res.data_ptr(), out.data_ptr(), rows, c, call.status, call.stream);
  });
  return wrap(out);
}

// x, weight, a_scale, w_scale, bias, kh .. dw (5-12), relu, residual, out_scale
PyObject* int8_conv2d(Args a) {
  const Tensor *x = plain_tensor(a[0]), *w = plain_tensor(a[1]), *as = plain_tensor(a[2]), *ws = plain_tensor(a[3]), *bias, *res, *os;
  if (x == nullptr || w == nullptr || as == nullptr || ws == nullptr) return nullptr;
  if (!optional_tensor(a[4], &bias) || !optional_tensor(a[14], &res) || !optional_tensor(a[15], &os)) return nullptr;
  FimConvGeometry g;
  int64_t sizes[4];
  FimConvEpilogue ep = {};
  if (x->scalar_type() != kI8 || w->scalar_type() != kI8 || !conv_geometry(*x, *w, a + 5, &g) || !out_sizes(g, sizes) ||
      !set_residual(res, sizes, &ep) || !scalar_f32(*as) || !vector_of(*ws, kF32, g.cout) || !at16(*ws) || !bias_ok(bias, g.cout) ||
      (os != nullptr && !scalar_f32(*os))) {
    return nullptr;
  }
  Call call;
  if (!call.begin(*x) || !call.here(w, as, ws, bias, res, os)) return nullptr;
  ep.bias = ptr(bias), ep.act = flag(a[13]) ? FIM_ACT_RELU : FIM_ACT_NONE;
  ep.out_mode = os == nullptr ? FIM_OUT_BF16 : FIM_OUT_INT8;
  ep.out_scale = static_cast<const float*>(ptr(os));
  Tensor out = call.empty(sizes, out_dtype(ep.out_mode));
  call.launch("int8_conv2d", [&] {
    return abi.fim_int8_conv2d(x->data_ptr(), w->data_ptr(), static_cast<const float*>(as->data_ptr()), static_cast<const float*>(ws->data_ptr()),
                               &g, &ep, out.data_ptr(), call.status, call.stream);
  });
  return wrap(out);
}

// x, weight, a_scale, w_scale, bias, kh .. dw (5-12), relu, out_scale
PyObject* int8_conv2d_maxpool(Args a) {
  const Tensor *x = plain_tensor(a[0]), *w = plain_tensor(a[1]), *as = plain_tensor(a[2]), *ws = plain_tensor(a[3]), *bias, *os = plain_tensor(a[14]);
  if (x == nullptr || w == nullptr || as == nullptr || ws == nullptr || os == nullptr || !optional_tensor(a[4], &bias)) return nullptr;
  FimConvGeometry g;
  int64_t sizes[4];
  if (x->scalar_type() != kI8 || w->scalar_type() != kI8 || !conv_geometry(*x, *w, a + 5, &g) || !out_sizes(g, sizes) || !scalar_f32(*as) ||
      !vector_of(*ws, kF32, g.cout) || !at16(*ws) || !bias_ok(bias, g.cout) || !scalar_f32(*os)) {
    return nullptr;
  }
  // one launch needs a whole window and 64-channel K steps (the general path runs the pooling pass otherwise)
  if (sizes[1] < 2 || sizes[2] < 2 || g.cin % 64 != 0) return nullptr;
  Call call;
  if (!call.begin(*x) || !call.here(w, as, ws, bias, os)) return nullptr;
  FimConvEpilogue ep = {};
  ep.bias = ptr(bias), ep.act = flag(a[13]) ? FIM_ACT_RELU : FIM_ACT_NONE, ep.out_mode = FIM_OUT_BF16;
  ep.out_scale = static_cast<const float*>(os->data_ptr());
  Tensor out = call.empty(sizes, kBF16), pooled = call.empty({sizes[0], sizes[1] / 2, sizes[2] / 2, sizes[3]}, kI8);
  call.launch("int8_conv2d_maxpool", [&] {
    return abi.fim_int8_conv2d_maxpool(x->data_ptr(), w->data_ptr(), static_cast<const float*>(as->data_ptr()),
                                       static_cast<const float*>(ws->data_ptr()), &g, &ep, out.data_ptr(), pooled.data_ptr(), call.status,
                                       call.stream);
  });
  return pair(out, pooled);
}

// -- GEMMs: a 1x1 conv over a one-row image of M pixels --

Tensor mx_gemm(const Tensor& a, int64_t rows, const Tensor* exponent, const Tensor* row_scales, const Tensor& weight, const Tensor& weight_scales,
               const Tensor* bias, const Call& call, const char* what) {
  const FimConvGeometry g = pointwise(rows, weight.size(1), weight.size(0));
  FimConvEpilogue ep = {};
  ep.bias = ptr(bias), ep.out_mode = FIM_OUT_BF16;
  Tensor out = call.empty({rows, weight.size(0)}, kBF16);
  call.launch(what, [&] {
    return abi.fim_mxfp8_conv2d(a.data_ptr(), static_cast<const int8_t*>(ptr(exponent)), ptr(row_scales), weight.data_ptr(),
                                weight_scales.data_ptr(), &g, &ep, out.data_ptr(), call.status, call.stream);
  });
  return out;
}

// an attribute of a container as a plain tensor (a borrowed reference is enough: the container outlives the call)
const Tensor* member(PyObject* o, PyObject* name) {
  if (o == nullptr || o == Py_None) return nullptr;
  PyObject* v = PyObject_GetAttr(o, name);
  if (v == nullptr) {
    PyErr_Clear();
    return nullptr;
  }
  const Tensor* t = Py_REFCNT(v) > 1 ? plain_tensor(v) : nullptr;
  Py_DECREF(v);
  return t;
}

bool linear_operands(const Tensor* values, const Tensor* exponent, const Tensor* w, const Tensor* we) {
  if (values == nullptr || exponent == nullptr || w == nullptr || we == nullptr || w->dim() != 2 || values->dim() < 1) return false;
  const int64_t n = w->size(0), k = w->size(1);
  return values->scalar_type() == kE4M3 && values->numel() > 0 && dense16(*values) && values->size(-1) == k && n > 0 && n % 32 == 0 &&
         k % 32 == 0 && matrix(*w, kE4M3, n, k) && exponent->dim() == 1 && vector_of(*exponent, kI8, k / 32) && we->dim() == 2 &&
         we->scalar_type() == kI8 && we->size(0) == n && we->size(1) == k / 32 && rows_fit(values->numel() / k);
}

PyObject* mxfp8_linear(Args a) {  // activation, bias, weight
  const Tensor *v = member(a[0], name_values), *e = member(a[0], name_scale_exponent), *w = member(a[2], name_values),
               *we = member(a[2], name_scale_exponent), *bias;
  if (!linear_operands(v, e, w, we) || !optional_tensor(a[1], &bias) || !bias_ok(bias, w->size(0))) return nullptr;
  Call call;
  if (!call.begin(*v) || !call.here(e, w, we, bias)) return nullptr;
  const Tensor packed = swizzled_scales(*we);
  if (!packed.defined()) return nullptr;
  return wrap(mx_gemm(*v, v->numel() / w->size(1), e, nullptr, *w, packed, bias, call, "mxfp8_linear"));
}

PyObject* mxfp8_gelu_mlp(Args a) {  // x, w1, b1, hidden_exponent, w2
  const Tensor *v = member(a[0], name_values), *e = member(a[0], name_scale_exponent), *w1 = member(a[1], name_values),
               *e1 = member(a[1], name_scale_exponent), *b1 = plain_tensor(a[2]), *he = plain_tensor(a[3]), *w2 = member(a[4], name_values),
               *e2 = member(a[4], name_scale_exponent);
  if (!linear_operands(v, e, w1, e1) || b1 == nullptr || he == nullptr || w2 == nullptr || e2 == nullptr) return nullptr;
  const int64_t hidden = w1->size(0), rows = v->numel() / w1->size(1);
  if (b1->numel() != hidden || he->dim() != 1 || !vector_of(*he, kI8, hidden / 32) || w2->dim() != 2 || w2->size(0) % 32 != 0 ||
      w2->size(0) == 0 || !matrix(*w2, kE4M3, w2->size(0), hidden) || e2->dim() != 2 || e2->scalar_type() != kI8 ||
      e2->size(0) != w2->size(0) || e2->size(1) != hidden / 32) {
    return nullptr;
  }
  Call call;
  if (!call.begin(*v) || !call.here(e, w1, e1, b1, he, w2, e2)) return nullptr;
  const Tensor packed1 = swizzled_scales(*e1), packed2 = swizzled_scales(*e2);
  if (!packed1.defined() || !packed2.defined()) return nullptr;
  // the reference's rounding points: the first product rounds to bf16 before b1 is added, GELU runs in fp32 on that sum,
  // and the second product has no bias
  Tensor q = call.empty({rows, hidden}, kE4M3);
  int code = FIM_ERR_UNSUPPORTED;
  if (b1->scalar_type() == kBF16 && b1->is_contiguous() && at16(*b1)) {  // all of it in the epilogue of the first product
    const FimConvGeometry g = pointwise(rows, w1->size(1), hidden);
    FimConvEpilogue ep = {};
    ep.bias = b1->data_ptr(), ep.act = FIM_ACT_GELU_SUM, ep.out_mode = FIM_OUT_E4M3_STATIC;
    ep.out_exponent = static_cast<const int8_t*>(he->data_ptr());
    call.launch("mxfp8_gelu_mlp", [&] {
      code = abi.fim_mxfp8_conv2d(v->data_ptr(), static_cast<const int8_t*>(e->data_ptr()), nullptr, w1->data_ptr(), packed1.data_ptr(), &g, &ep,
                                  q.data_ptr(), call.status, call.stream);
      return code == FIM_ERR_UNSUPPORTED ? 0 : code;
    });
  }
  if (code == FIM_ERR_UNSUPPORTED) {  // a bias of another type, a plan without 128-byte K steps or with 64-wide tiles
    const Tensor bias = b1->scalar_type() == kF32 && b1->is_contiguous() ? *b1 : b1->to(kF32).contiguous();
    Tensor h = mx_gemm(*v, rows, e, nullptr, *w1, packed1, nullptr, call, "mxfp8_gelu_mlp");
    call.launch("mxfp8_gelu_mlp", [&] {
      return abi.fim_gelu_quantize_mxfp8(h.data_ptr(), static_cast<const float*>(bias.data_ptr()), static_cast<const int8_t*>(he->data_ptr()),
                                         q.data_ptr(), rows, hidden, call.stream);
    });
  }
  return wrap(mx_gemm(q, rows, he, nullptr, *w2, packed2, nullptr, call, "mxfp8_gelu_mlp"));
}

PyObject* mxfp8_scaled_mm(Args a) {  // a, b_t, a_scale, b_scale, bias
  const Tensor *x = plain_tensor(a[0]), *bt = plain_tensor(a[1]), *as = plain_tensor(a[2]), *bs = plain_tensor(a[3]), *bias;
  if (x == nullptr || bt == nullptr || as == nullptr || bs == nullptr || !optional_tensor(a[4], &bias)) return nullptr;
  if (x->dim() != 2 || bt->dim() != 2 || x->scalar_type() != kE4M3 || bt->scalar_type() != kE4M3 || !dense16(*x) || !at16(*bt)) return nullptr;
  const int64_t m = x->size(0), k = x->size(1), n = bt->size(1);
  if (bt->size(0) != k || bt->stride(0) != 1 || bt->stride(1) != k || k % 32 != 0 || n % 32 != 0 || k == 0 || n == 0 || !rows_fit(m) ||
      as->element_size() != 1 || bs->element_size() != 1 || !dense16(*as) || !dense16(*bs) || as->numel() != swizzled_bytes(m, k / 32) ||
      bs->numel() != swizzled_bytes(n, k / 32) || !bias_ok(bias, n)) {
    return nullptr;
  }
  Call call;
  if (!call.begin(*x) || !call.here(bt, as, bs, bias)) return nullptr;
  return wrap(mx_gemm(*x, m, nullptr, as, bt->t(), *bs, bias, call, "mxfp8_scaled_mm"));
}

Tensor int8_gemm(const Tensor& a, int64_t rows, const Tensor& weight, const void* a_scale, const Tensor& w_scale, const Tensor* bias,
                 const Tensor* residual, int act, const Call& call, const char* what) {
  const FimConvGeometry g = pointwise(rows, weight.size(1), weight.size(0));
  FimConvEpilogue ep = {};
  ep.bias = ptr(bias), ep.act = act, ep.out_mode = FIM_OUT_BF16;
  if (residual != nullptr) {
    ep.residual = residual->data_ptr();
    ep.res_stride[0] = ep.res_stride[1] = rows * weight.size(0), ep.res_stride[2] = weight.size(0), ep.res_stride[3] = 1;
    ep.res_channels = weight.size(0);
  }
  Tensor out = call.empty({rows, weight.size(0)}, kBF16);
  call.launch(what, [&] {
    return abi.fim_int8_conv2d(a.data_ptr(), weight.data_ptr(), static_cast<const float*>(a_scale), static_cast<const float*>(w_scale.data_ptr()),
                               &g, &ep, out.data_ptr(), call.status, call.stream);
  });
  return out;
}

PyObject* int8_linear(Args a) {  // a, weight, a_scale, w_scale, bias, relu, gelu, residual
  const Tensor *x = plain_tensor(a[0]), *w = plain_tensor(a[1]), *as = plain_tensor(a[2]), *ws = plain_tensor(a[3]), *bias, *res;
  if (x == nullptr || w == nullptr || as == nullptr || ws == nullptr || !optional_tensor(a[4], &bias) || !optional_tensor(a[7], &res)) return nullptr;
  const bool relu = flag(a[5]), gelu = flag(a[6]);
  if (x->dim() != 2 || w->dim() != 2 || x->scalar_type() != kI8 || !dense16(*x) || (relu && gelu)) return nullptr;
  const int64_t m = x->size(0), k = x->size(1), n = w->size(0);
  if (!matrix(*w, kI8, n, k) || k % 32 != 0 || n % 32 != 0 || k == 0 || n == 0 || !rows_fit(m) || !scalar_f32(*as) || !vector_of(*ws, kF32, n) ||
      !at16(*ws) || !bias_ok(bias, n) || (res != nullptr && !matrix(*res, kBF16, m, n))) {
    return nullptr;
  }
  Call call;
  if (!call.begin(*x) || !call.here(w, as, ws, bias, res)) return nullptr;
  // the linear's order is ReLU -> bf16 -> GELU -> residual: its ReLU comes before the residual, the conv's after it
  return wrap(int8_gemm(*x, m, *w, as->data_ptr(), *ws, bias, res, gelu ? FIM_ACT_GELU : relu ? FIM_ACT_RELU_EARLY : FIM_ACT_NONE, call, "int8_linear"));
}

// -- depthwise --

// value [B, C, H, W] channels-last bf16, weight bf16 [25, C], bias fp32 [C]
bool depthwise_operands(const Tensor* v, const Tensor* w, const Tensor* bias) {
  if (v == nullptr || w == nullptr || bias == nullptr || v->dim() != 4 || v->scalar_type() != kBF16 || v->numel() == 0 || !at16(*v) ||
      v->size(1) % 32 != 0 || !channels_last(*v)) {
    return false;
  }
  for (int i = 0; i < 4; ++i) {
    if (v->size(i) >= INT32_MAX) return false;
  }
  return w->dim() == 2 && w->size(0) == 25 && w->size(1) == v->size(1) && w->scalar_type() == kBF16 && w->is_contiguous() &&
         bias->dim() == 1 && vector_of(*bias, kF32, v->size(1));
}

PyObject* depthwise_bf16(Args a) {  // value, weight, bias, act
  const Tensor *v = plain_tensor(a[0]), *w = plain_tensor(a[1]), *b = plain_tensor(a[2]);
  int act;
  if (!depthwise_operands(v, w, b) || !activation(a[3], FIM_ACT_GELU, &act)) return nullptr;
  Call call;
  if (!call.begin(*v) || !call.here(w, b)) return nullptr;
  Tensor out = call.empty({v->size(0), v->size(2), v->size(3), v->size(1)}, kBF16);
  call.launch("depthwise5x5_act", [&] {
    return abi.fim_dw5x5_bf16(v->data_ptr(), w->data_ptr(), static_cast<const float*>(b->data_ptr()), out.data_ptr(), v->size(0), v->size(2),
                              v->size(3), v->size(1), act, call.status, call.stream);
  });
  return wrap(out);
}

void depthwise_mx_launch(const Tensor& v, const Tensor& w, const Tensor& b, int act, Tensor& out, Tensor& scales, ScalarType scale_dtype,
                         const Call& call, const char* what) {
  const int64_t c = v.size(1), rows = v.size(0) * v.size(2) * v.size(3);
  out = call.empty({rows, c}, kE4M3);
  scales = call.empty({swizzled_bytes(rows, c / 32)}, scale_dtype);  // (the kernel writes the padding too)
  call.launch(what, [&] {
    return abi.fim_dw5x5_mxfp8(v.data_ptr(), w.data_ptr(), static_cast<const float*>(b.data_ptr()), out.data_ptr(), scales.data_ptr(), 1,
                               v.size(0), v.size(2), v.size(3), c, act, call.status, call.stream);
  });
}

PyObject* depthwise_mx(Args a, int fixed_act) {  // value, weight, bias(, act)
  const Tensor *v = plain_tensor(a[0]), *w = plain_tensor(a[1]), *b = plain_tensor(a[2]);
  int act = fixed_act;
  if (!depthwise_operands(v, w, b) || (fixed_act < 0 && !activation(a[3], FIM_ACT_GELU, &act))) return nullptr;
  Call call;
  if (!call.begin(*v) || !call.here(w, b)) return nullptr;
  Tensor out, scales;
  depthwise_mx_launch(*v, *w, *b, act, out, scales, fixed_act < 0 ? kU8 : kE8M0, call, "depthwise5x5_mxfp8");
  return pair(out, scales);
}
PyObject* depthwise_act_mx(Args a) { return depthwise_mx(a, -1); }
PyObject* depthwise_relu_mx(Args a) { return depthwise_mx(a, FIM_ACT_RELU); }

Tensor depthwise_int8_launch(const Tensor& v, const Tensor& w, const Tensor& b, const Tensor& scale, const Call& call, const char* what) {
  Tensor out = call.empty({v.size(0) * v.size(2) * v.size(3), v.size(1)}, kI8);
  call.launch(what, [&] {
    return abi.fim_dw5x5_relu_int8(v.data_ptr(), w.data_ptr(), static_cast<const float*>(b.data_ptr()), static_cast<const float*>(scale.data_ptr()),
                                   out.data_ptr(), v.size(0), v.size(2), v.size(3), v.size(1), call.status, call.stream);
  });
  return out;
}

PyObject* depthwise_relu_int8(Args a) {  // value, weight, bias, scale
  const Tensor *v = plain_tensor(a[0]), *w = plain_tensor(a[1]), *b = plain_tensor(a[2]), *s = plain_tensor(a[3]);
  if (!depthwise_operands(v, w, b) || s == nullptr || !scalar_f32(*s)) return nullptr;
  Call call;
  if (!call.begin(*v) || !call.here(w, b, s)) return nullptr;
  return wrap(depthwise_int8_launch(*v, *w, *b, *s, call, "depthwise5x5_relu_int8"));
}

// -- depthwise-separable blocks: the depthwise producer, then the pointwise product over its rows --

// rows [B * H * W, N] as the channels-last [B, N, H, W] tensor they are the memory of
Tensor as_image(const Tensor& rows, const Tensor& v) {
  const int64_t n = rows.size(1), h = v.size(2), w = v.size(3);
  return rows.as_strided({v.size(0), n, h, w}, {h * w * n, 1, w * n, n});
}

PyObject* separable_bf16(Args a) {  // value, dw_weight, dw_bias, pw_weight, pw_bias
  const Tensor *v = plain_tensor(a[0]), *w = plain_tensor(a[1]), *b = plain_tensor(a[2]), *pw = plain_tensor(a[3]), *pb = plain_tensor(a[4]);
  if (!depthwise_operands(v, w, b) || pw == nullptr || pb == nullptr || pw->dim() != 2 || pw->size(0) == 0 || pw->size(0) % 32 != 0 ||
      !matrix(*pw, kBF16, pw->size(0), v->size(1)) || !bias_ok(pb, pw->size(0))) {
    return nullptr;
  }
  const int64_t c = v->size(1), rows = v->size(0) * v->size(2) * v->size(3), n = pw->size(0);
  Call call;
  if (!rows_fit(rows) || !call.begin(*v) || !call.here(w, b, pw, pb)) return nullptr;
  Tensor hidden = call.empty({rows, c}, kBF16), out = call.empty({rows, n}, kBF16);
  call.launch("depthwise5x5_relu_pointwise", [&] {
    return abi.fim_dw5x5_bf16(v->data_ptr(), w->data_ptr(), static_cast<const float*>(b->data_ptr()), hidden.data_ptr(), v->size(0), v->size(2),
                              v->size(3), c, FIM_ACT_RELU, call.status, call.stream);
  });
  const FimConvGeometry g = pointwise(rows, c, n);
  FimConvEpilogue ep = {};
  ep.bias = pb->data_ptr(), ep.out_mode = FIM_OUT_BF16;
  call.launch("depthwise5x5_relu_pointwise", [&] {
    return abi.fim_bf16_conv2d(hidden.data_ptr(), pw->data_ptr(), &g, &ep, out.data_ptr(), call.status, call.stream);
  });
  return wrap(as_image(out, *v));
}

PyObject* separable_mx(Args a) {  // value, dw_weight, dw_bias, pw_weight, pw_scale_swizzled, pw_scale_u8, pw_bias
  const Tensor *v = plain_tensor(a[0]), *w = plain_tensor(a[1]), *b = plain_tensor(a[2]), *pw = plain_tensor(a[3]), *ps = plain_tensor(a[4]), *pb;
  if (!depthwise_operands(v, w, b) || pw == nullptr || ps == nullptr || !optional_tensor(a[6], &pb) || pw->dim() != 2 || pw->size(0) == 0 ||
      pw->size(0) % 32 != 0 || !matrix(*pw, kE4M3, pw->size(0), v->size(1)) || ps->element_size() != 1 || !dense16(*ps) ||
      ps->numel() != swizzled_bytes(pw->size(0), v->size(1) / 32) || !bias_ok(pb, pw->size(0))) {
    return nullptr;
  }
  const int64_t rows = v->size(0) * v->size(2) * v->size(3);
  Call call;
  if (!rows_fit(rows) || !call.begin(*v) || !call.here(w, b, pw, ps, pb)) return nullptr;
  Tensor q, scales;
  depthwise_mx_launch(*v, *w, *b, FIM_ACT_RELU, q, scales, kU8, call, "depthwise5x5_relu_pointwise_mxfp8");
  return wrap(as_image(mx_gemm(q, rows, nullptr, &scales, *pw, *ps, pb, call, "depthwise5x5_relu_pointwise_mxfp8"), *v));
}

PyObject* separable_int8(Args a) {  // value, dw_weight, dw_bias, pw_weight, pw_wscale, pw_bias, scale
  const Tensor *v = plain_tensor(a[0]), *w = plain_tensor(a[1]), *b = plain_tensor(a[2]), *pw = plain_tensor(a[3]), *ps = plain_tensor(a[4]),
               *pb, *s = plain_tensor(a[6]);
  if (!depthwise_operands(v, w, b) || pw == nullptr || ps == nullptr || s == nullptr || !optional_tensor(a[5], &pb) || pw->dim() != 2 ||
      pw->size(0) == 0 || pw->size(0) % 32 != 0 || !matrix(*pw, kI8, pw->size(0), v->size(1)) || !vector_of(*ps, kF32, pw->size(0)) ||
      !at16(*ps) || !bias_ok(pb, pw->size(0)) || !scalar_f32(*s)) {
    return nullptr;
  }
  const int64_t rows = v->size(0) * v->size(2) * v->size(3);
  Call call;
  if (!rows_fit(rows) || !call.begin(*v) || !call.here(w, b, pw, ps, pb, s)) return nullptr;
  Tensor q = depthwise_int8_launch(*v, *w, *b, *s, call, "depthwise5x5_relu_pointwise_int8");
  return wrap(as_image(int8_gemm(q, rows, *pw, s->data_ptr(), *ps, pb, nullptr, FIM_ACT_NONE, call, "depthwise5x5_relu_pointwise_int8"), *v));
}

// -- RoMaV2 refiner glue --

PyObject* refiner_input(Args a) {  // f_a, f_b, warp, emb_weight, emb_bias, scale_factor, radius, pair
  const Tensor *fa = plain_tensor(a[0]), *fb = plain_tensor(a[1]), *warp = plain_tensor(a[2]), *ew = plain_tensor(a[3]), *eb = plain_tensor(a[4]);
  int radius, pairs = 0;
  if (fa == nullptr || fb == nullptr || warp == nullptr || ew == nullptr || eb == nullptr || !integer(a[6], &radius) ||
      (a[7] != nullptr && !integer(a[7], &pairs))) {
    return nullptr;
  }
  // (a scale factor in a tensor is read back to the host by the general path)
  if (!(PyTuple_CheckExact(a[5]) || PyList_CheckExact(a[5])) || PySequence_Fast_GET_SIZE(a[5]) < 2) return nullptr;
  double sx, sy;
  if (!number(PySequence_Fast_GET_ITEM(a[5], 0), &sx) || !number(PySequence_Fast_GET_ITEM(a[5], 1), &sy)) return nullptr;
  if (fa->dim() != 4 || fa->numel() == 0 || fa->scalar_type() != kF32 || fb->scalar_type() != kF32 || warp->scalar_type() != kF32 ||
      !dense16(*fa) || !dense16(*fb) || fa->sizes() != fb->sizes() || !warp->is_contiguous()) {
    return nullptr;
  }
  const int64_t b = fa->size(0), h = fa->size(1), w = fa->size(2), p = fa->size(3), e = ew->dim() > 0 ? ew->size(0) : 0;
  if (p % 4 != 0 || p > 256 || radius > 3 || warp->numel() != b * h * w * 2 || e == 0 || !vector_of(*ew, kF32, 2 * e) || !vector_of(*eb, kF32, e) ||
      !(pairs == 0 || (pairs > 0 && b == 2 * static_cast<int64_t>(pairs)))) {
    return nullptr;
  }
  Call call;
  if (!call.begin(*fa) || !call.here(fb, warp, ew, eb)) return nullptr;
  const int64_t k = radius >= 0 ? (2 * radius + 1) * (2 * radius + 1) : 0, c = 2 * p + e + k;
  Tensor out = call.empty({b, h, w, c}, kBF16);
  call.launch("romav2_refiner_input", [&] {
    return abi.fim_romav2_refiner_input(static_cast<const float*>(fa->data_ptr()), static_cast<const float*>(fb->data_ptr()),
                                        static_cast<const float*>(warp->data_ptr()), static_cast<const float*>(ew->data_ptr()),
                                        static_cast<const float*>(eb->data_ptr()), static_cast<float>(sx), static_cast<float>(sy), out.data_ptr(),
                                        b, h, w, p, e, radius, pairs, call.stream);
  });
  return wrap(out.as_strided({b, c, h, w}, {h * w * c, 1, w * c, c}));
}

PyObject* refiner_heads(Args a) {  // z, weight, bias, prev_warp, prev_confidence, refine_init
  const Tensor *z = plain_tensor(a[0]), *w = plain_tensor(a[1]), *b = plain_tensor(a[2]), *pw = plain_tensor(a[3]), *pc = plain_tensor(a[4]);
  double init;
  if (z == nullptr || w == nullptr || b == nullptr || pw == nullptr || pc == nullptr || !number(a[5], &init) || init == 0.0) return nullptr;
  if (z->dim() != 4 || z->numel() == 0 || z->scalar_type() != kBF16 || !at16(*z) || !channels_last(*z)) return nullptr;
  const int64_t n = z->size(0), c = z->size(1), h = z->size(2), wd = z->size(3), rows = n * h * wd;
  if (c % 8 != 0 || c > 512 || w->dim() < 2 || w->size(0) != 6 || w->size(1) != c || !vector_of(*w, kF32, 6 * c) || !vector_of(*b, kF32, 6) ||
      !vector_of(*pw, kF32, 2 * rows) || pw->size(-1) != 2 || pc->dim() < 1 || (pc->size(-1) != 1 && pc->size(-1) != 4) ||
      !vector_of(*pc, kF32, rows * pc->size(-1))) {
    return nullptr;
  }
  Call call;
  if (!call.begin(*z) || !call.here(w, b, pw, pc)) return nullptr;
  Tensor warp = call.empty({n, h, wd, 2}, kF32), confidence = call.empty({n, h, wd, 4}, kF32);
  call.launch("romav2_refiner_heads", [&] {
    return abi.fim_romav2_refiner_heads(z->data_ptr(), static_cast<const float*>(w->data_ptr()), static_cast<const float*>(b->data_ptr()),
                                        static_cast<const float*>(pw->data_ptr()), static_cast<const float*>(pc->data_ptr()), pc->size(-1),
                                        static_cast<float*>(warp.data_ptr()), static_cast<float*>(confidence.data_ptr()), rows, c,
                                        static_cast<float>(1.0 / (init * wd)), static_cast<float>(1.0 / (init * h)), call.stream);
  });
  return pair(warp, confidence);
}

// ---- the module ------------------------------------------------------------------------------------------------------

template <PyObject* (*F)(Args), Signature* S>
PyObject* entry(PyObject*, PyObject* const* args, Py_ssize_t nargs, PyObject* kwnames) {
  PyObject* bound[20];
  try {
    PyObject* r = bind_arguments(*S, args, nargs, kwnames, bound) ? F(bound) : nullptr;
    return r != nullptr ? r : new_ref(Py_NotImplemented);
  } catch (const Failed&) {
    return nullptr;
  } catch (const c10::OutOfMemoryError& e) {
    PyObject* torch = PyImport_ImportModule("torch");
    PyObject* type = torch == nullptr ? nullptr : PyObject_GetAttrString(torch, "OutOfMemoryError");
    Py_XDECREF(torch);
    if (type != nullptr) PyErr_SetString(type, e.what_without_backtrace());
    Py_XDECREF(type);
    return nullptr;
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
}

#define GEOMETRY "kh", "kw", "sh", "sw", "ph", "pw", "dh", "dw"
// op name, function, required arguments, argument names
#define FIM_OPS(X)                                                                                                              \
  X(quantize_mxfp8, quantize_mxfp8, 2, "value", "scale_exponent")                                                               \
  X(quantize_int8, quantize_int8, 2, "value", "scale", "channel_scale")                                                         \
  X(quantize_mxfp8_dynamic, quantize_mxfp8_dynamic, 1, "value")                                                                 \
  X(gelu_quantize, gelu_quantize, 2, "value", "scale_exponent", "approximate", "input_bias")                                    \
  X(mxfp8_conv2d, mxfp8_conv2d, 13, "x", "channel_exponent", "weight", "weight_exponent", "bias", GEOMETRY, "relu", "residual", \
    "out_exponent")                                                                                                             \
  X(mxfp8_conv2d_fused, mxfp8_conv2d_fused, 13, "x", "act_scale", "weight", "weight_scales", "bias", GEOMETRY, "act", "residual", \
    "out_exponent", "dynamic_out", "out_fp32")                                                                                  \
  X(mxfp8_conv2d_bf16, mxfp8_conv2d_bf16, 5, "x", "act_exponent", "weight", "weight_scales", "bias", "act", "residual",         \
    "out_exponent", "dynamic_out", "out_fp32")                                                                                  \
  X(mxfp8_gelu_mlp_residual, mxfp8_gelu_mlp_residual, 9, "x", "x_scales", "w1", "w1_scales", "b1", "w2", "w2_scales", "b2", "residual") \
  X(int8_conv2d, int8_conv2d, 13, "x", "weight", "a_scale", "w_scale", "bias", GEOMETRY, "relu", "residual", "out_scale")       \
  X(int8_conv2d_maxpool, int8_conv2d_maxpool, 13, "x", "weight", "a_scale", "w_scale", "bias", GEOMETRY, "relu", "out_scale")   \
  X(mxfp8_linear, mxfp8_linear, 3, "activation", "bias", "weight")                                                              \
  X(mxfp8_gelu_mlp, mxfp8_gelu_mlp, 5, "x", "w1", "b1", "hidden_exponent", "w2")                                                \
  X(mxfp8_scaled_mm, mxfp8_scaled_mm, 4, "a", "b_t", "a_scale", "b_scale", "bias")                                              \
  X(int8_linear, int8_linear, 5, "a", "weight", "a_scale", "w_scale", "bias", "relu", "gelu", "residual")                       \
  X(depthwise5x5_act, depthwise_bf16, 3, "value", "weight", "bias", "act")                                                      \
  X(depthwise5x5_act_mxfp8, depthwise_act_mx, 3, "value", "weight", "bias", "act")                                              \
  X(depthwise5x5_relu_mxfp8, depthwise_relu_mx, 3, "value", "weight", "bias")                                                   \
  X(depthwise5x5_relu_int8, depthwise_relu_int8, 4, "value", "weight", "bias", "scale")                                         \
  X(depthwise5x5_relu_pointwise, separable_bf16, 5, "value", "dw_weight", "dw_bias", "pw_weight", "pw_bias")                    \
  X(depthwise5x5_relu_pointwise_mxfp8, separable_mx, 7, "value", "dw_weight", "dw_bias", "pw_weight", "pw_scale_swizzled",      \
    "pw_scale_u8", "pw_bias")                                                                                                   \
  X(depthwise5x5_relu_pointwise_int8, separable_int8, 7, "value", "dw_weight", "dw_bias", "pw_weight", "pw_wscale", "pw_bias", "scale") \
  X(romav2_refiner_input, refiner_input, 7, "f_a", "f_b", "warp", "emb_weight", "emb_bias", "scale_factor", "radius", "pair")   \
  X(romav2_refiner_heads, refiner_heads, 6, "z", "weight", "bias", "prev_warp", "prev_confidence", "refine_init")

template <typename... Names>
constexpr Signature signature(int required, Names... names) {
  return Signature{static_cast<int>(sizeof...(names)), required, {names...}, {}};
}
#define FIM_SIGNATURE(op, fn, required, ...) Signature signature_##op = signature(required, __VA_ARGS__);
FIM_OPS(FIM_SIGNATURE)
#undef FIM_SIGNATURE

// bind(library_path, status_word, check, check_status | None, swizzle_scales, QuantizedTensor, Int8Tensor)
PyObject* bind(PyObject*, PyObject* args) {
  const char* path;
  PyObject* objects[6];
  if (!PyArg_ParseTuple(args, "sOOOOOO", &path, &objects[0], &objects[1], &objects[2], &objects[3], &objects[4], &objects[5])) return nullptr;
  void* library = dlopen(path, RTLD_NOW | RTLD_LOCAL);  // the copy ctypes has loaded
  if (library == nullptr) {
    PyErr_SetString(PyExc_RuntimeError, dlerror());
    return nullptr;
  }
#define FIM_RESOLVE(name)                                                            \
  abi.name = reinterpret_cast<decltype(abi.name)>(dlsym(library, #name));            \
  if (abi.name == nullptr) {                                                         \
    PyErr_SetString(PyExc_RuntimeError, "missing entry point " #name);               \
    return nullptr;                                                                  \
  }
  FIM_ENTRIES(FIM_RESOLVE)
#undef FIM_RESOLVE
  PyObject** slots[6] = {&py_status_word, &py_check, &py_check_status, &py_swizzle, &py_quantized_tensor, &py_int8_tensor};
  for (int i = 0; i < 6; ++i) {
    Py_INCREF(objects[i]);
    Py_XSETREF(*slots[i], objects[i]);
  }
  Py_RETURN_NONE;
}

// swizzled_scales(exponent) -> tensor or None: the cache look-up for the Python implementations
PyObject* cached_swizzle(PyObject*, PyObject* o) {
  if (!THPVariable_Check(o)) Py_RETURN_NONE;
  try {
    Tensor t = swizzled_scales(THPVariable_Unpack(o));
    if (t.defined()) return wrap(std::move(t));
  } catch (const Failed&) {
    return nullptr;
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {
#define FIM_METHOD(op, fn, required, ...) \
  {#op, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(entry<fn, &signature_##op>)), METH_FASTCALL | METH_KEYWORDS, nullptr},
    FIM_OPS(FIM_METHOD)
#undef FIM_METHOD
    {"bind", bind, METH_VARARGS, "bind(library, status_word, check, check_status, swizzle_scales, QuantizedTensor, Int8Tensor)"},
    {"swizzled_scales", cached_swizzle, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fim_host", "Native host path of the flashim_b200 ops.", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__fim_host(void) {
#define FIM_INTERN(op, fn, required, ...) \
  for (int i = 0; i < signature_##op.count; ++i) signature_##op.interned[i] = PyUnicode_InternFromString(signature_##op.names[i]);
  FIM_OPS(FIM_INTERN)
#undef FIM_INTERN
  name_values = PyUnicode_InternFromString("values");
  name_scale = PyUnicode_InternFromString("scale");
  name_scale_exponent = PyUnicode_InternFromString("scale_exponent");
  name_logical_shape = PyUnicode_InternFromString("logical_shape");
  empty_tuple = PyTuple_New(0);
  return PyModule_Create(&module);
}
