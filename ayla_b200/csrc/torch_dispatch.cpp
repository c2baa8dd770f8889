// CUDA kernels of the torch ops for shapes that have been specialised: operand checks, the launch record of
// (device, shapes) and the call of the library, without entering Python.
//
// What bounds the smallest calls is the host.  A GEMM of 256 x 1024 x 1024 takes 5 us on the GPU; back-to-back
// calls of its op took 13.5 us through a Python kernel (boxed call into the interpreter, shape tuple, dict
// look-up, a ctypes call with seventeen arguments) and take 5.6 us through this one, whose own share is 4 us,
// the launch included.
//
// Everything that is not the plain repeated call stays in Python: an unseen shape, operands the op refuses, a
// launch reported as timed out by its status word, a stream other than the one the workspace belongs to, a capture of a
// launch with a workspace, another current device, a launch the library refuses.  Those go to the fallback with nothing
// done yet.
#include <algorithm>
#include <atomic>
#include <cstdint>
#include <memory>
#include <mutex>
#include <shared_mutex>
#include <unordered_map>
#include <vector>

#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/extension.h>
#include <torch/library.h>

namespace {

using GemmFn = int (*)(int, int, int, const void*, const void*, const void*, const void*, void*, int64_t, int64_t,
                       int64_t, int64_t, const void*, void*, size_t, uint32_t*, void*);
using SwigluFn = int (*)(int, const void*, const void*, const void*, void*, int64_t, int64_t, int64_t, const void*,
                         uint32_t*, void*);

// One specialised launch.  The pointers belong to the Python launcher, which `owner` keeps alive for good.
struct Launch {
  std::vector<int64_t> key;
  uintptr_t entry = 0;  // the library's function
  bool swiglu = false;
  int op = 0, dtype = 0, activation = 0;
  bool has_bias = false, gated = false;
  int64_t batch = 0, m = 0, n = 0, k = 0;
  const void* config = nullptr;
  const void* inside_config = nullptr;  // instead, if given, for results that start inside a 32-byte sector
  void* workspace = nullptr;
  size_t workspace_bytes = 0;
  uint32_t* status = nullptr;
  uintptr_t home_stream = 0;
  int device = 0;
  PyObject* owner = nullptr;
};

// Call `function` with the op's tensor and float arguments; its exception goes on to the op's caller.
void call_python(PyObject* function, c10::ArrayRef<c10::IValue> args) {
  py::gil_scoped_acquire gil;
  py::tuple values(args.size());
  for (size_t i = 0; i < args.size(); ++i) {
    PyObject* value =
        args[i].isTensor() ? THPVariable_Wrap(args[i].toTensor()) : PyFloat_FromDouble(args[i].toDouble());
    if (value == nullptr) throw python_error();
    PyTuple_SET_ITEM(values.ptr(), static_cast<Py_ssize_t>(i), value);
  }
  PyObject* result = PyObject_Call(function, values.ptr(), nullptr);
  if (result == nullptr) {
    python_error error;
    error.persist();
    throw error;
  }
  Py_DECREF(result);
}

// A captured launch gets a workspace of its graph's.
bool capturing(void* stream) {
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(static_cast<cudaStream_t>(stream), &status) != cudaSuccess) {
    (void)cudaGetLastError();
    return true;
  }
  return status != cudaStreamCaptureStatusNone;
}

constexpr size_t kMaxOperands = 5;
constexpr size_t kMaxKey = 1 + kMaxOperands * 4;  // the device, and of each operand its rank and up to three sizes

struct Key {
  int64_t values[kMaxKey];
  size_t size = 0;
  uint64_t hash = 1469598103934665603ull;
  void add(int64_t v) {
    values[size++] = v;
    hash = (hash ^ static_cast<uint64_t>(v)) * 1099511628211ull;
    hash ^= hash >> 29;
  }
};

class Dispatcher {
 public:
  Dispatcher(int64_t operands, py::object dtype, py::object fallback)
      : operands_(static_cast<size_t>(operands)),
        dtype_(reinterpret_cast<THPDtype*>(dtype.ptr())->scalar_type),
        fallback_(fallback.release().ptr()) {
    TORCH_CHECK(operands_ >= 1 && operands_ <= kMaxOperands, "unsupported operand count ", operands);
  }

  size_t operands() const { return operands_; }

  // The launch record of a call of the fast kind and the stream it goes to; null for any other.
  const Launch* ready(c10::ArrayRef<c10::IValue> args, void** stream) const {
    Key key;
    if (!key_of(args, &key)) return nullptr;
    const Launch* l = find(key);
    if (l == nullptr) return nullptr;
    if (*static_cast<volatile const uint32_t*>(l->status) != 0) return nullptr;
    if (c10::cuda::current_device() != l->device) return nullptr;
    *stream = c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(l->device)).stream();
    if (l->workspace_bytes != 0 && (reinterpret_cast<uintptr_t>(*stream) != l->home_stream || capturing(*stream))) return nullptr;
    return l;
  }

  // False: not a call of the fast kind; nothing has happened.
  bool launch(c10::ArrayRef<c10::IValue> args) const {
    void* stream = nullptr;
    const Launch* l = ready(args, &stream);
    if (l == nullptr) return false;
    const void* p[kMaxOperands];
    for (size_t i = 0; i + 1 < operands_; ++i) p[i] = args[i].toTensor().const_data_ptr();
    p[operands_ - 1] = args[operands_ - 1].toTensor().mutable_data_ptr();  // the last operand is written
    if (l->swiglu) {
      return reinterpret_cast<SwigluFn>(l->entry)(l->dtype, p[0], p[1], p[2], const_cast<void*>(p[3]), l->m, l->n,
                                                  l->k, l->config, l->status, stream) == 0;
    }
    const void* const* next = p;
    const void* bias = l->has_bias ? *next++ : nullptr;
    const void* a = *next++;
    const void* bt = *next++;
    const void* mul = l->gated ? *next++ : nullptr;
    const bool inside = l->inside_config != nullptr && (reinterpret_cast<uintptr_t>(*next) & 31) != 0;
    return reinterpret_cast<GemmFn>(l->entry)(l->op, l->dtype, l->activation, bias, a, bt, mul, const_cast<void*>(*next),
                                              l->batch, l->m, l->n, l->k, inside ? l->inside_config : l->config,
                                              l->workspace, l->workspace_bytes, l->status, stream) == 0;
  }

  void fallback(c10::ArrayRef<c10::IValue> args) const { call_python(fallback_, args); }

  // Remember the launch of these operands' shapes (once; the first one stays).
  void insert(const std::vector<at::Tensor>& tensors, py::object owner, const py::dict& fields) {
    std::vector<c10::IValue> args(tensors.begin(), tensors.end());
    Key key;
    if (args.size() != operands_ || !key_of(args, &key)) return;
    auto l = std::make_unique<Launch>();
    l->key.assign(key.values, key.values + key.size);
    l->entry = fields["entry"].cast<uintptr_t>();
    l->swiglu = fields["swiglu"].cast<bool>();
    l->op = fields["op"].cast<int>();
    l->dtype = fields["dtype"].cast<int>();
    l->activation = fields["activation"].cast<int>();
    l->has_bias = fields["has_bias"].cast<bool>();
    l->gated = fields["gated"].cast<bool>();
    l->batch = fields["batch"].cast<int64_t>();
    l->m = fields["m"].cast<int64_t>();
    l->n = fields["n"].cast<int64_t>();
    l->k = fields["k"].cast<int64_t>();
    l->config = reinterpret_cast<const void*>(fields["config"].cast<uintptr_t>());
    if (fields.contains("inside_config")) l->inside_config = reinterpret_cast<const void*>(fields["inside_config"].cast<uintptr_t>());
    l->workspace = reinterpret_cast<void*>(fields["workspace"].cast<uintptr_t>());
    l->workspace_bytes = fields["workspace_bytes"].cast<size_t>();
    l->status = reinterpret_cast<uint32_t*>(fields["status"].cast<uintptr_t>());
    l->home_stream = fields["home_stream"].cast<uintptr_t>();
    l->device = fields["device"].cast<int>();
    if (l->device != key.values[0]) return;
    const size_t expected = l->swiglu ? 4 : 3 + (l->has_bias ? 1 : 0) + (l->gated ? 1 : 0);
    TORCH_CHECK(expected == operands_, "a launch of ", expected, " operands for an op of ", operands_);
    std::unique_lock<std::shared_mutex> lock(mutex_);
    if (find_locked(key) != nullptr) return;
    l->owner = owner.release().ptr();
    launches_.emplace(key.hash, std::move(l));
  }

 private:
  // The operand checks of the Python dispatcher; a call that fails one is left to it, which raises.
  bool key_of(c10::ArrayRef<c10::IValue> args, Key* key) const {
    for (size_t i = 0; i < operands_; ++i) {
      if (!args[i].isTensor()) return false;
      const at::Tensor& t = args[i].toTensor();
      if (!t.defined() || !t.is_cuda() || t.scalar_type() != dtype_ || t.dim() > 3 || !t.is_contiguous()) return false;
      if (i == 0) {
        key->add(t.device().index());
      } else if (t.device().index() != key->values[0]) {
        return false;
      }
      key->add(t.dim());
      for (const int64_t s : t.sizes()) key->add(s);
    }
    return true;
  }

  const Launch* find_locked(const Key& key) const {
    const auto range = launches_.equal_range(key.hash);
    for (auto it = range.first; it != range.second; ++it) {
      const Launch& l = *it->second;
      if (l.key.size() == key.size && std::equal(l.key.begin(), l.key.end(), key.values)) return &l;
    }
    return nullptr;
  }
  const Launch* find(const Key& key) const {
    std::shared_lock<std::shared_mutex> lock(mutex_);  // launches are never removed: the pointer stays good
    return find_locked(key);
  }

  const size_t operands_;
  const at::ScalarType dtype_;
  PyObject* const fallback_;  // kept for good, as the op is
  mutable std::shared_mutex mutex_;
  std::unordered_multimap<uint64_t, std::unique_ptr<Launch>> launches_;
};

struct BoxedKernel final : c10::OperatorKernel {
  explicit BoxedKernel(const Dispatcher* dispatcher) : dispatcher_(dispatcher) {}
  void operator()(const c10::OperatorHandle&, c10::DispatchKeySet, torch::jit::Stack* stack) {
    const size_t n = dispatcher_->operands();
    const c10::ArrayRef<c10::IValue> args = torch::jit::last(*stack, n);
    if (!dispatcher_->launch(args)) dispatcher_->fallback(args);
    torch::jit::drop(*stack, n);
  }
  const Dispatcher* dispatcher_;
};

using RmsFactorsFn = int (*)(int, const void*, void*, int64_t, int64_t, float, void*);

// (x, eps, factors) -> (): the row factors of an RMS norm.
struct RmsFactorsKernel final : c10::OperatorKernel {
  RmsFactorsKernel(uintptr_t entry, int dtype_code, at::ScalarType dtype, PyObject* fallback)
      : entry_(reinterpret_cast<RmsFactorsFn>(entry)), dtype_code_(dtype_code), dtype_(dtype), fallback_(fallback) {}

  void operator()(const c10::OperatorHandle&, c10::DispatchKeySet, torch::jit::Stack* stack) {
    const c10::ArrayRef<c10::IValue> args = torch::jit::last(*stack, 3);
    if (!launch(args)) {
      call_python(fallback_, args);
      const int device = args[0].toTensor().device().index();
      if (device >= 0 && device < 64) ready_.fetch_or(uint64_t{1} << device);  // the library is set up there
    }
    torch::jit::drop(*stack, 3);
  }

 private:
  bool launch(c10::ArrayRef<c10::IValue> args) const {
    const at::Tensor& x = args[0].toTensor();
    const at::Tensor& factors = args[2].toTensor();
    if (!x.is_cuda() || x.dim() != 2 || x.scalar_type() != dtype_ || factors.scalar_type() != dtype_ ||
        !x.is_contiguous() || !factors.is_contiguous() || factors.device() != x.device() ||
        factors.numel() != x.size(0)) {
      return false;
    }
    const int device = x.device().index();
    if (device >= 64 || (ready_.load() >> device & 1) == 0 || c10::cuda::current_device() != device) return false;
    void* stream = c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(device)).stream();
    return entry_(dtype_code_, x.const_data_ptr(), factors.mutable_data_ptr(), x.size(0), x.size(1),
                  static_cast<float>(args[1].toDouble()), stream) == 0;
  }

  const RmsFactorsFn entry_;
  const int dtype_code_;
  const at::ScalarType dtype_;
  PyObject* const fallback_;
  std::atomic<uint64_t> ready_{0};
};

// (x, eps, weight, out) -> (): the row factors and the projection that takes them, whose launch record is that of the
// projection's own op on (x, weight, factors, out).  One op instead of two and an allocation from Python: what bounds the
// small calls is the host (us per call back to back, two ops -> one: 20x1216x1408 11.0 -> 7.9, 45x2112x1088 11.1 -> 8.2,
// 16x4096x4096 11.0 -> 10.5; replayed from a graph 6.8, 7.5 and 9.6 either way).
struct RmsLinearKernel final : c10::OperatorKernel {
  RmsLinearKernel(uintptr_t row_factors, const Dispatcher* projection, PyObject* fallback)
      : row_factors_(reinterpret_cast<RmsFactorsFn>(row_factors)), projection_(projection), fallback_(fallback) {}

  void operator()(const c10::OperatorHandle&, c10::DispatchKeySet, torch::jit::Stack* stack) {
    const c10::ArrayRef<c10::IValue> args = torch::jit::last(*stack, 4);
    if (!launch(args)) call_python(fallback_, args);
    torch::jit::drop(*stack, 4);
  }

 private:
  bool launch(c10::ArrayRef<c10::IValue> args) const {
    const at::Tensor& x = args[0].toTensor();
    if (!x.is_cuda() || x.dim() != 2) return false;
    const at::Tensor factors = at::detail::empty_cuda({x.size(0), 1}, x.scalar_type(), x.device(), std::nullopt);
    const c10::IValue operands[4] = {args[0], args[2], factors, args[3]};
    void* stream = nullptr;
    const Launch* l = projection_->ready(operands, &stream);
    if (l == nullptr) return false;
    if (row_factors_(l->dtype, x.const_data_ptr(), factors.mutable_data_ptr(), l->m, l->k,
                     static_cast<float>(args[1].toDouble()), stream) != 0) {
      return false;
    }
    return reinterpret_cast<GemmFn>(l->entry)(l->op, l->dtype, l->activation, nullptr, x.const_data_ptr(),
                                              args[2].toTensor().const_data_ptr(), factors.const_data_ptr(),
                                              args[3].toTensor().mutable_data_ptr(), l->batch, l->m, l->n, l->k, l->config,
                                              l->workspace, l->workspace_bytes, l->status, stream) == 0;
  }

  const RmsFactorsFn row_factors_;
  const Dispatcher* const projection_;  // both are kept for good, as the ops are
  PyObject* const fallback_;
};

void register_kernel(const std::string& ns, const std::string& name, torch::CppFunction&& kernel) {
  // Kept for good: dropping the library would take the kernel away.
  auto* library = new torch::Library(torch::Library::IMPL, ns, c10::DispatchKey::CUDA, __FILE__, __LINE__);
  library->impl(name.c_str(), std::move(kernel));
}

void register_rms_factors(const std::string& ns, const std::string& name, uintptr_t entry, int dtype_code,
                          py::object dtype, py::object fallback) {
  register_kernel(ns, name,
                  torch::CppFunction::makeFromBoxedFunctor(std::make_unique<RmsFactorsKernel>(
                      entry, dtype_code, reinterpret_cast<THPDtype*>(dtype.ptr())->scalar_type,
                      fallback.release().ptr())));
}

void register_rms_linear(const std::string& ns, const std::string& name, uintptr_t row_factors,
                         const Dispatcher* projection, py::object fallback) {
  TORCH_CHECK(projection->operands() == 4, "the projection's op takes x, weight, factors and out");
  register_kernel(ns, name,
                  torch::CppFunction::makeFromBoxedFunctor(
                      std::make_unique<RmsLinearKernel>(row_factors, projection, fallback.release().ptr())));
}

// Register the CUDA kernel of `name` (no results) and return its dispatcher, which lives as long as the process.
Dispatcher* register_op(const std::string& ns, const std::string& name, int64_t operands, py::object dtype,
                        py::object fallback) {
  auto* dispatcher = new Dispatcher(operands, std::move(dtype), std::move(fallback));
  register_kernel(ns, name, torch::CppFunction::makeFromBoxedFunctor(std::make_unique<BoxedKernel>(dispatcher)));
  return dispatcher;
}

}  // namespace

PYBIND11_MODULE(_torch_dispatch, m) {
  py::class_<Dispatcher, std::unique_ptr<Dispatcher, py::nodelete>>(m, "Dispatcher").def("insert", &Dispatcher::insert);
  m.def("register_op", &register_op, py::return_value_policy::reference);
  m.def("register_rms_factors", &register_rms_factors);
  m.def("register_rms_linear", &register_rms_linear);
}
