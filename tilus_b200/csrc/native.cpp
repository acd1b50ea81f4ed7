// Host path of QuantizedLinear as a CPython extension (tilus_b200._native): argument checks, output and
// workspace tensors, stream lookup and the call into libb200q, in one native function per call.
//
// A decode call occupies the GPU for 5..15 us, so a program that calls its layers one by one is bound by
// whatever the host spends per call.  The same steps written in Python around ctypes took 14 us (measured
// on M = 1, K = N = 8192, where the kernel takes 10.6 us); here they take about a third of that.
// The functions are entered through METH_FASTCALL and touch tensors through the C++ API; the library is
// called through addresses handed over by `bind`, so that whichever build _lib.load() opened is used.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAException.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/object_ptr.h>

#include <algorithm>
#include <memory>
#include <mutex>
#include <utility>
#include <vector>

#include "../../include/b200q.h"

namespace {

typedef decltype(&b200q_gemm) GemmFn;
typedef decltype(&b200q_gemm_host) GemmHostFn;
typedef decltype(&b200q_gemm_swiglu_cast) GemmCastFn;
typedef decltype(&b200q_workspace_bytes) WorkspaceFn;

GemmFn g_gemm = nullptr;
GemmHostFn g_gemm_host = nullptr;
GemmCastFn g_gemm_cast = nullptr;
WorkspaceFn g_workspace_bytes = nullptr;
PyObject* g_raise_status = nullptr;       // _lib.check
PyObject* g_raise_unsupported = nullptr;  // callable(M, N, K)

// what a layer's calls have in common: (dtype code, zero point, group size, in_features, out_features)
struct Layer { int code, zero_point, group, K, N; };

bool parse_layer(PyObject* t, Layer* l) {
  if (!PyTuple_CheckExact(t) || PyTuple_GET_SIZE(t) != 5) {
    PyErr_SetString(PyExc_TypeError, "layer constants are a tuple of five integers");
    return false;
  }
  int* dst[5] = {&l->code, &l->zero_point, &l->group, &l->K, &l->N};
  for (int i = 0; i < 5; ++i) *dst[i] = (int)PyLong_AsLong(PyTuple_GET_ITEM(t, i));
  return !PyErr_Occurred();
}

const at::Tensor* as_tensor(PyObject* o, const char* what) {
  if (!THPVariable_Check(o)) {
    PyErr_Format(PyExc_TypeError, "%s must be a torch.Tensor", what);
    return nullptr;
  }
  return &THPVariable_Unpack(o);
}

// activation dtype tag of the C ABI, -1 when it is neither float16 nor bfloat16
int act_code(at::ScalarType t) { return t == at::kHalf ? 0 : (t == at::kBFloat16 ? 1 : -1); }

bool check_weights(const at::Tensor& qw, const at::Tensor& scales, const c10::Device& dev) {
  if (qw.device() == dev && scales.device() == dev) return true;
  PyErr_SetString(PyExc_ValueError, "the layer's weights and the activations must be on one CUDA device");
  return false;
}

// Per (device, stream) buffers, grown on demand.  The kernels leave a workspace zeroed, so it is cleared
// only when it is (re)allocated; one stream's calls run one after the other, so they share one.  The
// staging pair holds the activations and results of host calls: decode batches (whose kernel fetches
// its own activations, so that consecutive calls overlap) have a pair of their own, so that a larger
// batch in between does not make the next decode call wait for it.
// A buffer that has become too small is replaced by one of at least twice its size, and kept: a captured graph may
// name its address, and b200q_gemm_host remembers staging buffers by theirs.  What is kept is less than what replaced it.
struct StreamBuffers {
  int device;
  cudaStream_t stream;
  at::Tensor workspace;
  at::Tensor staging[2][2];
  std::vector<at::Tensor> superseded;
  std::mutex host_call;  // a host call is several operations on one staging pair: one thread's at a time
};
std::mutex g_mutex;
std::vector<std::unique_ptr<StreamBuffers>>& pool() {
  static auto* p = new std::vector<std::unique_ptr<StreamBuffers>>();  // outlives the interpreter's teardown
  return *p;
}
StreamBuffers& buffers_of(int device, cudaStream_t stream) {  // g_mutex held; the entry stays where it is
  for (const auto& b : pool())
    if (b->device == device && b->stream == stream) return *b;
  pool().push_back(std::make_unique<StreamBuffers>());
  pool().back()->device = device;
  pool().back()->stream = stream;
  return *pool().back();
}
// Device memory for b's stream, which is b's device's current stream, zeroed if asked for.  While the stream is being
// captured the allocation and the zeroing are not part of the capture: memory of the graph's own pool would be cleared by that
// graph's replays only, and not before the first of them.  They take place on a stream of their own then, at once.
at::Tensor allocate(const StreamBuffers& b, int64_t size, bool zero) {
  const c10::Device dev(at::kCUDA, (c10::DeviceIndex)b.device);
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(b.stream, &capture) != cudaSuccess) (void)cudaGetLastError();  // (the launch will say what is wrong)
  if (capture == cudaStreamCaptureStatusNone) {
    at::Tensor t = at::detail::empty_cuda({size}, at::kByte, dev, std::nullopt);
    if (zero) C10_CUDA_CHECK(cudaMemsetAsync(t.mutable_data_ptr(), 0, (size_t)size, b.stream));
    return t;
  }
  const c10::cuda::CUDAStreamCaptureModeGuard relaxed(cudaStreamCaptureModeRelaxed);
  static auto* sides = new std::vector<std::pair<int, cudaStream_t>>();  // per device; g_mutex held
  cudaStream_t side = nullptr;
  for (const auto& s : *sides)
    if (s.first == b.device) side = s.second;
  if (side == nullptr) {
    C10_CUDA_CHECK(cudaStreamCreateWithFlags(&side, cudaStreamNonBlocking));
    sides->emplace_back(b.device, side);
  }
  const c10::cuda::CUDAStreamGuard guard(c10::cuda::getStreamFromExternal(side, dev.index()));
  at::Tensor t = at::detail::empty_cuda({size}, at::kByte, dev, std::nullopt);
  if (zero) C10_CUDA_CHECK(cudaMemsetAsync(t.mutable_data_ptr(), 0, (size_t)size, side));
  C10_CUDA_CHECK(cudaStreamSynchronize(side));
  return t;
}
// One of b's buffers with room for `need` bytes; g_mutex held, b's device current and b's stream its current stream.
at::Tensor with_room(StreamBuffers& b, at::Tensor& buffer, size_t need, bool zero) {
  const size_t have = buffer.defined() ? (size_t)buffer.numel() : 0;
  if (have < need || !buffer.defined()) {
    at::Tensor larger = allocate(b, (int64_t)std::max(need, 2 * have), zero);
    if (buffer.defined()) b.superseded.push_back(std::move(buffer));
    buffer = std::move(larger);
  }
  return buffer;
}
// `device` is current and `stream` its current stream
at::Tensor workspace_of(int device, cudaStream_t stream, size_t need) {
  std::lock_guard<std::mutex> lock(g_mutex);
  StreamBuffers& b = buffers_of(device, stream);
  return with_room(b, b.workspace, std::max(need, (size_t)1 << 20), true);
}

// Library calls run without the interpreter lock (as through ctypes): a launch into a full queue blocks, and a copy to
// pageable memory waits for everything queued before it.
class NoGil {
 public:
  NoGil() : state_(PyEval_SaveThread()) {}
  ~NoGil() { PyEval_RestoreThread(state_); }
  NoGil(const NoGil&) = delete;
  NoGil& operator=(const NoGil&) = delete;

 private:
  PyThreadState* state_;
};

PyObject* raise_status(int st) {
  PyObject* r = PyObject_CallFunction(g_raise_status, "i", st);
  Py_XDECREF(r);
  if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "b200q call failed");
  return nullptr;
}
PyObject* raise_unsupported(int M, int N, int K) {
  PyObject* r = PyObject_CallFunction(g_raise_unsupported, "iii", M, N, K);
  Py_XDECREF(r);
  if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "no kernel for this shape");
  return nullptr;
}

// activations as rows of K values: the tensor itself, or reshaped to two dimensions
bool as_rows(const at::Tensor& x, int K, at::Tensor* rows) {
  if (x.dim() == 0 || x.size(-1) != K) {
    PyErr_Format(PyExc_ValueError, "expected %d input features, got %lld", K,
                 x.dim() ? (long long)x.size(-1) : 1LL);
    return false;
  }
  *rows = x.dim() == 2 ? x : x.reshape({-1, (int64_t)K});
  return true;
}

// linear(x, quantized_weight, scales, layer) -> [..., out_features]
PyObject* linear(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 4) { PyErr_SetString(PyExc_TypeError, "linear takes 4 arguments"); return nullptr; }
  const at::Tensor* x = as_tensor(args[0], "activations");
  const at::Tensor* qw = as_tensor(args[1], "quantized_weight");
  const at::Tensor* scales = as_tensor(args[2], "scales");
  Layer l;
  if (!x || !qw || !scales || !parse_layer(args[3], &l)) return nullptr;
  at::Tensor rows;
  if (!as_rows(*x, l.K, &rows)) return nullptr;
  if (!rows.is_cuda()) {
    PyErr_SetString(PyExc_ValueError, "QuantizedLinear needs CUDA tensors (there is no CPU path)");
    return nullptr;
  }
  const at::ScalarType dtype = scales->scalar_type();
  const int act = act_code(dtype);
  if (rows.scalar_type() != dtype || act < 0 || rows.stride(1) != 1) {
    PyErr_Format(PyExc_TypeError, "activations must be %s with unit inner stride", c10::toString(dtype));
    return nullptr;
  }
  const c10::Device dev = rows.device();
  if (!check_weights(*qw, *scales, dev)) return nullptr;
  const int M = (int)rows.size(0);
  const c10::cuda::OptionalCUDAGuard guard(dev);
  at::Tensor out = at::detail::empty_cuda({(int64_t)M, (int64_t)l.N}, dtype, dev, std::nullopt);
  if (M > 0) {
    const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
    const size_t need = g_workspace_bytes(M, l.N, l.K, l.code, l.zero_point, l.group);
    if (need == 0) return raise_unsupported(M, l.N, l.K);
    const at::Tensor ws = workspace_of(dev.index(), stream, need);
    const void *a = rows.const_data_ptr(), *bq = qw->const_data_ptr(), *sc = scales->const_data_ptr();
    void *c = out.mutable_data_ptr(), *w = ws.mutable_data_ptr();
    const int lda = (int)rows.stride(0);
    int st;
    {
      const NoGil unlocked;
      st = g_gemm(a, lda, bq, sc, c, l.N, M, l.N, l.K, l.code, l.zero_point, l.group, act, w, (size_t)ws.numel(), stream);
    }
    if (st != 0) return raise_status(st);
  }
  if (x->dim() != 2) {
    std::vector<int64_t> shape(x->sizes().begin(), x->sizes().end());
    shape.back() = l.N;
    out = out.reshape(shape);
  }
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// linear_host(x_host, out_host, quantized_weight, scales, layer) -> out_host
PyObject* linear_host(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 5) { PyErr_SetString(PyExc_TypeError, "linear_host takes 5 arguments"); return nullptr; }
  const at::Tensor* x = as_tensor(args[0], "x_host");
  const at::Tensor* out = as_tensor(args[1], "out_host");
  const at::Tensor* qw = as_tensor(args[2], "quantized_weight");
  const at::Tensor* scales = as_tensor(args[3], "scales");
  Layer l;
  if (!x || !out || !qw || !scales || !parse_layer(args[4], &l)) return nullptr;
  if (x->is_cuda() || out->is_cuda()) {
    PyErr_SetString(PyExc_ValueError, "forward_host takes host tensors (use forward for device tensors)");
    return nullptr;
  }
  const at::ScalarType dtype = scales->scalar_type();
  const int act = act_code(dtype);
  if (x->scalar_type() != dtype || out->scalar_type() != dtype || act < 0) {
    PyErr_Format(PyExc_TypeError, "activations and result must be %s", c10::toString(dtype));
    return nullptr;
  }
  if (x->dim() != 2 || x->stride(1) != 1 || x->size(1) != l.K) {
    PyErr_Format(PyExc_ValueError, "x_host must be [M, %d] with unit inner stride", l.K);
    return nullptr;
  }
  const int M = (int)x->size(0);
  if (out->dim() != 2 || out->stride(1) != 1 || out->size(0) != M || out->size(1) != l.N) {
    PyErr_Format(PyExc_ValueError, "out_host must be [%d, %d] with unit inner stride", M, l.N);
    return nullptr;
  }
  const c10::Device dev = qw->device();
  if (!dev.is_cuda()) {
    PyErr_SetString(PyExc_ValueError, "QuantizedLinear needs its weights on a CUDA device (there is no CPU path)");
    return nullptr;
  }
  if (!check_weights(*qw, *scales, dev)) return nullptr;
  if (M > 0) {
    const c10::cuda::OptionalCUDAGuard guard(dev);
    const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
    const size_t need = g_workspace_bytes(M, l.N, l.K, l.code, l.zero_point, l.group);
    if (need == 0) return raise_unsupported(M, l.N, l.K);
    const at::Tensor ws = workspace_of(dev.index(), stream, need);
    at::Tensor sa, sc;
    StreamBuffers* buffers;
    {
      std::lock_guard<std::mutex> lock(g_mutex);
      buffers = &buffers_of(dev.index(), stream);
      at::Tensor* s = buffers->staging[M <= 16 ? 1 : 0];
      sa = with_room(*buffers, s[0], (size_t)M * l.K * 2, false);
      sc = with_room(*buffers, s[1], (size_t)M * l.N * 2, false);
    }
    const void *a = x->const_data_ptr(), *bq = qw->const_data_ptr(), *scp = scales->const_data_ptr();
    void *c = out->mutable_data_ptr(), *a_stage = sa.mutable_data_ptr(), *c_stage = sc.mutable_data_ptr();
    void* w = ws.mutable_data_ptr();
    const int lda = (int)x->stride(0), ldc = (int)out->stride(0);
    int st;
    {
      const NoGil unlocked;
      std::lock_guard<std::mutex> lock(buffers->host_call);
      st = g_gemm_host(a, lda, bq, scp, c, ldc, M, l.N, l.K, l.code, l.zero_point, l.group, act, a_stage, c_stage, w,
                       (size_t)ws.numel(), stream);
    }
    if (st != 0) return raise_status(st);
  }
  Py_INCREF(args[1]);
  return args[1];
  END_HANDLE_TH_ERRORS
}

// gate_up_cast(x, quantized_weight, scales, layer, channels per scale, clamp value or None)
//   -> (out e4m3 [M, N / 2], out_sf float32 [M, N / 2 / channels], gate_up [M, N])
PyObject* gate_up_cast(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 6) { PyErr_SetString(PyExc_TypeError, "gate_up_cast takes 6 arguments"); return nullptr; }
  const at::Tensor* x = as_tensor(args[0], "activations");
  const at::Tensor* qw = as_tensor(args[1], "quantized_weight");
  const at::Tensor* scales = as_tensor(args[2], "scales");
  Layer l;
  if (!x || !qw || !scales || !parse_layer(args[3], &l)) return nullptr;
  const long channels = PyLong_AsLong(args[4]);
  const bool clamp = args[5] != Py_None;
  const double clamp_value = clamp ? PyFloat_AsDouble(args[5]) : 0.0;
  if (PyErr_Occurred()) return nullptr;
  if (channels < 1) { PyErr_SetString(PyExc_ValueError, "channels per scale must be positive"); return nullptr; }
  // rows of K values: any shape whose elements make them up ([tokens, heads, head size] of an attention output), or the
  // first K columns of a wider matrix
  at::Tensor rows;
  if (x->dim() == 2 && x->size(1) >= l.K) {
    rows = *x;
  } else if (x->dim() != 2 && x->numel() % l.K == 0) {
    rows = x->reshape({-1, (int64_t)l.K});
  } else {
    PyErr_Format(PyExc_ValueError, "expected rows of %d input features", l.K);
    return nullptr;
  }
  const at::ScalarType dtype = scales->scalar_type();
  const int act = act_code(dtype);
  if (!rows.is_cuda() || rows.scalar_type() != dtype || act < 0 || rows.stride(1) != 1) {
    PyErr_Format(PyExc_ValueError, "activations must be CUDA %s with unit inner stride", c10::toString(dtype));
    return nullptr;
  }
  const c10::Device dev = rows.device();
  if (!check_weights(*qw, *scales, dev)) return nullptr;
  const int M = (int)rows.size(0), H = l.N / 2;
  const c10::cuda::OptionalCUDAGuard guard(dev);
  at::Tensor gate_up = at::detail::empty_cuda({M, l.N}, dtype, dev, std::nullopt);
  at::Tensor out = at::detail::empty_cuda({M, H}, at::kFloat8_e4m3fn, dev, std::nullopt);
  at::Tensor sf = at::detail::empty_cuda({M, H / channels}, at::kFloat, dev, std::nullopt);
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
  const size_t need = g_workspace_bytes(M, l.N, l.K, l.code, l.zero_point, l.group);
  if (need == 0) return raise_unsupported(M, l.N, l.K);
  const at::Tensor ws = workspace_of(dev.index(), stream, need);
  const void *a = rows.const_data_ptr(), *bq = qw->const_data_ptr(), *sc = scales->const_data_ptr();
  void *g = gate_up.mutable_data_ptr(), *o = out.mutable_data_ptr(), *f = sf.mutable_data_ptr(), *w = ws.mutable_data_ptr();
  const int lda = (int)rows.stride(0);
  int st;
  {
    const NoGil unlocked;
    st = g_gemm_cast(a, lda, bq, sc, g, l.N, o, H, static_cast<float*>(f), M, l.N, l.K, l.code, l.zero_point, l.group, act,
                     (int)channels, clamp ? 1 : 0, (float)clamp_value, w, (size_t)ws.numel(), stream);
  }
  if (st != 0) return raise_status(st);
  return PyTuple_Pack(3, THPObjectPtr(THPVariable_Wrap(std::move(out))).get(),
                      THPObjectPtr(THPVariable_Wrap(std::move(sf))).get(),
                      THPObjectPtr(THPVariable_Wrap(std::move(gate_up))).get());
  END_HANDLE_TH_ERRORS
}

// workspace(device index, bytes) -> the zeroed workspace of the device's current stream
PyObject* workspace(PyObject*, PyObject* args) {
  HANDLE_TH_ERRORS
  int device;
  Py_ssize_t bytes;
  if (!PyArg_ParseTuple(args, "in", &device, &bytes)) return nullptr;
  const c10::cuda::CUDAGuard guard((c10::DeviceIndex)device);
  return THPVariable_Wrap(
      workspace_of(device, c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)device).stream(), (size_t)bytes));
  END_HANDLE_TH_ERRORS
}

// bind(gemm, gemm_host, gemm_swiglu_cast, workspace_bytes, raise_status, raise_unsupported): addresses in
// libb200q and the Python callables that raise for a status
PyObject* bind(PyObject*, PyObject* args) {
  unsigned long long gemm, host, cast, ws;
  PyObject *status, *unsupported;
  if (!PyArg_ParseTuple(args, "KKKKOO", &gemm, &host, &cast, &ws, &status, &unsupported)) return nullptr;
  g_gemm = reinterpret_cast<GemmFn>(gemm);
  g_gemm_host = reinterpret_cast<GemmHostFn>(host);
  g_gemm_cast = reinterpret_cast<GemmCastFn>(cast);
  g_workspace_bytes = reinterpret_cast<WorkspaceFn>(ws);
  Py_INCREF(status);
  Py_INCREF(unsupported);
  Py_XSETREF(g_raise_status, status);
  Py_XSETREF(g_raise_unsupported, unsupported);
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"linear", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(linear)), METH_FASTCALL, nullptr},
    {"linear_host", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(linear_host)), METH_FASTCALL, nullptr},
    {"gate_up_cast", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(gate_up_cast)), METH_FASTCALL, nullptr},
    {"workspace", workspace, METH_VARARGS, nullptr},
    {"bind", bind, METH_VARARGS, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

extern "C" __attribute__((visibility("default"))) PyObject* PyInit__native() { return PyModule_Create(&module); }
