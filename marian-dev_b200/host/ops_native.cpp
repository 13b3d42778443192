// The per-call host path of ops.py / packed8.py in native code.
//
// A small affine takes a few microseconds of device time; argument checks, allocations, views and the ctypes call of the
// Python route took 40 us of host time per affine (measured, 4 x 256 x 1536), so the GPU idled between calls.  Here one call
// checks its arguments, takes output and scratch from torch's caching allocator and calls the C ABI: about 5 us.
//
// Every function returns None for arguments it does not take (another device, type or layout; wrong sizes; tensors without memory
// of their own, such as fake or vmapped ones): the caller then goes through the general Python route, which handles or rejects
// them.  A non-zero library status is returned as an int.  C++ exceptions (an allocation that fails) become torch's Python ones.
#include <Python.h>
#include <dlfcn.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/object_ptr.h>
#include <torch/version.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <vector>

#include "../../include/marian_i8.h"
#include "../../include/marian_packed8.h"

namespace {

// Entry points of the library the Python binding loaded (resolved by init(), so that MARIAN_I8_LIBRARY selects one for both).
struct Lib {
  decltype(&mi8_affine_f32) affine = nullptr;
  decltype(&mi8_prepare_b_f32) prepare_b = nullptr;
  decltype(&mi8p_packed_bytes) packed_bytes = nullptr;
  decltype(&mi8p_prepare_b_f32) p8_prepare_b = nullptr;
  decltype(&mi8p_unpack_b) p8_unpack_b = nullptr;
  decltype(&mi8p_scratch_bytes) p8_scratch_bytes = nullptr;
  decltype(&mi8p_gemm_int8_packed) p8_gemm = nullptr;
};
Lib g_lib;
PyObject* g_default_workspace = nullptr;   // ops.default_workspace, called once per (device, stream)

// The workspaces of default_workspace(), which keeps them for the life of the process; guarded by the GIL.
struct WsEntry {
  int device;
  cudaStream_t stream;
  void* ptr;
  size_t bytes;
};
std::vector<WsEntry> g_ws;

bool workspace(const at::Tensor& like, PyObject* like_obj, cudaStream_t stream, void** ptr, size_t* bytes) {
  const int dev = like.device().index();
  for(const WsEntry& e : g_ws)
    if(e.device == dev && e.stream == stream) {
      *ptr = e.ptr;
      *bytes = e.bytes;
      return true;
    }
  PyObject* device = PyObject_GetAttrString(like_obj, "device");
  if(device == nullptr)
    return false;
  PyObject* ws = PyObject_CallOneArg(g_default_workspace, device);
  Py_DECREF(device);
  if(ws == nullptr)
    return false;
  PyObject* p = PyObject_GetAttrString(ws, "ptr");
  PyObject* n = PyObject_GetAttrString(ws, "nbytes");
  bool ok = p != nullptr && n != nullptr;
  if(ok) {
    *ptr = PyLong_AsVoidPtr(p);
    *bytes = PyLong_AsSize_t(n);
    ok = PyErr_Occurred() == nullptr;
  }
  Py_XDECREF(p);
  Py_XDECREF(n);
  Py_DECREF(ws);
  if(ok)
    g_ws.push_back(WsEntry{dev, stream, *ptr, *bytes});
  return ok;
}

// A CUDA tensor of the current device, contiguous and of the given type, with its address; or nothing.
struct DeviceTensor {
  const at::Tensor* t = nullptr;
  void* ptr = nullptr;
  explicit operator bool() const { return t != nullptr; }
  const at::Tensor* operator->() const { return t; }
  template <typename T>
  T* as() const {
    return static_cast<T*>(ptr);
  }
};
DeviceTensor device_tensor(PyObject* o, at::ScalarType type) {
  if(!THPVariable_Check(o))
    return {};
  const at::Tensor& t = THPVariable_Unpack(o);
  try {
    if(!t.is_cuda() || t.scalar_type() != type || !t.is_contiguous() || t.device().index() != c10::cuda::current_device())
      return {};
    void* ptr = t.data_ptr();   // (throws, or is null, for a tensor without memory of its own)
    return ptr != nullptr || t.numel() == 0 ? DeviceTensor{&t, ptr} : DeviceTensor{};
  } catch(const std::exception&) {
    PyErr_Clear();
    return {};
  }
}

at::Tensor new_tensor(c10::IntArrayRef sizes, at::ScalarType type, c10::Device device) {
  return at::detail::empty_cuda(sizes, type, device, c10::nullopt);
}

// A contiguous tensor of `type` over the bytes of `storage_of` from byte `offset` on (a multiple of the element size).
at::Tensor view_bytes(const at::Tensor& storage_of, size_t offset, c10::IntArrayRef sizes, at::ScalarType type) {
  const caffe2::TypeMeta meta = c10::scalarTypeToTypeMeta(type);
  at::Tensor t = at::detail::make_tensor<c10::TensorImpl>(c10::Storage(storage_of.storage()), storage_of.key_set(), meta);
  c10::TensorImpl* impl = t.unsafeGetTensorImpl();
  impl->set_storage_offset(static_cast<int64_t>((static_cast<size_t>(storage_of.storage_offset()) * storage_of.element_size() + offset) / meta.itemsize()));
  impl->set_sizes_contiguous(sizes);
  return t;
}

size_t round256(size_t n) { return (n + 255) / 256 * 256; }

PyObject* status(int rc) { return PyLong_FromLong(rc); }

// The library's calls run without the GIL: a launch waits when the device's queue is full.
template <typename F>
int without_gil(F&& f) {
  struct Release {
    PyThreadState* st = PyEval_SaveThread();
    ~Release() { PyEval_RestoreThread(st); }
  } release;
  return f();
}

// Output sizes: the activation's leading dimensions and the weight's width.
void out_sizes(const at::Tensor& a, int64_t n, c10::SmallVector<int64_t, 6>& sizes) {
  sizes.assign(a.sizes().begin(), a.sizes().end());
  sizes.back() = n;
}

// affine(a, weight storage, K, N, bias or None, scale, relu, half) -> tensor [..., N]
PyObject* py_affine(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if(nargs != 8)
    Py_RETURN_NONE;
  const DeviceTensor a = device_tensor(args[0], at::kFloat), w = device_tensor(args[1], at::kByte);
  const int64_t K = PyLong_AsLongLong(args[2]), N = PyLong_AsLongLong(args[3]);
  const double scale = PyFloat_AsDouble(args[5]);
  if(PyErr_Occurred())
    return nullptr;
  if(!a || !w || K <= 0 || N <= 0 || a->dim() < 1 || a->size(-1) != K || a->numel() == 0 || w->numel() < N * K + 4)
    Py_RETURN_NONE;
  const float* bias = nullptr;
  if(args[4] != Py_None) {
    const DeviceTensor b = device_tensor(args[4], at::kFloat);
    if(!b || b->numel() != N)
      Py_RETURN_NONE;
    bias = b.as<float>();
  }
  const int64_t M = a->numel() / K;
  if(M > INT32_MAX || N > INT32_MAX || K > INT32_MAX)
    Py_RETURN_NONE;
  const bool half = args[7] == Py_True;
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream().stream();
  void* ws = nullptr;
  size_t ws_bytes = 0;
  if(!workspace(*a.t, args[0], stream, &ws, &ws_bytes))
    return nullptr;
  c10::SmallVector<int64_t, 6> sizes;
  out_sizes(*a.t, N, sizes);
  at::Tensor out = new_tensor(sizes, half ? at::kHalf : at::kFloat, a->device());
  const int64_t scratch_bytes = static_cast<int64_t>(round256(static_cast<size_t>(M) * K + 4));
  at::Tensor scratch = new_tensor({scratch_bytes}, at::kByte, a->device());
  const int8_t* bt = w.as<int8_t>();
  void* c = out.data_ptr();
  int8_t* aq = static_cast<int8_t*>(scratch.data_ptr());
  const int rc = without_gil([&] {
    return g_lib.affine(a.as<float>(), static_cast<int>(M), static_cast<int>(K), bt, reinterpret_cast<const float*>(bt + N * K), static_cast<int>(N), bias,
                        static_cast<float>(scale), args[6] == Py_True, c, half ? MI8_F16 : MI8_F32, aq, ws, ws_bytes, stream);
  });
  return rc == MI8_OK ? THPVariable_Wrap(std::move(out)) : status(rc);
  END_HANDLE_TH_ERRORS
}

// prepare_b(w, K, N, w_is_nk) -> uint8 storage: int8 [N, K], its multiplier behind it
PyObject* py_prepare_b(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if(nargs != 4)
    Py_RETURN_NONE;
  const DeviceTensor w = device_tensor(args[0], at::kFloat);
  const int64_t K = PyLong_AsLongLong(args[1]), N = PyLong_AsLongLong(args[2]);
  if(PyErr_Occurred())
    return nullptr;
  if(!w || K <= 0 || N <= 0 || K > INT32_MAX || N > INT32_MAX || (K * N) % 4 != 0 || w->numel() != K * N)
    Py_RETURN_NONE;
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream().stream();
  void* ws = nullptr;
  size_t ws_bytes = 0;
  if(!workspace(*w.t, args[0], stream, &ws, &ws_bytes))
    return nullptr;
  at::Tensor out = new_tensor({static_cast<int64_t>(round256(static_cast<size_t>(K) * N + 4))}, at::kByte, w->device());
  int8_t* bt = static_cast<int8_t*>(out.data_ptr());
  const int rc = without_gil([&] {
    return g_lib.prepare_b(w.as<float>(), static_cast<int>(K), static_cast<int>(N), args[3] == Py_True, bt, reinterpret_cast<float*>(bt + K * N), ws, ws_bytes, stream);
  });
  return rc == MI8_OK ? THPVariable_Wrap(std::move(out)) : status(rc);
  END_HANDLE_TH_ERRORS
}

// intgemm_views(storage, rows, cols) -> (int8 [rows, cols], float32 [1] behind it)
PyObject* py_intgemm_views(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if(nargs != 3 || !THPVariable_Check(args[0])) {
    PyErr_SetString(PyExc_TypeError, "intgemm_views(storage, rows, cols)");
    return nullptr;
  }
  const at::Tensor& s = THPVariable_Unpack(args[0]);
  const int64_t rows = PyLong_AsLongLong(args[1]), cols = PyLong_AsLongLong(args[2]);
  if(PyErr_Occurred())
    return nullptr;
  const size_t first = static_cast<size_t>(s.storage_offset()) * s.element_size();
  if(s.scalar_type() != at::kByte || s.dim() != 1 || !s.is_contiguous() || s.numel() < rows * cols + 4 || (first + static_cast<size_t>(rows) * cols) % 4 != 0)
    Py_RETURN_NONE;   // (an unusual storage: the caller takes views the general way, which says what is wrong)
  const THPObjectPtr data(THPVariable_Wrap(view_bytes(s, 0, {rows, cols}, at::kChar)));
  const THPObjectPtr mult(THPVariable_Wrap(view_bytes(s, static_cast<size_t>(rows) * cols, {1}, at::kFloat)));
  return data && mult ? PyTuple_Pack(2, data.get(), mult.get()) : nullptr;
  END_HANDLE_TH_ERRORS
}

// p8_prepare_b(w [K, N]) -> (item, bt, scale_b, zp_b, off_b): the packed8avx512 item, its row-major copy and its tail
PyObject* py_p8_prepare_b(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  const DeviceTensor w = nargs == 1 ? device_tensor(args[0], at::kFloat) : DeviceTensor{};
  if(!w || w->dim() != 2 || w->numel() == 0 || w->size(0) > INT32_MAX || w->size(1) > INT32_MAX)
    Py_RETURN_NONE;
  const int64_t K = w->size(0), N = w->size(1);
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream().stream();
  at::Tensor item = new_tensor({static_cast<int64_t>(g_lib.packed_bytes(static_cast<int>(K), static_cast<int>(N)))}, at::kChar, w->device());
  int8_t* p = static_cast<int8_t*>(item.data_ptr());
  int rc = without_gil([&] { return g_lib.p8_prepare_b(w.as<float>(), static_cast<int>(K), static_cast<int>(N), p, stream); });
  if(rc != MI8_OK)
    return status(rc);
  at::Tensor bt = new_tensor({N, K}, at::kChar, w->device());
  int8_t* pt = static_cast<int8_t*>(bt.data_ptr());
  rc = without_gil([&] { return g_lib.p8_unpack_b(p, static_cast<int>(K), static_cast<int>(N), pt, stream); });
  if(rc != MI8_OK)
    return status(rc);
  const size_t tail = static_cast<size_t>(K) * N;   // (K a multiple of 256, N of 32: the library takes no others)
  const THPObjectPtr scale(THPVariable_Wrap(view_bytes(item, tail, {N}, at::kFloat)));
  const THPObjectPtr zp(THPVariable_Wrap(view_bytes(item, tail + 4 * N, {N}, at::kInt)));
  const THPObjectPtr off(THPVariable_Wrap(view_bytes(item, tail + 8 * N, {N}, at::kInt)));
  const THPObjectPtr item_obj(THPVariable_Wrap(std::move(item))), bt_obj(THPVariable_Wrap(std::move(bt)));
  return scale && zp && off && item_obj && bt_obj ? PyTuple_Pack(5, item_obj.get(), bt_obj.get(), scale.get(), zp.get(), off.get()) : nullptr;
  END_HANDLE_TH_ERRORS
}

// p8_gemm(a, bt, scale_b, zp_b, off_b, bias or None) -> tensor [..., N]
PyObject* py_p8_gemm(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if(nargs != 6)
    Py_RETURN_NONE;
  const DeviceTensor a = device_tensor(args[0], at::kFloat), bt = device_tensor(args[1], at::kChar), sb = device_tensor(args[2], at::kFloat);
  const DeviceTensor zb = device_tensor(args[3], at::kInt), ob = device_tensor(args[4], at::kInt);
  if(!a || !bt || !sb || !zb || !ob || bt->dim() != 2)
    Py_RETURN_NONE;
  const int64_t N = bt->size(0), K = bt->size(1);
  if(a->dim() < 1 || a->numel() == 0 || a->size(-1) != K || sb->numel() != N || zb->numel() != N || ob->numel() != N || a->numel() / K > INT32_MAX)
    Py_RETURN_NONE;
  const float* bias = nullptr;
  if(args[5] != Py_None) {
    const DeviceTensor b = device_tensor(args[5], at::kFloat);
    if(!b || b->numel() != N)
      Py_RETURN_NONE;
    bias = b.as<float>();
  }
  const int M = static_cast<int>(a->numel() / K);
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream().stream();
  void* ws = nullptr;
  size_t ws_bytes = 0;
  if(!workspace(*a.t, args[0], stream, &ws, &ws_bytes))
    return nullptr;
  c10::SmallVector<int64_t, 6> sizes;
  out_sizes(*a.t, N, sizes);
  at::Tensor out = new_tensor(sizes, at::kFloat, a->device());
  const size_t need = std::max<size_t>(g_lib.p8_scratch_bytes(M, static_cast<int>(K)), 256);
  at::Tensor scratch = new_tensor({static_cast<int64_t>(need)}, at::kByte, a->device());
  float* c = static_cast<float*>(out.data_ptr());
  void* scratch_ptr = scratch.data_ptr();
  const int rc = without_gil([&] {
    return g_lib.p8_gemm(a.as<float>(), bt.as<int8_t>(), sb.as<float>(), zb.as<int32_t>(), ob.as<int32_t>(), bias, c, M, static_cast<int>(N),
                         static_cast<int>(K), scratch_ptr, need, ws, ws_bytes, stream);
  });
  return rc == MI8_OK ? THPVariable_Wrap(std::move(out)) : status(rc);
  END_HANDLE_TH_ERRORS
}

template <typename F>
bool resolve(void* handle, const char* name, F& fn) {
  fn = reinterpret_cast<F>(dlsym(handle, name));
  if(fn == nullptr)
    PyErr_Format(PyExc_ImportError, "the library does not export %s", name);
  return fn != nullptr;
}

// init(library path, default_workspace, torch's version): must be called once before anything else
PyObject* py_init(PyObject*, PyObject* args) {
  const char *path = nullptr, *torch_version = nullptr;
  PyObject* fn = nullptr;
  if(!PyArg_ParseTuple(args, "sOs", &path, &fn, &torch_version))
    return nullptr;
  const size_t n = std::strlen(TORCH_VERSION);   // "2.11.0", where the module says "2.11.0", "2.11.0+cu128" or "2.11.0a0+git..."
  if(std::strncmp(torch_version, TORCH_VERSION, n) != 0 || (torch_version[n] >= '0' && torch_version[n] <= '9')) {
    PyErr_Format(PyExc_ImportError, "_ops_native.so was built for torch %s, not %s", TORCH_VERSION, torch_version);
    return nullptr;
  }
  void* h = dlopen(path, RTLD_NOW);   // already loaded by the ctypes binding: the same handle
  if(h == nullptr) {
    PyErr_Format(PyExc_ImportError, "%s", dlerror());
    return nullptr;
  }
  if(!resolve(h, "mi8_affine_f32", g_lib.affine) || !resolve(h, "mi8_prepare_b_f32", g_lib.prepare_b) ||
     !resolve(h, "mi8p_packed_bytes", g_lib.packed_bytes) || !resolve(h, "mi8p_prepare_b_f32", g_lib.p8_prepare_b) ||
     !resolve(h, "mi8p_unpack_b", g_lib.p8_unpack_b) || !resolve(h, "mi8p_scratch_bytes", g_lib.p8_scratch_bytes) ||
     !resolve(h, "mi8p_gemm_int8_packed", g_lib.p8_gemm))
    return nullptr;
  Py_INCREF(fn);
  Py_XSETREF(g_default_workspace, fn);
  Py_RETURN_NONE;
}

PyCFunction fast(PyObject* (*f)(PyObject*, PyObject* const*, Py_ssize_t)) { return reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f)); }

PyMethodDef methods[] = {
    {"init", py_init, METH_VARARGS, "init(library path, default_workspace, torch version)"},
    {"affine", fast(py_affine), METH_FASTCALL, "affine(a, weight storage, K, N, bias, scale, relu, half)"},
    {"prepare_b", fast(py_prepare_b), METH_FASTCALL, "prepare_b(w, K, N, w_is_nk)"},
    {"intgemm_views", fast(py_intgemm_views), METH_FASTCALL, "intgemm_views(storage, rows, cols)"},
    {"p8_prepare_b", fast(py_p8_prepare_b), METH_FASTCALL, "p8_prepare_b(w)"},
    {"p8_gemm", fast(py_p8_gemm), METH_FASTCALL, "p8_gemm(a, bt, scale_b, zp_b, off_b, bias)"},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_ops_native", "per-call host path of ops.py and packed8.py", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__ops_native() { return PyModule_Create(&module); }
