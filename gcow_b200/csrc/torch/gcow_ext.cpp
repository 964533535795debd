// Native host path of the CUDA entry points: what lies between a Python call and a kernel launch.
//
// A call of the stand-alone codec on a small tensor is all host time: argument checks, an allocation, the current
// stream, the launch, the result object. In Python with ctypes that was 16 to 18 us per call (torch.cuda.device and
// current_stream alone 6 us) around 2.5 us of kernel; here it is the C++ calls those wrap.
//
// CPython C API on top of libtorch (tensors in and out) and the C ABI of libgcow_cuda.so (every kernel launch); errors
// are raised as Python exceptions.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/Exceptions.h>

#include "layers.h"

extern "C" {
int gcow_encode_1d_stream(const float* in, uint64_t n, int maxbits, void* out, void* stream);
int gcow_decode_1d_fixed(const void* in, float* out, uint64_t n, int maxbits, int shift, void* stream);
int gcow_tile_usable(const int32_t* params, uint64_t blocks, int dim);
uint64_t gcow_encode_tiles_scratch_bytes(const int32_t* params, uint64_t blocks, int dim);
int gcow_encode_tiles(const float* in, uint64_t nx, uint64_t ny, const int32_t* params, void* out, void* scratch,
                      uint64_t* block_bits, uint64_t* total_out, void* stream);
int gcow_decode_generic(const uint64_t* in, float* out, uint64_t nx, uint64_t ny, const int32_t* params,
                        const uint64_t* block_bits, int shift, void* stream);
int gcow_ar_launch_ef(const float* in, float* out, uint64_t n, int rank, int world, int variant, int bits, int ctas, int shift,
                      float postscale, void* const* arenas, void* mc_arena, uint64_t region_cap, uint32_t epoch,
                      uint64_t timeout_ns, uint32_t* status, uint32_t* abort_flag, unsigned long long* stamps, float* residual,
                      void* stream);
int gcow_ar_roundtrip(const float* in, float* out, uint64_t n, int bits, void* stream);
uint64_t gcow_max_stream_bytes(const int32_t* params, uint64_t blocks, int dim);
int gcow_host_word(uint64_t** word);
int gcow_wait_host_word(volatile uint64_t* word, void* stream, uint64_t* value);
}

namespace {

struct NoGil {
  PyThreadState* s;
  NoGil() : s(PyEval_SaveThread()) {}
  ~NoGil() { PyEval_RestoreThread(s); }
};

inline at::Tensor bytes_on(int64_t n, const at::Tensor& like) {
  return at::detail::empty_cuda({n}, at::kByte, like.device(), std::nullopt);
}
inline at::Tensor longs_on(int64_t n, const at::Tensor& like) {
  return at::detail::empty_cuda({n}, at::kLong, like.device(), std::nullopt);
}
inline void check(int err, const char* what) {
  TORCH_CHECK(err == 0, what, " failed with CUDA/launcher error ", err);
}
inline bool one_store_bits(int32_t bits) { return bits == 16 || bits == 32 || bits == 64 || bits == 128; }

bool read_params(PyObject* const* args, int32_t* p) {
  for (int i = 0; i < 4; i++) {
    const long v = PyLong_AsLong(args[i]);
    if (v == -1 && PyErr_Occurred()) return false;
    p[i] = (int32_t)v;
  }
  return true;
}

// compress(x, minbits, maxbits, maxprec, minexp, dim, want_index) -> (stream, index or None), or None when these
// parameters need the slot / scan / scatter kernels. x: contiguous float32 CUDA tensor (checked by the caller).
PyObject* compress(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(nargs == 7 && THPVariable_Check(args[0]), "compress: bad arguments");
  const at::Tensor& x = gcow_ext::in_memory(THPVariable_Unpack(args[0]));
  int32_t p[4];
  if (!read_params(args + 1, p)) return nullptr;
  const long dim = PyLong_AsLong(args[5]);
  const int want_index = PyObject_IsTrue(args[6]);
  if (PyErr_Occurred()) return nullptr;
  const uint64_t nx = dim == 1 ? x.numel() : x.size(1), ny = dim == 1 ? 0 : x.size(0);
  const uint64_t blocks = dim == 1 ? (nx + 3) / 4 : ((nx + 3) / 4) * ((ny + 3) / 4);
  const bool fixed = p[0] == p[1];
  const bool one_store = dim == 1 && fixed && one_store_bits(p[1]);
  if (!blocks || !(one_store || gcow_tile_usable(p, blocks, (int)dim))) Py_RETURN_NONE;
  const c10::cuda::CUDAGuard guard(x.device());
  void* const stream = c10::cuda::getCurrentCUDAStream(x.device().index()).stream();
  const float* const in = x.const_data_ptr<float>();
  at::Tensor out, index;
  if (fixed) {
    out = bytes_on((int64_t)((blocks * (uint64_t)p[1] + 63) / 64 * 8), x);
    if (one_store) {
      check(gcow_encode_1d_stream(in, nx, p[1], out.mutable_data_ptr(), stream), "gcow_encode_1d_stream");
    } else {
      if (want_index) index = longs_on((int64_t)blocks + 1, x);
      check(gcow_encode_tiles(in, nx, ny, p, out.mutable_data_ptr(), nullptr,
                              index.defined() ? (uint64_t*)index.mutable_data_ptr() : nullptr, nullptr, stream),
            "gcow_encode_tiles");
    }
  } else {
    at::Tensor cap = bytes_on((int64_t)gcow_max_stream_bytes(p, blocks, (int)dim), x);
    index = longs_on((int64_t)blocks + 1, x);
    const at::Tensor scratch = bytes_on((int64_t)gcow_encode_tiles_scratch_bytes(p, blocks, (int)dim), x);
    uint64_t* word = nullptr;
    check(gcow_host_word(&word), "gcow_host_word");
    check(gcow_encode_tiles(in, nx, ny, p, cap.mutable_data_ptr(), scratch.mutable_data_ptr(), (uint64_t*)index.mutable_data_ptr(),
                            word, stream),
          "gcow_encode_tiles");
    uint64_t bits = 0;
    int err;
    {
      NoGil free;
      err = gcow_wait_host_word(word, stream, &bits);
    }
    check(err, "waiting for the stream's length");
    out = cap.narrow(0, 0, (int64_t)((bits + 63) / 64 * 8));
  }
  PyObject* a = THPVariable_Wrap(std::move(out));
  PyObject* b = index.defined() ? THPVariable_Wrap(std::move(index)) : Py_NewRef(Py_None);
  PyObject* r = a && b ? PyTuple_Pack(2, a, b) : nullptr;
  Py_XDECREF(a);
  Py_XDECREF(b);
  return r;
  END_HANDLE_TH_ERRORS
}

// decompress(stream, index or None, minbits, maxbits, maxprec, minexp, shape, out or None, shift) -> out, or None when
// the call needs another path. stream: contiguous uint8 CUDA tensor; index: int64 on the same device.
PyObject* decompress(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(nargs == 9 && THPVariable_Check(args[0]) && PyTuple_Check(args[6]), "decompress: bad arguments");
  const at::Tensor& s = gcow_ext::in_memory(THPVariable_Unpack(args[0]));
  int32_t p[4];
  if (!read_params(args + 2, p)) return nullptr;
  const Py_ssize_t dim = PyTuple_GET_SIZE(args[6]);
  if (dim != 1 && dim != 2) Py_RETURN_NONE;
  int64_t shape[2] = {0, 0};
  for (Py_ssize_t i = 0; i < dim; i++) shape[i] = PyLong_AsLongLong(PyTuple_GET_ITEM(args[6], i));
  const long shift = PyLong_AsLong(args[8]);
  if (PyErr_Occurred()) return nullptr;
  const uint64_t nx = dim == 1 ? shape[0] : shape[1], ny = dim == 1 ? 0 : shape[0];
  const uint64_t blocks = dim == 1 ? (nx + 3) / 4 : ((nx + 3) / 4) * ((ny + 3) / 4);
  const bool fixed = p[0] == p[1];
  const bool one_store = dim == 1 && fixed && one_store_bits(p[1]);
  if (!blocks || !(one_store || gcow_tile_usable(p, blocks, (int)dim))) Py_RETURN_NONE;
  const uint64_t* index = nullptr;
  if (!fixed) {
    if (args[1] == Py_None) Py_RETURN_NONE;
    TORCH_CHECK_TYPE(THPVariable_Check(args[1]), "decompress: the index is no tensor");
    const at::Tensor& i = gcow_ext::in_memory(THPVariable_Unpack(args[1]));
    if (i.device() != s.device()) Py_RETURN_NONE;
    index = (const uint64_t*)i.const_data_ptr();
  }
  at::Tensor out;
  if (args[7] != Py_None) out = gcow_ext::in_memory(THPVariable_Unpack(args[7]));
  const c10::cuda::CUDAGuard guard(s.device());
  if (!out.defined()) out = at::detail::empty_cuda(c10::IntArrayRef(shape, (size_t)dim), at::kFloat, s.device(), std::nullopt);
  void* const stream = c10::cuda::getCurrentCUDAStream(s.device().index()).stream();
  if (one_store)
    check(gcow_decode_1d_fixed(s.const_data_ptr(), out.mutable_data_ptr<float>(), nx, p[1], (int)shift, stream), "gcow_decode_1d_fixed");
  else
    check(gcow_decode_generic((const uint64_t*)s.const_data_ptr(), out.mutable_data_ptr<float>(), nx, ny, p, index, (int)shift, stream), "gcow_decode_generic");
  if (args[7] != Py_None) return Py_NewRef(args[7]);
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// ar_launch(x, out, residual or None, first, count, stream or None, rank, world, variant, bits, ctas, shift, postscale, arenas,
//           mc_arena, region_cap, epoch, timeout_ns, status, stamps): one launch of the fused all-reduce over `count` values
// from `first` on. Addresses are ints; `stream` is a cudaStream_t as int, None for the current stream.
PyObject* ar_launch(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(nargs == 20 && THPVariable_Check(args[0]) && THPVariable_Check(args[1]), "ar_launch: bad arguments");
  const at::Tensor& x = gcow_ext::in_memory(THPVariable_Unpack(args[0]));
  const at::Tensor& out = gcow_ext::in_memory(THPVariable_Unpack(args[1]));
  uint64_t v[20];
  for (int i = 3; i < 20; i++) {
    if (i == 12 || (i == 5 && args[5] == Py_None)) continue;
    v[i] = PyLong_AsUnsignedLongLong(args[i]);
  }
  const double post = PyFloat_AsDouble(args[12]);
  if (PyErr_Occurred()) return nullptr;
  at::Tensor residual;
  if (args[2] != Py_None) residual = gcow_ext::in_memory(THPVariable_Unpack(args[2]));
  const c10::cuda::CUDAGuard guard(x.device());
  void* const stream = args[5] == Py_None ? c10::cuda::getCurrentCUDAStream(x.device().index()).stream() : (void*)v[5];
  float* const res = residual.defined() ? residual.mutable_data_ptr<float>() + v[3] : nullptr;
  uint32_t* const status = (uint32_t*)v[18];
  const int err = gcow_ar_launch_ef(x.const_data_ptr<float>() + v[3], out.mutable_data_ptr<float>() + v[3], v[4], (int)v[6], (int)v[7],
                                    (int)v[8], (int)v[9], (int)v[10], (int)v[11], (float)post, (void* const*)v[13], (void*)v[14],
                                    v[15], (uint32_t)v[16], v[17], status, status + 8, (unsigned long long*)v[19], res, stream);
  TORCH_CHECK(err == 0, "gcow_ar_launch failed: ", err);
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

// ar_roundtrip(x, out or None, stream or None, max_numel, bits) -> whether the call was the plain one and has been launched: one rank, no
// error feedback, contiguous float32 tensors of one device, as many values as an arena holds at most. What is not plain, mistakes
// among it, is the caller's.
PyObject* ar_roundtrip(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(nargs == 5, "ar_roundtrip: bad arguments");
  if (!THPVariable_Check(args[0]) || !(args[1] == Py_None || THPVariable_Check(args[1]))) Py_RETURN_FALSE;
  const at::Tensor& x0 = THPVariable_Unpack(args[0]);
  if (!x0.is_cuda() || x0.scalar_type() != at::kFloat || !x0.is_contiguous()) Py_RETURN_FALSE;
  const at::Tensor& x = gcow_ext::in_memory(x0);
  const bool own = args[1] == Py_None || args[1] == args[0];
  if (!own) {
    const at::Tensor& o = THPVariable_Unpack(args[1]);
    if (o.device() != x.device() || o.scalar_type() != at::kFloat || !o.is_contiguous() || o.numel() < x.numel()) Py_RETURN_FALSE;
  }
  const at::Tensor& out = own ? x : gcow_ext::in_memory(THPVariable_Unpack(args[1]));
  const int64_t n = x.numel(), most = PyLong_AsLongLong(args[3]);
  const long bits = PyLong_AsLong(args[4]);
  const uint64_t given = args[2] == Py_None ? 0 : PyLong_AsUnsignedLongLong(args[2]);
  if (PyErr_Occurred()) return nullptr;
  if (n < 1 || n > most) Py_RETURN_FALSE;
  const c10::cuda::CUDAGuard guard(x.device());
  void* const stream = args[2] == Py_None ? c10::cuda::getCurrentCUDAStream(x.device().index()).stream() : (void*)given;
  check(gcow_ar_roundtrip(x.const_data_ptr<float>(), out.mutable_data_ptr<float>(), (uint64_t)n, (int)bits, stream), "gcow_ar_roundtrip");
  Py_RETURN_TRUE;
  END_HANDLE_TH_ERRORS
}

PyMethodDef methods[] = {
    {"ar_roundtrip", (PyCFunction)(void (*)())ar_roundtrip, METH_FASTCALL, nullptr},
    {"ar_launch", (PyCFunction)(void (*)())ar_launch, METH_FASTCALL, nullptr},
    {"compress", (PyCFunction)(void (*)())compress, METH_FASTCALL, nullptr},
    {"decompress", (PyCFunction)(void (*)())decompress, METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "gcow_ext", "native host path of gcow_b200", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_gcow_ext(void) {
  PyObject* m = PyModule_Create(&module);
  if (m && PyModule_AddFunctions(m, gcow_ext::layer_methods)) Py_CLEAR(m);
  return m;
}
