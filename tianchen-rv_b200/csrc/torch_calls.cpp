// The Python package's hot calls as native functions: argument checks, the output's allocation
// and the current stream are taken from torch in C++, then the C ABI (include/tcrv_cuda.h) is
// called.  A decode step is dozens of launches of 3..10 us each; the same work done in the
// interpreter (attribute reads, torch.empty, a ctypes call of eleven arguments) cost 12.4 us per
// call, more than most of the kernels it launched.
//
// The functions take their arguments by position, exactly as the wrappers in __init__.py pass
// them; a non-zero status goes to the package's `_check`, which raises TcrvCudaError.
#include <Python.h>

#include <ATen/ops/empty.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "tcrv_cuda.h"

namespace {

constexpr int64_t kQK = TCRV_QK;

// What a module object keeps: the _check(status, where) of the package that loaded it.  (One package
// directory can be imported under several names; each raises its own TcrvCudaError.)
struct ModuleState {
  PyObject *check;
};
inline ModuleState &state(PyObject *module) { return *static_cast<ModuleState *>(PyModule_GetState(module)); }

struct PyError {};  // a Python exception is set

[[noreturn]] void fail(PyObject *type, const char *text) {
  PyErr_SetString(type, text);
  throw PyError{};
}

inline cudaStream_t stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

inline const at::Tensor &tensor(PyObject *o) {
  if (!THPVariable_Check(o))
    fail(PyExc_TypeError, "operands must be CUDA torch tensors (device pointers cross the C ABI)");
  const at::Tensor &t = THPVariable_Unpack(o);
  if (!t.is_cuda())
    fail(PyExc_TypeError, "operands must be CUDA torch tensors (device pointers cross the C ABI)");
  return t;
}

// What a kernel can read and write where it lies: a CUDA tensor, or one in page-locked host memory
// (mapped at the same address).  The GEMV and GEMM operands and the strided outputs may be either.
inline const at::Tensor &mapped(PyObject *o) {
  if (THPVariable_Check(o)) {
    const at::Tensor &t = THPVariable_Unpack(o);
    if (t.is_cuda() || t.is_pinned())
      return t;
  }
  return tensor(o);  // (refuses it)
}

// A contiguous CUDA tensor of the given type.
inline const at::Tensor &dense(PyObject *o, at::ScalarType type) {
  const at::Tensor &t = tensor(o);
  if (t.scalar_type() != type) {
    PyErr_Format(PyExc_TypeError, "expected dtype torch.%s, got %s",
                 type == at::kFloat ? "float32" : type == at::kInt ? "int32" : type == at::kByte ? "uint8" : "float64",
                 c10::toString(t.scalar_type()));
    throw PyError{};
  }
  if (!t.is_contiguous())
    fail(PyExc_ValueError, "operands must be contiguous");
  return t;
}

inline uint8_t *bytes(const at::Tensor &t) { return static_cast<uint8_t *>(t.data_ptr()); }
inline float *floats(const at::Tensor &t) { return static_cast<float *>(t.data_ptr()); }

inline at::Tensor empty(at::IntArrayRef shape, at::ScalarType type, const at::Tensor &like) {
  return at::empty(shape, like.options().dtype(type));
}

inline int64_t integer(PyObject *o) {
  const long long v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred())
    throw PyError{};
  return v;
}

inline double real(PyObject *o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred())
    throw PyError{};
  return v;
}

inline bool truth(PyObject *o) {
  const int v = PyObject_IsTrue(o);
  if (v < 0)
    throw PyError{};
  return v != 0;
}

void check(PyObject *module, int status, const char *where) {
  if (status == TCRV_CUDA_OK)
    return;
  PyObject *r = PyObject_CallFunction(state(module).check, "is", status, where);
  if (r != nullptr) {
    Py_DECREF(r);
    PyErr_SetString(PyExc_RuntimeError, where);
  }
  throw PyError{};
}

// The interpreter lock, given up as a ctypes call does and taken back however the scope is left:
// torch throws from data_ptr() for a tensor without storage (vmap, fake tensors), and what the
// handlers below do needs the lock.
class Unlocked {
 public:
  Unlocked() : state_(PyEval_SaveThread()) {}
  ~Unlocked() { PyEval_RestoreThread(state_); }
  Unlocked(const Unlocked &) = delete;
  Unlocked &operator=(const Unlocked &) = delete;

 private:
  PyThreadState *state_;
};

// Runs an allocation and a launch without the interpreter lock.
template <typename F>
inline int unlocked(F &&launch) {
  const Unlocked scope;
  return launch();
}

inline int64_t blocks_of(int64_t row_bytes, int64_t block_bytes) {
  if (row_bytes % block_bytes != 0) {
    PyErr_Format(PyExc_ValueError, "last dimension %lld is not a whole number of %lld-byte blocks",
                 static_cast<long long>(row_bytes), static_cast<long long>(block_bytes));
    throw PyError{};
  }
  return row_bytes / block_bytes;
}

// Elements from a tensor's first to its last one in memory.
inline int64_t extent(const at::Tensor &t) {
  if (t.numel() == 0)
    return 0;
  int64_t n = 1;
  for (int64_t d = 0; d < t.dim(); ++d)
    n += (t.size(d) - 1) * t.stride(d);
  return n;
}

// The output of a call: the caller's, or one that is made without the interpreter lock, in front of
// the launch (an allocation may have to wait for the device or flush torch's cache).
struct Output {
  PyObject *given;
  at::Tensor tensor;

  // `type` as dense() checks it
  Output(PyObject *o, at::ScalarType type) : given(o) {
    if (given != Py_None)
      tensor = dense(given, type);
  }
  // rows with a stride: a float32 tensor, in device or page-locked memory, whose last dimension is contiguous
  explicit Output(PyObject *o) : given(o) {
    if (given == Py_None)
      return;
    tensor = mapped(given);
    if (tensor.scalar_type() != at::kFloat)
      fail(PyExc_TypeError, "expected dtype torch.float32 for the output");
    if (tensor.dim() > 0 && tensor.size(-1) > 1 && tensor.stride(-1) != 1)
      fail(PyExc_ValueError, "the output's rows must be contiguous");
  }
  // A caller's tensor must hold what the launch writes: `count` elements from its first one on,
  void require(int64_t count) const {
    if (given != Py_None && count > extent(tensor))
      fail(PyExc_ValueError, "the output is too small for the result");
  }
  // or `rows` rows of `cols` elements, its row stride apart.
  void require_rows(int64_t rows, int64_t cols) const {
    if (given != Py_None && rows > 0 && cols > 0)
      require((rows - 1) * tensor.stride(0) + cols);
  }
  // An output that is made lies beside `like`, which has to be a CUDA tensor then.
  void beside(const at::Tensor &like) const {
    if (given == Py_None && !like.is_cuda())
      fail(PyExc_TypeError, "operands must be CUDA torch tensors (device pointers cross the C ABI)");
  }
  void make(at::IntArrayRef shape, at::ScalarType type, const at::Tensor &like) {
    if (given == Py_None)
      tensor = empty(shape, type, like);
  }
  float *floats() const { return ::floats(tensor); }
  size_t stride() const { return static_cast<size_t>(tensor.stride(0)); }
  PyObject *result() {
    if (given == Py_None)
      return THPVariable_Wrap(std::move(tensor));
    Py_INCREF(given);
    return given;
  }
};

#define TCRV_CALL(name, count) \
  PyObject *name##_body(PyObject *module, PyObject *const *a); \
  PyObject *name(PyObject *module, PyObject *const *a, Py_ssize_t n) { \
    if (n != (count)) { \
      PyErr_SetString(PyExc_TypeError, #name ": wrong number of arguments"); \
      return nullptr; \
    } \
    try { \
      return name##_body(module, a); \
    } catch (const PyError &) { \
      return nullptr; \
    } catch (...) { /* as torch's own functions raise it: OutOfMemoryError, IndexError, ... */ \
      torch::translate_exception_to_python(std::current_exception()); \
      return nullptr; \
    } \
  } \
  PyObject *name##_body([[maybe_unused]] PyObject *module, PyObject *const *a)

// add(lhs, rhs, out)
TCRV_CALL(add, 3) {
  const at::Tensor &lhs = tensor(a[0]);
  const at::ScalarType type = lhs.scalar_type();
  if (type != at::kFloat && type != at::kInt)
    fail(PyExc_TypeError, "add supports float32 and int32");
  const at::Tensor &l = dense(a[0], type), &r = dense(a[1], type);
  Output out(a[2], type);
  out.require(l.numel());
  if (r.numel() < l.numel())
    fail(PyExc_ValueError, "operands differ in size");
  const size_t n = static_cast<size_t>(l.numel());
  const cudaStream_t st = stream();
  check(module, unlocked([&] {
          out.make(l.sizes(), type, l);
          return type == at::kFloat
                     ? tcrv_cuda_add_f32(floats(l), floats(r), out.floats(), n, st)
                     : tcrv_cuda_add_i32(static_cast<const int32_t *>(l.data_ptr()), static_cast<const int32_t *>(r.data_ptr()),
                                         static_cast<int32_t *>(out.tensor.data_ptr()), n, st);
        }),
        type == at::kFloat ? "tcrv_cuda_add_f32" : "tcrv_cuda_add_i32");
  return out.result();
}

// dequantize(vx, out, block_bytes)
TCRV_CALL(dequantize, 3) {
  const int64_t block = integer(a[2]);
  const at::Tensor &vx = dense(a[0], at::kByte);
  if (vx.dim() == 0)
    fail(PyExc_ValueError, "blocks come in rows");
  const int64_t nb = blocks_of(vx.size(-1), block);
  auto shape = vx.sizes().vec();
  shape.back() = nb * kQK;
  Output out(a[1], at::kFloat);
  if (out.given != Py_None && out.tensor.numel() > vx.numel() / block * kQK)
    fail(PyExc_ValueError, "the output asks for more elements than the blocks hold");
  const cudaStream_t st = stream();
  const bool q8 = block == TCRV_Q8_0_BLOCK_BYTES;
  check(module, unlocked([&] {
          out.make(shape, at::kFloat, vx);
          return (q8 ? tcrv_cuda_dequantize_row_q8_0 : tcrv_cuda_dequantize_row_q4_0)(
              bytes(vx), out.floats(), static_cast<size_t>(out.tensor.numel()), st);
        }),
        q8 ? "tcrv_cuda_dequantize_row_q8_0" : "tcrv_cuda_dequantize_row_q4_0");
  return out.result();
}

// quantize(x, out, block_bytes)
TCRV_CALL(quantize, 3) {
  const int64_t block = integer(a[2]);
  const at::Tensor &x = tensor(a[0]);
  if (x.dim() == 0 || x.size(-1) % kQK != 0)
    fail(PyExc_ValueError, "last dimension must be a multiple of 32");
  dense(a[0], at::kFloat);
  auto shape = x.sizes().vec();
  shape.back() = shape.back() / kQK * block;
  Output out(a[1], at::kByte);
  out.require(x.numel() / kQK * block);
  const size_t n = static_cast<size_t>(x.numel());
  const cudaStream_t st = stream();
  const bool q8 = block == TCRV_Q8_0_BLOCK_BYTES;
  check(module, unlocked([&] {
          out.make(shape, at::kByte, x);
          return (q8 ? tcrv_cuda_quantize_row_q8_0 : tcrv_cuda_quantize_row_q4_0)(n, floats(x), bytes(out.tensor), st);
        }),
        q8 ? "tcrv_cuda_quantize_row_q8_0" : "tcrv_cuda_quantize_row_q4_0");
  return out.result();
}

// gemv(w, x, q8_weights, flags, out)
TCRV_CALL(gemv, 5) {
  const bool q8 = truth(a[2]);
  const unsigned flags = static_cast<unsigned>(integer(a[3]));
  const at::Tensor &w = mapped(a[0]), &x = mapped(a[1]);
  if (w.dim() != 2 || x.dim() != 2)
    fail(PyExc_ValueError, "weights are (rows, row_bytes), activations are (columns, column_bytes)");
  const int64_t nb = blocks_of(x.size(1), TCRV_Q8_0_BLOCK_BYTES);
  if (blocks_of(w.size(1), q8 ? TCRV_Q8_0_BLOCK_BYTES : TCRV_Q4_0_BLOCK_BYTES) != nb)
    fail(PyExc_ValueError, "weights and activations disagree on the number of blocks per row");
  const int64_t nr = w.size(0), nc = x.size(0);
  Output out(a[4], at::kFloat);
  out.require_rows(nr, nc);
  out.beside(w);
  const size_t n = static_cast<size_t>(nb * kQK), bx = static_cast<size_t>(w.stride(0)),
               by = static_cast<size_t>(x.stride(0));
  const cudaStream_t st = stream();
  check(module, unlocked([&] {
          out.make({nr, nc}, at::kFloat, w);
          return (q8 ? tcrv_cuda_gemv_q8_0_q8_0 : tcrv_cuda_gemv_q4_0_q8_0)(
              n, out.floats(), bytes(w), bytes(x), by, static_cast<size_t>(nr), static_cast<size_t>(nc), bx, out.stride(),
              flags, st);
        }),
        q8 ? "tcrv_cuda_gemv_q8_0_q8_0" : "tcrv_cuda_gemv_q4_0_q8_0");
  return out.result();
}

// gemv_group(address of the calls, count, q8_weights, flags)
TCRV_CALL(gemv_group, 4) {
  const auto *calls = reinterpret_cast<const tcrv_cuda_gemv_call *>(static_cast<uintptr_t>(PyLong_AsUnsignedLongLong(a[0])));
  if (PyErr_Occurred())
    throw PyError{};
  const size_t count = static_cast<size_t>(integer(a[1]));
  const bool q8 = truth(a[2]);
  const unsigned flags = static_cast<unsigned>(integer(a[3]));
  const cudaStream_t st = stream();
  check(module, unlocked([&] {
          return (q8 ? tcrv_cuda_gemv_group_q8_0_q8_0 : tcrv_cuda_gemv_group_q4_0_q8_0)(calls, count, flags, st);
        }),
        q8 ? "tcrv_cuda_gemv_group_q8_0_q8_0" : "tcrv_cuda_gemv_group_q4_0_q8_0");
  Py_RETURN_NONE;
}

// Device scratch of at least `need` bytes: the caller's tensor, or a new one.  (A new one may go
// back to torch's allocator as soon as the launches are queued: its next user on this stream
// runs behind them.)
struct Scratch {
  at::Tensor tensor;
  explicit Scratch(PyObject *given) {
    if (given != Py_None)
      tensor = mapped(given);
  }
  void make(size_t need, const at::Tensor &like) {
    if (!tensor.defined())
      tensor = empty({static_cast<int64_t>(need < 256 ? 256 : need)}, at::kByte, like);
  }
  size_t size() const { return static_cast<size_t>(tensor.numel()); }
};

// gemm(w, x, out, workspace)
TCRV_CALL(gemm, 4) {
  const at::Tensor &w = mapped(a[0]), &x = mapped(a[1]);
  if (w.dim() != 2 || x.dim() != 2)
    fail(PyExc_ValueError, "weights are (rows, row_bytes), activations are (columns, column_bytes)");
  const int64_t nb = blocks_of(x.size(1), TCRV_Q8_0_BLOCK_BYTES);
  if (blocks_of(w.size(1), TCRV_Q4_0_BLOCK_BYTES) != nb)
    fail(PyExc_ValueError, "weights and activations disagree on the number of blocks per row");
  const size_t n = static_cast<size_t>(nb * kQK), nr = static_cast<size_t>(w.size(0)), nc = static_cast<size_t>(x.size(0));
  Output out(a[2], at::kFloat);
  out.require_rows(w.size(0), x.size(0));
  out.beside(w);
  Scratch ws(a[3]);
  const size_t bx = static_cast<size_t>(w.stride(0)), by = static_cast<size_t>(x.stride(0));
  const cudaStream_t st = stream();
  check(module, unlocked([&] {
          out.make({w.size(0), x.size(0)}, at::kFloat, w);
          ws.make(tcrv_cuda_gemm_workspace_bytes(n, nr, nc), out.tensor);
          return tcrv_cuda_gemm_q4_0_q8_0(n, out.floats(), bytes(w), bytes(x), by, nr, nc, bx, out.stride(),
                                          ws.tensor.data_ptr(), ws.size(), 0, st);
        }),
        "tcrv_cuda_gemm_q4_0_q8_0");
  return out.result();
}

// gemm_prepared(buffer, n, nr, x, out, workspace)
TCRV_CALL(gemm_prepared, 6) {
  const at::Tensor &buffer = tensor(a[0]), &x = mapped(a[3]);
  const size_t n = static_cast<size_t>(integer(a[1])), nr = static_cast<size_t>(integer(a[2]));
  if (x.dim() != 2)
    fail(PyExc_ValueError, "activations are (columns, column_bytes)");
  if (static_cast<size_t>(blocks_of(x.size(1), TCRV_Q8_0_BLOCK_BYTES) * kQK) != n)
    fail(PyExc_ValueError, "weights and activations disagree on the number of blocks per row");
  const size_t nc = static_cast<size_t>(x.size(0));
  Output out(a[4], at::kFloat);
  out.require_rows(static_cast<int64_t>(nr), x.size(0));
  out.beside(x);
  Scratch ws(a[5]);
  const size_t by = static_cast<size_t>(x.stride(0));
  const cudaStream_t st = stream();
  check(module, unlocked([&] {
          out.make({static_cast<int64_t>(nr), x.size(0)}, at::kFloat, x);
          ws.make(tcrv_cuda_gemm_acts_workspace_bytes(n, nc), out.tensor);
          return tcrv_cuda_gemm_q4_0_q8_0_prepared(n, out.floats(), buffer.data_ptr(), bytes(x), by, nr, nc, out.stride(),
                                                   ws.tensor.data_ptr(), ws.size(), 0, st);
        }),
        "tcrv_cuda_gemm_q4_0_q8_0_prepared");
  return out.result();
}

// sibling_dot_rows(format, weight block bytes, activation block bytes, w, x, out)
TCRV_CALL(sibling_dot_rows, 6) {
  const int format = static_cast<int>(integer(a[0]));
  const int64_t wb = integer(a[1]), ab = integer(a[2]);
  const at::Tensor &w = dense(a[3], at::kByte), &x = dense(a[4], at::kByte);
  if (w.dim() != 2 || x.dim() != 2 || w.size(1) % wb != 0 || x.size(1) % ab != 0 || w.size(1) / wb != x.size(1) / ab)
    fail(PyExc_ValueError, "row bytes do not match the format's block sizes");
  const size_t n = static_cast<size_t>(w.size(1) / wb * kQK), nr = static_cast<size_t>(w.size(0)), nc = static_cast<size_t>(x.size(0));
  Output out(a[5], at::kFloat);
  out.require_rows(w.size(0), x.size(0));
  const cudaStream_t st = stream();
  check(module, unlocked([&] {
          out.make({w.size(0), x.size(0)}, at::kFloat, w);
          return tcrv_cuda_sibling_dot_rows(format, n, out.floats(), bytes(w), bytes(x), static_cast<size_t>(x.stride(0)), nr,
                                            nc, static_cast<size_t>(w.stride(0)), out.stride(), st);
        }),
        "tcrv_cuda_sibling_dot_rows");
  return out.result();
}

inline const at::Tensor &row_matrix(PyObject *o) {
  const bool is = THPVariable_Check(o);
  if (!is || !THPVariable_Unpack(o).is_cuda() || THPVariable_Unpack(o).dim() != 2 || THPVariable_Unpack(o).stride(1) != 1 ||
      THPVariable_Unpack(o).scalar_type() != at::kFloat)
    fail(PyExc_ValueError, "x must be a 2-D float32 CUDA tensor with unit inner stride");
  return THPVariable_Unpack(o);
}

// rms_norm(x, eps, out, flags)
TCRV_CALL(rms_norm, 4) {
  const at::Tensor &x = row_matrix(a[0]);
  const float eps = static_cast<float>(real(a[1]));
  const unsigned flags = static_cast<unsigned>(integer(a[3]));
  Output out(a[2]);
  out.require_rows(x.size(0), x.size(1));
  const cudaStream_t st = stream();
  check(module, unlocked([&] {
          out.make({x.size(0), x.size(1)}, at::kFloat, x);
          return tcrv_cuda_rms_norm_f32_flags(static_cast<size_t>(x.size(1)), floats(x), out.floats(), eps,
                                              static_cast<size_t>(x.size(0)), static_cast<size_t>(x.stride(0)),
                                              out.stride(), flags, st);
        }),
        "tcrv_cuda_rms_norm_f32_flags");
  return out.result();
}

// rope_apply(x, cache, out)
TCRV_CALL(rope_apply, 3) {
  const at::Tensor &x = row_matrix(a[0]);
  const at::Tensor &cache = dense(a[1], at::kFloat);
  if (cache.numel() < x.size(1))
    fail(PyExc_ValueError, "the angle cache is too small");
  Output out(a[2]);
  out.require_rows(x.size(0), x.size(1));
  const cudaStream_t st = stream();
  check(module, unlocked([&] {
          out.make({x.size(0), x.size(1)}, at::kFloat, x);
          return tcrv_cuda_rope_apply_f32(static_cast<size_t>(x.size(1)), floats(x), out.floats(), floats(cache),
                                          static_cast<size_t>(x.size(0)), static_cast<size_t>(x.stride(0)),
                                          out.stride(), st);
        }),
        "tcrv_cuda_rope_apply_f32");
  return out.result();
}

// vec_silu(x, out)
TCRV_CALL(vec_silu, 2) {
  const at::Tensor &x = dense(a[0], at::kFloat);
  Output out(a[1], at::kFloat);
  out.require(x.numel());
  const cudaStream_t st = stream();
  check(module, unlocked([&] {
          out.make(x.sizes(), at::kFloat, x);
          return tcrv_cuda_vec_silu_f32(static_cast<size_t>(x.numel()), floats(x), out.floats(), st);
        }),
        "tcrv_cuda_vec_silu_f32");
  return out.result();
}

// vec_scale_(y, v)
TCRV_CALL(vec_scale_, 2) {
  const at::Tensor &y = dense(a[0], at::kFloat);
  const float v = static_cast<float>(real(a[1]));
  const cudaStream_t st = stream();
  check(module, unlocked([&] { return tcrv_cuda_vec_scale_f32(static_cast<size_t>(y.numel()), floats(y), v, st); }),
        "tcrv_cuda_vec_scale_f32");
  Py_INCREF(a[0]);
  return a[0];
}

// repack_gemv(wx16, x, nc, q8_weights, out, flags)
TCRV_CALL(repack_gemv, 6) {
  const at::Tensor &w = tensor(a[0]), &x = tensor(a[1]);
  const int64_t nc = integer(a[2]);
  const bool q8 = truth(a[3]);
  const unsigned flags = static_cast<unsigned>(integer(a[5]));
  const int64_t nb = x.numel() / TCRV_Q8_0_BLOCK_BYTES;
  if (x.numel() % TCRV_Q8_0_BLOCK_BYTES != 0 || nc % 16 != 0 || w.numel() != nc / 16 * nb * (q8 ? 544 : 288))
    fail(PyExc_ValueError, "weights, activation and nc do not describe the same shape");
  dense(a[0], at::kByte);
  dense(a[1], at::kByte);
  Output out(a[4], at::kFloat);
  out.require(nc);
  const cudaStream_t st = stream();
  check(module, unlocked([&] {
          out.make({nc}, at::kFloat, w);
          return (q8 ? tcrv_cuda_repack_gemv_q8_0_q8_0 : tcrv_cuda_repack_gemv_q4_0_q8_0)(
              static_cast<size_t>(nb * kQK), out.floats(), bytes(w), bytes(x), static_cast<size_t>(nc), flags, st);
        }),
        "tcrv_cuda_repack_gemv");
  return out.result();
}

// bind(_check)
TCRV_CALL(bind, 1) {
  Py_INCREF(a[0]);
  Py_XSETREF(state(module).check, a[0]);
  Py_RETURN_NONE;
}

#define TCRV_METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {TCRV_METHOD(add),          TCRV_METHOD(dequantize),       TCRV_METHOD(quantize),
                         TCRV_METHOD(gemv),         TCRV_METHOD(gemv_group),       TCRV_METHOD(gemm),
                         TCRV_METHOD(gemm_prepared), TCRV_METHOD(sibling_dot_rows), TCRV_METHOD(rms_norm),
                         TCRV_METHOD(rope_apply),   TCRV_METHOD(vec_silu),         TCRV_METHOD(vec_scale_),
                         TCRV_METHOD(repack_gemv),  TCRV_METHOD(bind),             {nullptr, nullptr, 0, nullptr}};
int traverse(PyObject *module, visitproc visit, void *arg) {
  Py_VISIT(state(module).check);
  return 0;
}
int clear(PyObject *module) {
  Py_CLEAR(state(module).check);
  return 0;
}
void release(void *module) { clear(static_cast<PyObject *>(module)); }

PyModuleDef_Slot slots[] = {{0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_tcrv_torch", nullptr, sizeof(ModuleState), methods, slots, traverse, clear, release};

}  // namespace

PyMODINIT_FUNC PyInit__tcrv_torch() { return PyModuleDef_Init(&module_def); }
