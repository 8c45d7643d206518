// Native call path of the operators (Python extension module _qhost).
//
// A decode-sized call runs for 5 - 40 us on the GPU, while the same call made through Python checks, torch.empty,
// a device guard and ctypes took 17 - 30 us of host time, so every small call was host bound.  This module does the whole
// ordinary call natively: it reads the tensors' metadata, allocates the output and the scratch from torch's caching
// allocator, takes the current stream and enters the C ABI of libqgemm.so (through addresses handed to init(), so the
// module works with whichever build of the library was loaded).
//
// Every function returns None, without having launched anything, as soon as something is not ordinary (wrong type,
// shape, device or layout, an empty result, a rejected call); the Python operator then runs its full checks, which either
// raise the documented error or handle the rare case.  So there is exactly one place that words errors.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/cuda/EmptyTensor.h>
#include <ATen/core/Tensor.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstring>

#include "../../include/qgemm.h"

namespace {

struct Api {
  decltype(&qgemm_w8a8) w8a8 = nullptr;
  decltype(&qgemm_w8a8_grouped) w8a8_grouped = nullptr;
  decltype(&qgemm_w8a8_grouped_zeroed) w8a8_grouped_zeroed = nullptr;
  decltype(&qgemm_w4a16_call_workspace_bytes) w4a16_ws = nullptr;
  decltype(&qgemm_w4a16_ex) w4a16 = nullptr;
  decltype(&qgemm_w4a8) w4a8 = nullptr;
  decltype(&qgemm_w4a8_act_quant) w4a8_aq = nullptr;
  decltype(&qgemm_act_quant) act_quant = nullptr;
} api;

using at::ScalarType;

// A plain CUDA tensor: exactly torch.Tensor (no subclass with its own dispatch), contiguous, of the given type.
const at::Tensor* plain(PyObject* o, ScalarType st) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  if (!t.defined() || !t.is_cuda() || t.scalar_type() != st || t.layout() != at::kStrided || !t.is_contiguous() || t.is_conj() ||
      t.is_neg())
    return nullptr;
  return &t;
}
bool same_device(const at::Tensor& a, const at::Tensor* b) { return b->get_device() == a.get_device(); }

// f16 / bf16 as a torch.dtype or its name; Undefined for anything else.
ScalarType float16_kind(PyObject* o) {
  if (THPDtype_Check(o)) {
    const ScalarType st = reinterpret_cast<THPDtype*>(o)->scalar_type;
    return (st == at::kHalf || st == at::kBFloat16) ? st : ScalarType::Undefined;
  }
  if (PyUnicode_Check(o)) {
    if (PyUnicode_CompareWithASCIIString(o, "float16") == 0) return at::kHalf;
    if (PyUnicode_CompareWithASCIIString(o, "bfloat16") == 0) return at::kBFloat16;
  }
  return ScalarType::Undefined;
}
int abi_dt(ScalarType st) { return st == at::kHalf ? QGEMM_DT_F16 : QGEMM_DT_BF16; }

at::Tensor empty_cuda(at::IntArrayRef shape, ScalarType st, int dev) {
  return at::detail::empty_cuda(shape, st, c10::Device(c10::kCUDA, (c10::DeviceIndex)dev), std::nullopt);
}

int64_t as_int(PyObject* o) {  // -1 on anything that is not a non-negative int
  if (!PyLong_CheckExact(o)) return -1;
  int overflow = 0;
  const long long v = PyLong_AsLongLongAndOverflow(o, &overflow);
  return (overflow || v < 0) ? -1 : v;
}

// An int of any sign (-1: any size will do) into v; false, with no Python error set, for anything else - an integral float
// in a factory's shape, say, which the Python path compares by value.
bool plain_int(PyObject* o, int64_t* v) {
  if (!PyLong_CheckExact(o)) return false;
  int overflow = 0;
  *v = PyLong_AsLongLongAndOverflow(o, &overflow);
  return overflow == 0;
}

// The library call runs without the interpreter lock; a scope, so that an exception takes the lock back before it is caught.
struct WithoutGil {
  PyThreadState* state = PyEval_SaveThread();
  ~WithoutGil() { PyEval_RestoreThread(state); }
};

// C++ exceptions (out of memory, a tensor without storage under vmap or jvp, ...) must not cross into the interpreter: the
// Python path then meets the same condition and raises it in torch's own words.
#define QHOST_TRY try {
#define QHOST_CATCH                     \
  }                                     \
  catch (...) {                         \
    PyErr_Clear();                      \
    Py_RETURN_NONE;                     \
  }

PyObject* h_init(PyObject*, PyObject* const* args, Py_ssize_t n) {
  constexpr int kEntries = 8;
  if (n != kEntries) {
    PyErr_SetString(PyExc_TypeError, "init takes the addresses of the eight entry points");
    return nullptr;
  }
  void* p[kEntries];
  for (int i = 0; i < kEntries; ++i) {
    p[i] = PyLong_AsVoidPtr(args[i]);
    if (p[i] == nullptr) return nullptr;
  }
  api.w8a8 = reinterpret_cast<decltype(api.w8a8)>(p[0]);
  api.w8a8_grouped = reinterpret_cast<decltype(api.w8a8_grouped)>(p[1]);
  api.w4a16_ws = reinterpret_cast<decltype(api.w4a16_ws)>(p[2]);
  api.w4a16 = reinterpret_cast<decltype(api.w4a16)>(p[3]);
  api.w4a8 = reinterpret_cast<decltype(api.w4a8)>(p[4]);
  api.w4a8_aq = reinterpret_cast<decltype(api.w4a8_aq)>(p[5]);
  api.act_quant = reinterpret_cast<decltype(api.act_quant)>(p[6]);
  api.w8a8_grouped_zeroed = reinterpret_cast<decltype(api.w8a8_grouped_zeroed)>(p[7]);
  Py_RETURN_NONE;
}

// w8a8(A, B, scale, scale_a | None, out_dtype, nk: bool, batch, M, N, K) -> C; batch 0: 2-D, batch -1: any shape
PyObject* h_w8a8(PyObject*, PyObject* const* args, Py_ssize_t n) {
  QHOST_TRY
  if (n != 10) Py_RETURN_NONE;
  const at::Tensor* A = plain(args[0], at::kChar);
  const at::Tensor* B = plain(args[1], at::kChar);
  const at::Tensor* sb = plain(args[2], at::kFloat);
  if (A == nullptr || B == nullptr || sb == nullptr) Py_RETURN_NONE;
  const at::Tensor* sa = nullptr;
  if (args[3] != Py_None) {
    sa = plain(args[3], at::kFloat);
    if (sa == nullptr || !same_device(*A, sa)) Py_RETURN_NONE;
  }
  if (!same_device(*A, B) || !same_device(*A, sb)) Py_RETURN_NONE;
  const ScalarType out = float16_kind(args[4]);
  if (out == ScalarType::Undefined) Py_RETURN_NONE;
  const bool nk = args[5] == Py_True;
  const int64_t nd = A->dim();
  if ((nd != 2 && nd != 3) || B->dim() != nd) Py_RETURN_NONE;
  const bool batched = nd == 3;
  const int64_t batch = batched ? A->size(0) : 1, M = A->size(-2), K = A->size(-1);
  const int64_t N = nk ? B->size(-2) : B->size(-1);
  if ((nk ? B->size(-1) : B->size(-2)) != K || (batched && B->size(0) != batch)) Py_RETURN_NONE;
  int64_t want_batch;
  if (!plain_int(args[6], &want_batch)) Py_RETURN_NONE;
  if (want_batch >= 0) {  // a factory's static shape; its scale rule (what the scale length may be) is the caller's
    if ((want_batch > 0) != batched || (batched && batch != want_batch) || M != as_int(args[7]) || N != as_int(args[8]) ||
        K != as_int(args[9]))
      Py_RETURN_NONE;
  }
  const int64_t sb_len = sb->numel(), sa_len = sa ? sa->numel() : 0;
  if (sb_len != 1 && sb_len != N && sb_len != batch * N) Py_RETURN_NONE;
  if (sa != nullptr && sa_len != M && sa_len != batch * M) Py_RETURN_NONE;
  if (batch * M * N == 0) Py_RETURN_NONE;
  const int dev = A->get_device();
  c10::cuda::CUDAGuard guard((c10::DeviceIndex)dev);
  const int64_t shape[3] = {batch, M, N};
  at::Tensor C = empty_cuda(batched ? at::IntArrayRef(shape, 3) : at::IntArrayRef(shape + 1, 2), out, dev);
  void* st = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream();
  int rc;
  {
    WithoutGil unlocked;
    rc = api.w8a8(static_cast<const int8_t*>(A->const_data_ptr()), static_cast<const int8_t*>(B->const_data_ptr()),
                  static_cast<const float*>(sb->const_data_ptr()), sa ? static_cast<const float*>(sa->const_data_ptr()) : nullptr,
                  C.mutable_data_ptr(), nullptr, batch, M, N, K, sb_len, sa_len, abi_dt(out), nk ? QGEMM_B_NK : QGEMM_B_KN, nullptr, st);
  }
  if (rc != 0) Py_RETURN_NONE;
  return THPVariable_Wrap(std::move(C));
  QHOST_CATCH
}

// act_quant(x, round_scale) -> (y, s); want_n >= 0: x is [M, want_n] and s comes back as [M]
PyObject* h_act_quant(PyObject*, PyObject* const* args, Py_ssize_t n) {
  QHOST_TRY
  if (n != 3) Py_RETURN_NONE;
  const at::Tensor* x = plain(args[0], at::kBFloat16);
  if (x == nullptr) x = plain(args[0], at::kHalf);
  if (x == nullptr || (args[1] != Py_True && args[1] != Py_False)) Py_RETURN_NONE;
  int64_t want_n;
  if (!plain_int(args[2], &want_n)) Py_RETURN_NONE;
  const int64_t nd = x->dim();
  if (nd != 2 && nd != 3) Py_RETURN_NONE;
  const int64_t N = x->size(-1);
  if (N <= 0 || x->numel() == 0 || (want_n >= 0 && (nd != 2 || N != want_n))) Py_RETURN_NONE;
  const int64_t M = x->numel() / N;
  const int dev = x->get_device();
  c10::cuda::CUDAGuard guard((c10::DeviceIndex)dev);
  at::Tensor y = empty_cuda(x->sizes(), at::kChar, dev);
  const int64_t shape[3] = {x->size(0), nd == 3 ? x->size(1) : 1, 1};
  at::Tensor s = empty_cuda(want_n >= 0 ? at::IntArrayRef(shape, 1) : at::IntArrayRef(shape, (size_t)nd), at::kFloat, dev);
  void* st = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream();
  const int dt = abi_dt(x->scalar_type()), rs = args[1] == Py_True ? 1 : 0;
  int rc;
  {
    WithoutGil unlocked;
    rc = api.act_quant(x->const_data_ptr(), static_cast<int8_t*>(y.mutable_data_ptr()), static_cast<float*>(s.mutable_data_ptr()), M,
                       N, dt, rs, st);
  }
  if (rc != 0) Py_RETURN_NONE;
  PyObject* py = THPVariable_Wrap(std::move(y));
  PyObject* ps = THPVariable_Wrap(std::move(s));
  if (py == nullptr || ps == nullptr) {
    Py_XDECREF(py);
    Py_XDECREF(ps);
    return nullptr;
  }
  PyObject* res = PyTuple_New(2);
  if (res == nullptr) {
    Py_DECREF(py);
    Py_DECREF(ps);
    return nullptr;
  }
  PyTuple_SET_ITEM(res, 0, py);
  PyTuple_SET_ITEM(res, 1, ps);
  return res;
  QHOST_CATCH
}

// w4a16(A, B_packed, scales | None, zeros: int or tensor, group_size, out_dtype | None, zero_mode: int, layout: int,
//       M, N, K) -> C; M >= 0: the factory's static 2-D shape
PyObject* h_w4a16(PyObject*, PyObject* const* args, Py_ssize_t n) {
  QHOST_TRY
  if (n != 11) Py_RETURN_NONE;
  const at::Tensor* A = plain(args[0], at::kHalf);
  if (A == nullptr) A = plain(args[0], at::kBFloat16);
  const at::Tensor* B = plain(args[1], at::kByte);
  if (A == nullptr || B == nullptr || !same_device(*A, B)) Py_RETURN_NONE;
  const ScalarType out = args[5] == Py_None ? A->scalar_type() : float16_kind(args[5]);
  if (out == ScalarType::Undefined) Py_RETURN_NONE;
  const int64_t nd = A->dim();
  if ((nd != 2 && nd != 3) || B->dim() != nd) Py_RETURN_NONE;
  const bool batched = nd == 3;
  const int64_t batch = batched ? A->size(0) : 1, M = A->size(-2), K = A->size(-1), N = B->size(-2);
  if (K % 2 != 0 || B->size(-1) != K / 2 || (batched && B->size(0) != batch)) Py_RETURN_NONE;
  int64_t want_m, zero_mode, layout;
  if (!plain_int(args[8], &want_m) || !plain_int(args[6], &zero_mode) || !plain_int(args[7], &layout)) Py_RETURN_NONE;
  if (want_m >= 0 && (batched || M != want_m || N != as_int(args[9]) || K != as_int(args[10]))) Py_RETURN_NONE;
  if (zero_mode < 0 || layout < 0) Py_RETURN_NONE;
  int64_t group = K;
  int zero = 0;
  const at::Tensor* sc = nullptr;
  const at::Tensor* zt = nullptr;
  if (args[2] != Py_None) {
    if (args[4] != Py_None && PyLong_CheckExact(args[4])) {
      int overflow = 0;
      const long g = PyLong_AsLongAndOverflow(args[4], &overflow);
      if (overflow) Py_RETURN_NONE;
      group = g == -1 ? K : g;
    } else if (args[4] != Py_None) {
      Py_RETURN_NONE;
    }
    if (group <= 0 || K % group != 0) Py_RETURN_NONE;
    auto table = [&](PyObject* o) -> const at::Tensor* {  // [K / group, N] f16, with the batch in front
      const at::Tensor* t = plain(o, at::kHalf);
      if (t == nullptr || t->dim() != nd || t->size(-1) != N || t->size(-2) != K / group || (batched && t->size(0) != batch) ||
          !same_device(*A, t))
        return nullptr;
      return t;
    };
    if ((sc = table(args[2])) == nullptr) Py_RETURN_NONE;
    if (PyLong_CheckExact(args[3])) {
      const int64_t z = as_int(args[3]);
      if (z < 0 || z > 15 || zero_mode == QGEMM_ZERO_RESCALE) Py_RETURN_NONE;
      zero = (int)z;
    } else if ((zt = table(args[3])) == nullptr) {
      Py_RETURN_NONE;
    }
  } else if (!PyLong_CheckExact(args[3])) {
    Py_RETURN_NONE;
  }
  if (batch * M * N == 0) Py_RETURN_NONE;
  const int dev = A->get_device();
  c10::cuda::CUDAGuard guard((c10::DeviceIndex)dev);
  const int64_t need = api.w4a16_ws(batch, M, N, K, group, sc != nullptr, zt != nullptr, (int)zero_mode);
  if (need < 0) Py_RETURN_NONE;
  const int64_t shape[3] = {batch, M, N};
  at::Tensor C = empty_cuda(batched ? at::IntArrayRef(shape, 3) : at::IntArrayRef(shape + 1, 2), out, dev);
  const auto stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev);
  // scratch of this call: handed back to the stream-ordered caching allocator when the call returns
  const at::DataPtr ws = c10::cuda::CUDACachingAllocator::get()->allocate((size_t)(need > 0 ? need : 16));
  int rc;
  {
    WithoutGil unlocked;
    rc = api.w4a16(A->const_data_ptr(), static_cast<const uint8_t*>(B->const_data_ptr()), sc ? sc->const_data_ptr() : nullptr,
                   zt ? zt->const_data_ptr() : nullptr, zero, (int)zero_mode, (int)layout, group, C.mutable_data_ptr(), ws.get(), need,
                   batch, M, N, K, abi_dt(A->scalar_type()), abi_dt(out), nullptr, stream.stream());
  }
  if (rc != 0) Py_RETURN_NONE;
  return THPVariable_Wrap(std::move(C));
  QHOST_CATCH
}

// w4a8(A int8 [M, K], qB, workspace, C, M, N, K) -> True when launched (signed nibbles, int32 out)
// w4a8_aq(X bf16 / f16 [M, K], qB, workspace, C, M, N, K, round_scale) -> scale_a
PyObject* h_w4a8_common(PyObject* const* args, bool quant) {
  const at::Tensor* A = quant ? plain(args[0], at::kBFloat16) : plain(args[0], at::kChar);
  if (A == nullptr && quant) A = plain(args[0], at::kHalf);
  const at::Tensor* B = plain(args[1], at::kByte);
  const at::Tensor* W = plain(args[2], at::kChar);
  const at::Tensor* C = plain(args[3], at::kInt);
  if (A == nullptr || B == nullptr || W == nullptr || C == nullptr) Py_RETURN_NONE;
  const int64_t M = as_int(args[4]), N = as_int(args[5]), K = as_int(args[6]);
  if (M <= 0 || N <= 0 || K <= 0) Py_RETURN_NONE;
  auto is2d = [](const at::Tensor* t, int64_t r, int64_t c) { return t->dim() == 2 && t->size(0) == r && t->size(1) == c; };
  if (!is2d(A, M, K) || !is2d(B, N, K / 2) || !is2d(W, N, K) || !is2d(C, M, N)) Py_RETURN_NONE;
  if (!same_device(*A, B) || !same_device(*A, W) || !same_device(*A, C)) Py_RETURN_NONE;
  const int dev = A->get_device();
  c10::cuda::CUDAGuard guard((c10::DeviceIndex)dev);
  void* st = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream();
  // the caller's output and scratch tensors are written by data pointer, as the ctypes call does
  uint8_t* b = static_cast<uint8_t*>(B->data_ptr());
  int8_t* w = static_cast<int8_t*>(W->data_ptr());
  int rc;
  if (!quant) {
    {
    WithoutGil unlocked;
      rc = api.w4a8(static_cast<const int8_t*>(A->const_data_ptr()), b, w, C->data_ptr(), M, N, K, 1, QGEMM_DT_I32, nullptr, st);
    }
    if (rc != 0) Py_RETURN_NONE;
    Py_RETURN_TRUE;
  }
  if (args[7] != Py_True && args[7] != Py_False) Py_RETURN_NONE;
  at::Tensor s = empty_cuda({M}, at::kFloat, dev);
  const int rs = args[7] == Py_True ? 1 : 0, dt = abi_dt(A->scalar_type());
  {
    WithoutGil unlocked;
    rc = api.w4a8_aq(A->const_data_ptr(), dt, b, w, static_cast<int32_t*>(C->data_ptr()), static_cast<float*>(s.mutable_data_ptr()), rs,
                     M, N, K, 1, nullptr, st);
  }
  if (rc != 0) Py_RETURN_NONE;
  return THPVariable_Wrap(std::move(s));
}
PyObject* h_w4a8(PyObject*, PyObject* const* args, Py_ssize_t n) {
  QHOST_TRY
  if (n != 7) Py_RETURN_NONE;
  return h_w4a8_common(args, false);
  QHOST_CATCH
}
PyObject* h_w4a8_aq(PyObject*, PyObject* const* args, Py_ssize_t n) {
  QHOST_TRY
  if (n != 8) Py_RETURN_NONE;
  return h_w4a8_common(args, true);
  QHOST_CATCH
}

// grouped(A, B, block_metadata, scale, scale_a | None, out_dtype, nk: bool, out | None, total_M, K, groups, blocks) -> C
// total_M >= 0: the factory's static sizes.  Without `out` the rows that no block covers come back as zeros.
PyObject* h_grouped(PyObject*, PyObject* const* args, Py_ssize_t n) {
  QHOST_TRY
  if (n != 12) Py_RETURN_NONE;
  const at::Tensor* A = plain(args[0], at::kChar);
  const at::Tensor* B = plain(args[1], at::kChar);
  const at::Tensor* meta = plain(args[2], at::kInt);
  const at::Tensor* sb = plain(args[3], at::kFloat);
  if (A == nullptr || B == nullptr || meta == nullptr || sb == nullptr) Py_RETURN_NONE;
  const at::Tensor* sa = nullptr;
  if (args[4] != Py_None && (sa = plain(args[4], at::kFloat)) == nullptr) Py_RETURN_NONE;
  const ScalarType out = float16_kind(args[5]);
  if (out == ScalarType::Undefined) Py_RETURN_NONE;
  const bool nk = args[6] == Py_True;
  if (A->dim() != 2 || B->dim() != 3 || meta->dim() != 2 || meta->size(1) != 3) Py_RETURN_NONE;
  const int64_t M = A->size(0), K = A->size(1), G = B->size(0), N = nk ? B->size(1) : B->size(2), blocks = meta->size(0);
  if ((nk ? B->size(2) : B->size(1)) != K || blocks == 0 || M * N == 0) Py_RETURN_NONE;
  int64_t want_rows;
  if (!plain_int(args[8], &want_rows)) Py_RETURN_NONE;
  if (want_rows >= 0 &&
      (M != want_rows || K != as_int(args[9]) || G != as_int(args[10]) || blocks != as_int(args[11])))
    Py_RETURN_NONE;
  const int64_t sb_len = sb->numel(), sa_len = sa ? sa->numel() : 0;
  if ((sb_len != 1 && sb_len != N && sb_len != G * N) || (sa != nullptr && sa_len != M)) Py_RETURN_NONE;
  if (!same_device(*A, B) || !same_device(*A, meta) || !same_device(*A, sb) || (sa && !same_device(*A, sa))) Py_RETURN_NONE;
  const int dev = A->get_device();
  c10::cuda::CUDAGuard guard((c10::DeviceIndex)dev);
  const bool given = args[7] != Py_None;
  at::Tensor C;
  if (given) {
    const at::Tensor* o = plain(args[7], out);
    if (o == nullptr || o->dim() != 2 || o->size(0) != M || o->size(1) != N || !same_device(*A, o)) Py_RETURN_NONE;
    C = *o;
  } else {
    C = empty_cuda({M, N}, out, dev);
  }
  void* st = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream();
  const auto fn = given ? api.w8a8_grouped : api.w8a8_grouped_zeroed;
  int rc;
  {
    WithoutGil unlocked;
    rc = fn(static_cast<const int8_t*>(A->const_data_ptr()), static_cast<const int8_t*>(B->const_data_ptr()),
            static_cast<const float*>(sb->const_data_ptr()), sa ? static_cast<const float*>(sa->const_data_ptr()) : nullptr,
            C.data_ptr(), nullptr, static_cast<const int32_t*>(meta->const_data_ptr()), blocks, G, M, N, K, sb_len, sa_len,
            abi_dt(out), nk ? QGEMM_B_NK : QGEMM_B_KN, nullptr, st);
  }
  if (rc != 0) Py_RETURN_NONE;
  if (given) {
    Py_INCREF(args[7]);
    return args[7];
  }
  return THPVariable_Wrap(std::move(C));
  QHOST_CATCH
}

#define QHOST_FN(name, fn) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(fn)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {QHOST_FN("init", h_init),       QHOST_FN("w8a8", h_w8a8),     QHOST_FN("act_quant", h_act_quant),
                         QHOST_FN("w4a16", h_w4a16),     QHOST_FN("w4a8", h_w4a8),     QHOST_FN("w4a8_aq", h_w4a8_aq),
                         QHOST_FN("grouped", h_grouped), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_qhost", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__qhost(void) { return PyModule_Create(&module); }
