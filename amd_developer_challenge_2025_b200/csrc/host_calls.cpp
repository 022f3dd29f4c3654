// The per-call host work of the Python entry points, as a CPython module: the checks of the five (or two) tensors, the
// current stream, and the call of the C ABI. The operator is called in tight loops on problems that run for a few
// microseconds; the same checks and the argument conversion of a ctypes call took 12 to 15 us in Python and take about
// one here. Every call is checked in full, nothing is remembered between calls.
//
// A function returns True when the kernel has been launched. It returns False, having done nothing, for anything but
// the plain case (a check that fails, tensors that are not plain CUDA tensors on the current device, a workspace that
// does not exist yet, a code other than 0 from the library): the caller then goes through the checks in Python, which
// raise the error or handle the case.

#include <ATen/core/Tensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include "b200_fp8_mm.h"
#include "b200_mla_consumers.h"

namespace {

decltype(&b200_fp8_mm_strided) g_strided = nullptr;
decltype(&b200_fp8_mm_grouped) g_grouped = nullptr;
decltype(&b200_mla_rope) g_rope = nullptr;
decltype(&b200_mla_div_softmax) g_softmax = nullptr;

constexpr int64_t kScaleBlock = 128;

// The library's call without the GIL: a launch can block while the device's queue is full. (The caller holds the
// tensors; everything the call needs has been read out of them before.)
template <typename F, typename... Args>
bool launched(F fn, Args... args) {
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = fn(args...);
  Py_END_ALLOW_THREADS
  return rc == 0;
}

const at::Tensor* plain_tensor(PyObject* o) {
  return THPVariable_CheckExact(o) ? &THPVariable_Unpack(o) : nullptr;
}

// A strided CUDA tensor of the given type and rank on device `dev`.
bool is_cuda(const at::Tensor& t, c10::ScalarType type, int64_t rank, c10::DeviceIndex dev) {
  return t.is_cuda() && t.layout() == c10::kStrided && t.scalar_type() == type && t.dim() == rank && t.get_device() == dev;
}

bool aligned16(const at::Tensor& t) { return reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0; }

bool fits_int(int64_t v) { return v >= 0 && v <= 0x7fffffff; }

// The entry of `dict` for `key` (consumed), as a tensor; null when there is none.
const at::Tensor* lookup(PyObject* dict, PyObject* key) {
  if (key == nullptr) return nullptr;
  PyObject* v = PyDict_GetItemWithError(dict, key);  // borrowed
  Py_DECREF(key);
  return v != nullptr ? plain_tensor(v) : nullptr;
}

// fp8_mm(a, b, a_scale, b_scale, c, n_phase, workspaces, status[, address of the forced b200_fp8_mm_plan or 0])
bool run_fp8_mm(PyObject* const* args) {
  const at::Tensor *a = plain_tensor(args[0]), *b = plain_tensor(args[1]), *as = plain_tensor(args[2]),
                   *bs = plain_tensor(args[3]), *c = plain_tensor(args[4]);
  if (!a || !b || !as || !bs || !c || !PyIndex_Check(args[5])) return false;
  const c10::DeviceIndex dev = c10::cuda::current_device();
  if (!is_cuda(*a, at::kFloat8_e4m3fn, 2, dev) || !is_cuda(*b, at::kFloat8_e4m3fn, 2, dev) ||
      !is_cuda(*as, at::kFloat, 2, dev) || !is_cuda(*bs, at::kFloat, 2, dev) || !is_cuda(*c, at::kBFloat16, 2, dev))
    return false;
  const Py_ssize_t phase = PyNumber_AsSsize_t(args[5], nullptr);
  if (phase < 0 || phase >= kScaleBlock) return false;
  const auto* plan = static_cast<const b200_fp8_mm_plan*>(args[8] != nullptr ? PyLong_AsVoidPtr(args[8]) : nullptr);
  if (PyErr_Occurred()) return false;
  const int64_t m = a->size(0), k = a->size(1), n = b->size(0);
  if (m <= 0 || n <= 0 || k <= 0 || !fits_int(m) || !fits_int(n) || !fits_int(k) || k % kScaleBlock != 0) return false;
  const int64_t kb = k / kScaleBlock, nb = (n + phase + kScaleBlock - 1) / kScaleBlock;
  if (b->size(1) != k || c->size(0) != m || c->size(1) != n || as->size(0) != m || as->size(1) != kb ||
      bs->size(0) != nb || bs->size(1) != kb)
    return false;
  const int64_t a0 = a->stride(0), a1 = a->stride(1), b0 = b->stride(0), b1 = b->stride(1);
  const bool a_k = a1 == 1 && a0 >= k, b_k = b1 == 1 && b0 >= k;
  if (!a_k && !(a0 == 1 && a1 >= m)) return false;
  if (!b_k && !(b0 == 1 && b1 >= n)) return false;
  if ((a_k ? a0 : a1) % 16 != 0 || (b_k ? b0 : b1) % 16 != 0 || !aligned16(*a) || !aligned16(*b)) return false;
  if (c->stride(1) != 1) return false;
  cudaStream_t stream = c10::cuda::getCurrentCUDAStream(dev).stream();
  const at::Tensor* st = lookup(args[7], PyLong_FromLong(dev));
  if (st == nullptr) return false;
  const at::Tensor* ws = lookup(args[6], Py_BuildValue("(iK)", static_cast<int>(dev),
                                                       static_cast<unsigned long long>(reinterpret_cast<uintptr_t>(stream))));
  return launched(g_strided, a->data_ptr(), b->data_ptr(), static_cast<const float*>(as->data_ptr()),
                   static_cast<const float*>(bs->data_ptr()), c->data_ptr(), static_cast<int>(m), static_cast<int>(n),
                   static_cast<int>(k), a0, a1, b0, b1, as->stride(0), as->stride(1), bs->stride(0), bs->stride(1),
                   c->stride(0), static_cast<int>(phase), ws ? ws->data_ptr() : nullptr,
                   ws ? static_cast<size_t>(ws->numel()) : 0, static_cast<int*>(st->data_ptr()), stream,
                  plan);
}

// fp8_mm_grouped(a, b, a_scale, b_scale, c, m_valid or None, status)
bool run_grouped(PyObject* const* args) {
  const at::Tensor *a = plain_tensor(args[0]), *b = plain_tensor(args[1]), *as = plain_tensor(args[2]),
                   *bs = plain_tensor(args[3]), *c = plain_tensor(args[4]);
  if (!a || !b || !as || !bs || !c) return false;
  const c10::DeviceIndex dev = c10::cuda::current_device();
  if (!is_cuda(*a, at::kFloat8_e4m3fn, 3, dev) || !is_cuda(*b, at::kFloat8_e4m3fn, 3, dev) ||
      !is_cuda(*as, at::kFloat, 3, dev) || !is_cuda(*bs, at::kFloat, 3, dev) || !is_cuda(*c, at::kBFloat16, 3, dev))
    return false;
  const int64_t g = a->size(0), m = a->size(1), k = a->size(2), n = b->size(1);
  if (g <= 0 || m <= 0 || n <= 0 || k <= 0 || !fits_int(g) || !fits_int(m) || !fits_int(n) || !fits_int(k) ||
      k % kScaleBlock != 0)
    return false;
  const int64_t kb = k / kScaleBlock, nb = (n + kScaleBlock - 1) / kScaleBlock;
  if (b->size(0) != g || b->size(2) != k || c->size(0) != g || c->size(1) != m || c->size(2) != n || as->size(0) != g ||
      as->size(1) != m || as->size(2) != kb || bs->size(0) != g || bs->size(1) != nb || bs->size(2) != kb)
    return false;
  if (a->stride(2) != 1 || b->stride(2) != 1 || c->stride(2) != 1) return false;
  if (a->stride(1) % 16 != 0 || a->stride(0) % 16 != 0 || b->stride(1) % 16 != 0 || b->stride(0) % 16 != 0 ||
      !aligned16(*a) || !aligned16(*b))
    return false;
  const int* rows = nullptr;
  if (args[5] != Py_None) {
    const at::Tensor* mv = plain_tensor(args[5]);
    if (!mv || !is_cuda(*mv, at::kInt, 1, dev) || mv->size(0) != g || !mv->is_contiguous()) return false;
    rows = static_cast<const int*>(mv->data_ptr());
  }
  const at::Tensor* st = lookup(args[6], PyLong_FromLong(dev));
  if (st == nullptr) return false;
  cudaStream_t stream = c10::cuda::getCurrentCUDAStream(dev).stream();
  return launched(g_grouped, a->data_ptr(), b->data_ptr(), static_cast<const float*>(as->data_ptr()),
                   static_cast<const float*>(bs->data_ptr()), c->data_ptr(), static_cast<int>(g), static_cast<int>(m),
                   static_cast<int>(n), static_cast<int>(k), a->stride(1), a->stride(0), b->stride(1), b->stride(0),
                   as->stride(0), as->stride(1), as->stride(2), bs->stride(0), bs->stride(1), bs->stride(2), c->stride(1),
                   c->stride(0), rows, static_cast<int*>(st->data_ptr()),
                   stream, static_cast<const b200_fp8_mm_plan*>(nullptr));
}

// Reads `count` Python ints; false when one is none or does not fit `limit`.
bool ints(PyObject* const* args, int count, long long limit, long long* out) {
  for (int i = 0; i < count; ++i) {
    if (!PyLong_CheckExact(args[i])) return false;
    int overflow = 0;
    out[i] = PyLong_AsLongLongAndOverflow(args[i], &overflow);  // (beyond 64 bits the value itself would read as -1)
    if (overflow != 0 || out[i] > limit || out[i] < -limit) return false;
  }
  return true;
}

// Whether the elements off + [0, span1] + [0, span2] + [0, row) lie inside the bf16 tensor's storage (spans of either sign).
bool inside(const at::Tensor& t, long long off, long long span1, long long span2, long long row) {
  const long long first = off + (span1 < 0 ? span1 : 0) + (span2 < 0 ? span2 : 0);
  const long long last = off + (span1 > 0 ? span1 : 0) + (span2 > 0 ? span2 : 0) + row - 1;
  return t.storage_offset() + first >= 0 && t.storage_offset() + last < static_cast<long long>(t.storage().nbytes() / 2);
}

// mla_decode(x, y, pos, xoff, yoff, d0, d1, d2, xs1, xs2, ys1, ys2)
bool run_rope(PyObject* const* args) {
  const at::Tensor *x = plain_tensor(args[0]), *y = plain_tensor(args[1]);
  long long v[10];
  // (40 bits: the products below stay inside 64 bits once d0, d1 and d2 are known to fit 20)
  if (!x || !y || !ints(args + 2, 10, 1ll << 40, v)) return false;
  const long long pos = v[0], xoff = v[1], yoff = v[2], d0 = v[3], d1 = v[4], d2 = v[5], xs1 = v[6], xs2 = v[7],
                  ys1 = v[8], ys2 = v[9];
  const c10::DeviceIndex dev = c10::cuda::current_device();
  if (!x->is_cuda() || !y->is_cuda() || x->get_device() != dev || y->get_device() != dev ||
      x->layout() != c10::kStrided || y->layout() != c10::kStrided || x->scalar_type() != at::kBFloat16 ||
      y->scalar_type() != at::kBFloat16)
    return false;
  if (d0 <= 0 || d1 <= 0 || d2 <= 0 || d2 % 2 != 0 || d0 > (1 << 20) || d1 > (1 << 20) || d2 > (1 << 20) ||
      pos > 0x7fffffff || pos < -0x7fffffff || xoff < 0 || yoff < 0)
    return false;
  if (!inside(*x, xoff, (d0 - 1) * xs1, (d1 - 1) * xs2, d2) || !inside(*y, yoff, (d0 - 1) * ys1, (d1 - 1) * ys2, d2)) return false;
  cudaStream_t stream = c10::cuda::getCurrentCUDAStream(dev).stream();
  return launched(g_rope, static_cast<char*>(x->data_ptr()) + 2 * xoff, static_cast<char*>(y->data_ptr()) + 2 * yoff,
                static_cast<int>(pos), static_cast<int>(d0), static_cast<int>(d1), static_cast<int>(d2), xs1, xs2, ys1,
                ys2, stream);
}

// div_softmax(qk, bs, nh, sl, dnope, drope)
bool run_softmax(PyObject* const* args) {
  const at::Tensor* t = plain_tensor(args[0]);
  long long v[5];
  if (!t || !ints(args + 1, 5, 1 << 20, v)) return false;
  const c10::DeviceIndex dev = c10::cuda::current_device();
  if (!t->is_cuda() || t->get_device() != dev || t->layout() != c10::kStrided || t->scalar_type() != at::kBFloat16 ||
      !t->is_contiguous())
    return false;
  if (v[0] <= 0 || v[1] <= 0 || v[2] <= 0 || t->numel() != v[0] * v[1] * v[2]) return false;
  cudaStream_t stream = c10::cuda::getCurrentCUDAStream(dev).stream();
  return launched(g_softmax, t->data_ptr(), static_cast<int>(v[0]), static_cast<int>(v[1]), static_cast<int>(v[2]),
                   static_cast<int>(v[3]), static_cast<int>(v[4]), stream);
}

// A C++ exception (a tensor without storage, a device that is gone) is "not the plain case" too.
// The last `Optional` of the N arguments may be left out (null).
template <bool (*F)(PyObject* const*), Py_ssize_t N, Py_ssize_t Optional = 0>
PyObject* entry(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  bool done = false;
  if (nargs <= N && nargs >= N - Optional) {
    PyObject* all[N] = {};
    for (Py_ssize_t i = 0; i < nargs; ++i) all[i] = args[i];
    try {
      done = F(all);
    } catch (...) {
      done = false;
    }
    if (PyErr_Occurred()) {
      PyErr_Clear();
      done = false;
    }
  }
  return PyBool_FromLong(done);
}

// bind(strided, grouped, rope, softmax): addresses of the loaded library's functions.
PyObject* bind(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  void* f[4];
  if (nargs != 4) {
    PyErr_SetString(PyExc_TypeError, "bind takes four addresses");
    return nullptr;
  }
  for (int i = 0; i < 4; ++i) {
    f[i] = PyLong_AsVoidPtr(args[i]);
    if (PyErr_Occurred()) return nullptr;
  }
  g_strided = reinterpret_cast<decltype(g_strided)>(f[0]);
  g_grouped = reinterpret_cast<decltype(g_grouped)>(f[1]);
  g_rope = reinterpret_cast<decltype(g_rope)>(f[2]);
  g_softmax = reinterpret_cast<decltype(g_softmax)>(f[3]);
  Py_RETURN_NONE;
}

template <PyObject* (*F)(PyObject*, PyObject* const*, Py_ssize_t)>
PyCFunction fast() {
  return reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(F));
}

PyMethodDef methods[] = {
    {"bind", fast<bind>(), METH_FASTCALL, nullptr},
    {"fp8_mm", fast<entry<run_fp8_mm, 9, 1>>(), METH_FASTCALL, nullptr},
    {"fp8_mm_grouped", fast<entry<run_grouped, 7>>(), METH_FASTCALL, nullptr},
    {"mla_decode", fast<entry<run_rope, 12>>(), METH_FASTCALL, nullptr},
    {"div_softmax", fast<entry<run_softmax, 6>>(), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host() { return PyModule_Create(&module); }
