// The common calls of wmma_extension_b200/tcec.py without their interpreter time: one product, a strided batch, packing, and a
// product of packed operands on plain float32 CUDA tensors of the current device.  Anything else (and everything that has to raise)
// returns None, and tcec.py's own code, which accepts and checks it all, takes the call; so does every call before bind().  A status
// other than TCEC_OK comes back as an int.
//
// Calls in a row, us, interpreted and native: 32 x 32 x 32 10.6, 6.7 (the kernel: 6.5); pack_a of 64 x 4096 and the product with a packed
// 4096 x 4096 24.6, 22.7.
#include <ATen/ATen.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <optional>
#include <type_traits>

#include "../../include/tcec.h"

namespace {

// The types of the calls are those of the header that the library was built from.
typedef decltype(&tcec_sgemm) SgemmFn;
typedef decltype(&tcec_sgemm_strided_batched) StridedFn;
typedef decltype(&tcec_pack_a) PackFn;
static_assert(std::is_same<PackFn, decltype(&tcec_pack_b)>::value, "one type packs A and B");
typedef decltype(&tcec_sgemm_packed) PackedFn;
typedef decltype(&tcec_packed_bytes) PackedBytesFn;
SgemmFn g_sgemm = nullptr;
StridedFn g_strided = nullptr;
PackFn g_pack[2] = {nullptr, nullptr};
PackedFn g_packed = nullptr;
PackedBytesFn g_packed_bytes = nullptr;
bool g_bound = false;  // read and written with the GIL held

const at::Tensor* plain_tensor(PyObject* o) { return THPVariable_CheckExact(o) ? &THPVariable_Unpack(o) : nullptr; }
bool cuda_f32(const at::Tensor& t) { return t.is_cuda() && t.scalar_type() == at::kFloat; }
// Of the current device; other devices need a switch.
bool here(const at::Tensor& t) { return t.is_cuda() && t.device().index() == c10::cuda::current_device(); }
// A packed operand or room for one: `bytes` consecutive bytes on the current device, as _require_packed in tcec.py.
bool packed_here(const at::Tensor& t, size_t bytes) { return here(t) && t.is_contiguous() && t.nbytes() >= bytes; }

// Layout and leading dimension of the last two dimensions, as _layout_ld in tcec.py; false: neither.
struct Layout {
  int order;  // 0 row-major, 1 column-major
  long long ld;
};
bool layout_of(const at::Tensor& t, Layout& l) {
  const int64_t d = t.dim(), r = t.size(d - 2), c = t.size(d - 1), s0 = t.stride(d - 2), s1 = t.stride(d - 1);
  if (s1 == 1 && (s0 >= c || r == 1)) l = {0, s0 > c ? s0 : c};
  else if (s0 == 1 && (s1 >= r || c == 1)) l = {1, s1 > r ? s1 : r};
  else return false;
  return true;
}

bool scalar(PyObject* o, float& out) {
  if (PyFloat_CheckExact(o)) {
    out = static_cast<float>(PyFloat_AS_DOUBLE(o));
    return true;
  }
  return false;
}
bool extent(PyObject* o, int& out) {
  if (!PyLong_CheckExact(o)) return false;
  int overflow = 0;
  const long v = PyLong_AsLongAndOverflow(o, &overflow);
  if (overflow || v < 0 || v > 0x7fffffff) return false;
  out = static_cast<int>(v);
  return true;
}
bool fits(int64_t v) { return v >= 0 && v <= 0x7fffffff; }
bool policy_of(PyObject* o, int& out) {
  if (PyUnicode_CheckExact(o)) {
    static const char* const names[] = {"fp16_ec", "tf32_ec", "fp16_no_ec", "tf32_no_ec"};
    for (out = 0; out < 4; ++out)
      if (PyUnicode_CompareWithASCIIString(o, names[out]) == 0) return true;
    return false;
  }
  return extent(o, out);
}

void* stream_here() { return c10::cuda::getCurrentCUDAStream().stream(); }

// The result tensor of a call: `given` as it is, or a new one.
PyObject* answer(int status, PyObject* given, std::optional<at::Tensor>& made) {
  if (status != 0) return PyLong_FromLong(status);
  if (made) return THPVariable_Wrap(std::move(*made));
  Py_INCREF(given);
  return given;
}

// Other threads run while the library is called; back in, an exception on its way too.
class OthersRun {
 public:
  OthersRun() : state_(PyEval_SaveThread()) {}
  ~OthersRun() { PyEval_RestoreThread(state_); }
  OthersRun(const OthersRun&) = delete;
  OthersRun& operator=(const OthersRun&) = delete;

 private:
  PyThreadState* state_;
};

template <class Body>
PyObject* guarded(Body body) {
  try {
    return body();
  } catch (...) {  // a tensor without storage, out of memory: tcec.py meets the same and raises it
    PyErr_Clear();
    Py_RETURN_NONE;
  }
}

// sgemm(a, b, c, alpha, beta, policy) and strided(a, b, c, alpha, beta, policy)
template <int kDims>
PyObject* product(PyObject* const* args, Py_ssize_t n_args) {
  return guarded([&]() -> PyObject* {
    if (n_args != 6 || !g_bound) Py_RETURN_NONE;
    const at::Tensor *a = plain_tensor(args[0]), *b = plain_tensor(args[1]), *c = args[2] == Py_None ? nullptr : plain_tensor(args[2]);
    float alpha, beta;
    int policy;
    if (!a || !b || (!c && args[2] != Py_None) || !scalar(args[3], alpha) || !scalar(args[4], beta) || !policy_of(args[5], policy))
      Py_RETURN_NONE;
    if (a->dim() != kDims || b->dim() != kDims || (c && c->dim() != kDims) || !cuda_f32(*a) || !cuda_f32(*b) || (c && !cuda_f32(*c)) ||
        !here(*a) || !here(*b) || (c && !here(*c)))
      Py_RETURN_NONE;
    const int64_t batch = kDims == 3 ? a->size(0) : 1, m = a->size(kDims - 2), k = a->size(kDims - 1), n = b->size(kDims - 1);
    Layout la, lb, lc;
    if (b->size(kDims - 2) != k || (kDims == 3 && b->size(0) != batch) || !fits(m) || !fits(n) || !fits(k) || !fits(batch) ||
        !layout_of(*a, la) || !layout_of(*b, lb))
      Py_RETURN_NONE;
    if (c && (c->size(kDims - 2) < m || c->size(kDims - 1) < n || (kDims == 3 && c->size(0) < batch))) Py_RETURN_NONE;
    std::optional<at::Tensor> made;
    if (!c) made = kDims == 3 ? at::empty({batch, m, n}, a->options()) : at::empty({m, n}, a->options());
    const at::Tensor& out = c ? *c : *made;
    if (!layout_of(out, lc)) Py_RETURN_NONE;
    const float *pa = static_cast<const float*>(a->data_ptr()), *pb = static_cast<const float*>(b->data_ptr());
    float* pc = static_cast<float*>(out.data_ptr());
    void* stream = stream_here();
    int status;
    {
      const OthersRun others_run;
      if constexpr (kDims == 3)
        status = g_strided(la.order, lb.order, lc.order, m, n, k, alpha, pa, la.ld, a->stride(0), pb, lb.ld, b->stride(0), beta, pc, lc.ld,
                           out.stride(0), batch, policy, stream);
      else
        status = g_sgemm(la.order, lb.order, lc.order, m, n, k, alpha, pa, la.ld, pb, lb.ld, beta, pc, lc.ld, policy, stream);
    }
    return answer(status, args[2], made);
  });
}
PyObject* sgemm(PyObject*, PyObject* const* args, Py_ssize_t n) { return product<2>(args, n); }
PyObject* strided(PyObject*, PyObject* const* args, Py_ssize_t n) { return product<3>(args, n); }

// pack_a(a, policy, out) and pack_b(b, policy, out)
template <int kB>
PyObject* pack(PyObject*, PyObject* const* args, Py_ssize_t n_args) {
  return guarded([&]() -> PyObject* {
    if (n_args != 3 || !g_bound) Py_RETURN_NONE;
    const at::Tensor *x = plain_tensor(args[0]), *given = args[2] == Py_None ? nullptr : plain_tensor(args[2]);
    int policy;
    Layout l;
    if (!x || (!given && args[2] != Py_None) || !policy_of(args[1], policy) || policy > 3 || x->dim() != 2 || !cuda_f32(*x) || !here(*x) ||
        !fits(x->size(0)) || !fits(x->size(1)) || !layout_of(*x, l))
      Py_RETURN_NONE;
    const int first = x->size(0), second = x->size(1);
    std::optional<at::Tensor> made;
    const size_t bytes = kB ? g_packed_bytes(second, first, policy) : g_packed_bytes(first, second, policy);
    if (given && !packed_here(*given, bytes)) Py_RETURN_NONE;
    if (!given) made = at::empty({static_cast<int64_t>(bytes)}, x->options().dtype(at::kByte));
    const float* src = static_cast<const float*>(x->data_ptr());
    void *dst = (given ? *given : *made).data_ptr(), *stream = stream_here();
    int status;
    {
      const OthersRun others_run;
      status = g_pack[kB](l.order, first, second, src, l.ld, dst, policy, stream);
    }
    return answer(status, args[2], made);
  });
}

// sgemm_packed(a_packed, b_packed, m, n, k, c, alpha, beta, policy)
PyObject* sgemm_packed(PyObject*, PyObject* const* args, Py_ssize_t n_args) {
  return guarded([&]() -> PyObject* {
    if (n_args != 9 || !g_bound) Py_RETURN_NONE;
    const at::Tensor *a = plain_tensor(args[0]), *b = plain_tensor(args[1]), *c = args[5] == Py_None ? nullptr : plain_tensor(args[5]);
    int m, n, k, policy;
    float alpha, beta;
    if (!a || !b || (!c && args[5] != Py_None) || !extent(args[2], m) || !extent(args[3], n) || !extent(args[4], k) ||
        !scalar(args[6], alpha) || !scalar(args[7], beta) || !policy_of(args[8], policy))
      Py_RETURN_NONE;
    if (!packed_here(*a, g_packed_bytes(m, k, policy)) || !packed_here(*b, g_packed_bytes(n, k, policy))) Py_RETURN_NONE;
    if (c && (c->dim() != 2 || !cuda_f32(*c) || !here(*c) || c->size(0) < m || c->size(1) < n)) Py_RETURN_NONE;
    std::optional<at::Tensor> made;
    if (!c) made = at::empty({m, n}, a->options().dtype(at::kFloat));
    const at::Tensor& out = c ? *c : *made;
    Layout l;
    if (!layout_of(out, l)) Py_RETURN_NONE;
    const void *pa = a->data_ptr(), *pb = b->data_ptr();
    float* pc = static_cast<float*>(out.data_ptr());
    void* stream = stream_here();
    int status;
    {
      const OthersRun others_run;
      status = g_packed(l.order, m, n, k, alpha, pa, pb, beta, pc, l.ld, policy, stream);
    }
    return answer(status, args[5], made);
  });
}

// bind(sgemm, strided, pack_a, pack_b, packed, packed_bytes): addresses in the library that tcec.py has loaded
PyObject* bind(PyObject*, PyObject* const* args, Py_ssize_t n_args) {
  void* p[6] = {};
  if (n_args != 6) {
    PyErr_SetString(PyExc_TypeError, "bind() takes six addresses");
    return nullptr;
  }
  for (int i = 0; i < 6; ++i) {
    p[i] = PyLong_AsVoidPtr(args[i]);
    if (PyErr_Occurred()) return nullptr;
  }
  g_sgemm = reinterpret_cast<SgemmFn>(p[0]);
  g_strided = reinterpret_cast<StridedFn>(p[1]);
  g_pack[0] = reinterpret_cast<PackFn>(p[2]);
  g_pack[1] = reinterpret_cast<PackFn>(p[3]);
  g_packed = reinterpret_cast<PackedFn>(p[4]);
  g_packed_bytes = reinterpret_cast<PackedBytesFn>(p[5]);
  g_bound = true;
  Py_RETURN_NONE;
}

PyMethodDef kMethods[] = {
    {"bind", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(bind)), METH_FASTCALL, nullptr},
    {"sgemm", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(sgemm)), METH_FASTCALL, nullptr},
    {"strided", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(strided)), METH_FASTCALL, nullptr},
    {"pack_a", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(pack<0>)), METH_FASTCALL, nullptr},
    {"pack_b", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(pack<1>)), METH_FASTCALL, nullptr},
    {"sgemm_packed", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(sgemm_packed)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_binding", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__binding() {
  PyObject* module = PyModule_Create(&kModule);
  // What this was compiled against: tcec.py does not use it with another torch or another header.
  if (module && (PyModule_AddStringConstant(module, "built_for", TCEC_BINDING_BUILT_FOR) != 0)) {
    Py_DECREF(module);
    return nullptr;
  }
  return module;
}
