// CPython module `_q4torch`: the products of one quant linear as one native call each, on torch tensors.
//
// A call of the module costs the host more than the kernel takes on the GPU as soon as the rows are few: checked,
// allocated and marshalled from Python, one projection of one token took 19 us (its kernel: 4.2 us) and one projection
// of a 77-token prompt 42 us (20 us).  Here the checks that protect memory, the allocation of the output, the stream
// lookup and the library call are one C++ function; what is left in Python is the choice of the product.
//
// The module does not link against the CUDA library: `bind` receives the addresses of its entry points.  A function
// returns None - having done nothing - for operands it does not take (another dtype, not contiguous, shapes that do
// not describe one layer): the caller then takes the general path, which reports what is wrong.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../../include/q4b200.h"

namespace {

struct Entry {
  decltype(&q4_gemv) gemv;
  decltype(&q4_gemm_fwd_residual) fwd;
  decltype(&q4_gemm_bwd_table) bwd_table;
  decltype(&q4_gemm_bwd) bwd;
  decltype(&q4_swiglu_fwd) swiglu;
  decltype(&q4_last_error_string) error;
  decltype(&q4_gemm_fwd_v1) v1;
} g = {};

// A tensor argument, or null for None (and for anything that is no tensor).
const at::Tensor* tensor(PyObject* o) { return THPVariable_Check(o) ? &THPVariable_Unpack(o) : nullptr; }
bool plain(const at::Tensor& t, at::ScalarType dt, int dev) {
  return t.is_cuda() && t.scalar_type() == dt && t.get_device() == dev && t.is_contiguous();
}
// `t` has the leading dimensions of `x` and `cols` columns (not merely as many elements: the same numbers in another
// shape are another matrix).
bool rows_like(const at::Tensor& t, const at::Tensor& x, int64_t cols) {
  return t.dim() == x.dim() && t.size(-1) == cols && t.sizes().slice(0, t.dim() - 1) == x.sizes().slice(0, x.dim() - 1);
}
bool vector_of(const at::Tensor& t, int64_t n) { return t.dim() == 1 && t.size(0) == n; }
bool aligned(const at::Tensor& t) { return (uintptr_t)t.data_ptr() % 16 == 0; }
void* ptr(const at::Tensor* t) { return t ? t->data_ptr() : nullptr; }

PyObject* failed(const char* what, int rc) {
  return PyErr_Format(PyExc_RuntimeError, "q4b200 %s failed (%d): %s", what, rc, g.error());
}

// The packed tensors describe one layer [K, N] on device `dev`; groups out.  v1: one scale and one fp16 zero per column.
bool layer_ok(const at::Tensor& qw, const at::Tensor& sc, const at::Tensor& zr, bool v1, int dev, int64_t* K, int64_t* N, int64_t* G) {
  if (qw.dim() != 2 || !plain(qw, at::kInt, dev) || !plain(sc, at::kHalf, dev)) return false;
  *K = qw.size(0) * 8; *N = qw.size(1);
  if (v1) {
    *G = 1;
    return plain(zr, at::kHalf, dev) && sc.numel() == *N && zr.numel() == *N;
  }
  if (sc.dim() != 2 || zr.dim() != 2 || !plain(zr, at::kInt, dev)) return false;
  *G = sc.size(0);
  return sc.size(1) == *N && zr.size(0) == *G && zr.size(1) * 8 == *N;
}

at::Tensor new_rows(const at::Tensor& x, int64_t cols) {
  at::DimVector shape(x.sizes().begin(), x.sizes().end());
  shape.back() = cols;
  return at::empty(shape, x.options());
}

// gemv(x, qweight, scales, zeros, g_idx | None, bias | None, groupsize, flags, workspace) -> y | None:
// x [..., K] fp16 of 1..16 rows in all
PyObject* py_gemv(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const at::Tensor *x = nullptr, *qw, *sc, *zr, *gi, *bi, *ws;
  if (n != 9 || !(x = tensor(a[0])) || !(qw = tensor(a[1])) || !(sc = tensor(a[2])) || !(zr = tensor(a[3])) || !(ws = tensor(a[8]))) Py_RETURN_NONE;
  gi = tensor(a[4]); bi = tensor(a[5]);
  const long groupsize = PyLong_AsLong(a[6]), flags = PyLong_AsLong(a[7]);
  if (PyErr_Occurred()) return nullptr;
  if (!x->is_cuda()) Py_RETURN_NONE;
  const int dev = x->get_device();
  int64_t K, N, G;
  if (!plain(*x, at::kHalf, dev) || x->dim() < 1 || !layer_ok(*qw, *sc, *zr, flags & Q4_GEMV_V1, dev, &K, &N, &G) || x->size(-1) != K) Py_RETURN_NONE;
  if (gi && (!plain(*gi, at::kInt, dev) || gi->numel() < K)) Py_RETURN_NONE;
  if (bi && (!plain(*bi, at::kHalf, dev) || !vector_of(*bi, N))) Py_RETURN_NONE;
  const int64_t M = K ? x->numel() / K : 0;
  if (M < 1 || M > 16 || !ws->is_cuda() || ws->get_device() != dev) Py_RETURN_NONE;
  const c10::cuda::CUDAGuard guard(dev);
  at::Tensor y = new_rows(*x, N);
  const int rc = g.gemv(x->data_ptr(), (const int32_t*)qw->data_ptr(), y.data_ptr(), sc->data_ptr(), (const int32_t*)zr->data_ptr(),
                        (const int32_t*)ptr(gi), ptr(bi), (int)M, (int)K, (int)N, (int)G, (int)groupsize, Q4_F16, (unsigned)flags,
                        ws->data_ptr(), (size_t)ws->numel(), c10::cuda::getCurrentCUDAStream(dev).stream());
  if (rc) return failed("gemv", rc);
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

// gemm(x, qweight, out | None, scales, zeros, g_idx, bias | None, residual | None, lora_u | None, lora_w | None, transpose,
//      zero_terms | None, sequential_groupsize, workspace) -> out | None: x [..., K] (transpose: [..., N]) fp16
PyObject* py_gemm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const at::Tensor *x = nullptr, *qw, *sc, *zr, *gi, *ws;
  if (n != 14 || !(x = tensor(a[0])) || !(qw = tensor(a[1])) || !(sc = tensor(a[3])) || !(zr = tensor(a[4])) || !(gi = tensor(a[5])) ||
      !(ws = tensor(a[13]))) Py_RETURN_NONE;
  const at::Tensor *given = tensor(a[2]), *bi = tensor(a[6]), *res = tensor(a[7]), *lu = tensor(a[8]), *lw = tensor(a[9]), *zt = tensor(a[11]);
  const int transpose = PyObject_IsTrue(a[10]);
  const long seq = PyLong_AsLong(a[12]);
  if (PyErr_Occurred()) return nullptr;
  if (!x->is_cuda()) Py_RETURN_NONE;
  const int dev = x->get_device();
  int64_t K, N, G;
  if (!plain(*x, at::kHalf, dev) || x->dim() < 1 || !layer_ok(*qw, *sc, *zr, false, dev, &K, &N, &G)) Py_RETURN_NONE;
  const int64_t inner = transpose ? N : K, outer = transpose ? K : N;
  if (inner == 0 || x->size(-1) != inner || !plain(*gi, at::kInt, dev) || gi->numel() < K) Py_RETURN_NONE;
  const int64_t M = x->numel() / inner;
  if (M < 1 || M > INT32_MAX) Py_RETURN_NONE;
  if (given && (!plain(*given, at::kHalf, dev) || !rows_like(*given, *x, outer))) Py_RETURN_NONE;
  if (bi && (transpose || !plain(*bi, at::kHalf, dev) || !vector_of(*bi, N))) Py_RETURN_NONE;
  if (res && (transpose || !plain(*res, at::kHalf, dev) || !rows_like(*res, *x, N) || !aligned(*res))) Py_RETURN_NONE;
  int64_t r = 0;
  if (lu) {
    if (!lw || lw->dim() != 2) Py_RETURN_NONE;
    r = lw->size(transpose ? 0 : 1);
    if (!plain(*lu, at::kHalf, dev) || lu->dim() != 2 || lu->size(0) != M || lu->size(1) != 64 || !plain(*lw, at::kHalf, dev) || lw->size(transpose ? 1 : 0) != outer) Py_RETURN_NONE;
  }
  if (zt && (!plain(*zt, at::kHalf, dev) || zt->numel() != G * N)) Py_RETURN_NONE;
  if (!ws->is_cuda() || ws->get_device() != dev) Py_RETURN_NONE;
  const c10::cuda::CUDAGuard guard(dev);
  at::Tensor out = given ? *given : new_rows(*x, outer);
  const int32_t *qwp = (const int32_t*)qw->data_ptr(), *zrp = (const int32_t*)zr->data_ptr(), *gip = (const int32_t*)gi->data_ptr();
  void* const st = c10::cuda::getCurrentCUDAStream(dev).stream();
  int rc;
  if (!transpose)
    rc = g.fwd(x->data_ptr(), qwp, out.data_ptr(), sc->data_ptr(), zrp, ptr(zt), gip, ptr(bi), ptr(res), ptr(lu), ptr(lu ? lw : nullptr), (int)r,
               (int)M, (int)K, (int)N, (int)G, zt ? (int)seq : 0, ws->data_ptr(), (size_t)ws->numel(), st);
  else if (zt)
    rc = g.bwd_table(x->data_ptr(), qwp, out.data_ptr(), sc->data_ptr(), zrp, zt->data_ptr(), gip, ptr(lu), ptr(lu ? lw : nullptr), (int)r,
                     (int)M, (int)K, (int)N, (int)G, ws->data_ptr(), (size_t)ws->numel(), st);
  else
    rc = g.bwd(x->data_ptr(), qwp, out.data_ptr(), sc->data_ptr(), zrp, gip, ptr(lu), ptr(lu ? lw : nullptr), (int)r,
               (int)M, (int)K, (int)N, (int)G, ws->data_ptr(), (size_t)ws->numel(), st);
  if (rc) return failed("gemm", rc);
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// gemm_v1(x, qweight, scales, zeros, bias | None, residual | None, workspace) -> y | None: a layer of the first format;
// x [..., K] fp16
PyObject* py_gemm_v1(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const at::Tensor *x = nullptr, *qw, *sc, *zr, *ws;
  if (n != 7 || !(x = tensor(a[0])) || !(qw = tensor(a[1])) || !(sc = tensor(a[2])) || !(zr = tensor(a[3])) || !(ws = tensor(a[6]))) Py_RETURN_NONE;
  const at::Tensor *bi = tensor(a[4]), *res = tensor(a[5]);
  if (!x->is_cuda()) Py_RETURN_NONE;
  const int dev = x->get_device();
  int64_t K, N, G;
  if (!plain(*x, at::kHalf, dev) || x->dim() < 1 || !layer_ok(*qw, *sc, *zr, true, dev, &K, &N, &G)) Py_RETURN_NONE;
  if (K == 0 || N == 0 || K % 128 || N % 256 || x->size(-1) != K) Py_RETURN_NONE;
  const int64_t M = x->numel() / K;
  if (M < 1 || M > INT32_MAX) Py_RETURN_NONE;
  if (bi && (!plain(*bi, at::kHalf, dev) || !vector_of(*bi, N))) Py_RETURN_NONE;
  if (res && (!plain(*res, at::kHalf, dev) || !rows_like(*res, *x, N))) Py_RETURN_NONE;
  for (const at::Tensor* t : {x, qw, sc, zr, res})                 // (the bias is read by the element)
    if (t && !aligned(*t)) Py_RETURN_NONE;
  if (!ws->is_cuda() || ws->get_device() != dev) Py_RETURN_NONE;
  const c10::cuda::CUDAGuard guard(dev);
  at::Tensor out = new_rows(*x, N);
  const int rc = g.v1(x->data_ptr(), (const int32_t*)qw->data_ptr(), out.data_ptr(), sc->data_ptr(), zr->data_ptr(), ptr(bi), ptr(res),
                      (int)M, (int)K, (int)N, ws->data_ptr(), (size_t)ws->numel(), c10::cuda::getCurrentCUDAStream(dev).stream());
  if (rc) return failed("gemm_v1", rc);
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// swiglu(gu) -> silu(gate) * up | None for gu = [..., gate | up] fp16 (no gradient)
PyObject* py_swiglu(PyObject*, PyObject* arg) {
  HANDLE_TH_ERRORS
  const at::Tensor* gu = tensor(arg);
  if (!gu || !gu->is_cuda() || !plain(*gu, at::kHalf, gu->get_device()) || gu->dim() < 1 || gu->numel() == 0 || gu->size(-1) % 16 ||
      (uintptr_t)gu->data_ptr() % 16) Py_RETURN_NONE;
  const int dev = gu->get_device();
  const int64_t I = gu->size(-1) / 2, M = gu->numel() / (2 * I);
  const c10::cuda::CUDAGuard guard(dev);
  at::Tensor y = new_rows(*gu, I);
  const char* base = (const char*)gu->data_ptr();
  const int rc = g.swiglu(base, base + 2 * I, y.data_ptr(), (int)M, (int)I, (int)(2 * I), c10::cuda::getCurrentCUDAStream(dev).stream());
  if (rc) return failed("swiglu", rc);
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

// bind(addresses of q4_gemv, q4_gemm_fwd_residual, q4_gemm_bwd_table, q4_gemm_bwd, q4_swiglu_fwd, q4_last_error_string, q4_gemm_fwd_v1)
PyObject* py_bind(PyObject*, PyObject* const* a, Py_ssize_t n) {
  void* p[7];
  if (n != 7) { PyErr_SetString(PyExc_TypeError, "bind takes 7 addresses"); return nullptr; }
  for (int i = 0; i < 7; ++i) {
    p[i] = PyLong_AsVoidPtr(a[i]);
    if (!p[i]) { if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "bind: null address"); return nullptr; }
  }
  g.gemv = (decltype(g.gemv))p[0]; g.fwd = (decltype(g.fwd))p[1]; g.bwd_table = (decltype(g.bwd_table))p[2];
  g.bwd = (decltype(g.bwd))p[3]; g.swiglu = (decltype(g.swiglu))p[4]; g.error = (decltype(g.error))p[5]; g.v1 = (decltype(g.v1))p[6];
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"bind", (PyCFunction)(void (*)(void))py_bind, METH_FASTCALL, "addresses of the library's entry points"},
    {"gemv", (PyCFunction)(void (*)(void))py_gemv, METH_FASTCALL, "decode product of 1..16 rows"},
    {"gemm", (PyCFunction)(void (*)(void))py_gemm, METH_FASTCALL, "fused large-M product"},
    {"gemm_v1", (PyCFunction)(void (*)(void))py_gemm_v1, METH_FASTCALL, "fused large-M forward of a layer of the first format"},
    {"swiglu", py_swiglu, METH_O, "silu(gate) * up of a fused gate_up output"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_q4torch", nullptr, -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit__q4torch(void) { return PyModule_Create(&module); }
