// The launch wrappers of a step that is not replayed, in C++: checks, the output's allocation and the launch.
//
// Such a step (prompts, portions, decoded rows beside them) passes a few hundred wrappers one after the other.  In Python one took
// 10 to 14 us (the launch itself 2.4, the call through ctypes 1.2, an allocation 1.8, the rest checks and conversions), so that a
// prompt of 100 tokens of the 1.2B sizes took 2.2 ms on the host and 1.0 ms on the device.  Here it takes 6 us, with two launches 8,
// most of it the launches, and such a prompt 1.3 ms on the host.
//
// Every function takes the tensors as they are and returns the output, an int (the status of a launch that was refused), or
// None: something is not as these short checks want it, or the library is not loaded yet.  The caller's Python wrapper then goes
// its long way, which says what is wrong.  Nothing is kept from one call for the next but the addresses of the libraries'
// entry points (bind) and the count of launches.
#include <Python.h>
#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstring>

namespace {

typedef void* S;                                   // the stream
typedef int (*AddRmsnorm)(const void*, const void*, const void*, int, const void*, const void*, int, int, float, int, const void*,
                          const void*, const void*, int, float, const void*, int, int, S);
typedef int (*Skinny)(const void*, const void*, const void*, int, int, int, const void*, int, const void*, int, int, int, int, int, S);
typedef int (*Tc)(const void*, const void*, const void*, int, int, int, const void*, int, int, int, int, const void*, int, S);
typedef long long (*TcScratch)(int, int, int, int);
typedef int (*TcParts)(const void*, const void*, const void*, int, int, int, int*, int, S);
typedef int (*Tc2)(const void*, const void*, const void*, int, int, int, const void*, int, int, int, S);
typedef int (*Simt)(const void*, const void*, const void*, int, int, int, const void*, int, const void*, int, int, int, int, int, S);
typedef int (*Gather)(const void*, const void*, const void*, int, int, int, S);
typedef int (*ShortConv)(const void*, const void*, int, const void*, const void*, const void*, const void*, const void*, const void*,
                         int, int, int, int, int, int, S);
typedef int (*Rope)(const void*, const void*, const void*, int, int, float, const void*, int, const void*, const void*, const void*,
                    int, int, const void*, const void*, int, int, int, int, int, int, S);
typedef int (*Topk)(const void*, const void*, const void*, const void*, int, int, int, int, float, int, int, S);
typedef int (*Sort)(const void*, const void*, const void*, const void*, int, int, int, S);
typedef int (*Swiglu)(const void*, const void*, int, int, int, int, S);

AddRmsnorm f_norm;
Skinny f_skinny;
Tc f_tc;
TcScratch f_tc_scratch;
TcParts f_tc_parts;
Tc2 f_tc2;
Simt f_simt;
Gather f_gather;
ShortConv f_conv;
Rope f_rope;
Topk f_topk;
Sort f_sort;
Swiglu f_swiglu;

struct Entry { const char* name; void** at; } entries[] = {
    {"snk_add_rmsnorm", (void**)&f_norm}, {"snk_gemm_skinny", (void**)&f_skinny}, {"snk_gemm_tc", (void**)&f_tc},
    {"snk_gemm_tc_scratch_bytes", (void**)&f_tc_scratch}, {"snk_gemm_tc_parts", (void**)&f_tc_parts}, {"snk_gemm_tc2", (void**)&f_tc2},
    {"snk_gemm_simt", (void**)&f_simt}, {"snk_gather_rows_bf16", (void**)&f_gather}, {"snk_short_conv", (void**)&f_conv},
    {"snk_qk_norm_rope_cache", (void**)&f_rope}, {"snk_moe_topk", (void**)&f_topk}, {"snk_moe_sort", (void**)&f_sort},
    {"snk_swiglu", (void**)&f_swiglu},
};

long long launches = 0;

const at::ScalarType F32 = at::kFloat, BF16 = at::kBFloat16, I32 = at::kInt;

// The tensor behind `o` where it is a contiguous CUDA tensor, else null (None: null too).
inline const at::Tensor* tensor(PyObject* o) {
  if (!THPVariable_Check(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  return t.is_cuda() && t.is_contiguous() ? &t : nullptr;
}
inline const void* ptr(const at::Tensor* t) { return t ? t->data_ptr() : nullptr; }
inline bool is(const at::Tensor* t, at::ScalarType dtype) { return t && t->scalar_type() == dtype; }
inline bool is(const at::Tensor* t, at::ScalarType dtype, int64_t n) { return is(t, dtype) && t->dim() == 1 && t->size(0) == n; }
inline bool is(const at::Tensor* t, at::ScalarType dtype, int64_t m, int64_t n) {
  return is(t, dtype) && t->dim() == 2 && t->size(0) == m && t->size(1) == n;
}
// A small weight: float32 or the compute dtype.
inline bool small(const at::Tensor* t, at::ScalarType dtype) { return t && (t->scalar_type() == F32 || t->scalar_type() == dtype); }
inline bool aligned(const at::Tensor* t) { return ((uintptr_t)t->data_ptr() & 15) == 0; }
inline long to_int(PyObject* o) { return PyLong_AsLong(o); }
// Whether every number asked for so far was one; if not, the caller's long way meets it again and says so.
inline bool numbers() {
  if (!PyErr_Occurred()) return true;
  PyErr_Clear();
  return false;
}
inline S stream() { return (S)c10::cuda::getCurrentCUDAStream().stream(); }
inline at::Tensor empty(at::IntArrayRef sizes, at::ScalarType dtype, const at::Tensor& like) {
  return at::empty(sizes, at::TensorOptions().dtype(dtype).device(like.device()));
}
// What a wrapper returns: its output, or the status of a launch that was refused.
inline PyObject* result(int status, int n, const at::Tensor& out) {
  if (status) return PyLong_FromLong(status);
  launches += n;
  return THPVariable_Wrap(out);
}

// The interpreter's lock given back for as long as this stands, an exception's way out included: a tensor without memory throws
// where its pointer is asked for, and what catches that speaks to Python.
struct Unlocked {
  PyThreadState* state = PyEval_SaveThread();
  ~Unlocked() { PyEval_RestoreThread(state); }
};
#define LAUNCH(call)   \
  do {                 \
    Unlocked unlocked; \
    status = (call);   \
  } while (0)
#define GUARD_BEGIN try {
// Out of memory has to come out as torch's own error: the caller's long way meets it again and raises that.
#define GUARD_END                                      \
  }                                                    \
  catch (const c10::OutOfMemoryError&) { Py_RETURN_NONE; } \
  catch (const std::exception& e) {                    \
    PyErr_SetString(PyExc_RuntimeError, e.what());     \
    return nullptr;                                    \
  }

// (residual, delta | None, moe y | None, pair_pos | None, weights | None, gamma, eps, bf16, rows | None, w_ahead) -> the norm's rows
PyObject* add_rmsnorm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 10 || !f_norm) Py_RETURN_NONE;
  GUARD_BEGIN
  const at::Tensor *res = tensor(a[0]), *delta = tensor(a[1]), *y = tensor(a[2]), *pos = tensor(a[3]), *w = tensor(a[4]),
                   *gamma = tensor(a[5]), *rows = tensor(a[8]);
  const at::ScalarType dtype = a[7] == Py_True ? BF16 : F32;
  if (!is(res, F32) || res->dim() != 2 || !small(gamma, dtype)) Py_RETURN_NONE;
  const int64_t M = res->size(0), H = res->size(1);
  if (gamma->dim() != 1 || gamma->size(0) != H) Py_RETURN_NONE;
  if (a[1] != Py_None && !is(delta, F32, M, H)) Py_RETURN_NONE;
  int k = 0;
  if (a[2] != Py_None) {
    if (delta || H % 4 || !is(y, F32) || !is(w, F32) || w->dim() != 2 || w->size(0) != M || !is(pos, I32, M * w->size(1))) Py_RETURN_NONE;
    k = (int)w->size(1);
  }
  if (a[8] != Py_None && !is(rows, I32)) Py_RETURN_NONE;
  const int64_t R = rows ? rows->numel() : M;
  const float eps = (float)PyFloat_AsDouble(a[6]);
  const int ahead = a[9] == Py_True;
  if (!numbers()) Py_RETURN_NONE;
  at::Tensor out = empty({R, H}, dtype, *res);
  int status;
  LAUNCH(f_norm(ptr(res), ptr(delta), ptr(gamma), gamma->scalar_type() == F32, ptr(&out), ptr(rows), (int)R, (int)H, eps,
                dtype == BF16, ptr(y), ptr(pos), ptr(w), k, 1.f, nullptr, 0, ahead, stream()));
  return result(status, 1, out);
  GUARD_END
}

// (x, w, out_f32, act, w_ahead, route) -> x . w^T.  route 0: few rows, 1: tcgen05, 2: tcgen05 on pairs of SMs, 3: CUDA cores
// (float32).  act: the code of a gated store (out is then half as wide).
PyObject* linear(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 6) Py_RETURN_NONE;
  GUARD_BEGIN
  const at::Tensor *x = tensor(a[0]), *w = tensor(a[1]);
  const int f32 = (int)to_int(a[2]), act = (int)to_int(a[3]), ahead = (int)to_int(a[4]), route = (int)to_int(a[5]);
  if (!numbers() || !x || !w || x->dim() != 2 || w->dim() != 2) Py_RETURN_NONE;
  const at::ScalarType dtype = route == 3 ? F32 : BF16;
  const int64_t M = x->size(0), K = x->size(1), N = w->size(0);
  if (x->scalar_type() != dtype || w->scalar_type() != dtype || w->size(1) != K || M < 1 || (act && f32)) Py_RETURN_NONE;
  if (route != 3 && (K % 8 || !aligned(x) || !aligned(w))) Py_RETURN_NONE;
  int status = 0, count = 1;
  if (route == 1) {
    if (!f_tc || !f_tc_scratch) Py_RETURN_NONE;
    const long long need = f_tc_scratch((int)M, (int)N, (int)K, 0);
    at::Tensor out = empty({M, act ? N / 2 : N}, f32 ? F32 : BF16, *x), scratch;
    if (need) {
      scratch = empty({(int64_t)need}, at::kByte, *x);
      count = 2;
    }
    LAUNCH(f_tc(ptr(x), ptr(w), ptr(&out), (int)M, (int)N, (int)K, nullptr, 1, (int)((M + 127) / 128), f32, act,
                need ? ptr(&scratch) : nullptr, ahead, stream()));
    return result(status, count, out);
  }
  if (route == 2 ? !f_tc2 : route == 3 ? !f_simt || act : route == 0 ? !f_skinny : true) Py_RETURN_NONE;
  at::Tensor out = empty({M, act ? N / 2 : N}, f32 || route == 3 ? F32 : BF16, *x);
  if (route == 0)
    LAUNCH(f_skinny(ptr(x), ptr(w), ptr(&out), (int)M, (int)N, (int)K, nullptr, 1, nullptr, 1, (int)M, f32, act, ahead, stream()));
  else if (route == 2)
    LAUNCH(f_tc2(ptr(x), ptr(w), ptr(&out), (int)M, (int)N, (int)K, nullptr, 1, f32, act, stream()));
  else
    LAUNCH(f_simt(ptr(x), ptr(w), ptr(&out), (int)M, (int)N, (int)K, nullptr, 1, nullptr, 1, (int)M, 1, 0, ahead, stream()));
  return result(status, 1, out);
  GUARD_END
}

// (x, w, into, w_ahead, route 1 or 2) -> into, float [M, N], to which x . w^T has been added
PyObject* linear_add(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 5) Py_RETURN_NONE;
  GUARD_BEGIN
  const at::Tensor *x = tensor(a[0]), *w = tensor(a[1]), *into = tensor(a[2]);
  const int ahead = (int)to_int(a[3]), route = (int)to_int(a[4]);
  if (!numbers() || !is(x, BF16) || !is(w, BF16) || x->dim() != 2 || w->dim() != 2 || w->size(1) != x->size(1) ||
      !is(into, F32, x->size(0), w->size(0)) || x->size(0) < 1 || x->size(1) % 8 || !aligned(x) || !aligned(w) || !aligned(into)) Py_RETURN_NONE;
  const int M = (int)x->size(0), K = (int)x->size(1), N = (int)w->size(0);
  if (route == 2 ? !f_tc2 : route == 1 ? !f_tc || !f_tc_scratch : true) Py_RETURN_NONE;
  int status, count = 1;
  if (route == 2) {
    LAUNCH(f_tc2(ptr(x), ptr(w), ptr(into), M, N, K, nullptr, 1, 2, 0, stream()));
  } else {
    const long long need = f_tc_scratch(M, N, K, 0);
    at::Tensor scratch;
    if (need) {
      scratch = empty({(int64_t)need}, at::kByte, *x);
      count = 2;
    }
    LAUNCH(f_tc(ptr(x), ptr(w), ptr(into), M, N, K, nullptr, 1, (M + 127) / 128, 2, 0, need ? ptr(&scratch) : nullptr, ahead, stream()));
  }
  return result(status, count, *into);
  GUARD_END
}

// (x, w [G, N, K], offsets, rows | None, div, out_f32, act) -> the grouped product on pairs of SMs of x's rows in sorted order
// (gathered first where `rows` names them)
PyObject* grouped(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 7 || !f_tc2) Py_RETURN_NONE;
  GUARD_BEGIN
  const at::Tensor *x = tensor(a[0]), *w = tensor(a[1]), *offsets = tensor(a[2]), *rows = tensor(a[3]);
  const int div = (int)to_int(a[4]), f32 = (int)to_int(a[5]), act = (int)to_int(a[6]);
  if (!numbers() || !is(x, BF16) || !is(w, BF16) || x->dim() != 2 || w->dim() != 3 || w->size(2) != x->size(1) || !is(offsets, I32, w->size(0) + 1) ||
      (act && f32) || x->size(1) % 8 || !aligned(x) || !aligned(w)) Py_RETURN_NONE;
  const int64_t G = w->size(0), N = w->size(1), K = w->size(2);
  int status = 0, count = 1;
  at::Tensor sorted;
  int64_t M = x->size(0);
  if (a[3] != Py_None) {
    if (!f_gather || !is(rows, I32) || rows->numel() < 1) Py_RETURN_NONE;
    M = rows->numel();
    sorted = empty({M, K}, BF16, *x);
    LAUNCH(f_gather(ptr(x), ptr(&sorted), ptr(rows), div, (int)M, (int)K, stream()));
    if (status) return PyLong_FromLong(status);
    count = 2;
    x = &sorted;
  }
  if (M < 1) Py_RETURN_NONE;
  at::Tensor out = empty({M, act ? N / 2 : N}, f32 ? F32 : BF16, *x);
  LAUNCH(f_tc2(ptr(x), ptr(w), ptr(&out), (int)M, (int)N, (int)K, ptr(offsets), (int)G, f32, act, stream()));
  return result(status, count, out);
  GUARD_END
}

// (bcx, taps, state, cu_seqlens, seg_start, seg_slot, row_seg, w_ahead) -> y
PyObject* short_conv(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 8 || !f_conv) Py_RETURN_NONE;
  GUARD_BEGIN
  const at::Tensor *x = tensor(a[0]), *w = tensor(a[1]), *state = tensor(a[2]), *cu = tensor(a[3]), *start = tensor(a[4]),
                   *slot = tensor(a[5]), *seg = tensor(a[6]);
  if (!x || x->dim() != 2 || x->size(1) % 3 || (x->scalar_type() != F32 && x->scalar_type() != BF16)) Py_RETURN_NONE;
  const at::ScalarType dtype = x->scalar_type();
  const int64_t M = x->size(0), H = x->size(1) / 3;
  if (!small(w, dtype) || w->dim() != 2 || w->size(0) != H || !is(state, dtype) || state->dim() != 3 || state->size(2) != H ||
      state->size(1) != w->size(1) - 1 || !is(start, I32) || !is(seg, I32, M)) Py_RETURN_NONE;
  const int64_t B = start->numel(), L = w->size(1);
  if (!is(start, I32, B) || !is(slot, I32, B) || !is(cu, I32, B + 1)) Py_RETURN_NONE;
  const int ahead = a[7] == Py_True;
  at::Tensor out = empty({M, H}, dtype, *x);
  int status;
  LAUNCH(f_conv(ptr(x), ptr(w), w->scalar_type() == F32, ptr(state), ptr(cu), ptr(start), ptr(slot), ptr(seg), ptr(&out), (int)M,
                (int)B, (int)H, (int)L, dtype == BF16, ahead, stream()));
  return result(status, L > 1 && M != B ? 2 : 1, out);
  GUARD_END
}

// (qkv, q_gamma | None, k_gamma | None, eps, inv_freq | None, rot_dim, positions, row_seg, block_table, page_size, pool, heads,
//  kv heads, head_dim, write_kv) -> q
PyObject* rope(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 15 || !f_rope) Py_RETURN_NONE;
  GUARD_BEGIN
  const at::Tensor *qkv = tensor(a[0]), *qg = tensor(a[1]), *kg = tensor(a[2]), *freq = tensor(a[4]), *at_ = tensor(a[6]),
                   *seg = tensor(a[7]), *table = tensor(a[8]), *pool = tensor(a[10]);
  const int rot = (int)to_int(a[5]), page = (int)to_int(a[9]), nh = (int)to_int(a[11]), nkv = (int)to_int(a[12]), hd = (int)to_int(a[13]);
  const int write = a[14] == Py_True;
  if (!qkv || (qkv->scalar_type() != F32 && qkv->scalar_type() != BF16) || qkv->dim() != 2) Py_RETURN_NONE;
  const at::ScalarType dtype = qkv->scalar_type();
  const int64_t M = qkv->size(0);
  if (qkv->size(1) != (int64_t)(nh + (write ? 2 * nkv : 0)) * hd) Py_RETURN_NONE;
  const bool norm = a[1] != Py_None;
  if (norm && (!small(qg, dtype) || !kg || kg->scalar_type() != qg->scalar_type() || !is(qg, qg->scalar_type(), hd) ||
               !is(kg, qg->scalar_type(), hd))) Py_RETURN_NONE;
  if (a[4] != Py_None && !is(freq, F32, rot / 2)) Py_RETURN_NONE;
  if (!is(at_, I32, M) || !is(seg, I32, M) || !is(table, I32) || table->dim() != 2 || !is(pool, dtype) || pool->dim() != 5 ||
      pool->size(1) != 2 || pool->size(2) != nkv || pool->size(3) != page || pool->size(4) != hd) Py_RETURN_NONE;
  const float eps = (float)PyFloat_AsDouble(a[3]);
  if (!numbers()) Py_RETURN_NONE;
  at::Tensor q = empty({M, nh, hd}, dtype, *qkv);
  int status;
  LAUNCH(f_rope(ptr(qkv), norm ? ptr(qg) : nullptr, norm ? ptr(kg) : nullptr, norm && qg->scalar_type() == F32, norm, eps, ptr(freq),
                freq ? rot : 0, ptr(at_), ptr(seg), ptr(table), (int)table->size(1), page, ptr(pool), ptr(&q), (int)M, nh, nkv, hd, write,
                dtype == BF16, stream()));
  return result(status, 1, q);
  GUARD_END
}

// (x, router, bias | None, top_k, flags, scaling, identity, w_ahead) -> (ids, weights, offsets, pair_pos, sorted_pair): the router of
// many rows, a tcgen05 product split along K whose parts the selection adds, and the sort
PyObject* route_sort(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 8 || !f_tc_parts || !f_tc_scratch || !f_topk || !f_sort) Py_RETURN_NONE;
  GUARD_BEGIN
  const at::Tensor *x = tensor(a[0]), *w = tensor(a[1]), *bias = tensor(a[2]);
  const int k = (int)to_int(a[3]), flags = (int)to_int(a[4]), identity = (int)to_int(a[6]), ahead = (int)to_int(a[7]);
  if (!is(x, BF16) || !is(w, BF16) || x->dim() != 2 || w->dim() != 2 || x->size(1) != w->size(1) || x->size(1) % 8 || !aligned(x) ||
      !aligned(w)) Py_RETURN_NONE;
  const int64_t M = x->size(0), H = x->size(1), E = w->size(0), pairs = M * k;
  if (a[2] != Py_None && !is(bias, F32, E)) Py_RETURN_NONE;
  const long long need = f_tc_scratch((int)M, (int)E, (int)H, 0);
  if (need <= 0) Py_RETURN_NONE;
  const float scaling = (float)PyFloat_AsDouble(a[5]);
  if (!numbers()) Py_RETURN_NONE;
  at::Tensor parts = empty({(int64_t)need}, at::kByte, *x);
  at::Tensor ids = empty({M, k}, I32, *x), wts = empty({M, k}, F32, *x), offsets = empty({E + 1}, I32, *x),
             pos = empty({pairs}, I32, *x), sorted = empty({pairs}, I32, *x);
  int status, planes = 0;
  const S s = stream();
  {
    Unlocked unlocked;
    status = f_tc_parts(ptr(x), ptr(w), ptr(&parts), (int)M, (int)E, (int)H, &planes, ahead, s);
    if (!status) status = f_topk(ptr(&parts), ptr(bias), ptr(&ids), ptr(&wts), (int)M, (int)E, k, flags, scaling, 0, planes, s);
    if (!status) status = f_sort(ptr(&ids), ptr(&offsets), ptr(&pos), ptr(&sorted), (int)pairs, (int)E, (int)E - identity, s);
  }
  if (status) return PyLong_FromLong(status);
  launches += 3;
  PyObject* out = PyTuple_New(5);
  if (!out) return nullptr;
  const at::Tensor* all[5] = {&ids, &wts, &offsets, &pos, &sorted};
  for (int i = 0; i < 5; ++i) PyTuple_SET_ITEM(out, i, THPVariable_Wrap(*all[i]));
  return out;
  GUARD_END
}

// (gate_up, interleaved) -> silu(gate) * up
PyObject* swiglu(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 2 || !f_swiglu || !PyBool_Check(a[1])) Py_RETURN_NONE;       // (1 for True is the long way's)
  GUARD_BEGIN
  const at::Tensor* h = tensor(a[0]);
  if (!h || (h->scalar_type() != F32 && h->scalar_type() != BF16) || h->dim() != 2 || h->size(1) % 2) Py_RETURN_NONE;
  at::Tensor out = empty({h->size(0), h->size(1) / 2}, h->scalar_type(), *h);
  int status;
  LAUNCH(f_swiglu(ptr(h), ptr(&out), (int)h->size(0), (int)(h->size(1) / 2), a[1] == Py_True, h->scalar_type() == BF16, stream()));
  return result(status, 1, out);
  GUARD_END
}

// (name, address): an entry point of a loaded library; names that nothing here calls are ignored
PyObject* bind(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 2) Py_RETURN_NONE;
  const char* name = PyUnicode_AsUTF8(a[0]);
  if (!name) return nullptr;
  for (const Entry& e : entries)
    if (!strcmp(e.name, name)) *e.at = PyLong_AsVoidPtr(a[1]);
  Py_RETURN_NONE;
}

PyObject* count(PyObject*, PyObject* const*, Py_ssize_t) { return PyLong_FromLongLong(launches); }

#define METHOD(f) {#f, (PyCFunction)(void (*)(void))f, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {METHOD(add_rmsnorm), METHOD(linear), METHOD(linear_add), METHOD(grouped), METHOD(short_conv), METHOD(rope), METHOD(route_sort),
                         METHOD(swiglu), METHOD(bind), METHOD(count), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "snk_host", nullptr, -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit_snk_host() { return PyModule_Create(&module); }
