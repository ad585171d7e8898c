// The host side of the operator calls, between matconvnet_b200/nn.py and the C ABI (include/vlb.h): argument checks, output
// allocation and the call itself, in one native call per operator.  What the Python functions did per call -- descriptors, shape
// algebra through numpy, views, the stream look-up, ctypes marshalling -- took 20 to 40 us, more than the kernels of the small
// networks; here it is 2 to 4 us.  Nothing is kept from one call to the next.
//
// Tensors are column-major CUDA float32 torch tensors (matconvnet_b200/mat.py); memory comes from torch's allocator, work goes
// to torch's current stream.  Arguments are read under the interpreter lock; outputs are allocated and the engine is called without it.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <array>
#include <mutex>
#include <string>
#include <vector>
#include "../../include/vlb.h"

namespace {

struct PyFail {};        // a Python exception is set

[[noreturn]] void fail(PyObject* type, char const* msg) { PyErr_SetString(type, msg); throw PyFail(); }
[[noreturn]] void fail(PyObject* type, char const* fmt, char const* a) { PyErr_Format(type, fmt, a); throw PyFail(); }

PyObject* gHandleName;                // "_h": the context's vlb_ctx pointer as a Python int
PyObject *gPair, *gQuad;              // nn._pair, nn._quad: any sequence numpy understands, and the error messages
PyObject* gError;                     // capi.VlbError

// The interpreter lock let go of for a scope.
struct Unlocked {
  PyThreadState* const state = PyEval_SaveThread();
  Unlocked() = default;
  Unlocked(Unlocked const&) = delete;
  Unlocked& operator=(Unlocked const&) = delete;
  ~Unlocked() { PyEval_RestoreThread(state); }
};

// ---------------------------------------------------------------- tensors
struct Shape { int64_t d[4]; };

// size(t, 1..4): trailing dimensions folded into the fourth, missing ones 1 (reference bits/data.cu:585-601)
Shape shape4(at::Tensor const& t)
{
  Shape s = {{1, 1, 1, 1}};
  auto const sz = t.sizes();
  for (size_t i = 0; i < sz.size(); ++i) { if (i < 4) s.d[i] = sz[i]; else s.d[3] *= sz[i]; }
  return s;
}

bool column_major(at::Tensor const& t)
{
  if (t.numel() == 0) return true;
  int64_t want = 1;
  auto const sz = t.sizes(), st = t.strides();
  for (size_t i = 0; i < sz.size(); ++i) {
    if (sz[i] != 1 && st[i] != want) return false;
    want *= sz[i];
  }
  return true;
}

at::Tensor empty_cm(at::IntArrayRef sizes, at::Device device)
{
  std::array<int64_t, 8> st;
  int64_t s = 1;
  TORCH_CHECK(sizes.size() <= st.size(), "too many dimensions");
  for (size_t i = 0; i < sizes.size(); ++i) { st[i] = s; s *= sizes[i] > 0 ? sizes[i] : 1; }
  return at::empty_strided(sizes, at::IntArrayRef(st.data(), sizes.size()), at::TensorOptions().dtype(at::kFloat).device(device));
}

at::Tensor empty_cm(int64_t a, int64_t b, int64_t c, int64_t d, at::Device dev) { int64_t const s[4] = {a, b, c, d}; return empty_cm(at::IntArrayRef(s, 4), dev); }
at::Tensor empty_cm(int64_t a, int64_t b, at::Device dev) { int64_t const s[2] = {a, b}; return empty_cm(at::IntArrayRef(s, 2), dev); }

// A CUDA float32 tensor in column-major order (a copy when it is not); None gives an undefined tensor.
at::Tensor need(PyObject* o, char const* name)
{
  if (o == Py_None) return at::Tensor();
  if (!THPVariable_Check(o)) fail(PyExc_TypeError, "%s must be a CUDA float32 tensor (this engine has no CPU path)", name);
  at::Tensor const& t = THPVariable_Unpack(o);
  if (!t.is_cuda() || t.scalar_type() != at::kFloat) fail(PyExc_TypeError, "%s must be a CUDA float32 tensor (this engine has no CPU path)", name);
  if (column_major(t)) return t;
  Unlocked u;
  at::Tensor c = empty_cm(t.sizes(), t.device());
  c.copy_(t);
  return c;
}

at::Tensor flat32(PyObject* o, char const* name)
{
  if (!THPVariable_Check(o)) fail(PyExc_TypeError, "%s must be a CUDA float32 tensor", name);
  at::Tensor const& t = THPVariable_Unpack(o);
  if (!t.is_cuda() || t.scalar_type() != at::kFloat) fail(PyExc_TypeError, "%s must be a CUDA float32 tensor", name);
  return t;
}

// A new reference, let go of at the end of the scope.
struct PyRef {
  PyObject* p = nullptr;
  PyRef() = default;
  PyRef(PyRef const&) = delete;
  PyRef& operator=(PyRef const&) = delete;
  ~PyRef() { Py_XDECREF(p); }
};

// The two items of der_out = (first, second); `held` keeps them: the caller's sequence may make its items on access.
struct Pair { PyObject *first = nullptr, *second = nullptr; };

Pair two_items(PyObject* seq, PyRef& held)
{
  Pair r;
  if (seq == Py_None) return r;
  held.p = PySequence_Tuple(seq);
  if (!held.p) throw PyFail();
  if (PyTuple_GET_SIZE(held.p) != 2) fail(PyExc_ValueError, "der_out must have two items.");
  r.first = PyTuple_GET_ITEM(held.p, 0); r.second = PyTuple_GET_ITEM(held.p, 1);
  return r;
}

float* ptr(at::Tensor const& t) { return t.defined() ? static_cast<float*>(t.data_ptr()) : nullptr; }

// A caller-supplied output for a parameter derivative of `shape` (e.g. a view into a gradient bucket), checked; undefined without one.
at::Tensor der_out(PyObject* given, at::IntArrayRef shape, char const* name)
{
  if (given == nullptr || given == Py_None) return at::Tensor();
  int64_t n = 1;
  for (int64_t s : shape) n *= s;
  if (THPVariable_Check(given)) {
    at::Tensor const& t = THPVariable_Unpack(given);
    if (t.is_cuda() && t.scalar_type() == at::kFloat && column_major(t) && t.numel() == n && ((uintptr_t)t.data_ptr() & 15) == 0) return t;
  }
  PyErr_Format(PyExc_ValueError, "%s: the supplied output must be a dense 16-byte aligned CUDA float32 tensor of %lld elements", name, (long long)n);
  throw PyFail();
}

PyObject* wrap(at::Tensor const& t) { if (!t.defined()) Py_RETURN_NONE; return THPVariable_Wrap(t); }

PyObject* tuple_of(std::initializer_list<at::Tensor> ts)
{
  PyObject* r = PyTuple_New((Py_ssize_t)ts.size());
  if (!r) throw PyFail();
  Py_ssize_t i = 0;
  for (auto const& t : ts) PyTuple_SET_ITEM(r, i++, wrap(t));
  return r;
}

// ---------------------------------------------------------------- arguments
double as_double(PyObject* o)
{
  double const v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw PyFail();
  return v;
}

int as_int(PyObject* o)
{
  long const v = PyLong_AsLong(o);
  if (v == -1 && PyErr_Occurred()) throw PyFail();
  return (int)v;
}

bool as_bool(PyObject* o)
{
  int const v = PyObject_IsTrue(o);
  if (v < 0) throw PyFail();
  return v != 0;
}

// One or n (2 or 4) integers into out[0..n): ints and lists / tuples of ints here, anything else through nn._pair / nn._quad.
void ints(PyObject* o, int n, int* out, char const* name)
{
  if (PyLong_CheckExact(o)) {
    out[0] = as_int(o);
    for (int i = 1; i < n; ++i) out[i] = out[0];
    return;
  }
  if (PyList_CheckExact(o) || PyTuple_CheckExact(o)) {
    Py_ssize_t const len = PySequence_Fast_GET_SIZE(o);
    PyObject** const it = PySequence_Fast_ITEMS(o);
    bool plain = len == 1 || len == n;
    for (Py_ssize_t i = 0; plain && i < len; ++i) plain = PyLong_CheckExact(it[i]);
    if (plain) {
      for (int i = 0; i < n; ++i) out[i] = as_int(it[len == 1 ? 0 : i]);
      return;
    }
  }
  PyObject* t = PyObject_CallFunction(n == 2 ? gPair : gQuad, "Os", o, name);
  if (!t) throw PyFail();
  for (int i = 0; i < n; ++i) out[i] = (int)PyLong_AsLong(PyTuple_GetItem(t, i));
  Py_DECREF(t);
  if (PyErr_Occurred()) throw PyFail();
}

// The calls of one context come one at a time, whatever threads they come from: its stream, scratch and error message belong to the call.
// The locks stand in a fixed table; two contexts that share a place wait for one another's launches, nothing more.
std::mutex& lock_of(vlb_ctx* h)
{
  static std::mutex locks[61];
  return locks[((uintptr_t)h >> 4) % 61];
}

// The engine context behind a capi.Context, on torch's current stream.
struct Ctx {
  vlb_ctx* h;
  void* stream;
  explicit Ctx(PyObject* o)
  {
    PyObject* p = PyObject_GetAttr(o, gHandleName);
    if (!p) throw PyFail();
    h = static_cast<vlb_ctx*>(PyLong_AsVoidPtr(p));
    Py_DECREF(p);
    if (PyErr_Occurred()) throw PyFail();
    stream = c10::cuda::getCurrentCUDAStream().stream();
  }
  // f: allocates the outputs, calls the engine and returns its error code, which becomes capi.VlbError.  Without the interpreter lock, since it may wait: in the
  // allocator, for a place in the launch queue, for the stream when scratch grows.
  template <class F>
  void run(F f) const
  {
    int rc;
    std::string message;
    {
      Unlocked u;                                                  // (before the context's lock: a thread that waits for that one holds no other)
      std::lock_guard<std::mutex> one(lock_of(h));
      vlb_ctx_set_stream(h, stream);
      rc = f();
      if (rc) { message = vlb_ctx_last_error(h); vlb_ctx_reset_error(h); }
    }
    if (rc == 0) return;
    PyObject* e = PyObject_CallFunction(gError, "is", rc, message.c_str());
    if (e) PyErr_SetObject((PyObject*)Py_TYPE(e), e);
    Py_XDECREF(e);
    throw PyFail();
  }
};

using Args = PyObject* const*;

// Exceptions to Python exceptions; argument counts are those of the callers in nn.py.
template <class F>
PyObject* guarded(Py_ssize_t nargs, Py_ssize_t want, F f)
{
  if (nargs != want) { PyErr_Format(PyExc_TypeError, "%zd arguments expected, got %zd", want, nargs); return nullptr; }
  try {
    return f();
  } catch (PyFail const&) {
    return nullptr;
  } catch (python_error& e) {
    e.restore();
    return nullptr;
  } catch (c10::OutOfMemoryError const& e) {
    PyObject* torch = PyImport_ImportModule("torch");
    PyObject* type = torch ? PyObject_GetAttrString(torch, "OutOfMemoryError") : nullptr;
    if (type) PyErr_SetString(type, e.what_without_backtrace());
    Py_XDECREF(type);
    Py_XDECREF(torch);
    return nullptr;
  } catch (c10::Error const& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what_without_backtrace());
    return nullptr;
  } catch (std::exception const& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
}

// ---------------------------------------------------------------- vl_nnconv
// ctx, x, f, b, dzdy, stride, pad, dilate, no_der_data, no_der_filters, no_der_biases, relu, through_relu, der_out
PyObject* conv(PyObject*, Args a, Py_ssize_t n)
{
  return guarded(n, 14, [&]() -> PyObject* {
    Ctx ctx(a[0]);
    at::Tensor x = need(a[1], "x"), f = need(a[2], "f"), b = need(a[3], "b"), dzdy = need(a[4], "dzdy");
    if (!x.defined()) fail(PyExc_TypeError, "%s must be a CUDA float32 tensor (this engine has no CPU path)", "x");
    Shape const sx = shape4(x), sf = shape4(f);
    vlb_conv_desc d = {};
    d.H = (int)sx.d[0]; d.W = (int)sx.d[1]; d.C = (int)sx.d[2]; d.N = (int)sx.d[3];
    d.FH = (int)sf.d[0]; d.FW = (int)sf.d[1]; d.FC = (int)sf.d[2]; d.K = (int)sf.d[3];
    int v[4];
    ints(a[5], 2, v, "STRIDE"); d.strideY = v[0]; d.strideX = v[1];
    ints(a[6], 4, v, "PAD"); d.padTop = v[0]; d.padBottom = v[1]; d.padLeft = v[2]; d.padRight = v[3];
    ints(a[7], 2, v, "DILATE"); d.dilateY = v[0]; d.dilateX = v[1];
    if (b.defined() && b.numel() != d.K) fail(PyExc_ValueError, "The number of elements of BIASES is not the same as the number of filters.");
    int Ho = 0, Wo = 0;
    vlb_conv_output_shape(&d, &Ho, &Wo);
    // the gateway's fully connected case (reference matlab/src/vl_nnconv.cu:351-361)
    bool const fc = Ho == 1 && Wo == 1 && d.strideY == 1 && d.strideX == 1 && d.padTop == 0 && d.padBottom == 0 && d.padLeft == 0 && d.padRight == 0 &&
                    d.dilateY == 1 && d.dilateX == 1 && d.FC == d.C && d.FH == d.H && d.FW == d.W;
    if (!dzdy.defined()) {
      at::Tensor y;
      bool const relu = as_bool(a[11]);
      ctx.run([&] {
        y = empty_cm(Ho, Wo, d.K, d.N, x.device());
        if (relu) return vlb_conv_relu_forward(ctx.h, ptr(y), ptr(x), ptr(f), ptr(b), &d);
        if (fc)   return vlb_fc_forward(ctx.h, ptr(y), ptr(x), ptr(f), ptr(b), &d);
        return vlb_conv_forward(ctx.h, ptr(y), 0.0, ptr(x), 1.0, ptr(f), ptr(b), &d);
      });
      return wrap(y);
    }
    Shape const sd = shape4(dzdy);
    if (sd.d[0] != Ho || sd.d[1] != Wo || sd.d[2] != d.K || sd.d[3] != d.N)
      fail(PyExc_ValueError, "DEROUTPUT dimensions are incompatible with X and FILTERS.");
    PyRef held;
    Pair const given = two_items(a[13], held);
    bool const wantX = !as_bool(a[8]), wantF = !as_bool(a[9]), wantB = !as_bool(a[10]) && b.defined();
    int64_t const sb[2] = {1, d.K};
    at::Tensor dx, df, db;
    if (wantF) df = der_out(given.first, at::IntArrayRef(sf.d, 4), "DF");
    if (wantB) db = der_out(given.second, at::IntArrayRef(sb, 2), "DB");
    auto const fn = as_bool(a[12]) ? vlb_relu_conv_backward : (fc ? vlb_fc_backward : vlb_conv_backward);
    ctx.run([&] {
      if (wantX) dx = empty_cm(d.H, d.W, d.C, d.N, x.device());
      if (wantF && !df.defined()) df = empty_cm(at::IntArrayRef(sf.d, 4), x.device());
      if (wantB && !db.defined()) db = empty_cm(at::IntArrayRef(sb, 2), x.device());
      return fn(ctx.h, ptr(dx), ptr(df), ptr(db), ptr(x), ptr(f), ptr(dzdy), &d);
    });
    return tuple_of({dx, df, db});
  });
}

// ctx, x, f, b, dzdy, upsample, crop, num_groups, no_der_data, no_der_filters, no_der_biases
PyObject* convt(PyObject*, Args a, Py_ssize_t n)
{
  return guarded(n, 11, [&]() -> PyObject* {
    Ctx ctx(a[0]);
    at::Tensor x = need(a[1], "x"), f = need(a[2], "f"), b = need(a[3], "b"), dzdy = need(a[4], "dzdy");
    if (!x.defined() || !f.defined()) fail(PyExc_TypeError, "%s must be a CUDA float32 tensor (this engine has no CPU path)", x.defined() ? "f" : "x");
    Shape const sx = shape4(x), sf = shape4(f);
    vlb_convt_desc d = {};
    d.H = (int)sx.d[0]; d.W = (int)sx.d[1]; d.C = (int)sx.d[2]; d.N = (int)sx.d[3];
    d.FH = (int)sf.d[0]; d.FW = (int)sf.d[1]; d.FD = (int)sf.d[2]; d.FN = (int)sf.d[3];
    int v[4];
    ints(a[5], 2, v, "UPSAMPLE"); d.upsampleY = v[0]; d.upsampleX = v[1];
    ints(a[6], 4, v, "CROP"); d.cropTop = v[0]; d.cropBottom = v[1]; d.cropLeft = v[2]; d.cropRight = v[3];
    d.numGroups = as_int(a[7]);
    int const K = d.FD * d.numGroups;
    if (b.defined() && b.numel() != K) fail(PyExc_ValueError, "The number of elements of BIASES is not the same as the dimenison of the filters.");
    int Ho = 0, Wo = 0;
    vlb_convt_output_shape(&d, &Ho, &Wo);
    if (!dzdy.defined()) {
      at::Tensor y;
      ctx.run([&] {
        y = empty_cm(Ho > 0 ? Ho : 0, Wo > 0 ? Wo : 0, K > 0 ? K : 0, d.N, x.device());
        return vlb_convt_forward(ctx.h, ptr(y), ptr(x), ptr(f), ptr(b), &d);
      });
      return wrap(y);
    }
    Shape const sd = shape4(dzdy);
    if (sd.d[0] != Ho || sd.d[1] != Wo || sd.d[2] != K || sd.d[3] != d.N)
      fail(PyExc_ValueError, "DEROUTPUT dimensions are incompatible with X and FILTERS.");
    bool const wantX = !as_bool(a[8]), wantF = !as_bool(a[9]), wantB = !as_bool(a[10]) && b.defined();
    at::Tensor dx, df, db;
    ctx.run([&] {
      if (wantX) dx = empty_cm(d.H, d.W, d.C, d.N, x.device());
      if (wantF) df = empty_cm(at::IntArrayRef(sf.d, 4), x.device());
      if (wantB) db = empty_cm(1, K, x.device());
      return vlb_convt_backward(ctx.h, ptr(dx), ptr(df), ptr(db), ptr(x), ptr(f), ptr(dzdy), &d);
    });
    return tuple_of({dx, df, db});
  });
}

at::Tensor need_one(PyObject* o, char const* name)
{
  at::Tensor t = need(o, name);
  if (!t.defined()) fail(PyExc_TypeError, "%s must be a CUDA float32 tensor (this engine has no CPU path)", name);
  return t;
}

bool same4(Shape const& s, int64_t a, int64_t b, int64_t c, int64_t d) { return s.d[0] == a && s.d[1] == b && s.d[2] == c && s.d[3] == d; }
at::Tensor empty4(Shape const& s, at::Device dev) { return empty_cm(at::IntArrayRef(s.d, 4), dev); }

// ---------------------------------------------------------------- vl_nnbnorm
// ctx, x, g, b, dzdy, epsilon, moments, der_out, relu
PyObject* bnorm(PyObject*, Args a, Py_ssize_t n)
{
  return guarded(n, 9, [&]() -> PyObject* {
    Ctx ctx(a[0]);
    at::Tensor x = need_one(a[1], "x"), g = need_one(a[2], "g"), b = need_one(a[3], "b"), dzdy = need(a[4], "dzdy"), mom = need(a[6], "moments");
    double const eps = as_double(a[5]);
    Shape const s = shape4(x);
    int const H = (int)s.d[0], W = (int)s.d[1], C = (int)s.d[2], N = (int)s.d[3];
    if (g.numel() != C || b.numel() != C) fail(PyExc_ValueError, "The number of elements of MULTIPLIERS / BIASES is not the number of channels.");
    bool const given = mom.defined(), relu = as_bool(a[8]);
    if (given && mom.numel() != 2 * (int64_t)C) fail(PyExc_ValueError, "MOMENTS must have 2*C elements.");
    if (!dzdy.defined()) {
      at::Tensor y;
      ctx.run([&] {
        y = empty4(s, x.device());
        if (given) {
          int const rc = vlb_bnorm_forward_moment(ctx.h, ptr(y), ptr(mom), ptr(x), ptr(g), ptr(b), H, W, C, N, eps);
          return rc || !relu ? rc : vlb_relu_forward(ctx.h, ptr(y), ptr(y), (size_t)y.numel());
        }
        mom = empty_cm(C, 2, x.device());
        return (relu ? vlb_bnorm_relu_forward : vlb_bnorm_forward)(ctx.h, ptr(y), ptr(mom), ptr(x), ptr(g), ptr(b), H, W, C, N, eps);
      });
      return tuple_of({y, mom});
    }
    if (!same4(shape4(dzdy), H, W, C, N)) fail(PyExc_ValueError, "DZDY dimensions are incompatible with X.");
    PyRef held;
    Pair const own = two_items(a[7], held);
    int64_t const sc[2] = {C, 1};
    at::Tensor dx, dg = der_out(own.first, at::IntArrayRef(sc, 2), "DG"), db = der_out(own.second, at::IntArrayRef(sc, 2), "DB");
    ctx.run([&] {
      dx = empty4(s, x.device());
      if (!dg.defined()) dg = empty_cm(at::IntArrayRef(sc, 2), x.device());
      if (!db.defined()) db = empty_cm(at::IntArrayRef(sc, 2), x.device());
      if (given) return vlb_bnorm_backward_moment(ctx.h, ptr(dx), ptr(dg), ptr(db), ptr(mom), ptr(x), ptr(g), ptr(b), ptr(dzdy), H, W, C, N, eps);
      mom = empty_cm(C, 2, x.device());
      return vlb_bnorm_backward(ctx.h, ptr(dx), ptr(dg), ptr(db), ptr(mom), ptr(x), ptr(g), ptr(b), ptr(dzdy), H, W, C, N, eps);
    });
    return tuple_of({dx, dg, db, mom});
  });
}

// ---------------------------------------------------------------- vl_nnpool
// ctx, x, pool, dzdy, stride, pad, method (0 max, 1 avg), through_relu
PyObject* pool(PyObject*, Args a, Py_ssize_t n)
{
  return guarded(n, 8, [&]() -> PyObject* {
    Ctx ctx(a[0]);
    at::Tensor x = need_one(a[1], "x"), dzdy = need(a[3], "dzdy");
    Shape const s = shape4(x);
    vlb_pool_desc d = {};
    d.H = (int)s.d[0]; d.W = (int)s.d[1]; d.C = (int)s.d[2]; d.N = (int)s.d[3];
    int v[4];
    ints(a[2], 2, v, "POOL"); d.poolH = v[0]; d.poolW = v[1];
    ints(a[4], 2, v, "STRIDE"); d.strideY = v[0]; d.strideX = v[1];
    ints(a[5], 4, v, "PAD"); d.padTop = v[0]; d.padBottom = v[1]; d.padLeft = v[2]; d.padRight = v[3];
    d.method = as_int(a[6]);
    int Ho = 0, Wo = 0;
    vlb_pool_output_shape(&d, &Ho, &Wo);
    if (!dzdy.defined()) {
      at::Tensor y;
      ctx.run([&] {
        y = empty_cm(Ho > 0 ? Ho : 0, Wo > 0 ? Wo : 0, d.C, d.N, x.device());
        return vlb_pool_forward(ctx.h, ptr(y), ptr(x), &d);
      });
      return wrap(y);
    }
    if (!same4(shape4(dzdy), Ho, Wo, d.C, d.N)) fail(PyExc_ValueError, "DZDY dimensions are incompatible with X and POOL.");
    at::Tensor dx;
    auto const fn = as_bool(a[7]) ? vlb_relu_pool_backward : vlb_pool_backward;
    ctx.run([&] {
      dx = empty4(s, x.device());
      return fn(ctx.h, ptr(dx), ptr(x), ptr(dzdy), &d);
    });
    return wrap(dx);
  });
}

// ---------------------------------------------------------------- vl_nnroipool
// ctx, x, rois, dzdy, subdivisions, transform (6-tuple of floats, column-major 2 x 3), method
PyObject* roipool(PyObject*, Args a, Py_ssize_t n)
{
  return guarded(n, 7, [&]() -> PyObject* {
    Ctx ctx(a[0]);
    at::Tensor x = need_one(a[1], "x"), rois = need_one(a[2], "rois"), dzdy = need(a[3], "dzdy");
    Shape const s = shape4(x);
    int const H = (int)s.d[0], W = (int)s.d[1], C = (int)s.d[2], N = (int)s.d[3];
    if (rois.numel() % 5 != 0) fail(PyExc_ValueError, "ROIs is not a 5 x K array.");
    int const K = (int)(rois.numel() / 5), method = as_int(a[6]);
    int S[2];
    ints(a[4], 2, S, "SUBDIVISIONS");
    double tf[6];
    for (int i = 0; i < 6; ++i) tf[i] = as_double(PyTuple_GET_ITEM(a[5], i));
    if (!dzdy.defined()) {
      at::Tensor y;
      ctx.run([&] {
        y = empty_cm(S[0], S[1], C, K, x.device());
        return vlb_roipool_forward(ctx.h, ptr(y), ptr(x), ptr(rois), H, W, C, N, K, S[0], S[1], tf, method);
      });
      return wrap(y);
    }
    if (!same4(shape4(dzdy), S[0], S[1], C, K)) fail(PyExc_ValueError, "DZDY dimensions are incompatible with X and ROIS.");
    at::Tensor dx;
    ctx.run([&] {
      dx = empty4(s, x.device());
      return vlb_roipool_backward(ctx.h, ptr(dx), ptr(x), ptr(rois), ptr(dzdy), H, W, C, N, K, S[0], S[1], tf, method);
    });
    return wrap(dx);
  });
}

// ---------------------------------------------------------------- vl_nnbilinearsampler: ctx, x, grid, dzdy
PyObject* sampler(PyObject*, Args a, Py_ssize_t n)
{
  return guarded(n, 4, [&]() -> PyObject* {
    Ctx ctx(a[0]);
    at::Tensor x = need_one(a[1], "x"), grid = need_one(a[2], "grid"), dzdy = need(a[3], "dzdy");
    Shape const s = shape4(x), g = shape4(grid);
    int const H = (int)s.d[0], W = (int)s.d[1], C = (int)s.d[2], N = (int)s.d[3], Ho = (int)g.d[1], Wo = (int)g.d[2], Ng = (int)g.d[3];
    if (g.d[0] != 2) fail(PyExc_ValueError, "GRID has more than 2 channels.");
    if (N == 0 || Ng % N != 0) fail(PyExc_ValueError, "The number of GRIDs is not a multiple of the number of images.");
    if (!dzdy.defined()) {
      at::Tensor y;
      ctx.run([&] {
        y = empty_cm(Ho, Wo, C, Ng, x.device());
        return vlb_sampler_forward(ctx.h, ptr(y), ptr(x), ptr(grid), H, W, C, N, Ho, Wo, Ng);
      });
      return wrap(y);
    }
    if (!same4(shape4(dzdy), Ho, Wo, C, Ng)) fail(PyExc_ValueError, "DZDY dimensions are incompatible with X and GRID.");
    at::Tensor dx, dgrid;
    ctx.run([&] {
      dx = empty4(s, x.device()); dgrid = empty_cm(2, Ho, Wo, Ng, x.device());
      return vlb_sampler_backward(ctx.h, ptr(dx), ptr(dgrid), ptr(x), ptr(grid), ptr(dzdy), H, W, C, N, Ho, Wo, Ng);
    });
    return tuple_of({dx, dgrid});
  });
}

// ---------------------------------------------------------------- vl_nnrelu: ctx, x, dzdy
PyObject* relu(PyObject*, Args a, Py_ssize_t n)
{
  return guarded(n, 3, [&]() -> PyObject* {
    Ctx ctx(a[0]);
    at::Tensor x = need_one(a[1], "x"), dzdy = need(a[2], "dzdy"), out;
    if (dzdy.defined() && dzdy.numel() != x.numel()) fail(PyExc_ValueError, "DZDY dimensions are incompatible with X.");
    ctx.run([&] {
      out = empty_cm(x.sizes(), x.device());
      return dzdy.defined() ? vlb_relu_backward(ctx.h, ptr(out), ptr(x), ptr(dzdy), (size_t)x.numel()) : vlb_relu_forward(ctx.h, ptr(out), ptr(x), (size_t)x.numel());
    });
    return wrap(out);
  });
}

// ---------------------------------------------------------------- vl_nnnormalize: ctx, x, dzdy, depth, kappa, alpha, beta, through_relu
PyObject* normalize(PyObject*, Args a, Py_ssize_t n)
{
  return guarded(n, 8, [&]() -> PyObject* {
    Ctx ctx(a[0]);
    at::Tensor x = need_one(a[1], "x"), dzdy = need(a[2], "dzdy");
    Shape const s = shape4(x);
    int const H = (int)s.d[0], W = (int)s.d[1], C = (int)s.d[2], N = (int)s.d[3], depth = as_int(a[3]);
    double const kappa = as_double(a[4]), alpha = as_double(a[5]), beta = as_double(a[6]);
    if (dzdy.defined() && !same4(shape4(dzdy), H, W, C, N)) fail(PyExc_ValueError, "DZDY dimensions are incompatible with X.");
    auto const back = as_bool(a[7]) ? vlb_relu_lrn_backward : vlb_lrn_backward;
    at::Tensor out;
    ctx.run([&] {
      out = empty4(s, x.device());
      if (dzdy.defined()) return back(ctx.h, ptr(out), ptr(x), ptr(dzdy), H, W, C, N, depth, kappa, alpha, beta);
      return vlb_lrn_forward(ctx.h, ptr(out), ptr(x), H, W, C, N, depth, kappa, alpha, beta);
    });
    return wrap(out);
  });
}

// ---------------------------------------------------------------- vl_nnsoftmax: ctx, x, dzdy
PyObject* softmax(PyObject*, Args a, Py_ssize_t n)
{
  return guarded(n, 3, [&]() -> PyObject* {
    Ctx ctx(a[0]);
    at::Tensor x = need_one(a[1], "x"), dzdy = need(a[2], "dzdy");
    Shape const s = shape4(x);
    int const H = (int)s.d[0], W = (int)s.d[1], C = (int)s.d[2], N = (int)s.d[3];
    if (dzdy.defined() && dzdy.numel() != x.numel()) fail(PyExc_ValueError, "DZDY dimensions are incompatible with X.");
    at::Tensor out;
    ctx.run([&] {
      out = empty4(s, x.device());
      return dzdy.defined() ? vlb_softmax_backward(ctx.h, ptr(out), ptr(x), ptr(dzdy), H, W, C, N) : vlb_softmax_forward(ctx.h, ptr(out), ptr(x), H, W, C, N);
    });
    return wrap(out);
  });
}

// ---------------------------------------------------------------- vl_nndropout: ctx, x, dzdy, rate, mask, seed
PyObject* dropout(PyObject*, Args a, Py_ssize_t n)
{
  return guarded(n, 6, [&]() -> PyObject* {
    Ctx ctx(a[0]);
    at::Tensor x = need_one(a[1], "x"), dzdy = need(a[2], "dzdy"), mask = need(a[4], "mask");
    if (dzdy.defined() && dzdy.numel() != x.numel()) fail(PyExc_ValueError, "DZDY dimensions are incompatible with X.");
    bool const drawn = !mask.defined();
    unsigned long long seed = 0;
    double rate = 0;
    if (drawn) {
      seed = PyLong_AsUnsignedLongLongMask(a[5]);
      if (PyErr_Occurred()) throw PyFail();
      rate = as_double(a[3]);
    } else if (mask.numel() != x.numel()) {
      fail(PyExc_ValueError, "MASK and X do not have the same number of elements.");
    }
    at::Tensor out;
    ctx.run([&] {
      if (drawn) {
        mask = empty_cm(x.sizes(), x.device());
        int const rc = vlb_dropout_mask(ctx.h, ptr(mask), (size_t)x.numel(), rate, seed);
        if (rc) return rc;
      }
      out = empty_cm(x.sizes(), x.device());
      return vlb_mul(ctx.h, ptr(out), ptr(mask), ptr(dzdy.defined() ? dzdy : x), (size_t)x.numel());
    });
    return tuple_of({out, mask});
  });
}

// ---------------------------------------------------------------- vl_nnsoftmaxloss: ctx, x, c, dzdy (None or a number)
PyObject* softmaxloss(PyObject*, Args a, Py_ssize_t n)
{
  return guarded(n, 4, [&]() -> PyObject* {
    Ctx ctx(a[0]);
    at::Tensor x = need_one(a[1], "x"), c = need_one(a[2], "c");
    Shape const s = shape4(x);
    int const H = (int)s.d[0], W = (int)s.d[1], C = (int)s.d[2], N = (int)s.d[3];
    if (c.numel() != N) fail(PyExc_ValueError, "one label per image expected");
    if (a[3] == Py_None) {
      at::Tensor loss;
      ctx.run([&] {
        loss = at::empty({1}, x.options());
        return vlb_softmaxloss_forward(ctx.h, ptr(loss), ptr(x), ptr(c), H, W, C, N);
      });
      return wrap(loss);
    }
    double const dzdy = as_double(a[3]);
    at::Tensor dx;
    ctx.run([&] {
      dx = empty4(s, x.device());
      return vlb_softmaxloss_backward(ctx.h, ptr(dx), ptr(x), ptr(c), dzdy, H, W, C, N);
    });
    return wrap(dx);
  });
}

// ---------------------------------------------------------------- vl_taccum: ctx, alpha, a, beta, b, out
PyObject* taccum(PyObject*, Args a, Py_ssize_t n)
{
  return guarded(n, 6, [&]() -> PyObject* {
    Ctx ctx(a[0]);
    at::Tensor u = flat32(a[2], "a"), v = flat32(a[4], "b");
    if (u.numel() != v.numel()) fail(PyExc_ValueError, "A and B do not have the same number of elements.");
    at::Tensor y;
    if (a[5] != Py_None) y = flat32(a[5], "out");
    if (y.defined() && y.numel() != u.numel()) fail(PyExc_ValueError, "OUT and A do not have the same number of elements.");
    double const alpha = as_double(a[1]), beta = as_double(a[3]);
    ctx.run([&] {
      if (!y.defined()) y = at::empty_like(u);
      return vlb_taccum(ctx.h, ptr(y), alpha, ptr(u), beta, ptr(v), (size_t)u.numel());
    });
    return wrap(y);
  });
}

// ---------------------------------------------------------------- the trainer's update of several parameter tensors
// ctx, solver (-1: momentum SGD), [(w, s1, s2 or None, g, decay, lr, t)], grad_mult, momentum, nesterov, (rho, epsilon, beta1, beta2)
PyObject* update(PyObject*, Args a, Py_ssize_t n)
{
  return guarded(n, 7, [&]() -> PyObject* {
    Ctx ctx(a[0]);
    int const solver = as_int(a[1]);
    if (!PyList_CheckExact(a[2]) || !PyTuple_CheckExact(a[6]) || PyTuple_GET_SIZE(a[6]) != 4) fail(PyExc_TypeError, "a list of updates and four options expected");
    Py_ssize_t const count = PyList_GET_SIZE(a[2]);
    std::vector<vlb_param_update> u((size_t)count);
    std::vector<at::Tensor> held;                        // (another thread may change the list's tuples meanwhile)
    held.reserve(4 * (size_t)count);
    for (Py_ssize_t i = 0; i < count; ++i) {
      PyObject* t = PyList_GET_ITEM(a[2], i);
      if (!PyTuple_CheckExact(t) || PyTuple_GET_SIZE(t) != 7) fail(PyExc_TypeError, "an update is a tuple of seven");
      at::Tensor const w = flat32(PyTuple_GET_ITEM(t, 0), "w"), g = flat32(PyTuple_GET_ITEM(t, 3), "grad"), s1 = flat32(PyTuple_GET_ITEM(t, 1), "momentum_state");
      PyObject* const o2 = PyTuple_GET_ITEM(t, 2);
      at::Tensor const s2 = o2 == Py_None ? at::Tensor() : flat32(o2, "state");
      if (w.numel() != g.numel() || w.numel() != s1.numel() || (s2.defined() && s2.numel() != w.numel()))
        fail(PyExc_ValueError, solver < 0 ? "parameter, momentum and gradient do not have the same number of elements."
                                          : "parameter and gradient do not have the same number of elements.");
      vlb_param_update& p = u[(size_t)i];
      p.W = ptr(w); p.S1 = ptr(s1); p.S2 = ptr(s2); p.G = ptr(g); p.n = (size_t)w.numel();
      held.insert(held.end(), {w, s1, s2, g});
      p.decay = as_double(PyTuple_GET_ITEM(t, 4)); p.lr = as_double(PyTuple_GET_ITEM(t, 5));
      p.t = PyLong_AsLongLong(PyTuple_GET_ITEM(t, 6));
      if (PyErr_Occurred()) throw PyFail();
    }
    double const gm = as_double(a[3]), momentum = as_double(a[4]);
    vlb_solver_opts so = {};
    so.rho = as_double(PyTuple_GET_ITEM(a[6], 0)); so.epsilon = as_double(PyTuple_GET_ITEM(a[6], 1));
    so.beta1 = as_double(PyTuple_GET_ITEM(a[6], 2)); so.beta2 = as_double(PyTuple_GET_ITEM(a[6], 3));
    int const nesterov = as_bool(a[5]) ? 1 : 0;
    ctx.run([&] {
      return solver < 0 ? vlb_sgd_update_many(ctx.h, (int)count, u.data(), gm, momentum, nesterov) : vlb_solver_update_many(ctx.h, solver, (int)count, u.data(), gm, &so);
    });
    Py_RETURN_NONE;
  });
}

// ---------------------------------------------------------------- the module
PyObject* setup(PyObject*, Args a, Py_ssize_t n)      // nn._pair, nn._quad, capi.VlbError
{
  if (n != 3) { PyErr_SetString(PyExc_TypeError, "three callables expected"); return nullptr; }
  Py_INCREF(a[0]); Py_INCREF(a[1]); Py_INCREF(a[2]);
  Py_XSETREF(gPair, a[0]); Py_XSETREF(gQuad, a[1]); Py_XSETREF(gError, a[2]);
  Py_RETURN_NONE;
}

#define VLB_FN(name) {#name, (PyCFunction)(void*)name, METH_FASTCALL, nullptr}
PyMethodDef gMethods[] = {VLB_FN(setup), VLB_FN(conv), VLB_FN(convt), VLB_FN(bnorm), VLB_FN(pool), VLB_FN(roipool), VLB_FN(sampler), VLB_FN(relu),
                          VLB_FN(normalize), VLB_FN(softmax), VLB_FN(dropout), VLB_FN(softmaxloss), VLB_FN(taccum), VLB_FN(update),
                          {nullptr, nullptr, 0, nullptr}};
PyModuleDef gModule = {PyModuleDef_HEAD_INIT, "_hostpath", "Native host side of matconvnet_b200.nn", -1, gMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__hostpath(void)
{
  gHandleName = PyUnicode_InternFromString("_h");
  return PyModule_Create(&gModule);
}
