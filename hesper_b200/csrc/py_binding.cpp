// py_binding.cpp -- the layer API's calls as one C++ step: argument checks, output allocation,
// the caller's stream and the C ABI call.
//
// A one-token matvec is 3 to 5 us on the GPU.  Through ctypes a call cost 12 to 16 us of host time
// (a c_void_p per pointer, conversion of 13 arguments, torch.empty and current_stream from
// Python), so a decode loop written against the layer API was bound by the host.  Here the same
// call costs what the kernel launch costs.  Errors are those of the Python checks it replaces:
// ValueError for a tensor that is not on the GPU, not contiguous or of the wrong size, TypeError
// for a wrong dtype, HesperB200Error for what the library refuses.
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <string>
#include <vector>

#include "../../include/hesper_b200.h"

namespace {

PyObject* g_error = nullptr;  // hesper_b200._lib.HesperB200Error

PyObject* g_empty = nullptr;  // ()

struct Fail {};  // a Python error is set

[[noreturn]] void fail(PyObject* type, const std::string& msg) {
  PyErr_SetString(type, msg.c_str());
  throw Fail();
}

const at::Tensor& tensor(PyObject* o, const char* name) {
  if (!THPVariable_Check(o)) fail(PyExc_TypeError, std::string(name) + " must be a tensor");
  return THPVariable_Unpack(o);
}

const char* dtype_name(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return "torch.float32";
    case at::kHalf: return "torch.float16";
    case at::kInt: return "torch.int32";
    default: return "another dtype";
  }
}

const at::Tensor& need(PyObject* o, at::ScalarType dt, const char* name) {
  const at::Tensor& t = tensor(o, name);
  if (!t.is_cuda()) fail(PyExc_ValueError, std::string(name) + " must live on the GPU (there is no CPU fallback)");
  if (t.scalar_type() != dt)
    fail(PyExc_TypeError, std::string(name) + " must be " + dtype_name(dt) + ", got " + std::string(t.dtype().name()));
  if (!t.is_contiguous()) fail(PyExc_ValueError, std::string(name) + " must be contiguous");
  return t;
}

// Pointer of a tensor argument that may be None and is passed through unchecked.
void* ptr(PyObject* o, const char* name) { return o == Py_None ? nullptr : tensor(o, name).data_ptr(); }
float* fptr(PyObject* o, const char* name) { return static_cast<float*>(ptr(o, name)); }

long as_long(PyObject* o) {
  const long v = PyLong_AsLong(o);
  if (v == -1 && PyErr_Occurred()) throw Fail();
  return v;
}
float as_float(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw Fail();
  return static_cast<float>(v);
}
hb200_ctx* as_ctx(PyObject* o) {
  void* p = PyLong_AsVoidPtr(o);
  if (p == nullptr && PyErr_Occurred()) throw Fail();
  return static_cast<hb200_ctx*>(p);
}
// None: the current stream of the current device; else an object with `cuda_stream`.
hb200_stream as_stream(PyObject* o) {
  if (o == Py_None) return c10::cuda::getCurrentCUDAStream().stream();
  PyObject* h = PyObject_GetAttrString(o, "cuda_stream");
  if (!h) throw Fail();
  void* p = PyLong_AsVoidPtr(h);
  Py_DECREF(h);
  if (p == nullptr && PyErr_Occurred()) throw Fail();
  return p;
}

// Rows of x for layers of K inputs.
long rows(const at::Tensor& x, long K) {
  const int64_t n = x.numel();
  if (K == 0) fail(PyExc_ZeroDivisionError, "in_dim is zero");
  if (n % K) fail(PyExc_ValueError, "input size is not a multiple of in_dim");
  return n / K;
}
at::Tensor make(const at::Tensor& like, at::IntArrayRef shape, at::ScalarType dt = at::kFloat) {
  return at::empty(shape, like.options().dtype(dt));
}
// A new reference to the caller's `out`, or a new [M][N] f32 tensor.
PyObject* output(PyObject* out, const at::Tensor& x, long M, long N, float** p) {
  if (out != Py_None) {
    *p = fptr(out, "out");
    Py_INCREF(out);
    return out;
  }
  at::Tensor y = make(x, {M, N});
  *p = y.data_ptr<float>();
  return THPVariable_Wrap(std::move(y));
}

struct Ref {  // owns a Python reference until released
  PyObject* o;
  explicit Ref(PyObject* p) : o(p) {
    if (!p) throw Fail();
  }
  ~Ref() { Py_XDECREF(o); }
  PyObject* release() {
    PyObject* p = o;
    o = nullptr;
    return p;
  }
};

void check(int rc) {
  if (rc == HB200_OK) return;
  PyObject* e = PyObject_CallFunction(g_error, "is", rc, hb200_last_error());
  if (e) {
    PyErr_SetObject(g_error, e);
    Py_DECREF(e);
  }
  throw Fail();
}
template <typename F>
void call(F&& f) {
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = f();
  Py_END_ALLOW_THREADS
  check(rc);
}

template <typename F>
PyObject* guarded(Py_ssize_t n, Py_ssize_t want, F&& f) {
  if (n != want) {
    PyErr_Format(PyExc_TypeError, "%zd arguments expected, %zd given", want, n);
    return nullptr;
  }
  try {
    return f();
  } catch (const Fail&) {
  } catch (const c10::OutOfMemoryError& e) {  // as torch.empty raises it
    PyObject* torch = PyImport_ImportModule("torch");
    PyObject* type = torch ? PyObject_GetAttrString(torch, "OutOfMemoryError") : nullptr;
    if (type) PyErr_SetString(type, e.what_without_backtrace());
    Py_XDECREF(type);
    Py_XDECREF(torch);
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
  }
  return nullptr;
}

// (ctx, packed, scale, K, N, x, rms_gamma, eps, residual, return_acc, out, stream)
PyObject* bitlinear_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded(n, 12, [&]() -> PyObject* {
    const long K = as_long(a[3]), N = as_long(a[4]);
    const at::Tensor& x = need(a[5], at::kFloat, "input");
    const long M = rows(x, K);
    float* y;
    Ref out(output(a[10], x, M, N, &y));
    const bool acc = PyObject_IsTrue(a[9]);
    at::Tensor ta, td;
    if (acc) {
      ta = make(x, {M, N}, at::kInt);
      td = make(x, {M});
    }
    const float* res = a[8] == Py_None ? nullptr : need(a[8], at::kFloat, "residual").data_ptr<float>();
    const float* gam = a[6] == Py_None ? nullptr : need(a[6], at::kFloat, "rms_gamma").data_ptr<float>();
    const float eps = as_float(a[7]);
    hb200_ctx* ctx = as_ctx(a[0]);
    const void* w = ptr(a[1], "packed");
    const float* s = fptr(a[2], "scale");
    hb200_stream st = as_stream(a[11]);
    call([&] {
      return hb200_bitlinear_forward(ctx, w, s, (int)K, (int)N, x.data_ptr<float>(), (int)M, gam, eps, res,
                                     acc ? ta.data_ptr<int>() : nullptr, acc ? td.data_ptr<float>() : nullptr, y, st);
    });
    if (!acc) return out.release();
    Ref oa(THPVariable_Wrap(std::move(ta))), od(THPVariable_Wrap(std::move(td)));
    return PyTuple_Pack(3, out.o, oa.o, od.o);
  });
}

// (ctx, gate_packed, gate_scale, up_packed, up_scale, K, N, x, rms_gamma, eps, out, stream)
PyObject* bitlinear_gateup(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded(n, 12, [&]() -> PyObject* {
    const long K = as_long(a[5]), N = as_long(a[6]);
    const at::Tensor& x = need(a[7], at::kFloat, "input");
    const long M = rows(x, K);
    float* y;
    Ref out(output(a[10], x, M, N, &y));
    const void *wg = ptr(a[1], "packed"), *wu = ptr(a[3], "packed");
    const float *sg = fptr(a[2], "scale"), *su = fptr(a[4], "scale"), *gam = fptr(a[8], "rms_gamma");
    const float eps = as_float(a[9]);
    hb200_ctx* ctx = as_ctx(a[0]);
    hb200_stream st = as_stream(a[11]);
    call([&] {
      return hb200_bitlinear_gateup_relu2(ctx, wg, sg, wu, su, (int)K, (int)N, x.data_ptr<float>(), (int)M, gam,
                                          eps, y, st);
    });
    return out.release();
  });
}

PyObject* item(PyObject* seq, Py_ssize_t i) { return PySequence_Fast_GET_ITEM(seq, i); }

// (ctx, [(packed, scale, N)], K, x, rms_gamma, eps, residuals, return_acc, stream)
PyObject* bitlinear_multi(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded(n, 9, [&]() -> PyObject* {
    const long K = as_long(a[2]);
    const at::Tensor& x = need(a[3], at::kFloat, "input");
    const long M = rows(x, K);
    Ref ls(PySequence_Fast(a[1], "layers must be a sequence"));
    const Py_ssize_t nl = PySequence_Fast_GET_SIZE(ls.o);
    const bool acc = PyObject_IsTrue(a[7]);
    PyObject* rs = a[6] == Py_None ? nullptr : PySequence_Fast(a[6], "residuals must be a sequence");
    if (a[6] != Py_None && !rs) throw Fail();
    Ref hold(rs ? rs : (Py_INCREF(Py_None), Py_None));
    if (rs && PySequence_Fast_GET_SIZE(rs) < nl) fail(PyExc_IndexError, "fewer residuals than layers");
    Ref ys(PyList_New(nl)), accs(PyList_New(nl));
    std::vector<hb200_bitlinear_seg> segs(nl);
    for (Py_ssize_t i = 0; i < nl; ++i) {
      PyObject* l = item(ls.o, i);
      const long N = as_long(PyTuple_GET_ITEM(l, 2));
      at::Tensor y = make(x, {M, N});
      hb200_bitlinear_seg& s = segs[i];
      s.d_packed = ptr(PyTuple_GET_ITEM(l, 0), "packed");
      s.d_scale = fptr(PyTuple_GET_ITEM(l, 1), "scale");
      s.d_residual = rs ? fptr(item(rs, i), "residual") : nullptr;
      s.d_y = y.data_ptr<float>();
      s.d_acc = nullptr;
      s.N = (int)N;
      PyList_SET_ITEM(ys.o, i, THPVariable_Wrap(std::move(y)));
      PyObject* oa = Py_None;
      if (acc) {
        at::Tensor t = make(x, {M, N}, at::kInt);
        s.d_acc = t.data_ptr<int>();
        oa = THPVariable_Wrap(std::move(t));
      } else {
        Py_INCREF(oa);
      }
      PyList_SET_ITEM(accs.o, i, oa);
    }
    const float* gam = fptr(a[4], "rms_gamma");
    const float eps = as_float(a[5]);
    hb200_ctx* ctx = as_ctx(a[0]);
    hb200_stream st = as_stream(a[8]);
    call([&] {
      return hb200_bitlinear_forward_multi(ctx, segs.data(), (int)nl, (int)K, x.data_ptr<float>(), (int)M, gam, eps,
                                           nullptr, st);
    });
    return acc ? PyTuple_Pack(2, ys.o, accs.o) : ys.release();
  });
}

// (ctx, fmt, blocks, K, N, x, rms_gamma, eps, residual, out, stream)
PyObject* kquant_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded(n, 11, [&]() -> PyObject* {
    const long K = as_long(a[3]), N = as_long(a[4]);
    const at::Tensor& x = need(a[5], at::kFloat, "input");
    const long M = rows(x, K);
    float* y;
    Ref out(output(a[9], x, M, N, &y));
    const int fmt = (int)as_long(a[1]);
    const void* w = ptr(a[2], "blocks");
    const float *gam = fptr(a[6], "rms_gamma"), *res = fptr(a[8], "residual");
    const float eps = as_float(a[7]);
    hb200_ctx* ctx = as_ctx(a[0]);
    hb200_stream st = as_stream(a[10]);
    call([&] {
      return hb200_kquant_forward(ctx, fmt, w, (int)K, (int)N, x.data_ptr<float>(), (int)M, gam, eps, res, y, st);
    });
    return out.release();
  });
}

struct Pre {  // pre=(base, gamma) of a call, or None; what is missing in the pair the library refuses
  bool given;
  Ref hold;
  const float *base = nullptr, *gamma = nullptr;
  explicit Pre(PyObject* o) : given(o != Py_None), hold(PySequence_Fast(given ? o : g_empty, "pre must be a pair")) {
    if (!given) return;
    if (PySequence_Fast_GET_SIZE(hold.o) != 2) fail(PyExc_ValueError, "pre must be a pair (base, gamma)");
    base = fptr(PySequence_Fast_GET_ITEM(hold.o, 0), "pre base");
    gamma = fptr(PySequence_Fast_GET_ITEM(hold.o, 1), "pre gamma");
  }
};

// (ctx, fmt, gate_blocks, up_blocks, K, N, x, rms_gamma, eps, pre, out, stream); pre not None: returns (y, x')
PyObject* kquant_gateup(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded(n, 12, [&]() -> PyObject* {
    const long K = as_long(a[4]), N = as_long(a[5]);
    const at::Tensor& x = need(a[6], at::kFloat, "input");
    const long M = rows(x, K);
    float* y;
    const Pre pre(a[9]);
    Ref out(output(a[10], x, M, N, &y));
    const int fmt = (int)as_long(a[1]);
    const void *wg = ptr(a[2], "blocks"), *wu = ptr(a[3], "blocks");
    const float* gam = fptr(a[7], "rms_gamma");
    const float eps = as_float(a[8]);
    hb200_ctx* ctx = as_ctx(a[0]);
    hb200_stream st = as_stream(a[11]);
    if (!pre.given) {
      call([&] {
        return hb200_kquant_gateup_gelu(ctx, fmt, wg, wu, (int)K, (int)N, x.data_ptr<float>(), (int)M, gam, eps, y, st);
      });
      return out.release();
    }
    at::Tensor xo = at::empty_like(x);
    call([&] {
      return hb200_kquant_gateup_gelu_pre(ctx, fmt, wg, wu, (int)K, (int)N, x.data_ptr<float>(), (int)M, pre.base,
                                          pre.gamma, xo.data_ptr<float>(), gam, eps, y, st);
    });
    Ref o2(THPVariable_Wrap(std::move(xo)));
    return PyTuple_Pack(2, out.o, o2.o);
  });
}

// (ctx, fmt, [(blocks, N)], K, x, rms_gamma, eps, residuals, pre, stream); pre not None: returns (ys, x')
PyObject* kquant_multi(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded(n, 10, [&]() -> PyObject* {
    const long K = as_long(a[3]);
    const at::Tensor& x = need(a[4], at::kFloat, "input");
    const long M = rows(x, K);
    Ref ls(PySequence_Fast(a[2], "layers must be a sequence"));
    const Py_ssize_t nl = PySequence_Fast_GET_SIZE(ls.o);
    PyObject* rs = a[7] == Py_None ? nullptr : PySequence_Fast(a[7], "residuals must be a sequence");
    if (a[7] != Py_None && !rs) throw Fail();
    Ref hold(rs ? rs : (Py_INCREF(Py_None), Py_None));
    if (rs && PySequence_Fast_GET_SIZE(rs) < nl) fail(PyExc_IndexError, "fewer residuals than layers");
    Ref ys(PyList_New(nl));
    std::vector<hb200_kquant_seg> segs(nl);
    for (Py_ssize_t i = 0; i < nl; ++i) {
      PyObject* l = item(ls.o, i);
      const long N = as_long(PyTuple_GET_ITEM(l, 1));
      at::Tensor y = make(x, {M, N});
      segs[i] = {ptr(PyTuple_GET_ITEM(l, 0), "blocks"), rs ? fptr(item(rs, i), "residual") : nullptr,
                 y.data_ptr<float>(), (int)N};
      PyList_SET_ITEM(ys.o, i, THPVariable_Wrap(std::move(y)));
    }
    const int fmt = (int)as_long(a[1]);
    const float* gam = fptr(a[5], "rms_gamma");
    const float eps = as_float(a[6]);
    hb200_ctx* ctx = as_ctx(a[0]);
    hb200_stream st = as_stream(a[9]);
    const Pre pre(a[8]);
    if (!pre.given) {
      call([&] {
        return hb200_kquant_forward_multi(ctx, fmt, segs.data(), (int)nl, (int)K, x.data_ptr<float>(), (int)M, gam,
                                          eps, st);
      });
      return ys.release();
    }
    at::Tensor xo = at::empty_like(x);
    call([&] {
      return hb200_kquant_forward_multi_pre(ctx, fmt, segs.data(), (int)nl, (int)K, x.data_ptr<float>(), (int)M,
                                            pre.base, pre.gamma, xo.data_ptr<float>(), gam, eps, st);
    });
    Ref o2(THPVariable_Wrap(std::move(xo)));
    return PyTuple_Pack(2, ys.o, o2.o);
  });
}

struct AttnArgs {
  const at::Tensor *q, *k, *v, *len;
  int f16;
};
AttnArgs attn_args(PyObject* const* a, bool any_q) {
  const at::Tensor& q = tensor(a[0], "q");
  const at::ScalarType dt = q.scalar_type();
  if (!any_q && dt != at::kFloat && dt != at::kHalf) fail(PyExc_TypeError, "q must be f32 or f16");
  AttnArgs r;
  r.q = &need(a[0], dt, "q");
  r.k = &need(a[1], at::kHalf, "k_cache");
  r.v = &need(a[2], at::kHalf, "v_cache");
  r.len = &need(a[3], at::kInt, "seqlens");
  r.f16 = dt == at::kHalf;
  return r;
}

// (ctx, q, k_cache, v_cache, seqlens, H, Hkv, D, max_seq, scale, window, workspace, out, stream)
PyObject* attn_decode(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded(n, 14, [&]() -> PyObject* {
    const AttnArgs t = attn_args(a + 1, false);
    const int B = (int)t.len->numel(), H = (int)as_long(a[5]), Hkv = (int)as_long(a[6]), D = (int)as_long(a[7]);
    const int L = (int)as_long(a[8]), window = (int)as_long(a[10]);
    const float scale = as_float(a[9]);
    hb200_ctx* ctx = as_ctx(a[0]);
    at::Tensor own;
    if (a[11] == Py_None) {
      const size_t nb = hb200_attn_workspace_bytes(ctx, B, H, Hkv, D, L);
      own = make(*t.q, {(int64_t)(nb > 16 ? nb : 16)}, at::kByte);
    }
    const at::Tensor& ws = a[11] == Py_None ? own : tensor(a[11], "workspace");
    PyObject* out = a[12];
    at::Tensor y;
    float* o;
    if (out == Py_None) {
      y = make(*t.q, {B, H, D});
      o = y.data_ptr<float>();
    } else {
      o = fptr(out, "out");
    }
    hb200_stream st = as_stream(a[13]);
    call([&] {
      return hb200_attn_decode(ctx, t.q->data_ptr(), t.f16, t.k->data_ptr(), t.v->data_ptr(), t.len->data_ptr<int>(),
                               B, H, Hkv, D, L, window, scale, ws.data_ptr(), (size_t)ws.numel(), o, st);
    });
    if (out == Py_None) return THPVariable_Wrap(std::move(y));
    Py_INCREF(out);
    return out;
  });
}

// (ctx, q, k_cache, v_cache, seqlens, H, Hkv, D, max_seq, scale, window, stream)
PyObject* attn_prefill(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded(n, 12, [&]() -> PyObject* {
    const AttnArgs t = attn_args(a + 1, true);
    if (t.q->dim() < 2) fail(PyExc_IndexError, "q must be [B, T, H, D]");
    const int B = (int)t.q->size(0), T = (int)t.q->size(1);
    const int H = (int)as_long(a[5]), Hkv = (int)as_long(a[6]), D = (int)as_long(a[7]);
    const int L = (int)as_long(a[8]), window = (int)as_long(a[10]);
    const float scale = as_float(a[9]);
    hb200_ctx* ctx = as_ctx(a[0]);
    const size_t nb = hb200_attn_prefill_workspace_bytes(ctx, B, T, H, Hkv, D, L);
    at::Tensor ws = make(*t.q, {(int64_t)(nb > 16 ? nb : 16)}, at::kByte);
    at::Tensor y = make(*t.q, {B, T, H, D});
    hb200_stream st = as_stream(a[11]);
    call([&] {
      return hb200_attn_prefill(ctx, t.q->data_ptr(), t.f16, t.k->data_ptr(), t.v->data_ptr(), t.len->data_ptr<int>(),
                                B, T, H, Hkv, D, L, window, scale, ws.data_ptr(), (size_t)ws.numel(),
                                y.data_ptr<float>(), st);
    });
    return THPVariable_Wrap(std::move(y));
  });
}

PyObject* set_error_type(PyObject*, PyObject* type) {
  Py_INCREF(type);
  Py_XSETREF(g_error, type);
  Py_RETURN_NONE;
}

#define HB_FAST(f) {#f, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(f)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {HB_FAST(bitlinear_forward), HB_FAST(bitlinear_gateup), HB_FAST(bitlinear_multi),
                         HB_FAST(kquant_forward),    HB_FAST(kquant_gateup),    HB_FAST(kquant_multi),
                         HB_FAST(attn_decode),       HB_FAST(attn_prefill),
                         {"set_error_type", set_error_type, METH_O, nullptr},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_binding", "Layer API calls over the C ABI.", -1, methods,
                      nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__binding() {
  g_empty = PyTuple_New(0);
  return g_empty ? PyModule_Create(&module) : nullptr;
}
