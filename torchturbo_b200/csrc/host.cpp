// Launch functions of the hot operators as a CPython extension: shape checks, result allocation and the call into
// libttb200.so.  The same in Python (attribute reads, a ctypes object per argument, a structure field at a time) took 12 us for
// a GEMM, 16 us for a norm and 21 us for its backward, of which a launch is 3 us; a training step of a small model is made of
// hundreds of them.  kernels.py holds the documented Python entry points and keeps the keyword interface.
//
// Every function takes its arguments by position, holds the interpreter lock but for the launch itself, allocates from the
// framework's caching allocator on the current stream, and turns failures into kernels.KernelError (launches) or
// AssertionError (arguments).
#include <Python.h>
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/core/CachingHostAllocator.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "entries.h"

#include <atomic>
#include <cmath>
#include <string>

using at::Tensor;
using ttb::GemmArgs;

namespace {

PyObject* g_kernel_error = nullptr;    // kernels.KernelError
PyObject* g_oom_error = nullptr;       // torch.OutOfMemoryError
PyObject* g_gemm_splits = nullptr;     // kernels.gemm_splits: the rule lives there
std::atomic<long long> g_launches{0};

struct Raised {};                      // a Python error is set

[[noreturn]] void fail(PyObject* type, const std::string& text) {
  PyErr_SetString(type, text.c_str());
  throw Raised{};
}
void need(bool ok, const char* what) {
  if (!ok) fail(PyExc_AssertionError, what);
}

// positional arguments
struct Args {
  PyObject* const* a;
  Py_ssize_t n;
  Py_ssize_t i = 0;
  Args(PyObject* const* args, Py_ssize_t count, Py_ssize_t expected) : a(args), n(count) {
    if (count != expected) fail(PyExc_TypeError, "expected " + std::to_string(expected) + " arguments, got " + std::to_string(count));
  }
  const Tensor& tensor() {
    PyObject* o = a[i++];
    if (!THPVariable_Check(o)) fail(PyExc_TypeError, "argument " + std::to_string(i) + " must be a tensor");
    return THPVariable_Unpack(o);
  }
  Tensor optional() {
    if (a[i] == Py_None) { ++i; return Tensor(); }
    return tensor();
  }
  bool flag() {
    const int r = PyObject_IsTrue(a[i++]);
    if (r < 0) throw Raised{};
    return r != 0;
  }
  long long integer() {
    const long long v = PyLong_AsLongLong(a[i++]);
    if (v == -1 && PyErr_Occurred()) throw Raised{};
    return v;
  }
  double real() {
    const double v = PyFloat_AsDouble(a[i++]);
    if (v == -1.0 && PyErr_Occurred()) throw Raised{};
    return v;
  }
};

template <typename F>
PyObject* guarded(F body) {
  try {
    return body();
  } catch (const Raised&) {
  } catch (python_error& e) {
    e.restore();
  } catch (const c10::OutOfMemoryError& e) {
    PyErr_SetString(g_oom_error ? g_oom_error : PyExc_RuntimeError, e.what_without_backtrace());
  } catch (const c10::Error& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what_without_backtrace());
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
  }
  return nullptr;
}

const void* at_(const Tensor& t) { return t.defined() ? t.const_data_ptr() : nullptr; }
void* to_(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
const float* f32(const Tensor& t) { return static_cast<const float*>(at_(t)); }
const int* i32(const Tensor& t) { return static_cast<const int*>(at_(t)); }
float* f32w(const Tensor& t) { return static_cast<float*>(to_(t)); }

bool is_bf16(const Tensor& t) { return t.scalar_type() == at::kBFloat16; }
int sms(const Tensor& t) { return at::cuda::getDeviceProperties(t.get_device())->multiProcessorCount; }
at::TensorOptions plain(const Tensor& like) { return like.options().requires_grad(false); }
Tensor empty(at::IntArrayRef shape, at::ScalarType dt, const Tensor& like) { return at::empty(shape, plain(like).dtype(dt)); }
Tensor empty_rows(const Tensor& like) { return at::empty(like.sizes(), plain(like)); }

void check_device(const Tensor& t) {
  const int cur = c10::cuda::current_device();
  if (!t.is_cuda() || t.get_device() != cur)
    fail(g_kernel_error, "operand lives on " + t.device().str() + " but the current CUDA device is " + std::to_string(cur) +
                             "; call torch.cuda.set_device() for this process before using the ops");
}

// Gives the interpreter lock up for its lifetime.  An object, because a call may leave by an exception (the address of a tensor that has
// no storage, such as the batched gradients of `is_grads_batched`), and whoever turns that into a Python error needs the lock.
struct Unlocked {
  PyThreadState* state = PyEval_SaveThread();
  ~Unlocked() { PyEval_RestoreThread(state); }
};

// Runs a C entry on the current stream without the interpreter lock.
template <typename F>
void launch(const char* what, int kernels, F call) {
  void* stream = c10::cuda::getCurrentCUDAStream().stream();
  int code;
  {
    const Unlocked without_lock;
    code = call(stream);
  }
  if (code != 0) fail(g_kernel_error, std::string(what) + " failed with code " + std::to_string(code));
  g_launches.fetch_add(kernels, std::memory_order_relaxed);
}

PyObject* wrap(const Tensor& t) {
  if (!t.defined()) Py_RETURN_NONE;
  return THPVariable_Wrap(t);
}
template <typename... Ts>
PyObject* wrap_all(const Ts&... ts) {
  PyObject* out = PyTuple_New(sizeof...(Ts));
  if (!out) throw Raised{};
  Py_ssize_t i = 0;
  for (PyObject* o : {wrap(ts)...}) PyTuple_SET_ITEM(out, i++, o);
  return out;
}
// rows x last dimension
Tensor rows2d(const Tensor& t) { return t.dim() == 2 ? t.contiguous() : t.reshape({-1, t.size(-1)}).contiguous(); }
Tensor like_shape(const Tensor& t2, const Tensor& x) { return x.dim() == 2 ? t2 : t2.view(x.sizes()); }
int kda_gate_row_blocks(long long rows, int heads) { return ttb_kda_gate_row_blocks(rows, heads); }
int row_blocks(long long rows, const Tensor& t) { return static_cast<int>(std::max<long long>(1, std::min<long long>(rows, 2 * sms(t)))); }
at::ScalarType out_type(bool f32out) { return f32out ? at::kFloat : at::kBFloat16; }

// ---------------------------------------------------------------------------------------------
// GEMM
// ---------------------------------------------------------------------------------------------
PyObject* gemm(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args in(args, n, 15);
    const Tensor &a = in.tensor(), &b = in.tensor();
    const bool a_mn = in.flag(), b_mn = in.flag();
    Tensor out = in.optional();
    const bool want_f32 = in.flag(), accumulate = in.flag();
    const Tensor residual = in.optional(), tile_group = in.optional(), group_rows = in.optional();
    const bool swiglu = in.flag();
    const Tensor row_scale = in.optional(), preact = in.optional();
    const long long ep = in.integer();
    const Tensor alpha = in.optional();
    need(is_bf16(a) && is_bf16(b), "operands must be bf16");
    need(a.stride(-1) == 1 && b.stride(-1) == 1, "operands must be contiguous along their last dimension");
    check_device(a);
    GemmArgs g{};
    long long M, N, K;
    if (group_rows.defined()) {
      need(a_mn && b_mn && a.dim() == 2 && b.dim() == 2, "row groups need both operands as [rows, columns]");
      g.groups_k = static_cast<int>(group_rows.numel() - 1);
      M = a.size(1); N = b.size(1); K = 0;
      g.total_rows = a.size(0);
      need(b.size(0) == a.size(0), "operands differ in rows");
    } else {
      need(a.dim() == 2, "a must be a matrix");
      M = a.size(a_mn ? 1 : 0); K = a.size(a_mn ? 0 : 1);
      const long long Kb = b.size(b_mn ? -2 : -1), Nmem = b.size(b_mn ? -1 : -2);
      need(Kb == K, "operands differ in the contracted dimension");
      N = swiglu ? Nmem / 2 : Nmem;
    }
    g.A = a.const_data_ptr(); g.lda = a.stride(0);
    g.B = b.const_data_ptr(); g.ldb = b.stride(-2);
    if (b.dim() == 3) {
      g.b_groups = static_cast<int>(b.size(0)); g.b_group_stride = b.stride(0);
      need(tile_group.defined(), "a stack of matrices needs the tile map");
    } else {
      g.b_groups = 1;
    }
    if (!out.defined()) {
      out = g.groups_k ? empty({g.groups_k, M, N}, out_type(want_f32), a) : empty({M, N}, out_type(want_f32), a);
      need(!accumulate, "nothing to accumulate into");
    }
    need(out.stride(-1) == 1 && (is_bf16(out) || out.scalar_type() == at::kFloat), "out must be bf16 or fp32 with contiguous rows");
    g.C = out.data_ptr(); g.ldc = out.stride(-2);
    g.c_group_stride = g.groups_k ? out.stride(0) : 0;
    g.M = static_cast<int>(M); g.N = static_cast<int>(N); g.K = static_cast<int>(K);
    g.a_mn = a_mn; g.b_mn = b_mn;
    g.c_fp32 = !is_bf16(out); g.accumulate = accumulate;
    if (residual.defined()) {
      need(is_bf16(residual) && is_bf16(out), "the residual and its result are bf16");
      g.residual = residual.const_data_ptr(); g.ldr = residual.stride(0);
    }
    if (tile_group.defined()) {
      need(tile_group.scalar_type() == at::kInt, "the tile map is int32");
      g.tile_group = i32(tile_group); g.m_tiles_cap = static_cast<int>(tile_group.numel());
      need(M <= tile_group.numel() * 128, "more rows than the tile map covers");
    }
    if (group_rows.defined()) {
      need(group_rows.scalar_type() == at::kInt, "row groups are int32");
      g.group_rows = i32(group_rows);
    }
    g.epi = swiglu; g.F = swiglu ? g.N : 0;
    if (row_scale.defined()) {
      need(row_scale.scalar_type() == at::kFloat, "the row scale is fp32");
      g.row_scale = f32(row_scale);
    }
    if (preact.defined()) {
      need(is_bf16(preact), "pre-activations are bf16");
      g.preact = preact.data_ptr(); g.ld_preact = preact.stride(0);
    }
    g.num_sms = sms(a);
    if (alpha.defined()) {
      need(alpha.scalar_type() == at::kFloat && alpha.numel() == 1 && alpha.device() == a.device() && !swiglu, "alpha is one fp32 value on the device");
      g.alpha = f32(alpha);
    }
    g.ep = reinterpret_cast<const ttb::EpFuseArgs*>(ep);
    Tensor ws;
    int kernels = 1;
    if (K >= 4096 && !swiglu && !tile_group.defined() && !ep) {
      PyObject* r = PyObject_CallFunction(g_gemm_splits, "LLLi", M, N, K, g.num_sms);
      if (!r) throw Raised{};
      const long long s = PyLong_AsLongLong(r);
      Py_DECREF(r);
      if (s == -1 && PyErr_Occurred()) throw Raised{};
      if (s > 1) {
        ws = empty({s, M, N}, at::kFloat, a);
        g.split_ws = f32w(ws); g.k_splits = static_cast<int>(s);
        kernels = 2;
      }
    }
    launch("ttb_gemm_bf16", kernels, [&](void* st) { return ttb_gemm_bf16(&g, st); });
    return wrap(out);
  });
}

// ---------------------------------------------------------------------------------------------
// norms, bias + activation
// ---------------------------------------------------------------------------------------------
PyObject* rmsnorm_fwd(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args in(args, n, 5);
    const Tensor &x = in.tensor(), &w = in.tensor();
    const double eps = in.real();
    const Tensor residual = in.optional();
    const bool plus = in.flag();
    const Tensor x2 = rows2d(x), r2 = residual.defined() ? rows2d(residual) : Tensor();
    const long long T = x2.size(0);
    const Tensor y = empty_rows(x2), rstd = empty({T}, at::kFloat, x), sum = residual.defined() ? empty_rows(x2) : Tensor();
    launch("ttb_rmsnorm_fwd", 1, [&](void* st) {
      return ttb_rmsnorm_fwd(at_(x2), at_(r2), at_(w), to_(y), to_(sum), f32w(rstd), T, static_cast<int>(x2.size(1)), static_cast<float>(eps), plus, st);
    });
    return wrap_all(like_shape(y, x), rstd, sum.defined() ? like_shape(sum, x) : x);
  });
}

PyObject* rmsnorm_bwd(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args in(args, n, 7);
    const Tensor &dy = in.tensor(), &x = in.tensor(), &w = in.tensor(), &rstd = in.tensor();
    const Tensor dres = in.optional();
    const bool plus = in.flag(), f32out = in.flag();
    const Tensor x2 = rows2d(x), dy2 = rows2d(dy), d2 = dres.defined() ? rows2d(dres) : Tensor();
    const long long T = x2.size(0), H = x2.size(1);
    const int grid = row_blocks(T, x);
    const Tensor dx = empty_rows(x2), part = empty({grid, H}, at::kFloat, x), dw = empty({H}, out_type(f32out), x);
    launch("ttb_rmsnorm_bwd", 2, [&](void* st) {
      return ttb_rmsnorm_bwd(at_(dy2), at_(x2), at_(w), f32(rstd), at_(d2), to_(dx), f32w(part), to_(dw), !f32out, T, static_cast<int>(H), plus, grid, st);
    });
    return wrap_all(like_shape(dx, x), dw);
  });
}

PyObject* layernorm_fwd(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args in(args, n, 4);
    const Tensor &x = in.tensor(), &w = in.tensor(), &b = in.tensor();
    const double eps = in.real();
    const Tensor x2 = rows2d(x);
    const long long T = x2.size(0);
    const Tensor y = empty_rows(x2), mean = empty({T}, at::kFloat, x), rstd = empty({T}, at::kFloat, x);
    launch("ttb_layernorm_fwd", 1, [&](void* st) {
      return ttb_layernorm_fwd(at_(x2), at_(w), at_(b), to_(y), f32w(mean), f32w(rstd), T, static_cast<int>(x2.size(1)), static_cast<float>(eps), st);
    });
    return wrap_all(like_shape(y, x), mean, rstd);
  });
}

PyObject* layernorm_bwd(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args in(args, n, 6);
    const Tensor &dy = in.tensor(), &x = in.tensor(), &w = in.tensor(), &mean = in.tensor(), &rstd = in.tensor();
    const bool f32out = in.flag();
    const Tensor x2 = rows2d(x), dy2 = rows2d(dy);
    const long long T = x2.size(0), H = x2.size(1);
    const int grid = row_blocks(T, x);
    const Tensor dx = empty_rows(x2), part = empty({grid, 2 * H}, at::kFloat, x), dwdb = empty({2, H}, out_type(f32out), x);
    launch("ttb_layernorm_bwd", 2, [&](void* st) {
      return ttb_layernorm_bwd(at_(dy2), at_(x2), at_(w), f32(mean), f32(rstd), to_(dx), f32w(part), to_(dwdb), !f32out, T, static_cast<int>(H), grid, st);
    });
    return wrap_all(like_shape(dx, x), dwdb.select(0, 0), dwdb.select(0, 1));
  });
}

PyObject* bias_act_fwd(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args in(args, n, 4);
    const Tensor &x = in.tensor(), &bias = in.tensor();
    const int act = static_cast<int>(in.integer());
    const Tensor residual = in.optional();
    const Tensor x2 = rows2d(x), r2 = residual.defined() ? rows2d(residual) : Tensor(), y = empty_rows(x2);
    launch("ttb_bias_act_fwd", 1, [&](void* st) {
      return ttb_bias_act_fwd(at_(x2), at_(bias), at_(r2), to_(y), x2.size(0), static_cast<int>(x2.size(1)), act, st);
    });
    return wrap(like_shape(y, x));
  });
}

PyObject* bias_act_bwd(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args in(args, n, 5);
    const Tensor &dy = in.tensor(), &x = in.tensor(), &bias = in.tensor();
    const int act = static_cast<int>(in.integer());
    const bool f32out = in.flag();
    const Tensor x2 = rows2d(x), dy2 = rows2d(dy);
    const long long R = x2.size(0), C = x2.size(1);
    const int grid = row_blocks(R, x);
    const Tensor dx = act ? empty_rows(x2) : Tensor(), part = empty({grid, C}, at::kFloat, x), db = empty({C}, out_type(f32out), x);
    launch("ttb_bias_act_bwd", 2, [&](void* st) {
      return ttb_bias_act_bwd(at_(dy2), at_(x2), at_(bias), to_(dx), f32w(part), to_(db), !f32out, R, static_cast<int>(C), act, grid, st);
    });
    return wrap_all(act ? like_shape(dx, x) : dy, db);
  });
}

// ---------------------------------------------------------------------------------------------
// rotary embedding, SwiGLU
// ---------------------------------------------------------------------------------------------
PyObject* qknorm_rope_fwd(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args in(args, n, 10);
    const Tensor& qkv = in.tensor();
    const int nq = static_cast<int>(in.integer()), nkv = static_cast<int>(in.integer()), D = static_cast<int>(in.integer());
    const Tensor wq = in.optional(), wk = in.optional();
    const Tensor &cos = in.tensor(), &sin = in.tensor();
    const double eps = in.real();
    const bool norm = in.flag();
    const long long T = qkv.size(0);
    const auto dt = qkv.scalar_type();
    const Tensor q = empty({T, nq, D}, dt, qkv), k = empty({T, nkv, D}, dt, qkv), rstd = empty({T * (nq + nkv)}, at::kFloat, qkv);
    launch("ttb_qknorm_rope_fwd", 1, [&](void* st) {
      return ttb_qknorm_rope_fwd(at_(qkv), qkv.stride(0), nq, nkv, D, at_(wq), at_(wk), f32(cos), f32(sin), to_(q), to_(k), f32w(rstd), T,
                                 static_cast<float>(eps), norm, st);
    });
    return wrap_all(q, k, rstd);
  });
}

PyObject* qknorm_rope_bwd(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args in(args, n, 15);
    const Tensor &dq = in.tensor(), &dk = in.tensor();
    const Tensor dv = in.optional();
    const Tensor& qkv = in.tensor();
    const int nq = static_cast<int>(in.integer()), nkv = static_cast<int>(in.integer()), D = static_cast<int>(in.integer());
    const Tensor wq = in.optional(), wk = in.optional();
    const Tensor &cos = in.tensor(), &sin = in.tensor(), &rstd = in.tensor(), &dqkv = in.tensor();
    const bool norm = in.flag(), f32out = in.flag();
    const long long T = qkv.size(0), groups = (nq + nkv * (dv.defined() ? 2 : 1) + 3) / 4;     // a warp takes four heads of a token
    const int grid = static_cast<int>(std::max<long long>(1, std::min<long long>((T * groups + 7) / 8, 4 * sms(qkv))));
    const Tensor dw = norm && T ? empty({2, D}, out_type(f32out), qkv) : at::zeros({2, D}, plain(qkv).dtype(out_type(f32out)));
    const Tensor part = norm ? empty({grid, 2 * D}, at::kFloat, qkv) : Tensor();
    launch("ttb_qknorm_rope_bwd", norm ? 2 : 1, [&](void* st) {
      return ttb_qknorm_rope_bwd(at_(dq), at_(dk), at_(dv), at_(qkv), qkv.stride(0), nq, nkv, D, at_(wq), at_(wk), f32(cos), f32(sin), f32(rstd),
                                 to_(dqkv), dqkv.stride(0), f32w(part), to_(dw), !f32out, T, norm, grid, st);
    });
    return wrap_all(dw.select(0, 0), dw.select(0, 1));
  });
}

PyObject* qkv_rope_fwd(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args in(args, n, 5);
    const Tensor &x = in.tensor(), &bias = in.tensor();
    const int heads = static_cast<int>(in.integer());
    const Tensor &cos = in.tensor(), &sin = in.tensor();
    const long long T = x.size(0), D = x.size(1) / (3 * heads);
    need(x.dim() == 2 && x.is_contiguous() && bias.is_contiguous() && bias.numel() == x.size(1) && D * 3 * heads == x.size(1), "a row is q, k and v of all heads");
    const auto dt = x.scalar_type();
    const Tensor q = empty({T, heads, D}, dt, x), k = empty({T, heads, D}, dt, x), v = empty({T, heads, D}, dt, x);
    launch("ttb_qkv_rope_fwd", 1, [&](void* st) {
      return ttb_qkv_rope_fwd(at_(x), at_(bias), f32(cos), f32(sin), to_(q), to_(k), to_(v), T, heads, static_cast<int>(D / 2),
                              static_cast<int>(std::max<long long>(1, std::min<long long>(T, 4 * sms(x)))), st);
    });
    return wrap_all(q, k, v);
  });
}

PyObject* qkv_rope_bwd(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args in(args, n, 6);
    const Tensor &dq = in.tensor(), &dk = in.tensor(), &dv = in.tensor(), &cos = in.tensor(), &sin = in.tensor();
    const bool f32out = in.flag();
    const long long T = dq.size(0), heads = dq.size(1), D = dq.size(2), W = 3 * heads * D;
    need(dq.is_contiguous() && dk.is_contiguous() && dv.is_contiguous() && dk.sizes() == dq.sizes() && dv.sizes() == dq.sizes(), "gradients of one shape");
    const int grid = static_cast<int>(std::max<long long>(1, std::min<long long>(T, 2 * sms(dq))));
    const Tensor dx = empty({T, W}, dq.scalar_type(), dq), part = empty({grid, W}, at::kFloat, dq);
    const Tensor db = T ? empty({W}, out_type(f32out), dq) : at::zeros({W}, plain(dq).dtype(out_type(f32out)));
    launch("ttb_qkv_rope_bwd", 2, [&](void* st) {
      return ttb_qkv_rope_bwd(at_(dq), at_(dk), at_(dv), f32(cos), f32(sin), to_(dx), f32w(part), to_(db), !f32out, T, static_cast<int>(heads),
                              static_cast<int>(D / 2), grid, st);
    });
    return wrap_all(dx, db);
  });
}

PyObject* rope(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args in(args, n, 4);
    const Tensor &x = in.tensor(), &cos = in.tensor(), &sin = in.tensor();
    const double sign = in.real();
    const long long T = x.size(0), heads = x.size(1), D = x.size(2);
    const Tensor y = empty({T, heads, D}, x.scalar_type(), x);
    launch("ttb_rope", 1, [&](void* st) {
      return ttb_rope(at_(x), x.stride(0), x.stride(1), f32(cos), f32(sin), to_(y), T, static_cast<int>(heads), static_cast<int>(D / 2),
                      static_cast<float>(sign), st);
    });
    return wrap(y);
  });
}

PyObject* swiglu_fwd(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args in(args, n, 3);
    const Tensor& x = in.tensor();
    const Tensor scale = in.optional(), nrows = in.optional();
    const long long R = x.size(0), F = x.size(1) / 2;
    const Tensor y = empty({R, F}, x.scalar_type(), x);
    launch("ttb_swiglu_fwd", 1, [&](void* st) {
      return ttb_swiglu_fwd(at_(x), x.stride(0), to_(y), y.stride(0), f32(scale), R, static_cast<int>(F), i32(nrows), st);
    });
    return wrap(y);
  });
}

PyObject* swiglu_bwd(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args in(args, n, 6);
    const Tensor &dy = in.tensor(), &x = in.tensor();
    const Tensor scale = in.optional();
    const bool want = in.flag();
    const Tensor nrows = in.optional(), y = in.optional();
    const long long R = x.size(0), F = x.size(1) / 2;
    const Tensor dx = at::empty_like(x, plain(x)), ds = want ? empty({R}, at::kFloat, x) : Tensor();
    launch("ttb_swiglu_bwd", 1, [&](void* st) {
      return ttb_swiglu_bwd(at_(dy), dy.stride(0), at_(x), x.stride(0), f32(scale), to_(dx), dx.stride(0), f32w(ds), to_(y),
                            y.defined() ? y.stride(0) : 0, R, static_cast<int>(F), i32(nrows), st);
    });
    return wrap_all(dx, ds);
  });
}

// ---------------------------------------------------------------------------------------------
// gates of a gated delta net
// ---------------------------------------------------------------------------------------------
bool plain_type(const Tensor& t) { return is_bf16(t) || t.scalar_type() == at::kFloat; }

PyObject* gdn_gate_fwd(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args in(args, n, 4);
    const Tensor &a = in.tensor(), &b = in.tensor(), &A = in.tensor(), &dt = in.tensor();
    const long long T = a.size(0), H = a.size(1);
    need(is_bf16(a) && is_bf16(b) && b.sizes() == a.sizes() && (H == 1 || (a.stride(1) == 1 && b.stride(1) == 1)), "projections: bf16 rows of heads");
    need(A.numel() == H && dt.numel() == H && A.is_contiguous() && dt.is_contiguous() && plain_type(A) && plain_type(dt), "one value per head");
    const Tensor g = empty({T, H}, at::kFloat, a), beta = empty({T, H}, at::kFloat, a);
    launch("ttb_gdn_gate_fwd", 1, [&](void* st) {
      return ttb_gdn_gate_fwd(at_(a), a.stride(0), at_(b), b.stride(0), at_(A), is_bf16(A), at_(dt), is_bf16(dt), f32w(g), f32w(beta), T,
                              static_cast<int>(H), st);
    });
    return wrap_all(g, beta);
  });
}

PyObject* gdn_gate_bwd(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args in(args, n, 7);
    const Tensor &dg = in.tensor(), &dbeta = in.tensor(), &a = in.tensor(), &A = in.tensor(), &dt = in.tensor(), &beta = in.tensor();
    const bool f32out = in.flag();
    const long long T = a.size(0), H = a.size(1);
    need(dg.is_contiguous() && dbeta.is_contiguous() && dg.scalar_type() == at::kFloat && dbeta.scalar_type() == at::kFloat, "gradients: fp32 rows of heads");
    const int blocks = static_cast<int>(std::max<long long>(1, std::min<long long>((T + 7) / 8, 2 * sms(a))));
    const Tensor da = empty({T, H}, at::kBFloat16, a), db = empty({T, H}, at::kBFloat16, a), part = empty({blocks, 2, H}, at::kFloat, a);
    const Tensor sums = T ? empty({2, H}, out_type(f32out), a) : at::zeros({2, H}, plain(a).dtype(out_type(f32out)));
    launch("ttb_gdn_gate_bwd", 2, [&](void* st) {
      return ttb_gdn_gate_bwd(f32(dg), f32(dbeta), at_(a), a.stride(0), at_(A), is_bf16(A), at_(dt), is_bf16(dt), f32(beta), to_(da), to_(db),
                              f32w(part), to_(sums), !f32out, T, static_cast<int>(H), blocks, st);
    });
    return wrap_all(da, db, sums.select(0, 0), sums.select(0, 1));
  });
}

// ---------------------------------------------------------------------------------------------
// a tensor times a factor on the device
// ---------------------------------------------------------------------------------------------
PyObject* scale(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args in(args, n, 3);
    const Tensor &x = in.tensor(), &g = in.tensor();
    const bool bf16 = in.flag();
    check_device(x);
    check_device(g);
    need(x.is_contiguous() && (is_bf16(x) || x.scalar_type() == at::kFloat), "scale: a contiguous bf16 or fp32 tensor");
    need(g.numel() == 1 && g.scalar_type() == at::kFloat, "scale: one fp32 factor");
    const Tensor out = empty(x.sizes(), bf16 ? at::kBFloat16 : at::kFloat, x);
    launch("ttb_scale", 1, [&](void* st) { return ttb_scale(at_(x), is_bf16(x), f32(g), to_(out), bf16, x.numel(), sms(x), st); });
    return wrap(out);
  });
}

// ---------------------------------------------------------------------------------------------
// tables between pinned host memory and the device
// ---------------------------------------------------------------------------------------------
PyObject* copy_words(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args in(args, n, 2);
    const Tensor &dst = in.tensor(), &src = in.tensor();
    const long long bytes = static_cast<long long>(src.nbytes());
    need(dst.scalar_type() == src.scalar_type() && dst.numel() == src.numel() && dst.is_contiguous() && src.is_contiguous() && bytes % 4 == 0,
         "copy_words: two contiguous tensors of one type and of whole 32-bit words");
    for (const Tensor* t : {&dst, &src})
      if (t->is_cuda()) check_device(*t);
      else need(t->is_pinned(), "copy_words: host memory has to be pinned");
    launch("ttb_copy_words", 1, [&](void* st) { return ttb_copy_words(to_(dst), at_(src), bytes / 4, st); });
    // as a copy by torch does: pinned memory that is freed is not handed out again before the stream is past this launch
    for (const Tensor* t : {&dst, &src})
      if (!t->is_cuda()) {
        const auto& data = t->storage().data_ptr();
        at::getHostAllocator(at::kCUDA)->record_event(t->data_ptr(), data.get_context(), at::cuda::getCurrentCUDAStream().unwrap());
      }
    Py_RETURN_NONE;
  });
}

// ---------------------------------------------------------------------------------------------
// Kimi delta attention gate
// ---------------------------------------------------------------------------------------------
PyObject* kda_gate_fwd(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args in(args, n, 5);
    const Tensor &g = in.tensor(), &A = in.tensor();
    const Tensor dt = in.optional();
    const bool bounded = in.flag();
    const double bound = in.real();
    const Tensor out = empty(g.sizes(), at::kFloat, g);
    launch("ttb_kda_gate_fwd", 1, [&](void* st) {
      return ttb_kda_gate_fwd(at_(g), at_(A), is_bf16(A), at_(dt), dt.defined() && is_bf16(dt), f32w(out), g.size(0), static_cast<int>(g.size(1)),
                              bounded, static_cast<float>(bound), st);
    });
    return wrap(out);
  });
}

PyObject* kda_gate_bwd(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args in(args, n, 6);
    const Tensor &dd = in.tensor(), &g = in.tensor(), &A = in.tensor();
    const Tensor dt = in.optional();
    const bool bounded = in.flag();
    const double bound = in.real();
    const long long R = g.size(0), H = g.size(1), D = g.size(2);
    const int blocks = kda_gate_row_blocks(R, static_cast<int>(H));
    const Tensor dg = empty_rows(g), part = empty({std::max(blocks, 1), 2, H * D}, at::kFloat, g);
    const Tensor sums = R ? empty({2, H * D}, at::kFloat, g) : at::zeros({2, H * D}, plain(g).dtype(at::kFloat));
    launch("ttb_kda_gate_bwd", 2, [&](void* st) {
      return ttb_kda_gate_bwd(f32(dd), at_(g), at_(A), is_bf16(A), at_(dt), dt.defined() && is_bf16(dt), to_(dg), f32w(part), f32w(sums), R,
                              static_cast<int>(H), bounded, static_cast<float>(bound), st);
    });
    return wrap_all(dg, sums.select(0, 0), sums.select(0, 1).view({H, D}));
  });
}

// ---------------------------------------------------------------------------------------------
// delta rule
// ---------------------------------------------------------------------------------------------
// q, k, v, g, beta, chunk_rows of a call and what the kernels make of them (kernels.delta_prep)
struct DeltaIn {
  const Tensor &q, &k, &v, &g, &beta, &rows;
  ttb::DeltaChunkIn in{};
  explicit DeltaIn(Args& a) : q(a.tensor()), k(a.tensor()), v(a.tensor()), g(a.tensor()), beta(a.tensor()), rows(a.tensor()) {}
  // l2 and scale are a call's last arguments
  const ttb::DeltaChunkIn* fill(Args& a) {
    const bool l2 = a.flag();
    const double scale = a.real();
    need(v.dim() == 3 && q.dim() == 3 && k.dim() == 3 && rows.dim() == 2, "rows of heads");
    const long long R = v.size(0), H = v.size(1), Hk = q.size(1);
    check_device(q);
    auto heads = [&](const Tensor& t, long long n) { return is_bf16(t) && t.size(0) == R && t.size(1) == n && t.size(2) == 128 && t.stride(2) == 1; };
    need(heads(q, Hk) && heads(k, Hk) && heads(v, H), "q, k, v: bf16 rows of 128-wide heads");
    need(Hk > 0 && H % Hk == 0 && (Hk == H || g.dim() == 2), "key heads");
    need(g.scalar_type() == at::kFloat && g.is_contiguous() && (g.dim() == 2 || (g.dim() == 3 && g.size(2) == 128)) && g.size(0) == R && g.size(1) == H, "log decay");
    need(beta.scalar_type() == at::kFloat && beta.is_contiguous() && beta.dim() == 2 && beta.size(0) == R && beta.size(1) == H, "step size");
    need(rows.scalar_type() == at::kInt && rows.is_contiguous() && rows.size(1) == 3, "chunk table");
    auto bf = [](const Tensor& t) { return static_cast<const __nv_bfloat16*>(at_(t)); };
    in.q = bf(q); in.k = bf(k); in.v = bf(v);
    in.q_t = q.stride(0); in.q_h = q.stride(1);
    in.k_t = k.stride(0); in.k_h = k.stride(1);
    in.v_t = v.stride(0); in.v_h = v.stride(1);
    in.g = f32(g); in.beta = f32(beta); in.chunk_rows = i32(rows);
    in.H = static_cast<int>(H); in.NC = static_cast<int>(rows.size(0)); in.l2 = l2; in.scale = static_cast<float>(scale);
    in.rep = static_cast<int>(H / Hk);
    return &in;
  }
  bool vec() const { return g.dim() == 3; }
};

PyObject* delta_prep(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args in(args, n, 8);
    DeltaIn d(in);
    const ttb::DeltaChunkIn* a = d.fill(in);
    const long long H = a->H, NC = a->NC;
    const Tensor tri = empty({2, H, NC, 64, 64}, at::kFloat, d.q), u = empty({H, NC, 64, 128}, at::kFloat, d.q);
    const Tensor wk = empty({2, H, NC, 64, 128}, at::kBFloat16, d.q), decay = d.vec() ? empty({H, NC, 128}, at::kFloat, d.q) : empty({H, NC}, at::kFloat, d.q);
    const Tensor T = tri.select(0, 0), A = tri.select(0, 1), w = wk.select(0, 0), k_out = wk.select(0, 1);
    launch(d.vec() ? "ttb_delta_vec_prep" : "ttb_delta_prep", 1, [&](void* st) {
      if (d.vec()) return ttb_delta_vec_prep(a, f32w(T), f32w(A), f32w(u), to_(w), to_(k_out), f32w(decay), st);
      return ttb_delta_prep(a, f32w(T), f32w(A), f32w(u), to_(w), to_(k_out), f32w(decay), st);
    });
    return wrap_all(T, A, u, w, k_out, decay);
  });
}

PyObject* delta_out(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args in(args, n, 11);
    DeltaIn d(in);
    const Tensor &A = in.tensor(), &x = in.tensor(), &states = in.tensor();
    const ttb::DeltaChunkIn* a = d.fill(in);
    const Tensor o = empty(d.v.sizes(), at::kBFloat16, d.q);
    launch(d.vec() ? "ttb_delta_vec_out" : "ttb_delta_out", 1, [&](void* st) {
      if (d.vec()) return ttb_delta_vec_out(a, f32(A), f32(x), f32(states), static_cast<int>(states.size(1)) - a->NC, to_(o), st);
      return ttb_delta_out(a, f32(A), f32(x), f32(states), static_cast<int>(states.size(1)) - a->NC, to_(o), st);
    });
    return wrap(o);
  });
}

PyObject* delta_bwd_pre(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args in(args, n, 11);
    DeltaIn d(in);
    const Tensor &dout = in.tensor(), &A = in.tensor();
    const int nseq = static_cast<int>(in.integer());
    const ttb::DeltaChunkIn* a = d.fill(in);
    need(dout.is_contiguous() && is_bf16(dout) && dout.sizes() == d.v.sizes(), "the gradient has v's shape");
    const Tensor gx = empty({a->H, a->NC, 64, 128}, at::kFloat, d.q), gs = empty({a->H, a->NC + nseq, 128, 128}, at::kFloat, d.q);
    launch(d.vec() ? "ttb_delta_vec_bwd_pre" : "ttb_delta_bwd_pre", 1, [&](void* st) {
      if (d.vec()) return ttb_delta_vec_bwd_pre(a, at_(dout), f32(A), nseq, f32w(gx), f32w(gs), st);
      return ttb_delta_bwd_pre(a, at_(dout), f32(A), nseq, f32w(gx), f32w(gs), st);
    });
    return wrap_all(gx, gs);
  });
}

PyObject* delta_state_scan(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args in(args, n, 11);
    const Tensor &a = in.tensor(), &b = in.tensor(), &u0 = in.tensor(), &decay0 = in.tensor();
    const Tensor init0 = in.optional(), add0 = in.optional();
    const Tensor& seq0 = in.tensor();
    const int reverse = static_cast<int>(in.integer());
    const double s1 = in.real(), s2 = in.real();
    const int longest = static_cast<int>(in.integer());
    need(u0.dim() == 4 && seq0.dim() == 2 && (decay0.dim() == 2 || decay0.dim() == 3), "chunks of 64 rows");
    const long long H = u0.size(0), NC = u0.size(1), nseq = seq0.size(0);
    need(u0.size(2) == 64 && u0.size(3) == 128 && a.sizes() == u0.sizes() && b.sizes() == u0.sizes(), "chunks of 64 rows");
    need(is_bf16(a) && is_bf16(b) && u0.scalar_type() == at::kFloat && a.is_contiguous() && b.is_contiguous() && u0.is_contiguous(), "operands");
    need(decay0.is_contiguous() && decay0.scalar_type() == at::kFloat && decay0.size(0) == H && decay0.size(1) == NC, "decay");
    need(seq0.scalar_type() == at::kInt && seq0.is_contiguous() && seq0.size(1) == 2, "sequence table");
    check_device(u0);
    // the copy engine moves whole rows: tensors that start between 16-byte boundaries are copied
    auto placed = [](const Tensor& t) {
      if (!t.defined()) return t;
      const Tensor c = t.contiguous();
      return reinterpret_cast<uintptr_t>(c.const_data_ptr()) % 16 ? c.clone() : c;
    };
    const Tensor u = placed(u0), decay = placed(decay0), init = placed(init0), add = placed(add0), seq = placed(seq0);
    auto states_like = [&](const Tensor& t, long long slots) {
      return t.scalar_type() == at::kFloat && t.dim() == 4 && t.size(0) == H && t.size(1) == slots && t.size(2) == 128 && t.size(3) == 128;
    };
    need(!init.defined() || states_like(init, nseq), "first states");
    need(!add.defined() || states_like(add, NC + nseq), "added gradients");
    const Tensor x = empty_rows(u), states = empty({H, NC + nseq, 128, 128}, at::kFloat, u);
    launch("ttb_delta_state_scan", 1, [&](void* st) {
      return ttb_delta_state_scan(at_(a), at_(b), f32(u), f32w(x), f32(decay), decay.dim() == 3, f32(init), f32(add), f32w(states), i32(seq),
                                  static_cast<int>(nseq), static_cast<int>(H), static_cast<int>(NC), longest, reverse, static_cast<float>(s1),
                                  static_cast<float>(s2), st);
    });
    return wrap_all(x, states);
  });
}

// ---------------------------------------------------------------------------------------------
// attention
// ---------------------------------------------------------------------------------------------
// Rows that no sequence covers read as zero; [lo, hi) = covered rows, lo < 0 = unknown.
void zero_outside(const Tensor& t, long long lo, long long hi) {
  const long long rows = t.size(0);
  if (lo < 0) {
    t.zero_();
    return;
  }
  if (lo > 0) t.narrow(0, 0, std::min(lo, rows)).zero_();
  if (hi < rows) t.narrow(0, hi, rows - hi).zero_();
}
bool head_widths(long long D, long long Dv) { return (D <= 128 && Dv <= 128 && D % 8 == 0 && Dv % 8 == 0) || (D == 192 && Dv == 128); }

PyObject* attn_fwd(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args in(args, n, 11);
    const Tensor &q = in.tensor(), &k = in.tensor(), &v = in.tensor(), &tiles = in.tensor();
    const double scale = in.real();
    const bool causal = in.flag(), want_lse = in.flag(), want_max = in.flag();
    const long long lo = in.integer(), hi = in.integer();
    const int tile_rows = static_cast<int>(in.integer());
    const long long T = q.size(0), Hq = q.size(1), D = q.size(2), Hk = k.size(1), Dv = v.size(2);
    need(k.size(2) == D && head_widths(D, Dv), "head widths");
    need(q.stride(2) == 1 && q.stride(1) == D && k.stride(1) == D && k.stride(2) == 1 && v.stride(1) == Dv && v.stride(2) == 1, "heads must lie in a row");
    const Tensor out = empty({T, Hq, Dv}, q.scalar_type(), q);
    zero_outside(out, lo, hi);
    const auto f = plain(q).dtype(at::kFloat);
    const bool all = lo == 0 && hi == T;             // every row's logsumexp is written
    const Tensor lse = !want_lse ? Tensor() : all ? at::empty({Hq, T}, f) : at::full({Hq, T}, -INFINITY, f);
    const Tensor ml = want_max ? at::full({Hq}, -INFINITY, f) : Tensor();
    launch("ttb_attn_fwd", 1, [&](void* st) {
      return ttb_attn_fwd(at_(q), q.stride(0), at_(k), k.stride(0), at_(v), v.stride(0), to_(out), f32w(lse), f32w(ml), i32(tiles),
                          static_cast<int>(tiles.size(0)), tile_rows, T, static_cast<int>(Hq), static_cast<int>(Hk), static_cast<int>(D),
                          static_cast<int>(Dv), static_cast<float>(scale), causal, st);
    });
    return wrap_all(out, lse, ml);
  });
}

PyObject* attn_bwd(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args in(args, n, 13);
    const Tensor &dout = in.tensor(), &q = in.tensor(), &k = in.tensor(), &v = in.tensor(), &out = in.tensor(), &lse = in.tensor(), &kv = in.tensor();
    const double scale = in.real();
    const bool causal = in.flag();
    const Tensor q_tiles = in.optional();
    const bool deterministic = in.flag();
    const long long lo = in.integer(), hi = in.integer();
    const long long T = q.size(0), Hq = q.size(1), D = q.size(2), Hk = k.size(1), Dv = v.size(2);
    need(dout.is_contiguous() && out.is_contiguous() && q.is_contiguous(), "rows must be contiguous");
    need(k.stride(1) == D && k.stride(2) == 1 && v.stride(1) == Dv && v.stride(2) == 1, "heads must lie in a row");
    const bool split = deterministic || D > 128;
    if (split && !q_tiles.defined()) fail(PyExc_ValueError, "the query-major dQ pass needs the query tile table");
    const auto dt = plain(q);
    const auto f = dt.dtype(at::kFloat);
    if (kv.size(0) == 0)                             // no sequence covers a row
      return wrap_all(at::zeros(q.sizes(), dt), at::zeros({T, Hk, D}, dt), at::zeros({T, Hk, Dv}, dt));
    const Tensor delta = at::empty({Hq * T}, f);
    Tensor dq_acc, dk_acc, dv_acc, dq, dk, dv;
    const bool grouped = Hq != Hk && !deterministic;
    if (grouped) {
      // query heads of a group add into fp32 accumulators, cleared by the first launch and converted by the last; accumulators and
      // results lie back to back, so that they are converted in one
      const long long nq = split ? 0 : T * Hq * D, nk = T * Hk * D, nv = T * Hk * Dv;
      const Tensor acc = at::empty({nq + nk + nv}, f), res = at::empty({nq + nk + nv}, dt);
      auto part = [T](const Tensor& t, long long first, long long H, long long W) { return t.narrow(0, first, T * H * W).view({T, H, W}); };
      if (split) {
        dq = empty_rows(q);
        zero_outside(dq, lo, hi);
      } else {
        dq_acc = part(acc, 0, Hq, D); dq = part(res, 0, Hq, D);
      }
      dk_acc = part(acc, nq, Hk, D); dk = part(res, nq, Hk, D);
      dv_acc = part(acc, nq + nk, Hk, Dv); dv = part(res, nq + nk, Hk, Dv);
    } else {
      if (!split) dq_acc = at::empty({T, Hq, D}, f);
      dq = empty_rows(q);
      if (split) zero_outside(dq, lo, hi);
      dk = at::empty({T, Hk, D}, dt); zero_outside(dk, lo, hi);
      dv = at::empty({T, Hk, Dv}, dt); zero_outside(dv, lo, hi);
    }
    launch("ttb_attn_bwd", !split || grouped ? 3 : 2, [&](void* st) {
      return ttb_attn_bwd(at_(q), at_(k), k.stride(0), at_(v), v.stride(0), at_(out), at_(dout), f32(lse), f32w(delta), f32w(dq_acc), f32w(dk_acc),
                          f32w(dv_acc), to_(dq), to_(dk), to_(dv), i32(kv), static_cast<int>(kv.size(0)), T, static_cast<int>(Hq),
                          static_cast<int>(Hk), static_cast<int>(D), static_cast<int>(Dv), static_cast<float>(scale), causal,
                          split ? (deterministic ? 2 : 0) : 1, st);
    });
    if (split)
      launch("ttb_attn_bwd_dq", 1, [&](void* st) {
        return ttb_attn_bwd_dq(at_(q), at_(k), k.stride(0), at_(v), v.stride(0), at_(dout), f32(lse), f32(delta), to_(dq), i32(q_tiles),
                               static_cast<int>(q_tiles.size(0)), T, static_cast<int>(Hq), static_cast<int>(Hk), static_cast<int>(D),
                               static_cast<int>(Dv), static_cast<float>(scale), causal, st);
      });
    return wrap_all(dq, dk, dv);
  });
}

PyObject* setup(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args in(args, n, 3);
    for (int i = 0; i < 3; ++i) Py_INCREF(args[i]);
    g_kernel_error = args[0];
    g_oom_error = args[1];
    g_gemm_splits = args[2];
    Py_RETURN_NONE;
  });
}
PyObject* launches(PyObject*, PyObject* const*, Py_ssize_t) { return PyLong_FromLongLong(g_launches.load(std::memory_order_relaxed)); }

#define ENTRY(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {ENTRY(setup), ENTRY(launches), ENTRY(gemm), ENTRY(rmsnorm_fwd), ENTRY(rmsnorm_bwd), ENTRY(layernorm_fwd), ENTRY(layernorm_bwd),
                         ENTRY(bias_act_fwd), ENTRY(bias_act_bwd), ENTRY(qknorm_rope_fwd), ENTRY(qknorm_rope_bwd), ENTRY(qkv_rope_fwd), ENTRY(qkv_rope_bwd), ENTRY(gdn_gate_fwd),
                         ENTRY(gdn_gate_bwd), ENTRY(scale), ENTRY(copy_words), ENTRY(kda_gate_fwd), ENTRY(kda_gate_bwd), ENTRY(delta_prep), ENTRY(delta_out), ENTRY(delta_bwd_pre),
                         ENTRY(delta_state_scan), ENTRY(rope), ENTRY(swiglu_fwd),
                         ENTRY(swiglu_bwd), ENTRY(attn_fwd), ENTRY(attn_bwd), {nullptr, nullptr, 0, nullptr}};
#undef ENTRY
PyModuleDef module = {PyModuleDef_HEAD_INIT, "ttb_host", nullptr, -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit_ttb_host() { return PyModule_Create(&module); }
