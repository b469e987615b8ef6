// Host path of the torch operators: what Python did around the C ABI (include/mvpa.h) - checks, outputs, scratch, views and,
// for a block, the projections - as single calls.  A small operator call needs 10 us of the device; the same work took
// 25 us in Python, a training step of a block 1.1 ms where the device needs 0.6.
//
// Every function here works on ordinary CUDA tensors that nothing watches (no mode, transform or tracer) and answers None
// for anything else, which the callers then take through their Python path; results and errors are the same either way.
#include <Python.h>
#include <dlfcn.h>

#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <c10/core/GradMode.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/PyInterpreter.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>

#include <optional>
#include <stdexcept>
#include <string>
#include <vector>

#include "mvpa.h"

namespace {

using at::Tensor;

struct Api {
  decltype(&mvpa_fwd_workspace_bytes) fwd_bytes;
  decltype(&mvpa_bwd_workspace_bytes) bwd_bytes;
  decltype(&mvpa_fwd) fwd;
  decltype(&mvpa_bwd) bwd;
  decltype(&mvpa_rmsnorm) rmsnorm;
  decltype(&mvpa_rmsnorm_bwd) rmsnorm_bwd;
  decltype(&mvpa_rmsnorm_bwd_workspace_bytes) rmsnorm_bwd_bytes;
  decltype(&mvpa_silu_mul) silu_mul;
  decltype(&mvpa_silu_mul_bwd) silu_mul_bwd;
  decltype(&mvpa_workspace_status) fwd_status;
  decltype(&mvpa_bwd_status) bwd_status;
  decltype(&mvpa_last_error_string) last_error;
} api;

PyObject* device_mode = nullptr;  // torch.utils._device.DeviceContext

void check(int status, const char* what) {
  if (status != 0)
    throw std::runtime_error(std::string(what) + " failed (status " + std::to_string(status) + "): " + api.last_error());
}

// Nothing follows the current call operation by operation.  (Forward-mode levels and compilers are looked at in Python.)
bool watched() {
  using c10::DispatchKey;
  static constexpr c10::DispatchKeySet keys({DispatchKey::FuncTorchDynamicLayerFrontMode, DispatchKey::FuncTorchDynamicLayerBackMode,
                                             DispatchKey::FuncTorchVmapMode, DispatchKey::FuncTorchBatched, DispatchKey::Python,
                                             DispatchKey::Functionalize, DispatchKey::Tracer, DispatchKey::PreDispatch});
  return c10::impl::TorchDispatchModeTLS::any_modes_set() || !(c10::impl::tls_local_dispatch_key_set().included_ & keys).empty() ||
         torch::jit::tracer::isTracing();
}
// (A default device is a function mode as well; it only fills in where new tensors live.)
bool function_modes() {
  for (int64_t i = 0, n = at::impl::PythonTorchFunctionTLS::stack_len(); i < n; ++i) {
    const int device = PyObject_IsInstance(at::impl::PythonTorchFunctionTLS::get_stack_at(i)->ptr(getPyInterpreter()), device_mode);
    if (device < 0) throw python_error();
    if (device == 0) return true;
  }
  return false;
}

bool ordinary(const Tensor& t) {  // a strided CUDA tensor with storage and no wrapper or lazy bit
  using c10::DispatchKey;
  static constexpr c10::DispatchKeySet allowed =
      c10::DispatchKeySet(DispatchKey::CUDA) | c10::DispatchKeySet({DispatchKey::ADInplaceOrView, DispatchKey::AutogradCUDA, DispatchKey::AutocastCUDA});
  return t.defined() && t.is_cuda() && t.has_storage() && (t.key_set() | allowed) == allowed;
}

int dtype_code(const Tensor& t) {
  switch (t.scalar_type()) {
    case at::kBFloat16: return MVPA_BF16;
    case at::kFloat: return MVPA_F32;
    case at::kHalf: return MVPA_F16;
    default: return -1;
  }
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// (B, heads, N, D) as the kernels read it in place: contiguous last dimension, 16-byte aligned base and strides
bool rows_fit(const Tensor& t) {
  if (t.dim() != 4 || t.stride(3) != 1) return false;
  const int64_t es = t.element_size();
  return ((t.stride(0) | t.stride(1) | t.stride(2)) * es & 15) == 0 && aligned16(t.const_data_ptr());
}

mvpa_tensor view4(const Tensor& t) { return {t.data_ptr(), t.stride(0), t.stride(1), t.stride(2)}; }
// `heads` heads of D columns starting at column `col` of a (B * N, ld) matrix
mvpa_tensor columns(const Tensor& m, int64_t col, int64_t N, int64_t D) {
  const int64_t ld = m.stride(0);
  return {static_cast<char*>(m.data_ptr()) + col * m.element_size(), N * ld, D, ld};
}

void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

struct Ops {  // q, u, vt, z, k, r_time, r_chan, v
  Tensor t[8];
  bool take(PyObject* const* a, int64_t steps = 0) {  // `steps` time steps of queries, 0 for all
    for (int i = 0; i < 8; ++i) {
      if (!THPVariable_CheckExact(a[i])) return false;
      t[i] = THPVariable_Unpack(a[i]);
      if (!ordinary(t[i]) || t[i].device() != t[0].device() || t[i].scalar_type() != t[0].scalar_type() || t[i].numel() == 0) return false;
    }
    if (dtype_code(t[0]) < 0 || !rows_fit(t[0]) || !rows_fit(t[4]) || !rows_fit(t[7]) || t[5].dim() < 2 || t[6].dim() < 2) return false;
    for (int i : {1, 2, 3, 5, 6})
      if (!t[i].is_contiguous()) return false;
    const int64_t Hkv = t[4].size(1), N = t[4].size(2), D = t[4].size(3), T = t[5].size(-2), C = t[6].size(-2);
    return t[4].sizes() == t[7].sizes() && t[0].size(0) == t[4].size(0) && t[0].size(3) == D && T * C == N &&
           t[0].size(2) == (steps ? steps : T) * C && t[1].numel() == Hkv * D && t[2].numel() == Hkv * D && t[3].numel() == Hkv * D &&
           t[5].numel() == Hkv * T * D && t[6].numel() == Hkv * C * D;
  }
  mvpa_problem problem(double scale, int64_t window, int64_t t0, int64_t tn) const {
    mvpa_problem p = {};
    p.B = (int32_t)t[0].size(0); p.H = (int32_t)t[0].size(1); p.Hkv = (int32_t)t[4].size(1); p.D = (int32_t)t[0].size(3);
    p.T = (int32_t)t[5].size(-2); p.C = (int32_t)t[6].size(-2);
    p.window = (int32_t)window; p.dtype = dtype_code(t[0]); p.sm_scale = (float)scale;
    p.q_time_begin = (int32_t)t0; p.q_time_count = (int32_t)tn;
    return p;
  }
};

Tensor scratch(size_t bytes, const Tensor& like) { return at::empty({(int64_t)bytes}, like.options().dtype(at::kByte).requires_grad(false)); }

void launch_fwd(const mvpa_problem& p, const mvpa_tensor& q, const mvpa_tensor& k, const mvpa_tensor& v, const void* u, const void* vt,
                const void* z, const Tensor& rt, const Tensor& rc, const mvpa_tensor& o, float* lse, bool status) {
  const size_t bytes = api.fwd_bytes(&p);
  const Tensor ws = bytes ? scratch(bytes, rt) : Tensor();
  check(api.fwd(&p, &q, &k, &v, u, vt, z, rt.const_data_ptr(), rc.const_data_ptr(), &o, lse, bytes ? ws.data_ptr() : nullptr, bytes,
                stream_of(rt)), "mvpa_fwd");
  if (status && bytes) check(api.fwd_status(ws.data_ptr(), bytes, stream_of(rt)), "mvpa_fwd kernels");  // synchronises the stream
}

// Gradients of u, vt, z, r_time, r_chan one after the other, flat, in the operands' type (they leave the library as fp32; one
// buffer means one cast, and every piece is a whole number of rows of D >= 16 elements, hence 16-byte aligned).
Tensor launch_bwd(const mvpa_problem& p, const mvpa_tensor& q, const mvpa_tensor& k, const mvpa_tensor& v, const void* u, const void* vt,
                  const void* z, const Tensor& rt, const Tensor& rc, const mvpa_tensor& o, const Tensor& lse, const mvpa_tensor& d_o,
                  const mvpa_tensor& dq, const mvpa_tensor& dk, const mvpa_tensor& dv, bool status) {
  const int64_t nb = (int64_t)p.Hkv * p.D, nt = rt.numel(), nc = rc.numel();
  const Tensor small = at::empty({3 * nb + nt + nc}, rt.options().dtype(at::kFloat).requires_grad(false));
  float* f = small.data_ptr<float>();
  const size_t bytes = api.bwd_bytes(&p);
  const Tensor ws = scratch(bytes < 16 ? 16 : bytes, rt);
  check(api.bwd(&p, &q, &k, &v, u, vt, z, rt.const_data_ptr(), rc.const_data_ptr(), &o, lse.const_data_ptr<float>(), &d_o, &dq, &dk, &dv,
                f, f + nb, f + 2 * nb, f + 3 * nb, f + 3 * nb + nt, ws.data_ptr(), bytes, stream_of(rt)), "mvpa_bwd");
  if (status) check(api.bwd_status(&p, ws.data_ptr(), bytes, stream_of(rt)), "mvpa_bwd kernels");
  return small.to(rt.scalar_type());
}

bool numbers(PyObject* scale, PyObject* window, double* s, int64_t* w) {
  if (!PyFloat_Check(scale) || !PyLong_CheckExact(window)) return false;
  *s = PyFloat_AS_DOUBLE(scale);
  int overflow = 0;
  *w = PyLong_AsLongLongAndOverflow(window, &overflow);
  return !overflow && *w >= INT32_MIN && *w <= INT32_MAX;
}

PyObject* wrap(std::vector<Tensor>&& ts) {  // undefined tensors become None
  PyObject* out = PyTuple_New((Py_ssize_t)ts.size());
  if (!out) throw python_error();
  for (size_t i = 0; i < ts.size(); ++i) {
    PyObject* o;
    if (ts[i].defined()) o = THPVariable_Wrap(std::move(ts[i]));
    else { o = Py_None; Py_INCREF(o); }
    PyTuple_SET_ITEM(out, (Py_ssize_t)i, o);
  }
  return out;
}

bool arguments(Py_ssize_t given, Py_ssize_t wanted) {
  if (given == wanted) return true;
  PyErr_SetString(PyExc_TypeError, "mvpa_host: wrong number of arguments");
  return false;
}

// attend(q, u, vt, z, k, r_time, r_chan, v, sm_scale, window, status): the whole of an operator call that no gradient flows through,
// shapes as `flash_mvpa` wants them.  -> o or None
PyObject* attend(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!arguments(n, 11)) return nullptr;
  const bool status = a[10] == Py_True;
  Ops x;
  double scale;
  int64_t window;
  if (!numbers(a[8], a[9], &scale, &window) || function_modes() || watched() || !x.take(a)) Py_RETURN_NONE;
  const Tensor &q = x.t[0], &k = x.t[4], &rt = x.t[5], &rc = x.t[6];
  const int64_t D = q.size(3);
  if (c10::GradMode::is_enabled())
    for (const Tensor& t : x.t)
      if (t.requires_grad()) Py_RETURN_NONE;
  if (q.size(1) % k.size(1) != 0 || (D != 16 && D != 32 && D != 64 && D != 128) || rt.dim() != 4 || rc.dim() != 4)
    Py_RETURN_NONE;
  Tensor o;
  {
    pybind11::gil_scoped_release nogil;
    c10::cuda::CUDAGuard guard(q.device());
    c10::NoGradGuard no_grad;
    o = at::empty_like(q);
    launch_fwd(x.problem(scale, window, 0, 0), view4(q), view4(k), view4(x.t[7]), x.t[1].const_data_ptr(), x.t[2].const_data_ptr(),
               x.t[3].const_data_ptr(), rt, rc, view4(o), nullptr, status);
  }
  return THPVariable_Wrap(std::move(o));
  END_HANDLE_TH_ERRORS
}

// forward(q, u, vt, z, k, r_time, r_chan, v, sm_scale, window, t0, tn, status) -> (o, lse) or None
PyObject* forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!arguments(n, 13)) return nullptr;
  const bool status = a[12] == Py_True;
  Ops x;
  double scale;
  int64_t window;
  if (!numbers(a[8], a[9], &scale, &window) || !PyLong_CheckExact(a[10]) || !PyLong_CheckExact(a[11]) || function_modes() ||
      watched())
    Py_RETURN_NONE;
  const int64_t t0 = PyLong_AsLongLong(a[10]), tn = PyLong_AsLongLong(a[11]);
  if (PyErr_Occurred()) return nullptr;
  if (!x.take(a, tn)) Py_RETURN_NONE;
  const Tensor& q = x.t[0];
  Tensor o, lse;
  {
    pybind11::gil_scoped_release nogil;
    c10::cuda::CUDAGuard guard(q.device());
    c10::NoGradGuard no_grad;
    o = at::empty_like(q);
    lse = at::empty({q.size(0) * q.size(1), q.size(2)}, q.options().dtype(at::kFloat).requires_grad(false));
    launch_fwd(x.problem(scale, window, t0, tn), view4(q), view4(x.t[4]), view4(x.t[7]), x.t[1].const_data_ptr(),
               x.t[2].const_data_ptr(), x.t[3].const_data_ptr(), x.t[5], x.t[6], view4(o), lse.data_ptr<float>(), status);
  }
  return wrap({std::move(o), std::move(lse)});
  END_HANDLE_TH_ERRORS
}

// backward(do, q, u, vt, z, k, r_time, r_chan, v, o, lse, sm_scale, window, status) -> the eight gradients or None
PyObject* backward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!arguments(n, 14)) return nullptr;
  const bool status = a[13] == Py_True;
  Ops x;
  double scale;
  int64_t window;
  for (int i : {0, 9, 10})
    if (!THPVariable_CheckExact(a[i])) Py_RETURN_NONE;
  if (!numbers(a[11], a[12], &scale, &window) || function_modes() || watched() || !x.take(a + 1)) Py_RETURN_NONE;
  Tensor d_o = THPVariable_Unpack(a[0]);
  const Tensor o = THPVariable_Unpack(a[9]), lse = THPVariable_Unpack(a[10]);
  const Tensor &q = x.t[0], &k = x.t[4], &v = x.t[7];
  for (const Tensor& t : {d_o, o})
    if (!ordinary(t) || t.device() != q.device() || t.scalar_type() != q.scalar_type() || t.sizes() != q.sizes()) Py_RETURN_NONE;
  if (!ordinary(lse) || lse.scalar_type() != at::kFloat || lse.device() != q.device() || !lse.is_contiguous() ||
      lse.numel() != q.size(0) * q.size(1) * q.size(2) || !rows_fit(o))
    Py_RETURN_NONE;
  std::vector<Tensor> g(8);
  {
    pybind11::gil_scoped_release nogil;
    c10::cuda::CUDAGuard guard(q.device());
    c10::NoGradGuard no_grad;
    if (!rows_fit(d_o)) d_o = d_o.contiguous();
    g[0] = at::empty_like(q);
    g[4] = at::empty_like(k);
    g[7] = at::empty_like(v);
    const Tensor small = launch_bwd(x.problem(scale, window, 0, 0), view4(q), view4(k), view4(v), x.t[1].const_data_ptr(),
                                    x.t[2].const_data_ptr(), x.t[3].const_data_ptr(), x.t[5], x.t[6], view4(o), lse, view4(d_o),
                                    view4(g[0]), view4(g[4]), view4(g[7]), status);
    int64_t at = 0;
    for (int i : {1, 2, 3, 5, 6}) {
      g[i] = small.narrow(0, at, x.t[i].numel()).view(x.t[i].sizes());
      at += x.t[i].numel();
    }
  }
  return wrap(std::move(g));
  END_HANDLE_TH_ERRORS
}

// plain(*tensors): 1 if the kernels can take these contiguous tensors and nothing watches the call, 0 if not, -1 if Python has to look
PyObject* plain(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  long answer = 1;
  if (n == 0 || function_modes()) return PyLong_FromLong(-1);
  for (Py_ssize_t i = 0; i < n && answer == 1; ++i)
    if (!THPVariable_CheckExact(a[i])) answer = 0;
  if (answer == 1 && watched()) answer = 0;
  if (answer == 1) {
    const Tensor& t0 = THPVariable_Unpack(a[0]);
    for (Py_ssize_t i = 0; i < n && answer == 1; ++i) {
      const Tensor& t = THPVariable_Unpack(a[i]);
      if (!ordinary(t) || (t.scalar_type() != at::kBFloat16 && t.scalar_type() != at::kFloat) || t.scalar_type() != t0.scalar_type() ||
               t.device() != t0.device() || !t.is_contiguous() || t.numel() == 0 || !aligned16(t.const_data_ptr()))
        answer = 0;
    }
  }
  return PyLong_FromLong(answer);
  END_HANDLE_TH_ERRORS
}

struct Dims {
  int64_t B, T, C, E, H, Hkv, D, I, N, KV, rows;
  mvpa_problem problem(int dtype, double scale, int window) const {
    mvpa_problem p = {};
    p.B = (int32_t)B; p.H = (int32_t)H; p.Hkv = (int32_t)Hkv; p.T = (int32_t)T; p.C = (int32_t)C; p.D = (int32_t)D;
    p.window = window; p.dtype = dtype; p.sm_scale = (float)scale;
    return p;
  }
};

// What the kernels read of a block through pointers: one type and device, contiguous, 16-byte aligned, of the given sizes.
bool fits(const Tensor& t, const Tensor& like, at::ScalarType type, at::IntArrayRef sizes) {
  return ordinary(t) && t.scalar_type() == type && t.device() == like.device() && t.is_contiguous() && t.sizes() == sizes &&
         aligned16(t.const_data_ptr());
}

// The sizes of a block's call; false where an input (x, pos, chan, ln_w, wq, wkv, wpos, wchan, bias, wc, wg, wu, wd) is not of them.
bool block_dims(const Tensor* in, PyObject* const* heads, Dims& d) {
  const Tensor &x = in[0], &bias = in[8], &wg = in[10];
  d.H = PyLong_AsLongLong(heads[0]); d.Hkv = PyLong_AsLongLong(heads[1]); d.D = PyLong_AsLongLong(heads[2]);
  if (PyErr_Occurred()) throw python_error();
  if (!ordinary(x) || x.dim() != 4 || x.numel() == 0 || dtype_code(x) < 0 || !ordinary(wg) || wg.dim() != 2 || !ordinary(bias) ||
      d.H <= 0 || d.Hkv <= 0 || d.D <= 0)
    return false;
  d.B = x.size(0); d.T = x.size(1); d.C = x.size(2); d.E = x.size(3); d.I = wg.size(0);
  d.N = d.T * d.C; d.KV = d.Hkv * d.D; d.rows = d.B * d.N;
  const int64_t Q = d.H * d.D;
  const std::vector<int64_t> sizes[13] = {x.sizes().vec(), {1, d.T, d.E}, {1, d.C, d.E}, {d.E}, {Q, d.E}, {2 * d.KV, d.E}, {d.KV, d.E},
                                          {d.KV, d.E}, bias.sizes().vec(), {d.E, Q}, {d.I, d.E}, {d.I, d.E}, {d.E, d.I}};
  for (int i = 0; i < 13; ++i)
    if (!fits(in[i], x, x.scalar_type(), sizes[i])) return false;
  return bias.numel() == 3 * d.KV && d.I > 0 && d.I * x.element_size() % 16 == 0;
}

// What the body of a block's call runs under.  No autocast: a backward may run inside a region that the forward was outside of, and
// the kernels read every product as the type that the forward had.
struct Body {
  pybind11::gil_scoped_release nogil;
  c10::cuda::CUDAGuard guard;
  c10::NoGradGuard no_grad;
  c10::impl::ExcludeDispatchKeyGuard no_autocast{c10::autocast_dispatch_keyset};
  explicit Body(const Tensor& t) : guard(t.device()) {}
};

const char* part(const Tensor& t, int64_t elements) { return static_cast<const char*>(t.const_data_ptr()) + elements * t.element_size(); }

// block_forward(x, pos, chan, ln_w, wq, wkv, wpos, wchan, bias, wc, wg, wu, wd, eps, window, H, Hkv, D, status)
//   -> (h, xn, q, kv, g, up, rt, rc, o, lse, act): `block_grad.BlockFunction.forward`, or None
PyObject* block_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!arguments(n, 19)) return nullptr;
  const bool status = a[18] == Py_True;
  Tensor in[13];
  for (int i = 0; i < 13; ++i) {
    if (!THPVariable_CheckExact(a[i])) Py_RETURN_NONE;
    in[i] = THPVariable_Unpack(a[i]);
  }
  Dims d;
  if (watched() || !block_dims(in, a + 15, d)) Py_RETURN_NONE;
  const Tensor &x = in[0], &pos = in[1], &chan = in[2], &ln_w = in[3], &wq = in[4], &wkv = in[5], &wpos = in[6], &wchan = in[7],
               &bias = in[8], &wc = in[9], &wg = in[10], &wu = in[11], &wd = in[12];
  const double eps = PyFloat_AsDouble(a[13]);
  const int64_t window = PyLong_AsLongLong(a[14]);
  if (PyErr_Occurred()) return nullptr;
  Tensor h, xn, q, kv, g, up, rt, rc, o, lse, act;
  {
    const Body body(x);
    const int dt = dtype_code(x);
    const Tensor x2 = x.view({d.rows, d.E});
    xn = at::empty_like(x2);
    check(api.rmsnorm(x2.const_data_ptr(), nullptr, ln_w.const_data_ptr(), nullptr, xn.data_ptr(), d.rows, (int32_t)d.E, (float)eps, dt,
                      stream_of(x)), "mvpa_rmsnorm");
    q = at::mm(xn, wq.t());
    kv = at::mm(xn, wkv.t());
    g = at::mm(xn, wg.t());
    up = at::mm(xn, wu.t());
    const auto keys = [&](const Tensor& embeds, const Tensor& w) {  // (Hkv, rows, D)
      return at::mm(embeds.select(0, 0), w.t()).view({-1, d.Hkv, d.D}).transpose(0, 1).contiguous();
    };
    rt = keys(pos, wpos);
    rc = keys(chan, wchan);
    o = at::empty_like(q);
    lse = at::empty({d.B * d.H, d.N}, x.options().dtype(at::kFloat).requires_grad(false));
    launch_fwd(d.problem(dt, 1.0 / std::sqrt((double)d.D), (int)window), columns(q, 0, d.N, d.D), columns(kv, 0, d.N, d.D),
               columns(kv, d.KV, d.N, d.D), part(bias, 0), part(bias, d.KV), part(bias, 2 * d.KV), rt, rc, columns(o, 0, d.N, d.D),
               lse.data_ptr<float>(), status);
    act = at::empty_like(g);
    check(api.silu_mul(g.const_data_ptr(), up.const_data_ptr(), g.stride(0), act.data_ptr(), act.stride(0), d.rows, (int32_t)g.size(1), dt,
                       stream_of(x)), "mvpa_silu_mul");
    h = at::empty_like(x);  // (not a view of a matrix: the caller may change it in place)
    Tensor h2 = h.view({d.rows, d.E});
    at::addmm_out(h2, x2, act, wd.t());
    h2.addmm_(o, wc.t());
  }
  return wrap({h, xn, q, kv, g, up, rt, rc, o, lse, act});
  END_HANDLE_TH_ERRORS
}

// block_backward(dh, x, pos, chan, ln_w, wq, wkv, wpos, wchan, bias, wc, wg, wu, wd, xn, q, kv, g, up, rt, rc, o, lse, act, need, eps,
//   window, H, Hkv, D, status) -> the thirteen gradients (None where the bit of `need` is clear), or None
PyObject* block_backward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!arguments(n, 31)) return nullptr;
  const bool status = a[30] == Py_True;
  Tensor in[24];
  for (int i = 0; i < 24; ++i) {
    if (!THPVariable_CheckExact(a[i])) Py_RETURN_NONE;
    in[i] = THPVariable_Unpack(a[i]);
  }
  Dims d;
  if (watched() || !block_dims(in + 1, a + 27, d) || !ordinary(in[0]) || in[0].device() != in[1].device() ||
      in[0].scalar_type() != in[1].scalar_type() || in[0].sizes() != in[1].sizes())
    Py_RETURN_NONE;
  // (a saved-tensor hook may have brought anything back)
  const std::vector<int64_t> saved[10] = {{d.rows, d.E}, {d.rows, d.H * d.D}, {d.rows, 2 * d.KV}, {d.rows, d.I}, {d.rows, d.I},
                                          {d.Hkv, d.T, d.D}, {d.Hkv, d.C, d.D}, {d.rows, d.H * d.D}, {d.B * d.H, d.N}, {d.rows, d.I}};
  for (int i = 0; i < 10; ++i)
    if (!fits(in[14 + i], in[1], i == 8 ? at::kFloat : in[1].scalar_type(), saved[i])) Py_RETURN_NONE;
  const Tensor &x = in[1], &pos = in[2], &chan = in[3], &ln_w = in[4], &wq = in[5], &wkv = in[6], &wpos = in[7], &wchan = in[8],
               &bias = in[9], &wc = in[10], &wg = in[11], &wu = in[12], &wd = in[13], &xn = in[14], &q = in[15], &kv = in[16],
               &g = in[17], &up = in[18], &rt = in[19], &rc = in[20], &o = in[21], &lse = in[22], &act = in[23];
  const int64_t need = PyLong_AsLongLong(a[24]), window = PyLong_AsLongLong(a[26]);
  const double eps = PyFloat_AsDouble(a[25]);
  if (PyErr_Occurred()) return nullptr;
  std::vector<Tensor> grad(13);
  {
    const Body body(x);
    const int dt = dtype_code(x);
    const auto needs = [&](int i) { return (need >> i & 1) != 0; };
    const auto weight = [&](int i, const Tensor& dy, const Tensor& y) {  // d W = d^T input
      if (needs(i)) grad[i] = at::mm(dy.t(), y);
    };
    const Tensor dh = in[0].contiguous(), dh2 = dh.view({d.rows, d.E});
    weight(9, dh2, o);
    weight(12, dh2, act);
    const Tensor dact = at::mm(dh2, wd);
    const Tensor dg = at::empty({d.rows, g.size(1)}, g.options().requires_grad(false)), dup = at::empty_like(dg);
    check(api.silu_mul_bwd(g.const_data_ptr(), up.const_data_ptr(), g.stride(0), dact.const_data_ptr(), dact.stride(0), dg.data_ptr(),
                           dup.data_ptr(), g.size(1), d.rows, (int32_t)g.size(1), dt, stream_of(x)), "mvpa_silu_mul_bwd");
    const Tensor d_o = at::mm(dh2, wc), dq = at::empty_like(q), dkv = at::empty_like(kv);
    const auto q4 = [&](const Tensor& t) { return columns(t, 0, d.N, d.D); };
    const auto v4 = [&](const Tensor& t) { return columns(t, d.KV, d.N, d.D); };
    const Tensor small = launch_bwd(d.problem(dt, 1.0 / std::sqrt((double)d.D), (int)window), q4(q), q4(kv), v4(kv), part(bias, 0),
                                    part(bias, d.KV), part(bias, 2 * d.KV), rt, rc, q4(o), lse, q4(d_o), q4(dq), q4(dkv), v4(dkv), status);
    if (needs(8)) grad[8] = small.narrow(0, 0, 3 * d.KV).view(bias.sizes());
    const auto keys = [&](int64_t at, int64_t rows, const Tensor& e, int i_e, const Tensor& w, int i_w) {
      const Tensor dk = small.narrow(0, at, rows * d.KV).view({d.Hkv, rows, d.D}).transpose(0, 1).reshape({rows, d.KV});
      weight(i_w, dk, e.select(0, 0));
      if (needs(i_e)) grad[i_e] = at::mm(dk, w).view(e.sizes());
    };
    keys(3 * d.KV, d.T, pos, 1, wpos, 6);
    keys(3 * d.KV + d.T * d.KV, d.C, chan, 2, wchan, 7);
    weight(4, dq, xn);
    weight(5, dkv, xn);
    weight(10, dg, xn);
    weight(11, dup, xn);
    if (needs(0) || needs(3)) {
      Tensor dxn = at::mm(dq, wq);
      dxn.addmm_(dkv, wkv);
      dxn.addmm_(dg, wg);
      dxn.addmm_(dup, wu);
      grad[0] = at::empty(x.sizes(), x.options().requires_grad(false));
      grad[3] = at::empty_like(ln_w);
      const size_t bytes = api.rmsnorm_bwd_bytes(d.rows, (int32_t)d.E);
      const Tensor ws = scratch(bytes, x);
      check(api.rmsnorm_bwd(x.const_data_ptr(), ln_w.const_data_ptr(), dxn.const_data_ptr(), dh2.const_data_ptr(), grad[0].data_ptr(),
                            grad[3].data_ptr(), d.rows, (int32_t)d.E, (float)eps, dt, ws.data_ptr(), bytes, stream_of(x)), "mvpa_rmsnorm_bwd");
    }
  }
  return wrap(std::move(grad));
  END_HANDLE_TH_ERRORS
}

// branches(x, w_in, w_out, bias, r_time, r_chan, window, B, T, C, H, Hkv, D, status): MLP(x) + Attn(x) of the fused inference block
//   (`MVPFormerBlock.fused_branches`), or None
PyObject* branches(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!arguments(n, 14)) return nullptr;
  const bool status = a[13] == Py_True;
  Tensor in[6];
  for (int i = 0; i < 6; ++i) {
    if (!THPVariable_CheckExact(a[i])) Py_RETURN_NONE;
    in[i] = THPVariable_Unpack(a[i]);
    if (!ordinary(in[i]) || !in[i].is_contiguous() || in[i].device() != in[0].device() || in[i].scalar_type() != in[0].scalar_type() ||
        in[i].numel() == 0 || !aligned16(in[i].const_data_ptr()))
      Py_RETURN_NONE;
  }
  const Tensor &x = in[0], &w_in = in[1], &w_out = in[2], &bias = in[3], &rt = in[4], &rc = in[5];
  int64_t v[7];
  for (int i = 0; i < 7; ++i) v[i] = PyLong_AsLongLong(a[6 + i]);
  if (PyErr_Occurred()) return nullptr;
  Dims d;
  d.B = v[1]; d.T = v[2]; d.C = v[3]; d.H = v[4]; d.Hkv = v[5]; d.D = v[6];
  d.N = d.T * d.C; d.KV = d.Hkv * d.D; d.rows = d.B * d.N; d.E = d.H * d.D;
  const int dt = dtype_code(x);
  const int64_t I = x.dim() == 2 && w_in.dim() == 2 ? (w_in.size(0) - d.E - 2 * d.KV) / 2 : 0, es = x.element_size();
  if (I <= 0 || w_in.size(0) != d.E + 2 * (d.KV + I) || w_out.dim() != 2 || w_out.size(1) != d.E + I || d.KV <= 0 || d.rows <= 0 ||
      (dt != MVPA_BF16 && dt != MVPA_F32) || x.size(0) != d.rows || x.size(1) != d.E || I * es % 16 != 0 || bias.numel() != 3 * d.KV ||
      d.D * es % 16 != 0 || rt.numel() != d.T * d.KV || rc.numel() != d.C * d.KV || rt.size(-2) != d.T || rc.size(-2) != d.C ||
      function_modes() || watched())
    Py_RETURN_NONE;
  Tensor out;
  {
    pybind11::gil_scoped_release nogil;
    c10::cuda::CUDAGuard guard(x.device());
    c10::NoGradGuard no_grad;
    const Tensor big = at::linear(x, w_in);  // (rows, E + 2 KV + 2 I)
    if (big.scalar_type() == x.scalar_type()) {  // (autocast may have formed it in another type: Python's path follows that)
      const Tensor cat = at::empty({d.rows, d.E + I}, x.options().requires_grad(false));
      launch_fwd(d.problem(dt, 1.0 / std::sqrt((double)d.D), (int)v[0]), columns(big, 0, d.N, d.D), columns(big, d.E, d.N, d.D),
                 columns(big, d.E + d.KV, d.N, d.D), part(bias, 0), part(bias, d.KV), part(bias, 2 * d.KV), rt, rc,
                 columns(cat, 0, d.N, d.D), nullptr, status);
      const int64_t g0 = d.E + 2 * d.KV;
      check(api.silu_mul(part(big, g0), part(big, g0 + I), big.stride(0), const_cast<char*>(part(cat, d.E)), cat.stride(0), d.rows, (int32_t)I,
                         dt, stream_of(x)), "mvpa_silu_mul");
      out = at::linear(cat, w_out);
    }
  }
  if (!out.defined()) Py_RETURN_NONE;
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// init(path of libmvpa_b200.so, which is already loaded; the class of the mode that a default device is)
PyObject* init(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arguments(n, 2)) return nullptr;
  const char* p = PyUnicode_AsUTF8(a[0]);
  if (!p) return nullptr;
  Py_INCREF(a[1]);
  device_mode = a[1];
  void* so = dlopen(p, RTLD_NOW);
  if (!so) { PyErr_SetString(PyExc_ImportError, dlerror()); return nullptr; }
  const char* missing = nullptr;
  const auto get = [&](auto& f, const char* name) {
    f = reinterpret_cast<std::decay_t<decltype(f)>>(dlsym(so, name));
    if (!f) missing = name;
  };
  get(api.fwd_bytes, "mvpa_fwd_workspace_bytes"); get(api.bwd_bytes, "mvpa_bwd_workspace_bytes");
  get(api.fwd, "mvpa_fwd"); get(api.bwd, "mvpa_bwd");
  get(api.rmsnorm, "mvpa_rmsnorm"); get(api.rmsnorm_bwd, "mvpa_rmsnorm_bwd");
  get(api.rmsnorm_bwd_bytes, "mvpa_rmsnorm_bwd_workspace_bytes");
  get(api.silu_mul, "mvpa_silu_mul"); get(api.silu_mul_bwd, "mvpa_silu_mul_bwd");
  get(api.fwd_status, "mvpa_workspace_status"); get(api.bwd_status, "mvpa_bwd_status");
  get(api.last_error, "mvpa_last_error_string");
  if (missing) { PyErr_Format(PyExc_ImportError, "%s has no %s", p, missing); return nullptr; }
  Py_RETURN_NONE;
}

#define FAST(f) {#f, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {FAST(init), FAST(attend), FAST(forward), FAST(backward), FAST(plain), FAST(block_forward),
                         FAST(block_backward), FAST(branches), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "mvpa_host_b200", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_mvpa_host_b200() { return PyModule_Create(&module_def); }
