// Autograd nodes of the layers that most launches of a step come from (norms, linear layers, SwiGLU, attention), for the plain
// bf16 case of each: the same launchers, workspaces and results as the Python functions of ops/, which keep every other case
// (quantised operands, tensor parallelism, packed documents, other types) and run where this module is not built.
//
// Why: small layers wait for the host.  A Python function costs its call, a second one from the autograd thread, and a microsecond
// for every line and allocation between its launches, which is most of a layer of few tokens (200 x 2048 norm with residual, forward
// and backward: 125 us, here 93; a two-layer training step of 768 tokens 1560 and 890; a MoE layer of 64 tokens 640 and 375; an attention
// block of 128 tokens 500 and 240).
#include <torch/extension.h>

#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <dlfcn.h>

#include <atomic>
#include <map>
#include <mutex>
#include <tuple>

namespace py = pybind11;
using torch::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::Function;
using torch::autograd::variable_list;

namespace {

// ------------------------------------------------------------------ the launchers
void* library = nullptr;
PyObject *gemm_dict = nullptr, *autotune_dict = nullptr;      // module dictionaries (borrowed from modules that stay)
py::object *gemm_module = nullptr, *lib_module = nullptr;     // never released: used until the process ends
std::atomic<long> launches{0};

struct LaunchError : std::runtime_error {
  using std::runtime_error::runtime_error;
};

// A backward pass runs on a thread of the autograd engine: errors of Python code and of launches travel as Python errors.
template <typename F>
variable_list guarded(F f) {
  try {
    return f();
  } catch (py::error_already_set& e) {
    py::gil_scoped_acquire gil;
    e.restore();
    python_error err;
    err.persist();
    throw err;
  } catch (const LaunchError& e) {
    py::gil_scoped_acquire gil;
    PyErr_SetString(lib_module->attr("NativeLibraryError").ptr(), e.what());
    python_error err;
    err.persist();
    throw err;
  }
}

// An argument that the Python function refuses, with the class of error that it raises.
[[noreturn]] void refuse(PyObject* error, const char* why) {
  py::gil_scoped_acquire gil;
  PyErr_SetString(error, why);
  throw py::error_already_set();
}
void check_dims(const Tensor& t, long dims, const char* what) {      // (where it unpacks the shape)
  if (t.dim() != dims) refuse(PyExc_ValueError, what);
}

void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }
void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }

// What an argument travels as, as in launch.c: integers 64 bits wide (a launcher's 32-bit parameter reads the low half), pointers.
template <typename T>
std::enable_if_t<std::is_integral_v<T>, long> as_arg(T v) { return (long)v; }
inline float as_arg(float v) { return v; }
inline void* as_arg(void* v) { return v; }

void* symbol(const char* name) {        // pb_<name>
  static std::mutex m;
  static std::map<std::string, void*> known;
  std::lock_guard<std::mutex> g(m);
  void*& f = known[name];
  if (!f) f = dlsym(library, (std::string("pb_") + name).c_str());
  if (!f) throw LaunchError(std::string("pb_") + name + " not found");
  return f;
}

// pb_<name>(args..., stream); `kernels`: how many it launches
template <typename... A>
void launch(const char* name, int kernels, A... a) {
  using Fn = int (*)(decltype(as_arg(a))..., void*);
  const int rc = reinterpret_cast<Fn>(symbol(name))(as_arg(a)..., stream());
  launches.fetch_add(kernels, std::memory_order_relaxed);
  if (rc) throw LaunchError(std::string("pb_") + name + " failed with code " + std::to_string(rc));
}

// rows of partial sums that the norms' backward passes write for so many rows, as the library has it
long partial_rows(long rows) {
  static const auto f = reinterpret_cast<int (*)(long)>(symbol("rmsnorm_bwd_num_partials"));
  return f(rows);
}

// the device's status word, which ops/_lib.py owns
int* status_word(const Tensor& like) {
  static std::mutex m;
  static std::map<int, int*> words;
  const int dev = like.get_device();
  {
    std::lock_guard<std::mutex> g(m);
    auto it = words.find(dev);
    if (it != words.end()) return it->second;
  }
  py::gil_scoped_acquire gil;
  int* p = (int*)lib_module->attr("status_word")(dev).cast<Tensor>().data_ptr();
  std::lock_guard<std::mutex> g(m);
  return words[dev] = p;
}

Tensor empty(at::IntArrayRef sizes, const Tensor& like, at::ScalarType type) { return at::empty(sizes, like.options().dtype(type)); }

// ------------------------------------------------------------------ GEMM
// (with the GIL) whether every GEMM takes the plain bf16 route: no quantised recipe, no tuned or overridden tile options
bool plain_gemms() {
  auto none = [](PyObject* d, const char* k) { PyObject* v = PyDict_GetItemString(d, k); return v == Py_None; };
  auto no = [](PyObject* d, const char* k) { PyObject* v = PyDict_GetItemString(d, k); return v && PyObject_IsTrue(v) == 0; };
  return none(gemm_dict, "_FP8_RECIPE") && none(gemm_dict, "_BLOCK_N_OVERRIDE") && no(autotune_dict, "_TABLE") &&
         no(autotune_dict, "_RECORD") && no(autotune_dict, "_ONLINE");
}

bool matrix(const Tensor& t, at::ScalarType type) {
  return t.is_cuda() && t.dim() == 2 && t.scalar_type() == type && t.stride(1) == 1;
}

// ops/gemm.py's choice for these sizes, asked for once
int route_of(long M, long N, long K, bool both_mn, long ldb, int out_bytes) {
  static std::mutex m;
  static std::map<std::tuple<long, long, long, bool, long, int>, int> known;
  const auto key = std::make_tuple(M, N, K, both_mn, ldb, out_bytes);
  {
    std::lock_guard<std::mutex> g(m);
    auto it = known.find(key);
    if (it != known.end()) return it->second;
  }
  int r;
  {
    py::gil_scoped_acquire gil;
    r = gemm_module->attr("_bf16_route")(M, N, K, both_mn, ldb, out_bytes, 0).cast<int>();
  }
  std::lock_guard<std::mutex> g(m);
  if (known.size() > 4096) known.clear();
  return known[key] = r;
}

// out (+)= A . B^T as gemm.gemm computes it (a_mn / b_mn: the stored matrix is the transpose); `plain`: see above
void gemm(const Tensor& a, const Tensor& b, bool a_mn, bool b_mn, const Tensor& out, bool accumulate, bool plain) {
  const long M = a.size(a_mn ? 1 : 0), K = a.size(a_mn ? 0 : 1), N = b.size(b_mn ? 1 : 0);
  const bool f32 = out.scalar_type() == at::kFloat;
  if (!plain || !matrix(a, at::kBFloat16) || !matrix(b, at::kBFloat16) || !out.is_cuda() || out.stride(1) != 1 ||
      (!f32 && out.scalar_type() != at::kBFloat16) || (accumulate && !f32) || K != b.size(b_mn ? 0 : 1) || out.size(0) != M ||
      out.size(1) != N) {
    py::gil_scoped_acquire gil;
    gemm_module->attr("gemm")(a, b, a_mn, b_mn, py::arg("out") = out, py::arg("accumulate") = accumulate);
    return;
  }
  if (M == 0 || N == 0) return;
  if (K == 0) {
    if (!accumulate) out.zero_();
    return;
  }
  const int mode = !f32 ? 0 : accumulate ? 2 : 1, am = a_mn, bm = b_mn, m = (int)M, n = (int)N, k = (int)K;
  const long lda = a.stride(0), ldb = b.stride(0), ldo = out.stride(0);
  const int block_n = N <= 128 ? 128 : 256;
  static constexpr int out_bytes[] = {2, 4, 8};
  const int route = block_n == 256 ? route_of(M, N, K, a_mn && b_mn, ldb, out_bytes[mode]) : 0;
  int* status = status_word(a);
  if (route > 1) {
    const Tensor ws = empty({route * ((M + 255) / 256 * 256) * N}, a, at::kFloat);
    launch("gemm_bf16_splitk", 2, ptr(a), ptr(b), ptr(out), ptr(ws), m, n, k, lda, ldb, ldo, am, bm, mode, route, (void*)status);
  } else if (route == 1) {
    launch("gemm_bf16_2cta", 1, ptr(a), ptr(b), ptr(out), m, n, k, lda, ldb, ldo, am, bm, mode, 0, (void*)status);
  } else {
    launch("gemm_bf16", 1, ptr(a), ptr(b), ptr(out), m, n, k, lda, ldb, ldo, am, bm, mode, block_n, 0, (void*)status);
  }
}

// dW = dy^T x as gemm.wgrad: into the weight's main_grad (undefined is returned), else as a gradient of its type
Tensor wgrad(const Tensor& dy, const Tensor& x, const Tensor& weight) {
  py::gil_scoped_acquire gil;
  py::object w = py::cast(weight);
  const bool plain = plain_gemms() && gemm_module->attr("WGRAD_STORE").attr("current").is_none();
  py::object main_grad = py::getattr(w, "main_grad", py::none());
  if (!plain || (main_grad.is_none() && weight.scalar_type() != at::kBFloat16)) {
    py::object r = gemm_module->attr("wgrad")(dy, x, w);
    return r.is_none() ? Tensor() : r.cast<Tensor>();
  }
  if (main_grad.is_none()) {
    Tensor out = empty({dy.size(1), x.size(1)}, dy, at::kBFloat16);
    gemm(dy, x, true, true, out, false, plain);
    return out;
  }
  gemm(dy, x, true, true, main_grad.cast<Tensor>(), true, plain);
  py::setattr(w, "grad_added_to_main_grad", py::bool_(true));
  py::object ready = py::getattr(w, "_grad_ready_cb", py::none());
  if (!ready.is_none()) ready(w);
  return Tensor();
}

// the fp32 buffer that a parameter's gradient is added to, if it owns one
Tensor main_grad_of(const Tensor& weight) {
  py::gil_scoped_acquire gil;
  py::object g = py::getattr(py::cast(weight), "main_grad", py::none());
  return g.is_none() ? Tensor() : g.cast<Tensor>();
}

bool plain_now() {
  py::gil_scoped_acquire gil;
  return plain_gemms();
}

// ------------------------------------------------------------------ norms
bool aligned(const Tensor& t) { return (uintptr_t)t.data_ptr() % 16 == 0; }
Tensor as_rows(const Tensor& t, long H) { return t.dim() == 2 ? t : t.reshape({-1, H}); }
Tensor as_shape(const Tensor& t, at::IntArrayRef shape) { return t.sizes() == shape ? t : t.view(shape); }
Tensor dense_rows(const Tensor& t) { return t.is_contiguous() ? (aligned(t) ? t : t.clone()) : t.contiguous(); }

// (an input that may be missing is an optional: the nodes take no undefined tensors)
using Opt = std::optional<Tensor>;
Tensor given(const Opt& t) { return t ? *t : Tensor(); }

struct NormOut {
  Tensor y, xsum, rstd;
};
NormOut norm_forward(const Tensor& x, const Tensor& w, double eps, const Tensor& residual) {
  const long H = x.size(-1);
  Tensor x2 = as_rows(x, H), r2;
  if (residual.defined()) {
    x2 = dense_rows(x2);
    r2 = dense_rows(as_rows(residual, H));
  } else if (x2.stride(1) != 1 || !aligned(x2)) {
    x2 = dense_rows(x2);
  }
  NormOut o;
  const long rows = x2.size(0);
  o.y = at::empty_like(x2);
  o.rstd = empty({rows}, x2, at::kFloat);
  if (residual.defined()) o.xsum = at::empty_like(x2);
  launch("rmsnorm_fwd", 1, ptr(x2), ptr(r2), ptr(w), ptr(o.y), ptr(o.xsum), ptr(o.rstd), rows, (int)H, (long)x2.stride(0),
         (long)o.y.stride(0), (float)eps);
  if (!residual.defined()) o.xsum = x2;
  return o;
}

struct NormGrads {
  Tensor dx, dx2, dw;
};
// fused.norm_backward; y (undefined: not wanted) receives the normalised rows
NormGrads norm_backward(const Tensor& dy, const Tensor& xin_, const Tensor& w, const Tensor& rstd, const Tensor& dres, bool two,
                        at::IntArrayRef shape, const Tensor& y) {
  const Tensor xin = xin_.contiguous();
  const long rows = xin.size(0), H = xin.size(1);
  Tensor target = main_grad_of(w);
  int mode;
  NormGrads g;
  if (target.defined()) {
    mode = 1;
  } else if (w.scalar_type() == at::kBFloat16) {
    target = g.dw = empty({H}, xin, at::kBFloat16);
    mode = 2;
  } else {
    target = empty({H}, xin, at::kFloat);
    mode = 0;
  }
  g.dx = at::empty_like(xin);
  if (two) g.dx2 = at::empty_like(xin);
  const Tensor partial = empty({partial_rows(rows) * H}, xin, at::kFloat);
  const long ldx = xin.stride(0), ldy = dy.stride(0);
  if (y.defined())
    launch("rmsnorm_bwd_y", 2, ptr(dy), ptr(xin), ptr(w), ptr(rstd), ptr(dres), ptr(g.dx), ptr(g.dx2), ptr(y), ptr(target), ptr(partial),
           rows, (int)H, ldx, ldy, mode);
  else if (two)
    launch("rmsnorm_bwd_two", 2, ptr(dy), ptr(xin), ptr(w), ptr(rstd), ptr(dres), ptr(g.dx), ptr(g.dx2), ptr(target), ptr(partial), rows,
           (int)H, ldx, ldy, mode);
  else
    launch("rmsnorm_bwd", 2, ptr(dy), ptr(xin), ptr(w), ptr(rstd), ptr(dres), ptr(g.dx), ptr(target), ptr(partial), rows, (int)H, ldx,
           ldy, mode);
  if (mode == 0) g.dw = target.to(w.scalar_type());
  g.dx = as_shape(g.dx, shape);
  g.dx2 = two ? as_shape(g.dx2, shape) : g.dx;
  return g;
}

// Two leaves that both lack a gradient get tensors of their own (fused.two_leaves; where autograd hands the gradients out instead of
// accumulating them that is only a store more).
void remember_leaves(AutogradContext* ctx, const Tensor& a, const Tensor& b) {
  if (b.defined() && a.is_leaf() && b.is_leaf() && a.requires_grad() && b.requires_grad() && !a.is_same(b)) {
    ctx->saved_data["leaf_a"] = a;
    ctx->saved_data["leaf_b"] = b;
  }
}
bool two_leaves(AutogradContext* ctx) {
  auto a = ctx->saved_data.find("leaf_a");
  return a != ctx->saved_data.end() && !a->second.toTensor().grad().defined() && !ctx->saved_data["leaf_b"].toTensor().grad().defined();
}
// inputs that autograd does not save: parameters, whose attributes the backward pass reads
void keep(AutogradContext* ctx, const char* name, const Tensor& t) { ctx->saved_data[name] = t; }
Tensor kept(AutogradContext* ctx, const char* name) { return ctx->saved_data[name].toTensor(); }

struct RMSNorm : Function<RMSNorm> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, const Opt& residual_, double eps) {
    const Tensor residual = given(residual_);
    const NormOut o = norm_forward(x, w, eps, residual);
    ctx->save_for_backward({o.xsum, w, o.rstd});
    keep(ctx, "w", w);
    ctx->saved_data["shape"] = x.sizes().vec();
    ctx->saved_data["res"] = residual.defined();
    ctx->set_materialize_grads(false);
    remember_leaves(ctx, x, residual);
    if (!residual.defined()) return {as_shape(o.y, x.sizes())};
    return {as_shape(o.y, x.sizes()), as_shape(o.xsum, x.sizes())};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    return guarded([&]() -> variable_list {
      const auto saved = ctx->get_saved_variables();
      const Tensor &xin = saved[0], &rstd = saved[2];
      const long H = xin.size(-1);
      const bool res = ctx->saved_data["res"].toBool();
      Tensor dres, dy = grads[0].defined() ? dense_rows(as_rows(grads[0], H)) : at::zeros_like(xin, {}, at::MemoryFormat::Contiguous);
      if (res && grads[1].defined()) dres = dense_rows(as_rows(grads[1], H));
      const auto shape = ctx->saved_data["shape"].toIntVector();
      const NormGrads g = norm_backward(dy, xin, kept(ctx, "w"), rstd, dres, dres.defined() && two_leaves(ctx), shape, Tensor());
      return {g.dx, g.dw, res ? g.dx2 : Tensor(), Tensor()};
    });
  }
};

struct NormLinear : Function<NormLinear> {
  static variable_list forward(AutogradContext* ctx, const Tensor& hidden, const Tensor& norm_w, const Tensor& weight,
                               const Opt& residual_, double eps) {
    const Tensor residual = given(residual_);
    const NormOut o = norm_forward(hidden, norm_w, eps, residual);
    Tensor out = empty({o.y.size(0), weight.size(0)}, o.y, at::kBFloat16);
    gemm(o.y, weight, false, false, out, false, true);
    ctx->save_for_backward({o.xsum, norm_w, weight, o.rstd});
    keep(ctx, "norm_w", norm_w);
    keep(ctx, "w", weight);
    ctx->saved_data["shape"] = hidden.sizes().vec();
    ctx->saved_data["res"] = residual.defined();
    ctx->saved_data["eps"] = eps;
    ctx->set_materialize_grads(false);
    remember_leaves(ctx, hidden, residual);
    return {out, residual.defined() ? as_shape(o.xsum, hidden.sizes()) : hidden};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    return guarded([&]() -> variable_list {
      const auto saved = ctx->get_saved_variables();
      const Tensor &xsum = saved[0], &norm_w = saved[1], &weight = saved[2], &rstd = saved[3];
      const long rows = xsum.size(0), H = xsum.size(1);
      Tensor dout = grads[0].defined() ? as_rows(grads[0], weight.size(0)).contiguous()
                                       : at::zeros({rows, weight.size(0)}, xsum.options());
      const bool plain = plain_now(), early = H <= 64;
      Tensor y, dw;
      if (early) {                         // (rows that the norm's kernel for few channels takes: recomputed on their own)
        y = at::empty_like(xsum);
        launch("rmsnorm_fwd", 1, ptr(xsum), (void*)nullptr, ptr(norm_w), ptr(y), (void*)nullptr, (void*)nullptr, rows, (int)H,
               (long)xsum.stride(0), (long)y.stride(0), (float)ctx->saved_data["eps"].toDouble());
        dw = wgrad(dout, y, kept(ctx, "w"));
      } else {
        y = empty({rows, H}, xsum, at::kBFloat16);
      }
      Tensor dy = empty({rows, H}, xsum, at::kBFloat16);
      gemm(dout, weight, false, true, dy, false, plain);
      Tensor dres;
      if (grads[1].defined()) dres = dense_rows(as_rows(grads[1], H));
      const auto shape = ctx->saved_data["shape"].toIntVector();
      const NormGrads g = norm_backward(dy, xsum, kept(ctx, "norm_w"), rstd, dres, dres.defined() && two_leaves(ctx), shape,
                                        early ? Tensor() : y);
      if (!early) dw = wgrad(dout, y, kept(ctx, "w"));
      return {g.dx, g.dw, dw, ctx->saved_data["res"].toBool() ? g.dx2 : Tensor(), Tensor()};
    });
  }
};

// ------------------------------------------------------------------ linear, SwiGLU
// channels of one half of [gate | up]
long half_of(long I2) {
  TORCH_CHECK(I2 % 2 == 0, "gated rows of ", I2, " values have no two halves");
  return I2 / 2;
}

struct Linear : Function<Linear> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& weight) {
    const Tensor x2 = as_rows(x, x.size(-1));
    Tensor y = empty({x2.size(0), weight.size(0)}, x, at::kBFloat16);
    gemm(x2, weight, false, false, y, false, true);
    ctx->save_for_backward({x2, weight});
    keep(ctx, "w", weight);
    ctx->saved_data["shape"] = x.sizes().vec();
    auto shape = x.sizes().vec();
    shape.back() = weight.size(0);
    return as_shape(y, shape);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    return guarded([&]() -> variable_list {
      const auto saved = ctx->get_saved_variables();
      const Tensor &x2 = saved[0], &weight = saved[1];
      const Tensor dy = as_rows(grads[0], grads[0].size(-1)).contiguous();
      Tensor dx, dw;
      if (ctx->needs_input_grad(0)) {
        dx = empty({dy.size(0), weight.size(1)}, dy, at::kBFloat16);
        gemm(dy, weight, false, true, dx, false, plain_now());
        dx = as_shape(dx, ctx->saved_data["shape"].toIntVector());
      }
      if (ctx->needs_input_grad(1)) dw = wgrad(dy, x2, kept(ctx, "w"));
      return {dx, dw};
    });
  }
};

struct SwiGLULinear : Function<SwiGLULinear> {
  static Tensor forward(AutogradContext* ctx, const Tensor& h1, const Tensor& weight, double clamp, int64_t kind) {
    const long I2 = h1.size(-1), I = half_of(I2);
    const Tensor x2 = as_rows(h1, I2);
    const long T = x2.size(0);
    const Tensor act = empty({T, I}, h1, at::kBFloat16);
    launch("swiglu_fwd", 1, ptr(x2), (void*)nullptr, ptr(act), T, (int)I, (float)clamp, (int)kind);
    Tensor out = empty({T, weight.size(0)}, h1, at::kBFloat16);
    gemm(act, weight, false, false, out, false, true);
    ctx->save_for_backward({x2, weight});
    keep(ctx, "w", weight);
    ctx->saved_data["clamp"] = clamp;
    ctx->saved_data["kind"] = kind;
    ctx->saved_data["shape"] = h1.sizes().vec();
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    return guarded([&]() -> variable_list {
      const auto saved = ctx->get_saved_variables();
      const Tensor &x2 = saved[0], &weight = saved[1];
      const long T = x2.size(0), I = x2.size(1) / 2;
      const Tensor dout = as_rows(grads[0], grads[0].size(-1)).contiguous();
      Tensor dact = empty({T, I}, x2, at::kBFloat16);
      gemm(dout, weight, false, true, dact, false, plain_now());
      const Tensor din = at::empty_like(x2);
      // (the activation for the weight gradient, in the place of its own gradient)
      launch("swiglu_bwd_act", 1, ptr(dact), ptr(x2), (void*)nullptr, ptr(din), (void*)nullptr, ptr(dact), T, (int)I,
             (float)ctx->saved_data["clamp"].toDouble(), (int)ctx->saved_data["kind"].toInt());
      const Tensor dw = wgrad(dout, dact, kept(ctx, "w"));
      return {as_shape(din, ctx->saved_data["shape"].toIntVector()), dw, Tensor(), Tensor()};
    });
  }
};

// ------------------------------------------------------------------ attention
void check_view(const Tensor& t, long d) {     // (attention._check_view, and its class of error)
  if (t.dim() < 3) refuse(PyExc_IndexError, "heads must be [T, H, D]");
  if (t.stride(2) != 1 || t.stride(1) != d || !aligned(t))
    refuse(PyExc_AssertionError, "heads must be contiguous [.., H, D] views");
}

struct AttnArgs {
  long batch;
  bool causal;
  double scale;
  long q_off, window;
  double softcap;
};
AttnArgs attn_args(long batch, bool causal, double scale, long q_off, long window, double softcap) {
  if (batch == 0) refuse(PyExc_ZeroDivisionError, "attention of rows that belong to no sequence");    // (as T // batch does)
  return {batch, causal, scale, q_off, window, softcap};
}
void save_args(AutogradContext* ctx, const AttnArgs& a) {
  ctx->saved_data["args"] = std::vector<int64_t>{a.batch, a.causal, a.q_off, a.window};
  ctx->saved_data["fargs"] = std::vector<double>{a.scale, a.softcap};
}
AttnArgs load_args(AutogradContext* ctx) {
  const auto i = ctx->saved_data["args"].toIntVector();
  const auto f = ctx->saved_data["fargs"].toDoubleVector();
  return {i[0], i[1] != 0, f[0], i[2], i[3], f[1]};
}

std::pair<Tensor, Tensor> attn_forward(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& sinks, const AttnArgs& a) {
  const long T = q.size(0), hq = q.size(1), dqk = q.size(2), hkv = k.size(1), dv = v.size(2), S = T / a.batch, SK = k.size(0) / a.batch;
  check_view(q, dqk);
  check_view(k, dqk);
  check_view(v, dv);
  Tensor o = empty({T, hq, dv}, q, at::kBFloat16), lse = empty({a.batch, hq, S}, q, at::kFloat);
  launch("flash_attn_fwd_cap", 1, ptr(q), ptr(k), ptr(v), ptr(o), ptr(lse), (int)a.batch, (int)S, (int)SK, (int)a.q_off, (int)hq, (int)hkv,
         (int)dqk, (int)dv, (long)q.stride(0), (long)k.stride(0), (long)v.stride(0), (long)o.stride(0), (float)a.scale, (int)a.causal,
         (int)a.window, ptr(sinks), (float)a.softcap, (void*)status_word(q));
  return {o, lse};
}

// returns the gradient of the sinks (undefined without any)
Tensor attn_backward(const Tensor& dout, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o, const Tensor& lse,
                     const Tensor& sinks, const AttnArgs& a, const Tensor& dq, const Tensor& dk, const Tensor& dv) {
  const long T = q.size(0), hq = q.size(1), dqk = q.size(2), hkv = k.size(1), dvd = v.size(2), S = T / a.batch, SK = k.size(0) / a.batch;
  const Tensor d = dout.stride(2) == 1 && dout.stride(1) == dvd ? dout : dout.contiguous();
  for (const Tensor* t : {&q, &k, &dq, &dk}) check_view(*t, dqk);
  for (const Tensor* t : {&v, &o, &d, &dv}) check_view(*t, dvd);
  const Tensor delta = empty({2, a.batch, hq, S}, q, at::kFloat);   // row sums of dO * O; log-sum-exp in base 2
  launch("flash_attn_bwd_cap", 3, ptr(d), ptr(q), ptr(k), ptr(v), ptr(o), ptr(lse), ptr(delta), ptr(dq), ptr(dk), ptr(dv), (int)a.batch,
         (int)S, (int)SK, (int)a.q_off, (int)hq, (int)hkv, (int)dqk, (int)dvd, (long)q.stride(0), (long)k.stride(0), (long)v.stride(0),
         (long)o.stride(0), (long)d.stride(0), (long)dq.stride(0), (long)dk.stride(0), (long)dv.stride(0), (float)a.scale, (int)a.causal,
         (int)a.window, (float)a.softcap, (void*)status_word(q));
  if (!sinks.defined()) return Tensor();
  const Tensor dsinks = at::empty_like(sinks);
  launch("attn_sink_grad", 1, ptr(delta), ptr(lse), ptr(sinks), ptr(dsinks), (int)a.batch, (int)S, (int)hq);
  return dsinks;
}

struct FlashAttention : Function<FlashAttention> {
  static Tensor forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const Opt& sinks_, int64_t batch,
                        bool causal, double scale, int64_t q_off, int64_t window, double softcap) {
    const Tensor sinks = given(sinks_);
    check_dims(q, 3, "queries must be [T, H, D]");
    const AttnArgs a = attn_args(batch, causal, scale, q_off, window, softcap);
    const auto [o, lse] = attn_forward(q, k, v, sinks, a);
    ctx->save_for_backward({q, k, v, o, lse, sinks});
    save_args(ctx, a);
    return o;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    return guarded([&]() -> variable_list {
      const auto s = ctx->get_saved_variables();
      const Tensor dq = empty(s[0].sizes(), s[0], at::kBFloat16), dk = empty(s[1].sizes(), s[1], at::kBFloat16),
                   dv = empty(s[2].sizes(), s[2], at::kBFloat16);
      const Tensor ds = attn_backward(grads[0], s[0], s[1], s[2], s[3], s[4], s[5], load_args(ctx), dq, dk, dv);
      return {dq, dk, dv, ds, Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
    });
  }
};

// What heads() takes for granted (the Python function's slices and views refuse the rest)
void check_packed(const Tensor& qkv, long hq, long hkv, long d) {
  if (qkv.dim() != 2 || qkv.size(1) != (hq + 2 * hkv) * d) refuse(PyExc_RuntimeError, "packed heads must be [T, (Hq + 2 Hkv) D]");
  if (qkv.stride(1) != 1 || !aligned(qkv)) refuse(PyExc_AssertionError, "packed heads must be contiguous rows");
}
// q, k and v heads inside a packed [T, (hq + 2 hkv) d] tensor
std::tuple<Tensor, Tensor, Tensor> heads(const Tensor& qkv, long hq, long hkv, long d) {
  const long T = qkv.size(0), ld = qkv.stride(0);
  auto part = [&](long first, long n) { return qkv.as_strided({T, n, d}, {ld, d, 1}, qkv.storage_offset() + first * d); };
  return {part(0, hq), part(hq, hkv), part(hq + hkv, hkv)};
}

struct RopeAttention : Function<RopeAttention> {
  static Tensor forward(AutogradContext* ctx, const Tensor& qkv, const Opt& sinks_, const Opt& cos_, const Opt& sin_, const Opt& pos_,
                        int64_t batch, int64_t hq, int64_t hkv, int64_t d, int64_t rot_dim, bool causal, double scale, int64_t window,
                        double softcap) {
    const Tensor sinks = given(sinks_), cos = given(cos_), sin = given(sin_), pos = given(pos_);
    const AttnArgs a = attn_args(batch, causal, scale, 0, window, softcap);
    check_packed(qkv, hq, hkv, d);
    const auto [q, k, v] = heads(qkv, hq, hkv, d);
    // (in place: the projection's output has no other consumer; q and k heads are neighbours)
    if (cos.defined())
      launch("rope", 1, ptr(qkv), ptr(pos), ptr(cos), ptr(sin), (long)qkv.size(0), (int)(hq + hkv), (int)d, (int)rot_dim, (long)qkv.stride(0), 0);
    const auto [o, lse] = attn_forward(q, k, v, sinks, a);
    ctx->save_for_backward({qkv, o, lse, cos, sin, pos, sinks});
    save_args(ctx, a);
    ctx->saved_data["dims"] = std::vector<int64_t>{hq, hkv, d, rot_dim};
    return o.view({qkv.size(0), hq * d});
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    return guarded([&]() -> variable_list {
      const auto s = ctx->get_saved_variables();
      const auto dims = ctx->saved_data["dims"].toIntVector();
      const long hq = dims[0], hkv = dims[1], d = dims[2], T = s[0].size(0);
      const Tensor dqkv = at::empty_like(s[0]);
      const auto [q, k, v] = heads(s[0], hq, hkv, d);
      const auto [dq, dk, dv] = heads(dqkv, hq, hkv, d);
      const Tensor ds = attn_backward(grads[0].reshape({T, hq, d}), q, k, v, s[1], s[2], s[6], load_args(ctx), dq, dk, dv);
      if (s[3].defined())
        launch("rope", 1, ptr(dqkv), ptr(s[5]), ptr(s[3]), ptr(s[4]), T, (int)(hq + hkv), (int)d, (int)dims[3], (long)dqkv.stride(0), 1);
      variable_list out(14);
      out[0] = dqkv;
      out[1] = ds;
      return out;
    });
  }
};

struct QKNorm : Function<QKNorm> {
  static Tensor forward(AutogradContext* ctx, const Tensor& qkv, const Tensor& wq, const Tensor& wk, const Opt& cos_, const Opt& sin_,
                        const Opt& pos_, int64_t hq, int64_t hkv, int64_t d, double eps, int64_t rot_dim) {
    const Tensor cos = given(cos_), sin = given(sin_), pos = given(pos_);
    const long T = qkv.size(0);
    const Tensor out = empty({T, (hq + 2 * hkv) * d}, qkv, at::kBFloat16), rstd = empty({T, hq + hkv}, qkv, at::kFloat);
    launch("qk_norm_rope_fwd", 1, ptr(qkv), ptr(wq), ptr(wk), ptr(out), ptr(rstd), T, (int)hq, (int)hkv, (int)d, (long)qkv.stride(0),
           (long)out.stride(0), (float)eps, ptr(pos), ptr(cos), ptr(sin), (int)rot_dim);
    ctx->save_for_backward({qkv, wq, wk, rstd, cos, sin, pos});
    keep(ctx, "wq", wq);
    keep(ctx, "wk", wk);
    ctx->saved_data["dims"] = std::vector<int64_t>{hq, hkv, d, rot_dim};
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    return guarded([&]() -> variable_list {
      const auto s = ctx->get_saved_variables();
      const Tensor &qkv = s[0], &wq = s[1], &wk = s[2];
      const auto dims = ctx->saved_data["dims"].toIntVector();
      const long hq = dims[0], hkv = dims[1], d = dims[2], T = qkv.size(0);
      const Tensor dy = dense_rows(grads[0]), dx = empty({T, (hq + 2 * hkv) * d}, qkv, at::kBFloat16);
      Tensor target[2] = {main_grad_of(kept(ctx, "wq")), main_grad_of(kept(ctx, "wk"))}, dw[2];
      for (int i = 0; i < 2; ++i)
        if (!target[i].defined()) target[i] = dw[i] = at::zeros({d}, qkv.options().dtype(at::kFloat));
      const Tensor partial = empty({partial_rows(T) * 2 * d}, qkv, at::kFloat);
      launch("qk_norm_rope_bwd", 3, ptr(dy), ptr(qkv), ptr(wq), ptr(wk), ptr(s[3]), ptr(dx), ptr(target[0]), ptr(target[1]), ptr(partial), T,
             (int)hq, (int)hkv, (int)d, (long)qkv.stride(0), (long)dy.stride(0), (long)dx.stride(0), 1, ptr(s[6]), ptr(s[4]), ptr(s[5]),
             (int)dims[3]);
      variable_list out(11);
      out[0] = dx;
      for (int i = 0; i < 2; ++i)
        if (dw[i].defined()) out[1 + i] = dw[i].to((i ? wk : wq).scalar_type());
      return out;
    });
  }
};

// ------------------------------------------------------------------ embedding, loss
struct Embedding : Function<Embedding> {
  static Tensor forward(AutogradContext* ctx, const Tensor& tokens, const Tensor& weight) {
    ctx->save_for_backward({tokens});
    keep(ctx, "w", weight);
    return at::embedding(weight, tokens);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    return guarded([&]() -> variable_list {
      const Tensor w = kept(ctx, "w"), tokens = ctx->get_saved_variables()[0].reshape({-1}).contiguous();
      const Tensor dy = grads[0].reshape({-1, w.size(1)}).contiguous();
      Tensor target = main_grad_of(w);
      const bool own = !target.defined();
      if (own) target = at::zeros(w.sizes(), w.options().dtype(at::kFloat));
      launch("embedding_bwd", 1, ptr(dy), ptr(tokens), ptr(target), tokens.numel(), w.size(1), 0, w.size(0));
      return {Tensor(), own ? target.to(w.scalar_type()) : Tensor()};
    });
  }
};

// fused.CrossEntropyFn of one rank: the gradient takes the place of the logits in the forward pass
struct CrossEntropy : Function<CrossEntropy> {
  static Tensor forward(AutogradContext* ctx, const Tensor& logits, const Tensor& labels, const Opt& weights, bool unit) {
    const long V = logits.size(-1);
    const Tensor l2 = as_rows(logits, V), lab = labels.reshape({-1}).contiguous();
    const long rows = l2.size(0);
    TORCH_CHECK(lab.numel() == rows && (!weights || weights->numel() == rows), "cross entropy of ", rows, " rows: ", lab.numel(), " labels, ",
                weights ? weights->numel() : rows, " weights");
    const Tensor scale = weights ? weights->reshape({-1}).to(at::kFloat).contiguous() : at::ones({rows}, logits.options().dtype(at::kFloat));
    const Tensor loss = empty({rows}, logits, at::kFloat);
    launch("ce_fused", 1, ptr(l2), ptr(lab), ptr(scale), ptr(loss), rows, V, l2.stride(0));
    ctx->save_for_backward({l2});
    ctx->saved_data["shape"] = logits.sizes().vec();
    ctx->saved_data["unit"] = unit && weights.has_value();
    ctx->saved_data["weighted"] = weights.has_value();
    if (!weights) return loss.view(labels.sizes());
    const Tensor total = empty({}, logits, at::kFloat);
    launch("weighted_sum", 1, ptr(loss), ptr(scale), ptr(total), rows);
    return total;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    return guarded([&]() -> variable_list {
      Tensor g = ctx->get_saved_variables()[0];
      if (!ctx->saved_data["unit"].toBool())
        g.mul_((ctx->saved_data["weighted"].toBool() ? grads[0] : grads[0].reshape({-1, 1})).to(g.scalar_type()));
      return {g.view(ctx->saved_data["shape"].toIntVector()), Tensor(), Tensor(), Tensor()};
    });
  }
};

// ------------------------------------------------------------------ mixture of experts (ops/moe.py)
struct Router : Function<Router> {
  static variable_list forward(AutogradContext* ctx, const Tensor& logits_, const Opt& bias_, int64_t topk, bool sigmoid, bool pre_softmax,
                               int64_t groups, int64_t group_topk, double scale, const std::optional<double>& aux_coeff) {
    check_dims(logits_, 2, "logits must be [T, E]");
    const Tensor logits = logits_.contiguous();
    const long T = logits.size(0), E = logits.size(1);
    Tensor bias, aux, sums;
    if (bias_) bias = bias_->to(at::kFloat).contiguous();
    const Tensor probs = empty({T, topk}, logits, at::kFloat), idx = empty({T, topk}, logits, at::kInt), idx64 = empty({T, topk}, logits, at::kLong),
                 full = empty({T, E}, logits, at::kFloat), ws = empty({E + 33}, logits, at::kInt);
    double factor = 0.0;
    if (aux_coeff) {
      aux = empty({}, logits, at::kFloat);
      sums = empty({(T + 7) / 8, E}, logits, at::kFloat);
      factor = *aux_coeff * (double)E;
    }
    launch("moe_route", aux_coeff ? 2 : 1, ptr(logits), 1, ptr(bias), T, E, topk, sigmoid, pre_softmax, groups, group_topk, (float)scale,
           ptr(probs), ptr(idx), ptr(idx64), ptr(full), ptr(ws), ptr(aux), ptr(sums), (float)factor);
    const Tensor counts = ws.narrow(0, 0, E);
    ctx->save_for_backward({full, idx, probs, counts});
    ctx->saved_data["cfg"] = std::vector<int64_t>{topk, sigmoid, pre_softmax};
    ctx->saved_data["fcfg"] = std::vector<double>{scale, factor};
    ctx->mark_non_differentiable({idx64, counts});
    ctx->set_materialize_grads(false);
    if (!aux_coeff) return {probs, idx64, full, counts};
    return {probs, idx64, full, counts, aux};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    return guarded([&]() -> variable_list {
      const auto s = ctx->get_saved_variables();
      const auto cfg = ctx->saved_data["cfg"].toIntVector();
      const auto f = ctx->saved_data["fcfg"].toDoubleVector();
      const long T = s[0].size(0), E = s[0].size(1);
      const Tensor dlogits = empty({T, E}, s[0], at::kBFloat16);
      const Tensor dp = grads[0].defined() ? grads[0].to(at::kFloat).contiguous() : at::zeros_like(s[2]);
      const Tensor df = grads[2].defined() ? grads[2].to(at::kFloat).contiguous() : Tensor(), da = grads.size() > 4 ? grads[4] : Tensor();
      launch("router_bwd", 1, ptr(dp), ptr(df), ptr(s[0]), ptr(s[1]), ptr(s[2]), T, E, cfg[0], cfg[1], cfg[2], (float)f[0], ptr(da),
             ptr(s[3]), (float)f[1], 1, ptr(dlogits));
      variable_list out(9);
      out[0] = dlogits;
      return out;
    });
  }
};

struct LocalPlan : Function<LocalPlan> {
  static variable_list forward(AutogradContext* ctx, const Tensor& probs, const Tensor& idx, const Tensor& counts, int64_t topk, int64_t rows_cap) {
    const long E = counts.numel(), R = idx.numel(), blocks = rows_cap / 128;
    const auto ints = empty({R + 2 * rows_cap + blocks + 2 * E + 1}, probs, at::kInt).split_with_sizes({R, rows_cap, rows_cap, blocks, E, E, 1});
    const Tensor &src = ints[1], &src_token = ints[2], &mblock = ints[3], &row_start = ints[4], &padded = ints[5], &total = ints[6];
    const Tensor pos = ints[0].view({-1, topk}), out = empty({rows_cap}, probs, at::kFloat);
    launch("moe_local_plan", 1, ptr(idx), ptr(counts), ptr(probs), R, topk, E, rows_cap, blocks, ptr(padded), ptr(row_start), ptr(mblock),
           ptr(total), ptr(src), ptr(src_token), ptr(pos), ptr(out));
    ctx->save_for_backward({pos});
    ctx->saved_data["shape"] = probs.sizes().vec();
    ctx->mark_non_differentiable({pos, src_token, padded, row_start, mblock, total});
    ctx->set_materialize_grads(false);
    return {out, pos, src_token, padded, row_start, mblock, total};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    return guarded([&]() -> variable_list {
      variable_list out(5);
      if (!grads[0].defined()) return out;
      const Tensor pos = ctx->get_saved_variables()[0], d = grads[0].to(at::kFloat).contiguous();
      out[0] = empty(ctx->saved_data["shape"].toIntVector(), d, at::kFloat);
      launch("gather_f32", 1, ptr(d), ptr(pos), ptr(out[0]), pos.numel());
      return out;
    });
  }
};

Tensor gather(const Tensor& x, const Tensor& src) {
  const long R = src.numel(), H = x.size(-1);
  const Tensor out = empty({R, H}, x, at::kBFloat16);
  launch("moe_gather_rows", 1, ptr(x), ptr(src), (void*)nullptr, ptr(out), R, H, (void*)nullptr);
  return out;
}
Tensor combine(const Tensor& y, const Tensor& pos, long T, long k) {
  const long H = y.size(-1);
  const Tensor out = empty({T, H}, y, at::kBFloat16);
  launch("moe_combine_rows", 1, ptr(y), ptr(pos), ptr(out), T, k, H);
  return out;
}
struct GatherRows : Function<GatherRows> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& src, const Tensor& inv_pos) {
    ctx->save_for_backward({inv_pos});
    ctx->saved_data["T"] = x.size(0);
    return gather(x, src);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    return guarded([&]() -> variable_list {
      const Tensor pos = ctx->get_saved_variables()[0];
      const long T = ctx->saved_data["T"].toInt();
      return {combine(grads[0].contiguous(), pos, T, T ? pos.numel() / T : 0), Tensor(), Tensor()};
    });
  }
};
struct CombineRows : Function<CombineRows> {
  static Tensor forward(AutogradContext* ctx, const Tensor& y, const Tensor& pos, const Tensor& src_token) {
    check_dims(pos, 2, "positions must be [T, k]");
    ctx->save_for_backward({src_token});
    return combine(y, pos.contiguous(), pos.size(0), pos.size(1));
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    return guarded([&]() -> variable_list {
      return {gather(grads[0].contiguous(), ctx->get_saved_variables()[0]), Tensor(), Tensor()};
    });
  }
};

// y[rows of e] = x[rows of e] @ w[e]^T over the layout's row blocks
struct GroupedLinear : Function<GroupedLinear> {
  static void run(int mode, const Tensor& a, const Tensor& b, const Tensor& out, long rows, long N, long K, long E, const Tensor& mblock,
                  const Tensor& row_start, const Tensor& padded, bool accumulate) {
    launch("grouped_gemm", 1, mode, ptr(a), ptr(b), ptr(out), rows, N, K, E, ptr(mblock), ptr(row_start), ptr(padded), accumulate,
           (void*)status_word(a));
  }
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, const Tensor& mblock, const Tensor& row_start,
                        const Tensor& padded) {
    check_dims(w, 3, "weights must be [E, N, K]");
    const long E = w.size(0), N = w.size(1), K = w.size(2);
    const Tensor out = empty({x.size(0), N}, x, at::kBFloat16);
    run(0, x, w, out, x.size(0), N, K, E, mblock, row_start, padded, false);
    ctx->save_for_backward({x, w, mblock, row_start, padded});
    keep(ctx, "w", w);
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    return guarded([&]() -> variable_list {
      const auto s = ctx->get_saved_variables();
      const Tensor &x = s[0], &w = s[1], dy = grads[0].contiguous();
      const long E = w.size(0), N = w.size(1), K = w.size(2), rows = x.size(0);
      variable_list out(5);
      if (ctx->needs_input_grad(0)) {
        out[0] = at::empty_like(x);
        run(1, dy, w, out[0], rows, K, N, E, s[2], s[3], s[4], false);
      }
      if (ctx->needs_input_grad(1)) {
        const Tensor weight = kept(ctx, "w");
        Tensor target = main_grad_of(weight);
        const bool own = !target.defined();
        if (own) target = empty({E, N, K}, x, at::kFloat);
        run(2, dy, x, target, rows, N, K, E, s[2], s[3], s[4], !own);
        if (own) {
          out[1] = target.to(w.scalar_type());
        } else {
          py::gil_scoped_acquire gil;
          py::object p = py::cast(weight), ready = py::getattr(p, "_grad_ready_cb", py::none());
          if (!ready.is_none()) ready(p);
        }
      }
      return out;
    });
  }
};

struct SwiGLU : Function<SwiGLU> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Opt& probs_, double clamp, int64_t kind) {
    const long I2 = x.size(-1), I = half_of(I2);
    const Tensor x2 = as_rows(x, I2);
    Tensor probs;
    if (probs_) probs = probs_->reshape({-1}).to(at::kFloat).contiguous();
    const Tensor out = empty({x2.size(0), I}, x, at::kBFloat16);
    launch("swiglu_fwd", 1, ptr(x2), ptr(probs), ptr(out), x2.size(0), I, (float)clamp, kind);
    ctx->save_for_backward({x2, probs});
    ctx->saved_data["clamp"] = clamp;
    ctx->saved_data["kind"] = kind;
    ctx->saved_data["shape"] = x.sizes().vec();
    if (probs_) {
      ctx->saved_data["pshape"] = probs_->sizes().vec();
      ctx->saved_data["ptype"] = (int64_t)probs_->scalar_type();
    }
    auto shape = x.sizes().vec();
    shape.back() = I;
    return as_shape(out, shape);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    return guarded([&]() -> variable_list {
      const auto s = ctx->get_saved_variables();
      const Tensor &x2 = s[0], &probs = s[1];
      const long T = x2.size(0), I = x2.size(1) / 2;
      const Tensor dy = as_rows(grads[0], I).contiguous(), din = at::empty_like(x2);
      Tensor dprobs;
      if (probs.defined()) dprobs = empty({T}, x2, at::kFloat);
      launch("swiglu_bwd", 1, ptr(dy), ptr(x2), ptr(probs), ptr(din), ptr(dprobs), T, I, (float)ctx->saved_data["clamp"].toDouble(),
             ctx->saved_data["kind"].toInt());
      if (dprobs.defined())
        dprobs = as_shape(dprobs, ctx->saved_data["pshape"].toIntVector()).to((at::ScalarType)ctx->saved_data["ptype"].toInt());
      return {as_shape(din, ctx->saved_data["shape"].toIntVector()), dprobs, Tensor(), Tensor()};
    });
  }
};

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  py::register_exception_translator([](std::exception_ptr p) {
    try {
      if (p) std::rethrow_exception(p);
    } catch (const LaunchError& e) {
      PyErr_SetString(lib_module->attr("NativeLibraryError").ptr(), e.what());
    }
  });
  m.def("init", [](const std::string& path, py::object lib, py::object gemm_mod, py::object autotune_mod) {
    library = dlopen(path.c_str(), RTLD_NOW | RTLD_GLOBAL);
    if (!library) throw std::runtime_error(dlerror());
    lib_module = new py::object(std::move(lib));
    gemm_module = new py::object(std::move(gemm_mod));
    gemm_dict = PyModule_GetDict(gemm_module->ptr());
    autotune_dict = PyModule_GetDict((new py::object(std::move(autotune_mod)))->ptr());
  });
  m.def("launches", [] { return launches.load(); });
  m.def("plain_gemms", [] { return plain_gemms(); });
  m.def("partial_rows", &partial_rows);
  m.def("rmsnorm", [](const Tensor& x, const Tensor& w, double eps, const Opt& residual) -> py::object {
    auto r = RMSNorm::apply(x, w, residual, eps);
    if (r.size() == 1) return py::cast(r[0]);
    return py::make_tuple(r[0], r[1]);
  });
  m.def("norm_linear", [](const Tensor& hidden, const Opt& residual, const Tensor& norm_w, const Tensor& weight, double eps) {
    auto r = NormLinear::apply(hidden, norm_w, weight, residual, eps);
    return py::make_tuple(r[0], r[1]);
  });
  m.def("linear", [](const Tensor& x, const Tensor& w) { return Linear::apply(x, w); });
  m.def("swiglu_linear", [](const Tensor& h1, const Tensor& w, double clamp, int64_t kind) { return SwiGLULinear::apply(h1, w, clamp, kind); });
  m.def("flash_attention", [](const Tensor& q, const Tensor& k, const Tensor& v, int64_t batch, bool causal, double scale, int64_t q_off,
                              int64_t window, const Opt& sinks, double softcap) {
    return FlashAttention::apply(q, k, v, sinks, batch, causal, scale, q_off, window, softcap);
  });
  m.def("rope_attention", [](const Tensor& qkv, const Opt& cos, const Opt& sin, const Opt& pos, int64_t batch, int64_t hq, int64_t hkv,
                             int64_t d, int64_t rot_dim, bool causal, double scale, int64_t window, const Opt& sinks, double softcap) {
    return RopeAttention::apply(qkv, sinks, cos, sin, pos, batch, hq, hkv, d, rot_dim, causal, scale, window,
                                softcap);
  });
  m.def("qk_norm", [](const Tensor& qkv, const Tensor& wq, const Tensor& wk, int64_t hq, int64_t hkv, int64_t d, double eps, const Opt& cos,
                      const Opt& sin, const Opt& pos, int64_t rot_dim) {
    return QKNorm::apply(qkv, wq, wk, cos, sin, pos, hq, hkv, d, eps, rot_dim);
  });
  m.def("embedding", [](const Tensor& tokens, const Tensor& w) { return Embedding::apply(tokens, w); });
  m.def("cross_entropy", [](const Tensor& logits, const Tensor& labels, const Opt& weights, bool unit) {
    return CrossEntropy::apply(logits, labels, weights, unit);
  });
  m.def("router", [](const Tensor& logits, const Opt& bias, int64_t topk, bool sigmoid, bool pre_softmax, int64_t groups, int64_t group_topk,
                     double scale, const std::optional<double>& aux_coeff) {
    auto r = Router::apply(logits, bias, topk, sigmoid, pre_softmax, groups, group_topk, scale, aux_coeff);
    return py::make_tuple(r[0], r[1], r[2], r[3], r.size() > 4 ? py::cast(r[4]) : py::none());
  });
  m.def("local_plan", [](const Tensor& probs, const Tensor& idx, const Tensor& counts, int64_t topk, int64_t rows_cap) {
    auto r = LocalPlan::apply(probs, idx, counts, topk, rows_cap);
    return py::make_tuple(r[0], r[1], r[2], r[3], r[4], r[5], r[6]);
  });
  m.def("gather_rows", [](const Tensor& x, const Tensor& src, const Tensor& inv_pos) { return GatherRows::apply(x, src, inv_pos); });
  m.def("combine_rows", [](const Tensor& y, const Tensor& pos, const Tensor& src_token) { return CombineRows::apply(y, pos, src_token); });
  m.def("grouped_linear", [](const Tensor& x, const Tensor& w, const Tensor& mblock, const Tensor& row_start, const Tensor& padded) {
    return GroupedLinear::apply(x, w, mblock, row_start, padded);
  });
  m.def("swiglu", [](const Tensor& x, const Opt& probs, double clamp, int64_t kind) { return SwiGLU::apply(x, probs, clamp, kind); });
}
