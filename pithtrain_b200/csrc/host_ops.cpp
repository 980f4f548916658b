// Operators of the training step whose host side is C++: allocation, checks, kernel launches and the autograd nodes of RMSNorm,
// linear layers, QK-norm with RoPE, attention, the router and the expert block.
//
// These run once or more per layer and micro-batch. From Python an operator spent 5 to 8 us in its launches and 15 to 30 us around
// them (argument checks, views, autograd.Function, ctypes): without gradients an RMSNorm took 19 us and takes 7, a linear layer 24
// and 8. Two micro-batches of 512 tokens through four narrow layers (forward and backward, some 400 launches) 13.7 -> 7.2 ms, the
// 64-token forward of two Qwen3 layers 2.87 -> 1.45 ms, of which the device works 1.17.
//
// The kernels stay in libpithb200.so; their entry points are looked up by name (bind) in the library that Python has loaded. What
// a user can replace or observe is asked from Python when it is needed: the gradient buffer of a parameter (main_grad, else .grad)
// and the deferral of weight gradients. The nodes keep tensors (through SavedVariable: version checks and saved-tensor hooks as
// for any operator), never raw pointers, and no state outlives a call. A parameter that a node adds gradients to is kept beside its
// saved value: under hooks, the memory trace's or a checkpoint's, unpacking hands out another tensor, without main_grad and .grad.
#include <c10/cuda/CUDAStream.h>
#include <dlfcn.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/extension.h>

#include <atomic>

namespace {

namespace py = pybind11;
using at::Tensor;
using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;
using OptTensor = std::optional<Tensor>;

// ------------------------------------------------------------------------------------------------
// kernel entry points
// ------------------------------------------------------------------------------------------------
using P = const void*;
using I = int;
using L = long long;
using F = float;
#define PITH_ENTRY_POINTS(X)                                                                                             \
  X(pt_rmsnorm_fwd, P, P, P, P, P, P, I, I, F, I, P)                                                                     \
  X(pt_rmsnorm_bwd_grid, I)                                                                                              \
  X(pt_rmsnorm_bwd, P, P, P, P, P, P, P, I, I, I, P)                                                                     \
  X(pt_colsum_accumulate, P, I, I, I, P, I, P)                                                                           \
  X(pt_colsum_accumulate_pair, P, I, I, I, P, P, I, P)                                                                   \
  X(pt_gemm2cta_nt, P, P, P, I, I, I, L, L, L, P)                                                                        \
  X(pt_dense_nn, P, P, P, I, I, I, L, L, L, P)                                                                           \
  X(pt_dense_tn, P, P, P, I, I, I, I, I, L, L, L, P)                                                                     \
  X(pt_gemm_bf16, P, P, P, I, I, I, I, I, I, L, L, L, L, L, L, L, L, P, I, I, L, I, I, I, I, I, I, P, I, L, P)           \
  X(pt_qk_norm_rope_fwd, P, P, P, P, P, P, P, P, P, P, I, I, I, I, I, L, F, I, P)                                        \
  X(pt_qk_norm_rope_bwd_grid, I, I, I, I)                                                                                \
  X(pt_qk_norm_rope_bwd, P, P, P, P, P, P, P, P, P, P, P, P, P, I, I, I, I, I, L, L, I, P)                               \
  X(pt_attn_fwd, P, P, P, P, P, P, P, I, I, I, I, I, I, I, L, L, L, L, F, I, I, P)                                       \
  X(pt_attn_bwd, P, P, P, P, P, P, P, P, P, P, P, P, P, P, P, I, I, I, I, I, I, L, L, L, L, L, F, I, I, P)               \
  X(pt_attn_bwd_split_reach, P, P, P, P, P, P, P, P, P, P, P, P, P, I, I, I, I, I, I, I, L, L, L, L, L, F, I, I, I, P)   \
  X(pt_router_topk_fwd, P, I, P, P, P, I, I, I, I, I, F, P)                                                              \
  X(pt_router_given_fwd, P, I, P, P, P, I, I, I, I, F, P)                                                                \
  X(pt_router_topk_bwd, P, P, P, P, P, P, I, I, I, I, I, I, F, P)                                                        \
  X(pt_route_sort, P, P, I, I, I, P, L, P, P, P, I, P)                                                                   \
  X(pt_gather_rows, P, P, I, P, P, I, I, L, P)                                                                           \
  X(pt_combine, P, P, P, P, P, P, I, I, I, P)                                                                            \
  X(pt_swiglu_fwd, P, P, P, I, I, I, F, F, P)                                                                            \
  X(pt_swiglu_bwd, P, P, P, P, P, P, P, I, I, I, F, F, P, P)
struct Api {
#define PITH_DECLARE(name, ...) int (*name)(__VA_ARGS__) = nullptr;
  PITH_ENTRY_POINTS(PITH_DECLARE)
#undef PITH_DECLARE
} api;

void bind(const std::string& path) {
  void* lib = dlopen(path.c_str(), RTLD_NOW | RTLD_LOCAL);
  TORCH_CHECK(lib != nullptr, "dlopen: ", dlerror());
#define PITH_LOOKUP(name, ...)                                       \
  api.name = reinterpret_cast<decltype(api.name)>(dlsym(lib, #name)); \
  TORCH_CHECK(api.name != nullptr, #name " is missing in ", path);
  PITH_ENTRY_POINTS(PITH_LOOKUP)
#undef PITH_LOOKUP
}

std::atomic<long long> launches{0};

void check(int rc, const char* what, int kernels = 1) {
  TORCH_CHECK(rc == 0, what, " failed with code ", rc);
  launches.fetch_add(kernels, std::memory_order_relaxed);
}
P current_stream() { return c10::cuda::getCurrentCUDAStream().stream(); }
P ptr(const Tensor& t) { return t.defined() ? t.const_data_ptr() : nullptr; }

// ------------------------------------------------------------------------------------------------
// helpers
// ------------------------------------------------------------------------------------------------
// A custom operator without a vmap or jvp rule refuses transformed and dual inputs, as autograd.Function does.
void refuse_transforms(std::initializer_list<const Tensor*> inputs) {
  TORCH_CHECK(!c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode),
              "this operator does not support functorch transforms (vmap, grad, jvp, jacrev, ...)");
  for (const Tensor* t : inputs)
    TORCH_CHECK_NOT_IMPLEMENTED(!t->defined() || !t->_fw_grad(0).defined(), "forward-mode differentiation is not implemented for this operator");
}
// The kernels take raw pointers. Operands on the host or on different devices are refused, and those without memory of their own
// (fake tensors, subclasses that wrap others).
void check_operands(const Tensor& x, std::initializer_list<const Tensor*> others) {
  TORCH_CHECK(x.is_cuda(), "the first operand must be on a CUDA device, is on ", x.device());
  const auto has_memory = [](const Tensor& t) { return t.const_data_ptr() != nullptr || t.numel() == 0; };
  bool memory = has_memory(x);
  for (const Tensor* t : others) {
    if (!t->defined()) continue;
    TORCH_CHECK(t->device() == x.device(), "operands on ", x.device(), " and ", t->device());
    memory = memory && has_memory(*t);
  }
  TORCH_CHECK(memory, "an operand has no memory");
}
Tensor opt(const OptTensor& t) { return t.has_value() ? *t : Tensor(); }
Tensor empty(at::IntArrayRef sizes, const Tensor& like, at::ScalarType type) { return at::empty(sizes, like.options().dtype(type)); }
void check_rows(const Tensor& t, const char* name) {
  TORCH_CHECK(t.dim() == 2 && t.stride(1) == 1 && t.scalar_type() == at::kBFloat16, name, " must be a row-major bf16 matrix");
  TORCH_CHECK(t.stride(0) % 8 == 0 && reinterpret_cast<uintptr_t>(t.const_data_ptr()) % 16 == 0, name, " must be 16-byte aligned");
}
void check_aligned(const Tensor& t, const char* name) {
  TORCH_CHECK(reinterpret_cast<uintptr_t>(t.const_data_ptr()) % 16 == 0, name, " must be 16-byte aligned");
}

// Contiguous and 16-byte aligned, as the vector loads of the elementwise kernels want it.
Tensor dense(const Tensor& t) {
  Tensor c = t.contiguous();
  return reinterpret_cast<uintptr_t>(c.const_data_ptr()) % 16 == 0 ? c : c.clone(at::MemoryFormat::Contiguous);
}

// A Python object that a node keeps: dropped under the interpreter lock, which the autograd engine does not hold.
class PyRef {
 public:
  PyRef() = default;
  explicit PyRef(const py::object& o) : obj_(o.ptr()) { Py_XINCREF(obj_); }
  PyRef(const PyRef&) = delete;
  PyRef& operator=(PyRef&& o) noexcept {
    std::swap(obj_, o.obj_);
    return *this;
  }
  ~PyRef() {
    if (obj_ && Py_IsInitialized()) {
      py::gil_scoped_acquire gil;
      Py_DECREF(obj_);
    }
  }
  py::object get() const { return py::reinterpret_borrow<py::object>(obj_); }  // under the lock

 private:
  PyObject* obj_ = nullptr;
};

py::object python(const char* module, const char* name) { return py::module_::import(module).attr(name); }
py::object wrap(const Tensor& t) { return py::reinterpret_steal<py::object>(THPVariable_Wrap(t)); }

// The flat gradient buffer of a parameter, if it has one that the column-sum kernels can add to.
Tensor colsum_target(const Tensor& param, int64_t n) {
  py::object o = wrap(param);
  if (!py::hasattr(o, "main_grad")) return {};
  py::object g = o.attr("main_grad");
  if (!THPVariable_Check(g.ptr())) return {};
  const Tensor& t = THPVariable_Unpack(g.ptr());
  const bool ok = t.is_cuda() && t.is_contiguous() && (t.scalar_type() == at::kFloat || t.scalar_type() == at::kBFloat16) && t.numel() == n;
  return ok ? t : Tensor();
}
// grad(param) += part.sum(0), part [G, n] fp32
void accumulate_colsum(const Tensor& param, const Tensor& part) {
  py::gil_scoped_acquire gil;
  const Tensor g = colsum_target(param, part.size(1));
  if (!g.defined()) {
    python("pithtrain_b200.ops.common", "accumulate_colsum")(wrap(param), part);
    return;
  }
  check(api.pt_colsum_accumulate(ptr(part), part.size(0), part.stride(0), part.size(1), g.data_ptr(), g.scalar_type() == at::kFloat, current_stream()),
        "pt_colsum_accumulate");
}
// the same of part[:, :d] into p0 and part[:, d:] into p1
void accumulate_colsum_pair(const Tensor& p0, const Tensor& p1, const Tensor& part, int64_t d) {
  py::gil_scoped_acquire gil;
  const Tensor g0 = colsum_target(p0, d), g1 = colsum_target(p1, d);
  if (!g0.defined() || !g1.defined() || g0.scalar_type() != g1.scalar_type() || p0.is_same(p1)) {
    python("pithtrain_b200.ops.common", "accumulate_colsum_pair")(wrap(p0), wrap(p1), part, d);
    return;
  }
  check(api.pt_colsum_accumulate_pair(ptr(part), part.size(0), part.stride(0), d, g0.data_ptr(), g1.data_ptr(),
                                      g0.scalar_type() == at::kFloat, current_stream()),
        "pt_colsum_accumulate_pair");
}

// While a torch.jit.trace is recorded, an operator hands itself to Python, which makes one step of the trace of it.
thread_local bool in_traced_step = false;
template <class R, class... A>
R traced(const char* name, const A&... args) {
  struct Step {
    Step() { in_traced_step = true; }
    ~Step() { in_traced_step = false; }
  } step;
  return python("pithtrain_b200._native", "_traced")(name, args...).template cast<R>();
}
bool tracing() { return torch::jit::tracer::isTracing() && !in_traced_step; }

template <class N, class... T>
std::shared_ptr<N> make_node(const T&... inputs) {
  if (!torch::autograd::compute_requires_grad(inputs...)) return nullptr;
  std::shared_ptr<N> node(new N(), torch::autograd::deleteNode);
  node->set_next_edges(torch::autograd::collect_next_edges(inputs...));
  return node;
}
using Below = at::AutoDispatchBelowADInplaceOrView;

// ------------------------------------------------------------------------------------------------
// RMSNorm, optionally of x + residual
// ------------------------------------------------------------------------------------------------
struct RmsNormBackward : Node {
  SavedVariable h, w, rstd;
  Tensor weight;  // the parameter
  bool residual = false, h_is_output = false, zero_centered = false;

  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    const Tensor hv = h_is_output ? h.unpack(shared_from_this()) : h.unpack(), wv = w.unpack(), r = rstd.unpack();
    Tensor dx, part;
    {
      Below guard;
      const Tensor wd = dense(wv);
      const int64_t H = hv.size(-1), n = H ? hv.numel() / H : 0;
      const Tensor dy = grads[0].defined() ? dense(grads[0]) : at::zeros_like(hv);
      const Tensor dh = residual && grads[1].defined() ? dense(grads[1]) : Tensor();
      dx = at::empty_like(hv);
      part = empty({api.pt_rmsnorm_bwd_grid(n), H}, hv, at::kFloat);
      check(api.pt_rmsnorm_bwd(ptr(dy), ptr(dh), ptr(hv), ptr(wd), ptr(r), ptr(dx), ptr(part), n, H, zero_centered, current_stream()), "pt_rmsnorm_bwd");
    }
    if (task_should_compute_output(1)) accumulate_colsum(weight, part);
    return {dx, Tensor(), residual ? dx : Tensor()};
  }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    h.reset_data();
    w.reset_data();
    rstd.reset_data();
    weight.reset();
  }
};

py::object rmsnorm(const Tensor& x, const Tensor& w, double eps, const OptTensor& residual_, bool zero_centered) {
  if (tracing()) return traced<py::object>("rmsnorm", x, w, eps, residual_, zero_centered);
  const Tensor residual = opt(residual_);
  refuse_transforms({&x, &w, &residual});
  check_operands(x, {&w, &residual});
  TORCH_CHECK(x.size(-1) > 0, "rmsnorm: rows of no elements");
  auto node = make_node<RmsNormBackward>(x, w, residual);
  Tensor xc, h, y, rstd;
  {
    Below guard;
    const int64_t H = x.size(-1), n = H ? x.numel() / H : 0;
    xc = dense(x);
    const Tensor rc = residual.defined() ? dense(residual) : Tensor();
    TORCH_CHECK(!rc.defined() || (rc.numel() == xc.numel() && rc.scalar_type() == at::kBFloat16), "rmsnorm: residual ", rc.sizes());
    TORCH_CHECK(w.numel() == H && w.is_contiguous(), "rmsnorm: weight ", w.sizes(), " for rows of ", H);
    const Tensor wd = dense(w);
    y = at::empty_like(xc);
    if (rc.defined()) h = at::empty_like(xc);
    rstd = empty({n}, xc, at::kFloat);
    check(api.pt_rmsnorm_fwd(ptr(xc), ptr(rc), ptr(wd), ptr(y), ptr(h), ptr(rstd), n, H, static_cast<float>(eps), zero_centered, current_stream()),
          "pt_rmsnorm_fwd");
  }
  if (node) {
    torch::autograd::set_history(y, node);
    if (h.defined()) torch::autograd::set_history(h, node);
    node->residual = node->h_is_output = h.defined();
    node->h = h.defined() ? SavedVariable(h, true) : SavedVariable(xc, false);
    node->w = SavedVariable(w, false);
    node->weight = w;
    node->rstd = SavedVariable(rstd, false);
    node->zero_centered = zero_centered;
  }
  if (h.defined()) return py::make_tuple(y, h);
  return py::cast(y);
}

// ------------------------------------------------------------------------------------------------
// linear layers
// ------------------------------------------------------------------------------------------------
struct LinearBackward : Node {
  SavedVariable x, w;
  PyRef grad_getter, bias_param;
  bool has_bias = false;

  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    if (!grads[0].defined()) return {Tensor(), Tensor(), Tensor()};
    const Tensor xv = x.unpack(), wv = w.unpack();
    Tensor dx, dy, x2;
    {
      Below guard;
      const int64_t K = wv.size(1), N = wv.size(0);
      dy = grads[0].contiguous().view({-1, N});
      x2 = xv.view({-1, K});
      if (task_should_compute_output(0)) {
        check_aligned(dy, "dy");
        dx = at::empty_like(xv);
        check(api.pt_dense_nn(ptr(dy), ptr(wv), ptr(dx), dy.size(0), K, N, N, wv.stride(0), K, current_stream()), "pt_dense_nn");
      }
    }
    py::gil_scoped_acquire gil;
    if (has_bias && !bias_param.get().is_none())
      python("pithtrain_b200.ops.common", "accumulate_grad")(bias_param.get(), dy.to(at::kFloat).sum(0));
    python("pithtrain_b200.ops.linear", "_queue_wgrad")(dy, x2, grad_getter.get());
    return {dx, Tensor(), Tensor()};
  }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    x.reset_data();
    w.reset_data();
  }
};

// x [..., K], w [N, K]; the weight gradient goes where grad_getter() says, the bias gradient to bias_param.
Tensor linear(const Tensor& x, const Tensor& w, const OptTensor& bias_, const py::object& grad_getter, const py::object& bias_param) {
  if (tracing()) return traced<Tensor>("linear", x, w, bias_, grad_getter, bias_param);
  const Tensor bias = opt(bias_);
  refuse_transforms({&x, &w, &bias});
  check_operands(x, {&w, &bias});
  auto node = make_node<LinearBackward>(x, w, bias);
  Tensor xc, y;
  {
    Below guard;
    const int64_t K = w.size(1), N = w.size(0);
    TORCH_CHECK(x.size(-1) == K && K > 0, "linear: ", x.sizes(), " x ", w.sizes());
    xc = x.contiguous();
    check_aligned(xc, "x");
    check_rows(w, "w");
    auto sizes = x.sizes().vec();
    sizes.back() = N;
    y = empty(sizes, xc, at::kBFloat16);
    check(api.pt_gemm2cta_nt(ptr(xc), ptr(w), ptr(y), xc.numel() / K, N, K, K, w.stride(0), N, current_stream()), "pt_gemm2cta_nt");
    if (bias.defined()) y.add_(bias);
  }
  if (node) {
    torch::autograd::set_history(y, node);
    node->x = SavedVariable(xc, false);
    node->w = SavedVariable(w, false);
    node->grad_getter = PyRef(grad_getter);
    node->bias_param = PyRef(bias_param);
    node->has_bias = bias.defined();
  }
  return y;
}

// target [N, K] += dy^T x, both contiguous with 16-byte aligned rows.
void wgrad_into(const Tensor& dy, const Tensor& x, const Tensor& target, bool fp32_sums) {
  check_rows(dy, "dy");
  check_rows(x, "x");
  check_operands(dy, {&x, &target});
  check(api.pt_dense_tn(ptr(dy), ptr(x), target.data_ptr(), target.scalar_type() == at::kFloat, fp32_sums, dy.size(1), x.size(1), dy.size(0),
                        dy.stride(0), x.stride(0), target.stride(0), current_stream()),
        "pt_dense_tn");
}

// ------------------------------------------------------------------------------------------------
// per-head RMSNorm of q and k with RoPE, on the packed projection
// ------------------------------------------------------------------------------------------------
struct QkNormRopeBackward : Node {
  SavedVariable qkv, q_w, k_w, cos, sin, pos, rq, rk;
  Tensor q_weight, k_weight;  // the parameters
  int64_t Hq = 0, Hkv = 0, D = 0, S = 0;
  bool norm = false, zero_centered = false;

  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    const Tensor x = qkv.unpack(), qw = q_w.unpack(), kw = k_w.unpack(), c = cos.unpack(), s = sin.unpack(), p = pos.unpack();
    const Tensor rqv = rq.unpack(), rkv = rk.unpack();
    Tensor dx, part;
    {
      Below guard;
      const int64_t n = x.size(0);
      const Tensor dq = grads[0].defined() ? dense(grads[0]) : at::zeros({n, Hq, D}, x.options());
      const Tensor dk = grads[1].defined() ? dense(grads[1]) : at::zeros({n, Hkv, D}, x.options());
      const Tensor dv = grads[2].defined() ? dense(grads[2]) : Tensor();
      const Tensor qd = norm ? dense(qw) : qw, kd = norm ? dense(kw) : kw;
      dx = at::empty_like(x);
      if (norm) part = empty({api.pt_qk_norm_rope_bwd_grid(n, Hq, Hkv, D), 2 * D}, x, at::kFloat);
      check(api.pt_qk_norm_rope_bwd(ptr(dq), ptr(dk), ptr(dv), ptr(x), ptr(dx), ptr(qd), ptr(kd), ptr(c), ptr(s), ptr(p), ptr(rqv), ptr(rkv),
                                    ptr(part), n, S, Hq, Hkv, D, x.stride(0), dx.stride(0), zero_centered, current_stream()),
            "pt_qk_norm_rope_bwd");
    }
    if (norm) accumulate_colsum_pair(q_weight, k_weight, part, D);
    return {dx, Tensor(), Tensor()};
  }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    for (SavedVariable* v : {&qkv, &q_w, &k_w, &cos, &sin, &pos, &rq, &rk}) v->reset_data();
    q_weight.reset();
    k_weight.reset();
  }
};

py::tuple qk_norm_rope(const Tensor& qkv_, const OptTensor& q_w_, const OptTensor& k_w_, const Tensor& cos_, const Tensor& sin_,
                       const OptTensor& positions, int64_t Hq, int64_t Hkv, int64_t D, double eps, int64_t S, bool zero_centered) {
  if (tracing()) return traced<py::tuple>("qk_norm_rope", qkv_, q_w_, k_w_, cos_, sin_, positions, Hq, Hkv, D, eps, S, zero_centered);
  const Tensor q_w = opt(q_w_), k_w = opt(k_w_);
  refuse_transforms({&qkv_, &q_w, &k_w});
  const Tensor positions_ = opt(positions);
  check_operands(qkv_, {&q_w, &k_w, &cos_, &sin_, &positions_});
  auto node = make_node<QkNormRopeBackward>(qkv_, q_w, k_w);
  Tensor qkv = qkv_, cos, sin, q, k, v, rq, rk, pos;
  {
    Below guard;
    // rows of any 16-byte pitch, as a projection's slice has them
    if (qkv.stride(0) % 8 != 0 || reinterpret_cast<uintptr_t>(qkv.const_data_ptr()) % 16 != 0) qkv = qkv.clone(at::MemoryFormat::Contiguous);
    cos = dense(cos_);
    sin = dense(sin_);
    const Tensor qd = q_w.defined() ? dense(q_w) : q_w, kd = k_w.defined() ? dense(k_w) : k_w;
    const int64_t n = qkv.size(0);
    q = empty({n, Hq, D}, qkv, at::kBFloat16);
    k = empty({n, Hkv, D}, qkv, at::kBFloat16);
    if (q_w.defined()) {
      rq = empty({n, Hq}, qkv, at::kFloat);
      rk = empty({n, Hkv}, qkv, at::kFloat);
    }
    if (positions.has_value()) pos = positions->to(at::kInt).contiguous();
    check(api.pt_qk_norm_rope_fwd(ptr(qkv), ptr(q), ptr(k), ptr(qd), ptr(kd), ptr(cos), ptr(sin), ptr(pos), ptr(rq), ptr(rk), n, S, Hq, Hkv, D,
                                  qkv.stride(0), static_cast<float>(eps), zero_centered, current_stream()),
          "pt_qk_norm_rope_fwd");
    // v is not rotated: the rows of the projection themselves, whose changes it has to show (version counter)
    v = qkv.as_strided({n, Hkv, D}, {qkv.stride(0), D, 1}, qkv.storage_offset() + (Hq + Hkv) * D);
    v.unsafeGetTensorImpl()->set_version_counter(qkv.unsafeGetTensorImpl()->version_counter());
  }
  if (node) {
    for (Tensor* t : {&q, &k, &v}) torch::autograd::set_history(*t, node);
    node->qkv = SavedVariable(qkv, false);
    node->q_w = SavedVariable(q_w, false);
    node->k_w = SavedVariable(k_w, false);
    node->q_weight = q_w;
    node->k_weight = k_w;
    node->cos = SavedVariable(cos, false);
    node->sin = SavedVariable(sin, false);
    node->pos = SavedVariable(pos, false);
    node->rq = SavedVariable(rq, false);
    node->rk = SavedVariable(rk, false);
    node->Hq = Hq; node->Hkv = Hkv; node->D = D; node->S = S;
    node->norm = q_w.defined();
    node->zero_centered = zero_centered;
  }
  return py::make_tuple(q, k, v);
}

// ------------------------------------------------------------------------------------------------
// attention
// ------------------------------------------------------------------------------------------------
// [B, S, H, D] whose (H, D) block is contiguous and whose tokens are equally spaced (a slice of a fused projection qualifies)
bool token_major(const Tensor& t) {
  const int64_t B = t.size(0), S = t.size(1), H = t.size(2), D = t.size(3);
  return t.stride(3) == 1 && (H == 1 || t.stride(2) == D) && (B == 1 || t.stride(0) == S * t.stride(1)) && t.stride(1) % 8 == 0 &&
         reinterpret_cast<uintptr_t>(t.const_data_ptr()) % 16 == 0;
}
Tensor as_token_major(const Tensor& t) { return token_major(t) ? t : t.contiguous(); }

struct Grads {
  Tensor dq, dk, dv, delta;
};

Grads attention_backward(const Tensor& grad, const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& out_, const Tensor& lse_, double scale,
                         bool causal, int64_t q_off, const Tensor& row_lo, int64_t reach) {
  const Tensor q = as_token_major(q_), k = as_token_major(k_), v = as_token_major(v_), out = as_token_major(out_), lse = lse_.contiguous();
  // Unlike q, k and v the gradient comes to no tensor map that refuses a misaligned base or pitch
  Tensor d = as_token_major(grad);
  if (!token_major(d)) d = d.clone(at::MemoryFormat::Contiguous);
  const int64_t B = q.size(0), Sq = q.size(1), Hq = q.size(2), D = q.size(3), Sk = k.size(1), Hkv = k.size(2), Dv = v.size(3);
  Tensor dq = empty(q.sizes(), q, at::kBFloat16), dk = empty(k.sizes(), q, at::kBFloat16), dv = empty(v.sizes(), q, at::kBFloat16);
  const float sc = static_cast<float>(scale);
  // csrc/attention_bwd.cu has head dims 64 and 128 and lengths that are a multiple of 4 (its row statistics move in 16-byte pieces
  // without a padded pitch): five tile products, P and dS rounded to bf16, gradients 2.3e-3 to 2.9e-3 off the 64-bit ones. All other
  // gradients came from fp32 products before they had kernels (1.7e-3, the rounding of the result) and keep that in
  // csrc/attention_bwd_split.cu with 14 tile products. 32/4 heads x 128 at 4096 / 4093 tokens, backward: 439 / 1177 us.
  if (D == Dv && (D == 64 || D == 128) && Sq % 4 == 0) {
    // one zeroed buffer: the fp32 accumulators (dq over key tiles; dk and dv over the heads of a group), then the row statistics,
    // padded by one tile because the kernel reads them in whole 128-row tiles
    const int64_t nq = B * Sq * Hq * D, nk = B * Sk * Hkv * D, ns = B * Hq * Sq;
    Tensor buf = at::zeros({nq + 2 * nk + 2 * (ns + 128)}, q.options().dtype(at::kFloat));
    float* b = buf.data_ptr<float>();
    float *delta = b + nq + 2 * nk, *lse2 = delta + ns + 128;
    check(api.pt_attn_bwd(ptr(q), ptr(k), ptr(v), ptr(out), ptr(d), ptr(lse), ptr(row_lo), b, b + nq, b + nq + nk, ptr(dq), ptr(dk), ptr(dv), delta,
                          lse2, B, Sq, Sk, Hq, Hkv, D, q.stride(1), k.stride(1), v.stride(1), out.stride(1), d.stride(1), sc, causal, q_off, current_stream()),
          "pt_attn_bwd", 3);
    return {dq, dk, dv, buf.narrow(0, nq + 2 * nk, ns).view({B, Hq, Sq})};
  }
  const int64_t Sp = (Sq + 3) / 4 * 4, ns = B * Hq * Sp;
  Tensor stats = empty({2 * (ns + 128)}, q, at::kFloat);  // read in whole 64-row tiles: padded
  float* delta = stats.data_ptr<float>();
  Tensor part;
  if (Hq != Hkv) part = empty({B * Sk * Hq * (D > Dv ? D : Dv)}, q, at::kFloat);
  check(api.pt_attn_bwd_split_reach(ptr(q), ptr(k), ptr(v), ptr(out), ptr(d), ptr(lse), ptr(row_lo), ptr(dq), ptr(dk), ptr(dv), delta,
                                    delta + ns + 128, ptr(part), B, Sq, Sk, Hq, Hkv, D, Dv, q.stride(1), k.stride(1), v.stride(1), out.stride(1),
                                    d.stride(1), sc, causal, q_off, reach, current_stream()),
        "pt_attn_bwd_split", part.defined() ? 6 : 4);
  return {dq, dk, dv, stats.narrow(0, 0, ns).view({B, Hq, Sp}).narrow(2, 0, Sq)};
}

struct AttentionBackward : Node {
  SavedVariable q, k, v, sinks, row_lo, out, lse;
  double scale = 0;
  bool causal = false;
  int64_t q_off = 0, reach = 0;

  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    if (!grads[0].defined()) return {Tensor(), Tensor(), Tensor(), Tensor()};
    const Tensor qv = q.unpack(), kv = k.unpack(), vv = v.unpack(), sv = sinks.unpack(), rv = row_lo.unpack();
    const Tensor ov = out.unpack(shared_from_this()), lv = lse.unpack();
    Below guard;
    Grads g = attention_backward(grads[0], qv, kv, vv, ov, lv, scale, causal, q_off, rv, reach);
    Tensor ds;
    if (sv.defined())  // of the lse-normalised weight of the sink column, -exp(sink - lse) * delta, over batch and rows
      ds = ((sv.to(at::kFloat).view({1, -1, 1}) - lv).exp() * g.delta).sum(at::IntArrayRef{0, 2}).neg().to(sv.scalar_type());
    return {g.dq, g.dk, g.dv, ds};
  }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    for (SavedVariable* s : {&q, &k, &v, &sinks, &row_lo, &out, &lse}) s->reset_data();
  }
};

// out [B, Sq, Hq, Dv] bf16, lse [B, Hq, Sq] fp32 (not differentiable); reach: about how many keys a query sees
py::tuple attention(const Tensor& q, const Tensor& k, const Tensor& v, const OptTensor& sinks_, const OptTensor& row_lo_, double scale, bool causal,
                    int64_t q_off, int64_t reach) {
  if (tracing()) return traced<py::tuple>("attention", q, k, v, sinks_, row_lo_, scale, causal, q_off, reach);
  const Tensor sinks = opt(sinks_), row_lo = opt(row_lo_);
  refuse_transforms({&q, &k, &v, &sinks});
  check_operands(q, {&k, &v, &sinks, &row_lo});
  auto node = make_node<AttentionBackward>(q, k, v, sinks);
  Tensor out, lse;
  {
    Below guard;
    const Tensor qc = as_token_major(q), kc = as_token_major(k), vc = as_token_major(v);
    const int64_t B = q.size(0), Sq = q.size(1), Hq = q.size(2), D = q.size(3), Sk = k.size(1), Hkv = k.size(2), Dv = v.size(3);
    out = empty({B, Sq, Hq, Dv}, q, at::kBFloat16);
    lse = empty({B, Hq, Sq}, q, at::kFloat);
    const Tensor sk = sinks.defined() ? sinks.to(at::kFloat).contiguous() : Tensor();
    check(api.pt_attn_fwd(ptr(qc), ptr(kc), ptr(vc), ptr(out), ptr(lse), ptr(row_lo), ptr(sk), B, Sq, Sk, Hq, Hkv, D, Dv, qc.stride(1), kc.stride(1),
                          vc.stride(1), out.stride(1), static_cast<float>(scale), causal, q_off, current_stream()),
          "pt_attn_fwd");
  }
  if (node) {
    torch::autograd::set_history(out, node);
    node->q = SavedVariable(q, false);
    node->k = SavedVariable(k, false);
    node->v = SavedVariable(v, false);
    node->sinks = SavedVariable(sinks, false);
    node->row_lo = SavedVariable(row_lo, false);
    node->out = SavedVariable(out, true);
    node->lse = SavedVariable(lse, false);
    node->scale = scale; node->causal = causal; node->q_off = q_off; node->reach = reach;
  }
  return py::make_tuple(out, lse);
}

// ------------------------------------------------------------------------------------------------
// router
// ------------------------------------------------------------------------------------------------
enum RouterMode : int { SOFTMAX_TOPK = 0, TOPK_SOFTMAX = 1 };

struct RouterBackward : Node {
  SavedVariable probs, idx, w;
  int mode = SOFTMAX_TOPK;
  bool renorm = false;
  double scale = 1;
  int64_t experts = 0;
  at::ScalarType type = at::kFloat;

  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    const Tensor pv = probs.unpack(shared_from_this()), iv = idx.unpack(), wv = w.unpack(shared_from_this());
    Below guard;
    const int64_t n = wv.size(0), k = wv.size(1);
    const Tensor dw = grads[0].defined() ? grads[0].contiguous().to(at::kFloat) : at::zeros_like(wv);
    const Tensor dp = mode == SOFTMAX_TOPK && grads[1].defined() ? grads[1].contiguous() : Tensor();
    Tensor dl = empty({n, experts}, wv, type);
    check(api.pt_router_topk_bwd(ptr(pv), ptr(iv), ptr(wv), ptr(dw), ptr(dp), ptr(dl), type == at::kFloat, n, experts, k, mode, renorm,
                                 static_cast<float>(scale), current_stream()),
          "pt_router_topk_bwd");
    return {dl};
  }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    probs.reset_data();
    idx.reset_data();
    w.reset_data();
  }
};

// (weights [n, k] fp32, picks [n, k] int32, probabilities [n, E] fp32 or None); given: the picks, else they are the top k
py::tuple router(const Tensor& logits, const OptTensor& given, int64_t k, int64_t mode, bool renorm, double scale) {
  if (tracing()) return traced<py::tuple>("router", logits, given, k, mode, renorm, scale);
  refuse_transforms({&logits});
  const Tensor picks = opt(given);
  check_operands(logits, {&picks});
  auto node = make_node<RouterBackward>(logits);
  Tensor probs, idx, w;
  const int64_t n = logits.size(0), E = logits.size(1);
  const bool fp32 = logits.scalar_type() == at::kFloat;
  {
    Below guard;
    const Tensor lg = logits.contiguous();
    if (mode == SOFTMAX_TOPK) probs = empty({n, E}, lg, at::kFloat);
    if (given.has_value()) {
      idx = *given;
      w = empty({n, idx.size(1)}, lg, at::kFloat);
      check(api.pt_router_given_fwd(ptr(lg), fp32, ptr(probs), ptr(idx), ptr(w), n, E, idx.size(1), renorm, static_cast<float>(scale), current_stream()),
            "pt_router_given_fwd");
    } else {
      idx = empty({n, k}, lg, at::kInt);
      w = empty({n, k}, lg, at::kFloat);
      check(api.pt_router_topk_fwd(ptr(lg), fp32, ptr(probs), ptr(idx), ptr(w), n, E, k, mode, renorm, static_cast<float>(scale), current_stream()),
            "pt_router_topk_fwd");
    }
  }
  if (node) {
    torch::autograd::set_history(w, node);
    if (probs.defined()) torch::autograd::set_history(probs, node);
    node->probs = SavedVariable(probs, probs.defined());
    node->idx = SavedVariable(idx, false);
    node->w = SavedVariable(w, true);
    node->mode = static_cast<int>(mode);
    node->renorm = renorm; node->scale = scale; node->experts = E; node->type = logits.scalar_type();
  }
  return py::make_tuple(w, idx, probs.defined() ? py::cast(probs) : py::none());
}

// The top k alone, [n, k] int32: what a replay of the routing is handed.
Tensor router_picks(const Tensor& logits, int64_t k) {
  if (tracing()) return traced<Tensor>("router_picks", logits, k);
  refuse_transforms({&logits});
  check_operands(logits, {});
  Below guard;
  const Tensor lg = logits.contiguous();
  const int64_t n = lg.size(0), E = lg.size(1);
  Tensor idx = empty({n, k}, lg, at::kInt), w = empty({n, k}, lg, at::kFloat);
  check(api.pt_router_topk_fwd(ptr(lg), lg.scalar_type() == at::kFloat, nullptr, ptr(idx), ptr(w), n, E, k, SOFTMAX_TOPK, 0, 1.f, current_stream()),
        "pt_router_topk_fwd");
  return idx;
}

// ------------------------------------------------------------------------------------------------
// expert block (bf16, no biases; every slot has a local expert)
// ------------------------------------------------------------------------------------------------
// Rows of group g times w[g]: D = X W^T (w [E, N, K]) or, w_mn, D = X W (w [E, K, N]); K the reduction.
Tensor grouped(const Tensor& x, const Tensor& w, const Tensor& offs, bool w_mn) {
  const int64_t R = x.size(0), K = x.size(1), E = w.size(0), N = w_mn ? w.size(2) : w.size(1);
  TORCH_CHECK(w.is_contiguous(), "expert weights must be contiguous");
  Tensor out = empty({R, N}, x, at::kBFloat16);
  check(api.pt_gemm_bf16(ptr(x), ptr(w), ptr(out), 1, R, N, K, 0, w_mn, R, K, K, E * w.size(1), w.size(2), w.size(2), R, N, ptr(offs), E, w.size(1), 0, 0, 0,
                         1, 2, 0, 0, nullptr, 1, 0, current_stream()),
        "pt_gemm_bf16");
  return out;
}
Tensor gather(const Tensor& src, const Tensor& idx, int64_t div, const Tensor& n_rows) {
  Tensor dst = empty({idx.numel(), src.size(1)}, src, at::kBFloat16);
  check(api.pt_gather_rows(ptr(src), ptr(idx), div, ptr(dst), ptr(n_rows), dst.size(0), dst.size(1), src.stride(0), current_stream()), "pt_gather_rows");
  return dst;
}
Tensor combine(const Tensor& y, const Tensor& row_of_slot, const Tensor& w, int64_t k) {
  const int64_t n = row_of_slot.numel() / k;
  Tensor out = empty({n, y.size(1)}, y, at::kBFloat16);
  check(api.pt_combine(ptr(y), ptr(row_of_slot), ptr(w), nullptr, ptr(out), nullptr, n, k, y.size(1), current_stream()), "pt_combine");
  return out;
}

struct ExpertsBackward : Node {
  SavedVariable x, w, gu, offs, row_of_slot, slot_of_row;
  Tensor w1, w2;  // parameters, not activations: saved-tensor hooks would copy or count them for every micro-batch
  PyRef queue_wgrad;  // (dyg, act, dgu, x, slot_of_row, offs, n_rows)
  int64_t k = 0;
  bool interleaved = false;
  double alpha = 1, limit = 0;

  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    if (!grads[0].defined()) return {Tensor(), Tensor()};
    const Tensor xv = x.unpack(), wv = w.unpack(), g = gu.unpack(), o = offs.unpack();
    const Tensor ros = row_of_slot.unpack(), sor = slot_of_row.unpack();
    Tensor dx, dw, dyg, dgu, act, n_rows;
    {
      Below guard;
      const Tensor d_out = dense(grads[0]);
      n_rows = o.narrow(0, w1.size(0), 1);
      const int64_t R = g.size(0), inter = g.size(1) / 2;
      dyg = gather(d_out, sor, k, n_rows);  // output gradient of each sorted row, without its routing weight
      const Tensor da = grouped(dyg, w2, o, true);
      // routing weights and their gradients are looked up and scattered through the slot index in the kernel
      dgu = at::empty_like(g);
      act = empty({R, inter}, g, at::kBFloat16);
      const Tensor wf = wv.to(at::kFloat).contiguous();
      dw = at::zeros({wf.numel()}, wf.options());
      check(api.pt_swiglu_bwd(ptr(g), ptr(da), ptr(wf), ptr(dgu), ptr(act), ptr(dw), ptr(n_rows), R, inter, interleaved, static_cast<float>(alpha),
                              static_cast<float>(limit), ptr(sor), current_stream()),
            "pt_swiglu_bwd");
      const Tensor dxs = grouped(dgu, w1, o, true);
      if (task_should_compute_output(0)) dx = combine(dxs, ros, Tensor(), k);
      dw = dw.view(wv.sizes()).to(wv.scalar_type());
    }
    py::gil_scoped_acquire gil;
    queue_wgrad.get()(dyg, act, dgu, xv, sor, o, n_rows);
    return {dx, dw};
  }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    for (SavedVariable* s : {&x, &w, &gu, &offs, &row_of_slot, &slot_of_row}) s->reset_data();
    w1.reset();
    w2.reset();
  }
};

// g1 [E, 2I, H] += dgu^T x, g2 [E, H, I] += dyg^T act over the rows of each group, x gathered into their order.
void expert_wgrads(const Tensor& dyg, const Tensor& act, const Tensor& dgu, const Tensor& x, const Tensor& slot_of_row, const Tensor& offs,
                   const Tensor& n_rows, int64_t k, const Tensor& g1, const Tensor& g2) {
  Below guard;
  const auto add = [&](const Tensor& dy, const Tensor& a, const Tensor& g) {
    const int64_t R = dy.size(0), N = dy.size(1), K = a.size(1), E = g.size(0);
    TORCH_CHECK(g.dim() == 3 && g.size(1) == N && g.size(2) == K && g.is_contiguous(), "expert_wgrads: gradient buffer ", g.sizes());
    check_aligned(g, "the gradient buffer");
    check_operands(dy, {&g});
    check(api.pt_gemm_bf16(ptr(dy), ptr(a), g.data_ptr(), 2, N, K, 0, 1, 1, R, N, dy.stride(0), R, K, a.stride(0), N, K, ptr(offs), E, 0, N * K,
                           g.scalar_type() == at::kFloat, 1, 1, 2, 0, 0, nullptr, 1, 0, current_stream()),
          "pt_gemm_bf16");
  };
  add(dyg, act, g2);
  add(dgu, gather(x, slot_of_row, k, n_rows), g1);
}

// out[t] = sum_j w[t, j] * expert_{eids[t, j]}(x[t]); x [n, H], w and eids [n, k], w1 [E, 2I, H], w2 [E, H, I]
Tensor moe_experts(const Tensor& x, const Tensor& w, const Tensor& eids, const Tensor& w1, const Tensor& w2, int64_t align, int64_t r_cap,
                   bool interleaved, double alpha, double limit, const py::object& queue_wgrad) {
  if (tracing()) return traced<Tensor>("moe_experts", x, w, eids, w1, w2, align, r_cap, interleaved, alpha, limit, queue_wgrad);
  refuse_transforms({&x, &w, &w1, &w2});
  check_operands(x, {&w, &eids, &w1, &w2});
  auto node = make_node<ExpertsBackward>(x, w);
  Tensor gu, out, offs, row_of_slot, slot_of_row;
  const int64_t n = eids.size(0), k = eids.size(1), E = w1.size(0), slots = n * k;
  {
    Below guard;
    check_rows(x, "x");
    check_aligned(w1, "w1");
    check_aligned(w2, "w2");
    const Tensor flat = eids.to(at::kInt).contiguous();
    const Tensor counts = E > 1024 ? empty({E}, flat, at::kInt) : Tensor();  // scratch of the sort beyond that many experts
    offs = empty({E + 1}, flat, at::kInt);
    row_of_slot = empty({slots}, flat, at::kInt);
    slot_of_row = empty({r_cap}, flat, at::kInt);
    check(api.pt_route_sort(ptr(flat), nullptr, slots, E, align, ptr(counts), E, ptr(offs), ptr(row_of_slot), ptr(slot_of_row), r_cap,
                            current_stream()),
          "pt_route_sort", E > 1024 ? 3 : 1);
    const Tensor n_rows = offs.narrow(0, E, 1);
    gu = grouped(gather(x, slot_of_row, k, n_rows), w1, offs, false);
    const int64_t inter = gu.size(1) / 2;
    Tensor act = empty({r_cap, inter}, x, at::kBFloat16);
    check(api.pt_swiglu_fwd(ptr(gu), ptr(act), ptr(n_rows), r_cap, inter, interleaved, static_cast<float>(alpha), static_cast<float>(limit), current_stream()),
          "pt_swiglu_fwd");
    const Tensor y = grouped(act, w2, offs, false);
    out = combine(y, row_of_slot, w.to(at::kFloat).contiguous(), k);
  }
  if (node) {
    torch::autograd::set_history(out, node);
    node->x = SavedVariable(x, false);
    node->w = SavedVariable(w, false);
    node->w1 = w1;
    node->w2 = w2;
    node->gu = SavedVariable(gu, false);
    node->offs = SavedVariable(offs, false);
    node->row_of_slot = SavedVariable(row_of_slot, false);
    node->slot_of_row = SavedVariable(slot_of_row, false);
    node->queue_wgrad = PyRef(queue_wgrad);
    node->k = k; node->interleaved = interleaved; node->alpha = alpha; node->limit = limit;
  }
  return out;
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.def("bind", &bind);
  m.def("launches", [] { return launches.load(); });
  m.def("rmsnorm", &rmsnorm);
  m.def("linear", &linear);
  m.def("wgrad_into", &wgrad_into);
  m.def("qk_norm_rope", &qk_norm_rope);
  m.def("attention", &attention);
  m.def("router", &router);
  m.def("router_picks", &router_picks);
  m.def("moe_experts", &moe_experts);
  m.def("expert_wgrads", &expert_wgrads);
}
