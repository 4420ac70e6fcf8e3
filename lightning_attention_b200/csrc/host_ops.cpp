// Native call path of the Python operators: argument checks, output allocation, stream look-up, the autograd nodes and the C-ABI
// calls for the common form of a call, in one step from Python. A call whose arguments or surroundings are of any other form is
// answered with None, and the Python operators (ops/cuda/*.py) then take it through their own code, which makes the copies and
// raises the errors; both paths run the same kernels through the same C ABI.
//
// Why: with the operators in Python a forward and backward of a small problem (b1 h4 n256 d64: 25 us of kernels) took 180 us, of
// which ~75 were torch.autograd's for any Python Function and ~100 the operators' own (context managers, allocations and stream
// look-ups through Python, ctypes argument conversion); one decode step took 21 us around a 2.4 us kernel.
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/forward_grad.h>
#include <torch/extension.h>

#include "../../include/lightning_b200.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

// Entry points of the C-ABI library the Python side has loaded (bind()).
struct Api {
  decltype(&lab200_error_string) error_string;
  decltype(&lab200_last_status) last_status;
  decltype(&lab200_la_plan_chunks) plan_chunks;
  decltype(&lab200_la_workspace_bytes) workspace_bytes;
  decltype(&lab200_la_generic) generic;
  decltype(&lab200_la_decode_step) decode_step;
  decltype(&lab200_la2_fwd) la2_fwd;
  decltype(&lab200_la2_bwd) la2_bwd;
  decltype(&lab200_la2_bwd_workspace_bytes) la2_bwd_workspace_bytes;
  decltype(&lab200_la2_bwd_kept) la2_bwd_kept;
  decltype(&lab200_srmsnorm_fwd) srms_fwd;
  decltype(&lab200_srmsnorm_bwd) srms_bwd;
  decltype(&lab200_srmsnorm_gate_fwd) gate_fwd;
  decltype(&lab200_srmsnorm_gate_bwd) gate_bwd;
};
Api g_api{};

template <class F>
void set_entry(const std::unordered_map<std::string, uintptr_t>& table, const char* name, F& slot) {
  const auto it = table.find(name);
  TORCH_CHECK(it != table.end() && it->second != 0, "missing entry point ", name);
  slot = reinterpret_cast<F>(it->second);
}

void bind(const std::unordered_map<std::string, uintptr_t>& t) {
  Api a{};
  set_entry(t, "lab200_error_string", a.error_string);
  set_entry(t, "lab200_last_status", a.last_status);
  set_entry(t, "lab200_la_plan_chunks", a.plan_chunks);
  set_entry(t, "lab200_la_workspace_bytes", a.workspace_bytes);
  set_entry(t, "lab200_la_generic", a.generic);
  set_entry(t, "lab200_la_decode_step", a.decode_step);
  set_entry(t, "lab200_la2_fwd", a.la2_fwd);
  set_entry(t, "lab200_la2_bwd", a.la2_bwd);
  set_entry(t, "lab200_la2_bwd_workspace_bytes", a.la2_bwd_workspace_bytes);
  set_entry(t, "lab200_la2_bwd_kept", a.la2_bwd_kept);
  set_entry(t, "lab200_srmsnorm_fwd", a.srms_fwd);
  set_entry(t, "lab200_srmsnorm_bwd", a.srms_bwd);
  set_entry(t, "lab200_srmsnorm_gate_fwd", a.gate_fwd);
  set_entry(t, "lab200_srmsnorm_gate_bwd", a.gate_bwd);
  g_api = a;
}

void check(int rc, const char* what) {
  TORCH_CHECK(rc == LAB200_OK, what, " failed with code ", rc, ": ", g_api.error_string(rc));
}

// An earlier call's expired device wait (see _lib.raise_on_device_status); the device of `t` is current.
void raise_on_device_status(const Tensor& t) {
  const int rc = g_api.last_status();
  TORCH_CHECK(rc == LAB200_OK, "an earlier lightning attention call on ", t.device().str(), " failed on the device with code ", rc, " (",
              g_api.error_string(rc), "); its outputs are invalid");
}

// ---- the common form -------------------------------------------------------------------------------------------------------
// Ordinary strided CUDA tensors, and no tracing, dispatch mode, functional transform or forward-mode level around the call: under
// those the Python autograd Functions run, so that what they support and what they refuse stays theirs.
bool plain(const Tensor& t) {
  constexpr c10::DispatchKeySet special({c10::DispatchKey::Python, c10::DispatchKey::PythonTLSSnapshot, c10::DispatchKey::FuncTorchBatched,
                                         c10::DispatchKey::FuncTorchGradWrapper, c10::DispatchKey::BatchedNestedTensor,
                                         c10::DispatchKey::Functionalize, c10::DispatchKey::Conjugate, c10::DispatchKey::Negative,
                                         c10::DispatchKey::ZeroTensor});
  return t.defined() && t.is_cuda() && t.layout() == c10::kStrided && !t.key_set().has_any(special);
}
bool plain_surroundings() {
  const c10::DispatchKeySet extra = c10::impl::tls_local_dispatch_key_set().included_ - c10::default_included_set;
  return extra.empty() && !torch::autograd::ForwardADLevel::try_get_by_idx(0);
}

bool half_type(const Tensor& t) { return t.scalar_type() == at::kBFloat16 || t.scalar_type() == at::kHalf; }
bool aligned16(const Tensor& t) { return (reinterpret_cast<uintptr_t>(t.const_data_ptr()) & 15u) == 0; }
int dtype_code(const Tensor& t) {
  return t.scalar_type() == at::kBFloat16 ? LAB200_BF16 : t.scalar_type() == at::kHalf ? LAB200_F16 : LAB200_F32;
}

// (b, h, n, dim) view of a contiguous (b, n, h, dim) tensor (lightning_attn2.py:_is_bnhd)
bool is_bnhd(const Tensor& t) {
  const int64_t h = t.size(1), n = t.size(2), d = t.size(3);
  return h > 1 && n > 1 && t.stride(0) == n * h * d && t.stride(1) == d && t.stride(2) == h * d && t.stride(3) == 1 && aligned16(t);
}
Tensor empty_like_layout(int64_t b, int64_t h, int64_t n, int64_t d, const Tensor& like, bool bnhd) {
  const auto opt = like.options().requires_grad(false);
  return bnhd ? at::empty({b, n, h, d}, opt).transpose(1, 2) : at::empty({b, h, n, d}, opt);
}

// The layout of an attention call, or -1 when the tensors need a copy or are refused.
int call_layout(const Tensor& q, const Tensor& k, const Tensor& v) {
  if (!plain(q) || !plain(k) || !plain(v) || q.dim() != 4 || v.dim() != 4 || !half_type(q) || k.scalar_type() != q.scalar_type() ||
      v.scalar_type() != q.scalar_type() || k.sizes() != q.sizes() || k.device() != q.device() || v.device() != q.device())
    return -1;
  for (int i = 0; i < 3; ++i)
    if (v.size(i) != q.size(i)) return -1;
  if (q.numel() == 0 || v.numel() == 0 || q.size(0) * q.size(1) > 65535 || q.size(2) > (1 << 30)) return -1;
  if (q.is_contiguous() && k.is_contiguous() && v.is_contiguous()) return 0;
  const int64_t d = q.size(3), e = v.size(3);
  if (d <= 128 && e <= 128 && d % 16 == 0 && e % 16 == 0 && is_bnhd(q) && is_bnhd(k) && is_bnhd(v)) return 1;
  return -1;
}
bool plain_slopes(const Tensor& s, const Tensor& q) {
  return plain(s) && s.scalar_type() == at::kFloat && s.device() == q.device() && s.is_contiguous() && s.numel() >= q.size(1);
}

Tensor workspace(size_t bytes, const Tensor& like) {
  return at::empty({static_cast<int64_t>(bytes)}, like.options().dtype(at::kByte).requires_grad(false));
}

struct Sizes {
  int b, h, n, d, e, dt;
  Sizes(const Tensor& q, const Tensor& v, bool bnhd)
      : b(q.size(0)), h(q.size(1)), n(q.size(2)), d(q.size(3)), e(v.size(3)), dt(dtype_code(q) | (bnhd ? LAB200_LAYOUT_BNHD : 0)) {}
};
void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }
const float* float_ptr(const Tensor& s) { return s.defined() ? static_cast<const float*>(s.const_data_ptr()) : nullptr; }

// `t` in the layout of the call, copied if it has another one: a gradient, or a saved tensor. What saved-tensor hooks return has the
// values of what was packed but often other strides (a copy through pinned host memory comes back contiguous).
Tensor in_layout(const Tensor& t, bool bnhd) {
  if (!bnhd) return t.contiguous();
  return is_bnhd(t) ? t : empty_like_layout(t.size(0), t.size(1), t.size(2), t.size(3), t, true).copy_(t);
}

// ---- attention -------------------------------------------------------------------------------------------------------------
// Where the library cuts the sequence into chunks and d == e, the forward pass saves its workspace too, and backward passes read its
// chunk states transposed (they leave them as they are). It is saved like the other tensors, so that saved-tensor hooks have it as
// well: checkpointing then keeps none from the forward pass, and takes the one of the recomputed pass.
struct Attention : torch::autograd::Function<Attention> {
  static Tensor forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const std::optional<Tensor>& s_opt, bool bnhd) {
    const Tensor s = s_opt.has_value() ? *s_opt : Tensor();
    const c10::cuda::CUDAGuard guard(q.device());
    raise_on_device_status(q);
    const Sizes z(q, v, bnhd);
    Tensor o = empty_like_layout(z.b, z.h, z.n, z.e, q, bnhd);
    const size_t bytes = g_api.workspace_bytes(z.b * z.h, z.n, z.d, z.e, 0);
    Tensor ws = workspace(bytes, q);
    check(g_api.la2_fwd(q.const_data_ptr(), k.const_data_ptr(), v.const_data_ptr(), float_ptr(s), o.mutable_data_ptr(), ws.mutable_data_ptr(),
                        bytes, z.b, z.h, z.n, z.d, z.e, 0, z.dt, stream_of(q)), "lab200_la2_fwd");
    const bool keep = z.d == z.e && g_api.plan_chunks(z.b * z.h, z.n, z.d, z.e) > 1;
    ctx->saved_data["bnhd"] = bnhd;
    ctx->save_for_backward({q, k, v, s, keep ? ws : Tensor()});
    return o;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list saved = ctx->get_saved_variables();
    const bool bnhd = ctx->saved_data["bnhd"].toBool();
    Tensor go = grads[0], s = saved[3], kept = saved[4];
    const at::IntArrayRef lead = go.sizes().slice(0, 3);
    for (int i = 0; i < 3; ++i)
      TORCH_CHECK(saved[i].defined() && saved[i].dim() == 4 && saved[i].sizes().slice(0, 3) == lead && saved[i].scalar_type() == go.scalar_type() &&
                  saved[i].device() == go.device(), "lightning attention backward: saved-tensor hooks returned another shape, dtype or device");
    TORCH_CHECK(saved[1].sizes() == saved[0].sizes() && saved[2].sizes() == go.sizes() && (!s.defined() || s.numel() >= go.size(1)),
                "lightning attention backward: saved-tensor hooks returned another shape, dtype or device");
    const c10::cuda::CUDAGuard guard(go.device());
    if (s.defined() && !plain_slopes(s, go)) s = s.to(go.device(), at::kFloat).contiguous();
    const Tensor q = in_layout(saved[0], bnhd), k = in_layout(saved[1], bnhd), v = in_layout(saved[2], bnhd);
    go = in_layout(go, bnhd);
    const Sizes z(q, v, bnhd);
    if (kept.defined() && !(kept.scalar_type() == at::kByte && kept.device() == q.device() && kept.is_contiguous() && aligned16(kept) &&
                            static_cast<size_t>(kept.numel()) == g_api.workspace_bytes(z.b * z.h, z.n, z.d, z.e, 0)))
      kept = Tensor();  // not what was saved: the states are computed again
    raise_on_device_status(q);
    Tensor dq = empty_like_layout(z.b, z.h, z.n, z.d, q, bnhd), dk = empty_like_layout(z.b, z.h, z.n, z.d, q, bnhd);
    Tensor dv = empty_like_layout(z.b, z.h, z.n, z.e, q, bnhd);
    const float* sl = float_ptr(s);
    const void *qp = q.const_data_ptr(), *kp = k.const_data_ptr(), *vp = v.const_data_ptr(), *gp = go.const_data_ptr();
    void *dqp = dq.mutable_data_ptr(), *dkp = dk.mutable_data_ptr(), *dvp = dv.mutable_data_ptr(), *st = stream_of(q);
    const size_t bytes = g_api.la2_bwd_workspace_bytes(z.b, z.h, z.n, z.d, z.e, 0);
    Tensor ws = workspace(bytes, q);
    if (kept.defined()) {
      check(g_api.la2_bwd_kept(qp, kp, vp, sl, gp, dqp, dkp, dvp, kept.mutable_data_ptr(), kept.numel(), ws.mutable_data_ptr(), bytes, z.b, z.h,
                               z.n, z.d, 0, z.dt, st), "lab200_la2_bwd_kept");
    } else {
      check(g_api.la2_bwd(qp, kp, vp, sl, gp, dqp, dkp, dvp, ws.mutable_data_ptr(), bytes, z.b, z.h, z.n, z.d, z.e, 0, z.dt, st), "lab200_la2_bwd");
    }
    return {dq, dk, dv, Tensor(), Tensor()};
  }
};

std::optional<Tensor> attn(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& s) {
  const int layout = call_layout(q, k, v);
  if (layout < 0 || !plain_slopes(s, q) || !plain_surroundings()) return std::nullopt;
  return Attention::apply(q, k, v, std::optional<Tensor>(s), layout == 1);
}
std::optional<Tensor> attn_no_decay(const Tensor& q, const Tensor& k, const Tensor& v) {
  const int layout = call_layout(q, k, v);
  if (layout < 0 || !plain_surroundings()) return std::nullopt;
  return Attention::apply(q, k, v, std::optional<Tensor>(), layout == 1);
}

// ---- inference: no autograd nodes ------------------------------------------------------------------------------------------
std::optional<std::tuple<Tensor, Tensor>> prefill(const Tensor& q, const Tensor& k, const Tensor& v, const std::optional<Tensor>& s,
                                                  const std::optional<Tensor>& kv) {
  const int layout = call_layout(q, k, v);
  if (layout < 0 || (s && !plain_slopes(*s, q)) || !plain_surroundings()) return std::nullopt;
  const Sizes z(q, v, layout == 1);
  const std::array<int64_t, 4> shape{z.b, z.h, z.e, z.d};
  if (kv && !(plain(*kv) && kv->scalar_type() == at::kFloat && kv->device() == q.device() && kv->is_contiguous() && kv->sizes() == at::IntArrayRef(shape)))
    return std::nullopt;
  const c10::cuda::CUDAGuard guard(q.device());
  raise_on_device_status(q);
  Tensor o = empty_like_layout(z.b, z.h, z.n, z.e, q, layout == 1);
  Tensor out = at::empty(shape, q.options().dtype(at::kFloat).requires_grad(false));
  const size_t bytes = g_api.workspace_bytes(z.b * z.h, z.n, z.d, z.e, 0);
  Tensor ws = workspace(bytes, q);
  check(g_api.generic(q.const_data_ptr(), k.const_data_ptr(), v.const_data_ptr(), s ? float_ptr(*s) : nullptr, o.mutable_data_ptr(),
                      kv ? float_ptr(*kv) : nullptr, static_cast<float*>(out.mutable_data_ptr()), ws.mutable_data_ptr(), bytes, z.b * z.h, z.h,
                      z.n, z.d, z.e, 0, 0, 0, z.dt, stream_of(q)), "lab200_la_generic");
  return std::make_tuple(o, out);
}

std::optional<Tensor> decode(const Tensor& q, const Tensor& k, const Tensor& v, const std::optional<Tensor>& s, const Tensor& kv) {
  const int64_t nd = q.dim();
  if (!plain(q) || !plain(k) || !plain(v) || !plain(kv) || (nd != 3 && nd != 4) || v.dim() != nd || k.sizes() != q.sizes() || !half_type(q) ||
      k.scalar_type() != q.scalar_type() || v.scalar_type() != q.scalar_type() || v.size(0) != q.size(0) || v.size(1) != q.size(1) ||
      (nd == 4 && (q.size(2) != 1 || v.size(2) != 1)) || !q.is_contiguous() || !k.is_contiguous() || !v.is_contiguous() ||
      k.device() != q.device() || v.device() != q.device() || kv.device() != q.device() || q.numel() == 0 || v.numel() == 0 ||
      q.size(0) * q.size(1) > 65535 || (s && !plain_slopes(*s, q)) || !plain_surroundings())
    return std::nullopt;
  const int b = q.size(0), h = q.size(1), d = q.size(nd - 1), e = v.size(nd - 1);
  if (kv.dim() != 4 || kv.size(0) != b || kv.size(1) != h || kv.size(2) != e || kv.size(3) != d || kv.scalar_type() != at::kFloat || !kv.is_contiguous())
    return std::nullopt;
  const c10::cuda::CUDAGuard guard(q.device());
  Tensor o = at::empty(v.sizes(), v.options().requires_grad(false));
  check(g_api.decode_step(q.const_data_ptr(), k.const_data_ptr(), v.const_data_ptr(), s ? float_ptr(*s) : nullptr,
                          static_cast<float*>(kv.mutable_data_ptr()), o.mutable_data_ptr(), b * h, h, d, e, dtype_code(q), stream_of(q)),
        "lab200_la_decode_step");
  return o;
}

// ---- SimpleRMSNorm and its gated form --------------------------------------------------------------------------------------
// Rows of a contiguous tensor; the gradient is brought into the same form.
bool plain_rows(const Tensor& x) {
  const auto t = x.scalar_type();
  return plain(x) && (t == at::kFloat || t == at::kHalf || t == at::kBFloat16) && x.dim() >= 1 && x.numel() > 0 && x.is_contiguous() &&
         x.numel() / x.size(-1) <= INT_MAX && x.size(-1) * x.element_size() <= 65536;
}
float row_eps(const Tensor& x, double eps) { return static_cast<float>(x.scalar_type() == at::kHalf ? std::max(eps, 1.6e-5) : eps); }
Tensor row_grad(const Tensor& g, const Tensor& x) {
  TORCH_CHECK(g.numel() == x.numel(), "gradient and input sizes differ");
  return g.contiguous().to(x.scalar_type());
}

// Saved rows and their 1 / rms, from whatever strides saved-tensor hooks return.
Tensor saved_rows(const Tensor& x, const Tensor& g) {
  TORCH_CHECK(x.defined() && x.dim() >= 1 && x.numel() == g.numel() && x.device() == g.device(), "norm backward: saved-tensor hooks returned another shape or device");
  return x.contiguous();
}
Tensor saved_rstd(const Tensor& r, const Tensor& x) {
  TORCH_CHECK(r.defined() && r.scalar_type() == at::kFloat && r.numel() == x.numel() / x.size(-1) && r.device() == x.device(),
              "norm backward: saved-tensor hooks returned another shape, dtype or device");
  return r.contiguous();
}

struct Norm : torch::autograd::Function<Norm> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, double eps) {
    const c10::cuda::CUDAGuard guard(x.device());
    const int64_t N = x.size(-1), M = x.numel() / N;
    Tensor y = at::empty(x.sizes(), x.options().requires_grad(false)), rstd = at::empty({M}, y.options().dtype(at::kFloat));
    check(g_api.srms_fwd(x.const_data_ptr(), y.mutable_data_ptr(), static_cast<float*>(rstd.mutable_data_ptr()), M, static_cast<int>(N),
                         row_eps(x, eps), dtype_code(x), stream_of(x)), "lab200_srmsnorm_fwd");
    ctx->save_for_backward({x, rstd});
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list saved = ctx->get_saved_variables();
    const c10::cuda::CUDAGuard guard(grads[0].device());
    const Tensor x = saved_rows(saved[0], grads[0]), rstd = saved_rstd(saved[1], x);
    const int64_t N = x.size(-1), M = x.numel() / N;
    const Tensor dy = row_grad(grads[0], x);
    Tensor dx = at::empty(dy.sizes(), x.options().requires_grad(false));
    check(g_api.srms_bwd(x.const_data_ptr(), dy.const_data_ptr(), float_ptr(rstd), dx.mutable_data_ptr(), M, static_cast<int>(N), dtype_code(x),
                         stream_of(x)), "lab200_srmsnorm_bwd");
    return {dx, Tensor()};
  }
};

struct NormGate : torch::autograd::Function<NormGate> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& gate, double eps) {
    const c10::cuda::CUDAGuard guard(x.device());
    const int64_t N = x.size(-1), M = x.numel() / N;
    Tensor y = at::empty(x.sizes(), x.options().requires_grad(false)), rstd = at::empty({M}, y.options().dtype(at::kFloat));
    check(g_api.gate_fwd(x.const_data_ptr(), gate.const_data_ptr(), y.mutable_data_ptr(), static_cast<float*>(rstd.mutable_data_ptr()), M,
                         static_cast<int>(N), row_eps(x, eps), dtype_code(x), stream_of(x)), "lab200_srmsnorm_gate_fwd");
    ctx->save_for_backward({x, gate, rstd});
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list saved = ctx->get_saved_variables();
    const c10::cuda::CUDAGuard guard(grads[0].device());
    Tensor x = saved_rows(saved[0], grads[0]), gate = saved_rows(saved[1], grads[0]), rstd = saved_rstd(saved[2], x);
    TORCH_CHECK(gate.scalar_type() == x.scalar_type() && gate.sizes() == x.sizes(), "norm backward: saved-tensor hooks returned another shape or dtype");
    if (!aligned16(x)) x = x.clone();
    if (!aligned16(gate)) gate = gate.clone();
    const int64_t N = x.size(-1), M = x.numel() / N;
    Tensor dy = row_grad(grads[0], x);
    if (!aligned16(dy)) dy = dy.clone();
    Tensor dx = at::empty(x.sizes(), x.options().requires_grad(false)), dg = at::empty(x.sizes(), dx.options());
    check(g_api.gate_bwd(x.const_data_ptr(), gate.const_data_ptr(), dy.const_data_ptr(), float_ptr(rstd), dx.mutable_data_ptr(),
                         dg.mutable_data_ptr(), M, static_cast<int>(N), dtype_code(x), stream_of(x)), "lab200_srmsnorm_gate_bwd");
    return {dx, dg, Tensor()};
  }
};

std::optional<Tensor> norm(const Tensor& x, double eps) {
  if (!plain_rows(x) || !plain_surroundings()) return std::nullopt;
  return Norm::apply(x, eps);
}
std::optional<Tensor> norm_gate(const Tensor& x, const Tensor& gate, double eps) {
  if (!plain_rows(x) || !plain_rows(gate) || gate.sizes() != x.sizes() || gate.scalar_type() != x.scalar_type() || gate.device() != x.device() ||
      !aligned16(x) || !aligned16(gate) || !plain_surroundings())
    return std::nullopt;
  return NormGate::apply(x, gate, eps);
}

}  // namespace

// What this file was compiled for, for a look before it is imported (_lib.py:host_abi).
extern "C" __attribute__((visibility("default"))) const char* lab200_host_built_for() { return LAB200_HOST_ABI; }

PYBIND11_MODULE(_host_ops, m) {
  m.def("bind", &bind);
  // The GIL is released, as ctypes does: a launch may have to wait for room in the stream's queue.
  using nogil = py::call_guard<py::gil_scoped_release>;
  m.def("attn", &attn, nogil());
  m.def("attn_no_decay", &attn_no_decay, nogil());
  m.def("prefill", &prefill, nogil());
  m.def("decode", &decode, nogil());
  m.def("norm", &norm, nogil());
  m.def("norm_gate", &norm_gate, nogil());
}
