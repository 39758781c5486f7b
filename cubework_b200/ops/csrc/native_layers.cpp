// Autograd nodes of the local linear layer, the layer norms and the packed attention in C++.
//
// The kernels of a small layer take 2 to 20 us each; a Python autograd.Function around them takes 15 to 30 us of host time
// per direction (argument handling, views, the GIL in the engine's thread), so small batches and decoding ran at the
// host's pace.  These nodes hold the same tensors and launch the same kernels as the Python functions of
// parallel/functional.py and ops/__init__.py, which stay for everything the kernels do not take (host tensors, fp32
// compute, extents that need padding); the callers there decide.
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include <atomic>

namespace cw {

std::vector<torch::Tensor> gemm(torch::Tensor a, torch::Tensor b, bool trans_a, bool trans_b, c10::optional<torch::Tensor> bias,
                                const std::string& act, bool out_f32, bool want_z);
std::vector<torch::Tensor> act_backward(torch::Tensor dy, c10::optional<torch::Tensor> z, int64_t act, bool want_dz, bool want_sum);
std::vector<torch::Tensor> layer_norm_fwd_res(torch::Tensor x, c10::optional<torch::Tensor> residual, torch::Tensor gamma,
                                              torch::Tensor beta, double eps);
std::vector<torch::Tensor> layer_norm_bwd_res(torch::Tensor dy, torch::Tensor x, torch::Tensor mean, torch::Tensor rstd,
                                              torch::Tensor gamma, c10::optional<torch::Tensor> dres);

std::vector<torch::Tensor> attention_fwd(torch::Tensor qkv, bool causal, c10::optional<torch::Tensor> key_bias, double scale,
                                         int64_t status_ptr, c10::optional<torch::Tensor> trace);
torch::Tensor attention_bwd(torch::Tensor dout, torch::Tensor qkv, torch::Tensor out, torch::Tensor lse, bool causal,
                            c10::optional<torch::Tensor> key_bias, double scale, int64_t status_ptr,
                            c10::optional<torch::Tensor> packed, c10::optional<torch::Tensor> trace);
int64_t status_device_ptr();

using torch::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

static std::atomic<int64_t> g_native_launches{0};
int64_t native_launch_count() { return g_native_launches.load(); }

// 2-D, of the compute dtype, contiguous, and on a 16-byte boundary (TMA and the vector loads)
static Tensor as_rows(const Tensor& t, at::ScalarType cd) {
  Tensor r = t.reshape({-1, t.size(-1)});
  if (r.scalar_type() != cd) r = r.to(cd);
  r = r.contiguous();
  return reinterpret_cast<uintptr_t>(r.data_ptr()) % 16 == 0 ? r : r.clone();
}
static Tensor as_f32(const Tensor& t) { return t.scalar_type() == at::kFloat && t.is_contiguous() ? t : t.to(at::kFloat).contiguous(); }
static Tensor cast_to(Tensor t, int64_t dtype) {
  const auto d = static_cast<at::ScalarType>(dtype);
  return t.scalar_type() == d ? t : t.to(d);
}

// y = act(x op(w) + b); `wc` is w in the compute dtype.
struct LinearFn : public torch::autograd::Function<LinearFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, const c10::optional<Tensor>& bias, const Tensor& wc,
                        bool out_in, int64_t act, bool keep) {
    const auto cd = wc.scalar_type();
    const c10::cuda::CUDAGuard guard(x.device());
    Tensor x2 = as_rows(x, cd);
    const Tensor wa = as_rows(wc, cd);
    static const std::string names[3] = {"", "gelu", "relu"};
    g_native_launches += 1;
    auto r = gemm(x2, wa, false, out_in, bias, names[act], false, keep && act != 0);
    if (keep) {
      // Saved as the Python function saves them.  The 16-bit copy of the weight is not the graph's (it is the parameter's, and
      // stays): hooks on saved tensors, which may move them to the host, are not asked about it.
      ctx->save_for_backward({x2, w, r[1].defined() ? r[1] : Tensor()});
      ctx->saved_data["wc"] = wc;
      ctx->saved_data["out_in"] = out_in;
      ctx->saved_data["act"] = act;
      ctx->saved_data["b"] = bias.has_value() ? static_cast<int64_t>(bias->scalar_type()) : int64_t{-1};
      ctx->saved_data["x"] = static_cast<int64_t>(x.scalar_type());
      ctx->saved_data["shape"] = x.sizes().vec();
    }
    auto shape = x.sizes().vec();
    shape.back() = r[0].size(1);
    return r[0].view(shape);
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor x2 = saved[0], w = saved[1], z = saved[2], wc = ctx->saved_data["wc"].toTensor();
    const bool out_in = ctx->saved_data["out_in"].toBool();
    const int64_t act = ctx->saved_data["act"].toInt(), bt = ctx->saved_data["b"].toInt();
    const auto cd = wc.scalar_type();
    const c10::cuda::CUDAGuard guard(x2.device());
    Tensor dy = as_rows(grads[0], cd), db, dx, dw;
    if (act != 0) {
      g_native_launches += bt >= 0 ? 2 : 1;
      auto r = act_backward(dy, z, act, true, bt >= 0);
      dy = r[0];
      if (bt >= 0) db = cast_to(r[1], bt);
    } else if (bt >= 0) {
      g_native_launches += 2;
      db = cast_to(act_backward(dy, c10::nullopt, 0, false, true)[1], bt);
    }
    if (ctx->needs_input_grad(0)) {
      g_native_launches += 1;
      dx = gemm(dy, as_rows(wc, cd), false, !out_in, c10::nullopt, "", false, false)[0];
      dx = cast_to(dx.view(ctx->saved_data["shape"].toIntVector()), ctx->saved_data["x"].toInt());
    }
    if (ctx->needs_input_grad(1)) {
      g_native_launches += 1;
      const bool f32 = w.scalar_type() == at::kFloat;
      dw = out_in ? gemm(dy, x2, true, false, c10::nullopt, "", f32, false)[0] : gemm(x2, dy, true, false, c10::nullopt, "", f32, false)[0];
    }
    return {dx, dw, db, Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

// (LN(x)) or, with a residual, (x + r, LN(x + r)); see _LayerNorm and _AddLayerNorm.
struct NormFn : public torch::autograd::Function<NormFn> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const c10::optional<Tensor>& r, const Tensor& gamma,
                               const Tensor& beta, double eps, int64_t cdi) {
    const auto cd = static_cast<at::ScalarType>(cdi);
    const c10::cuda::CUDAGuard guard(x.device());
    const Tensor x2 = as_rows(x, cd);
    c10::optional<Tensor> r2;
    if (r.has_value()) r2 = as_rows(*r, cd);
    g_native_launches += 1;
    // the kernels read 16-bit parameters of the rows' type as they are
    const bool raw = gamma.scalar_type() == cd && beta.scalar_type() == cd && gamma.is_contiguous() && beta.is_contiguous();
    auto o = layer_norm_fwd_res(x2, r2, raw ? gamma : as_f32(gamma), raw ? beta : as_f32(beta), eps);
    ctx->save_for_backward({r.has_value() ? o[3] : x2, o[1], o[2], gamma});
    ctx->saved_data["x"] = static_cast<int64_t>(x.scalar_type());
    ctx->saved_data["r"] = r.has_value() ? static_cast<int64_t>(r->scalar_type()) : int64_t{-1};
    ctx->saved_data["shape"] = x.sizes().vec();
    if (r.has_value()) return {o[3].view(x.sizes()), o[0].view(x.sizes())};
    return {o[0].view(x.sizes())};
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor x2 = saved[0], gamma = saved[3];
    const auto cd = x2.scalar_type();
    const int64_t rt = ctx->saved_data["r"].toInt();
    const c10::cuda::CUDAGuard guard(x2.device());
    c10::optional<Tensor> dres;
    if (rt >= 0) dres = as_rows(grads[0], cd);
    const Tensor dy = as_rows(grads[rt >= 0 ? 1 : 0], cd);
    g_native_launches += 2;
    auto o = layer_norm_bwd_res(dy, x2, saved[1], saved[2], as_f32(gamma), dres);
    const Tensor dx = o[0].view(ctx->saved_data["shape"].toIntVector());
    const auto pt = static_cast<int64_t>(gamma.scalar_type());
    return {cast_to(dx, ctx->saved_data["x"].toInt()), rt >= 0 ? cast_to(dx, rt) : Tensor(), cast_to(o[1], pt), cast_to(o[2], pt),
            Tensor(), Tensor()};
  }
};

// Fused attention over packed QKV [B, T, heads, 3*dh] -> [B, T, heads, dh]; see _AttentionFn.
struct AttentionFn : public torch::autograd::Function<AttentionFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& qkv, bool causal, const c10::optional<Tensor>& bias, double scale) {
    const c10::cuda::CUDAGuard guard(qkv.device());
    auto r = attention_fwd(qkv, causal, bias, scale, status_device_ptr(), c10::nullopt);
    g_native_launches += r[2].defined() ? 2 : 1;
    // r[2] is the padded, TMA-aligned copy of QKV that odd head dims need; the backward takes it back
    ctx->save_for_backward({qkv, r[0], r[1], bias.has_value() ? *bias : Tensor(), r[2]});
    ctx->saved_data["causal"] = causal;
    ctx->saved_data["scale"] = scale;
    return r[0];
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const c10::cuda::CUDAGuard guard(saved[0].device());
    c10::optional<Tensor> bias, packed;
    if (saved[3].defined()) bias = saved[3];
    if (saved[4].defined()) packed = saved[4];
    g_native_launches += packed.has_value() ? 4 : 3;
    return {attention_bwd(grads[0].contiguous(), saved[0], saved[1], saved[2], ctx->saved_data["causal"].toBool(), bias,
                          ctx->saved_data["scale"].toDouble(), status_device_ptr(), packed, c10::nullopt),
            Tensor(), Tensor(), Tensor()};
  }
};

Tensor native_linear(const Tensor& x, const Tensor& w, const c10::optional<Tensor>& b, const Tensor& wc, bool out_in, int64_t act) {
  return LinearFn::apply(x, w, b, wc, out_in, act, at::GradMode::is_enabled());
}
std::vector<Tensor> native_norm(const Tensor& x, const c10::optional<Tensor>& residual, const Tensor& gamma, const Tensor& beta,
                                double eps, torch::ScalarType cd) {
  return NormFn::apply(x, residual, gamma, beta, eps, static_cast<int64_t>(cd));
}
Tensor native_attention(const Tensor& qkv, bool causal, const c10::optional<Tensor>& bias, double scale) {
  return AttentionFn::apply(qkv, causal, bias, scale);
}

}  // namespace cw
