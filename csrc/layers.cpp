// Whole layers, one call per pass: the launches of a Gated DeltaNet layer, an attention layer with its indexer, an expert block, the entry of a
// residual-stream sub-layer and the vocabulary loss, in the order and with the kernels of the op-by-op path (q38/ops/backend.py), so results
// have the same bits.  At a few hundred tokens a pass is bound by the host: each op from Python costs 10 to 30 us (argument
// parsing, an autograd node, views, small allocations), a launch from here about 4.
//
// Everything that a backward pass needs is returned and saved by the caller's autograd node; nothing is kept here.  Inputs are not returned (a result
// that shares memory with an argument would need a schema that says so): the caller saves them itself, `saved` begins with them.  Weight gradients go to the
// parameters' fp32 gradient buffers (`grads`, `grad_of[i]` = position of weight i's buffer, -1: return a fresh fp32 gradient, -2: not wanted),
// on a second stream when one is given: it waits for the work issued so far, and the tensors it reads are recorded on it.  A pass says whether it
// put anything there: the caller joins the stream only then.
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/CUDAEvent.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/library.h>

#include "host.h"

namespace q38 {
at::Tensor qsa_first_query_lp(const at::Tensor& q_first, const at::Tensor& ki, const at::Tensor& w_first, double scale);   // qsa_first.cu

namespace {

using at::Tensor;
using OptTensor = c10::optional<Tensor>;
using Tensors = std::vector<Tensor>;
using BwdResult = std::tuple<Tensors, bool>;                             // gradients; whether work went to the second stream

Tensor f32(const Tensor& t) { return t.to(at::kFloat).contiguous(); }
Tensor rows_of(const Tensor& x) { return x.reshape({-1, x.size(-1)}).to(at::kBFloat16).contiguous(); }

// A 2-D tensor whose row stride TMA accepts: narrow matrices (one column per head, say) are copied into rows padded to 16 bytes.
Tensor tma_rows(const Tensor& t) {
  const int64_t n = t.size(1), per16 = 16 / t.element_size();
  if (t.stride(1) == 1 && t.stride(0) >= n && t.stride(0) % per16 == 0 && (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0) return t;
  auto view = at::empty({t.size(0), (n + per16 - 1) / per16 * per16}, t.options()).narrow(1, 0, n);
  view.copy_(t);
  return view;
}

Tensor mm_nt(const Tensor& a, const Tensor& b, const Tensor& err) {       // a[M,K] b[N,K]^T
  auto c = at::empty({a.size(0), b.size(0)}, a.options());
  gemm_bf16_persistent(a, b, c, false, false, 1.0, false, err, -1);
  return c;
}
Tensor mm_nn(const Tensor& a, const Tensor& b, const Tensor& err) {       // a[M,K] b[K,N]
  auto c = at::empty({a.size(0), b.size(1)}, a.options());
  gemm_bf16_persistent(tma_rows(a), b, c, false, true, 1.0, false, err, -1);
  return c;
}

// The weight gradients of one backward pass.
struct WeightGrads {
  at::TensorList grads;
  at::IntArrayRef grad_of;
  c10::optional<c10::cuda::CUDAStream> side;
  bool deterministic;
  const Tensor& err;
  mutable bool on_side = false;

  WeightGrads(at::TensorList g, at::IntArrayRef of, at::IntArrayRef stream, bool det, const Tensor& e) : grads(g), grad_of(of), deterministic(det), err(e) {
    if (!stream.empty()) {
      TORCH_CHECK(stream.size() == 3, "layers: a stream is {id, device index, device type}");
      side = c10::cuda::CUDAStream(c10::Stream::unpack3(stream[0], (c10::DeviceIndex)stream[1], (c10::DeviceType)stream[2]));
    }
  }
  bool wanted(size_t i) const { return grad_of[i] != -2; }
  const Tensor* buffer(size_t i, bool matrix) const {
    if (grad_of[i] < 0) return nullptr;
    const Tensor& g = grads[grad_of[i]];
    if (g.scalar_type() != at::kFloat || !g.is_contiguous()) return nullptr;
    if (matrix && (g.dim() != 2 || g.size(1) % 4 != 0 || (reinterpret_cast<uintptr_t>(g.data_ptr()) & 15) != 0)) return nullptr;
    return &g;
  }
  template <typename F> void run(F&& launch, std::initializer_list<Tensor> used) const {
    if (!side.has_value()) { launch(); return; }
    at::cuda::CUDAEvent issued;
    issued.record(at::cuda::getCurrentCUDAStream());
    issued.block(*side);
    {
      const c10::cuda::CUDAStreamGuard on(*side);
      launch();
    }
    for (const Tensor& t : used) t.record_stream(*side);
    on_side = true;
  }
  // dW_i = dy^T x.  Returns an undefined tensor when it went into the buffer or is not wanted.
  Tensor linear(size_t i, const Tensor& dy, const Tensor& x) const {
    if (!wanted(i)) return {};
    const Tensor a = tma_rows(dy), b = tma_rows(x);
    if (const Tensor* g = buffer(i, true)) {
      run([&] { gemm_bf16_persistent(a, b, *g, true, true, 1.0, true, err, deterministic ? -1 : 0); }, {a, b});
      return {};
    }
    auto out = at::empty({dy.size(1), x.size(1)}, dy.options().dtype(at::kFloat));
    gemm_bf16_persistent(a, b, out, true, true, 1.0, false, err, -1);
    return out;
  }
};

// Input gradient of several projections of one input: the later products add their tiles onto the first one's output.
struct InputGrad {
  const Tensor& err;
  Tensor dx;
  void add(const Tensor& dy, const Tensor& w) {
    if (!dx.defined()) dx = mm_nn(dy, w, err);
    else gemm_bf16_persistent(tma_rows(dy), w, dx, false, true, 1.0, true, err, -1);
  }
};

}  // namespace

// ---- Gated DeltaNet -----------------------------------------------------------------------------------------------------------
// w = {qkv, z, b, a, out} (bf16).  Returns {y} or, with `save`, {y, p_qkv, z, p_b, p_a, qkv, beta, g, o, on, (the delta rule's nine)}.
Tensors gdn_layer_fwd(const Tensor& x, at::TensorList w, const Tensor& conv_w, const Tensor& A_log, const Tensor& dt_bias, const Tensor& norm_w, int64_t Hk, int64_t Hv,
                      double eps, const Tensor& err, bool save) {
  const c10::cuda::CUDAGuard guard(x.device());
  TORCH_CHECK(x.dim() == 3 && w.size() == 5, "gdn_layer_fwd: [B,S,hidden] input and five weights required");
  const int64_t B = x.size(0), S = x.size(1);
  const Tensor x2 = rows_of(x);
  Tensor p[4];
  for (int i = 0; i < 4; ++i) p[i] = mm_nt(x2, w[i], err).view({B, S, w[i].size(0)});
  auto qkv = conv_silu_fwd(p[0], f32(conv_w.reshape({conv_w.size(0), -1})));
  auto gates = gdn_gates_fwd(p[2], p[3], f32(A_log), f32(dt_bias));
  if (!save) p[0].reset(), p[2].reset(), p[3].reset();
  auto rule = gdn_rule_fwd(qkv, gates[1], gates[0], Hk, Hv, err, save);
  if (!save) { qkv.reset(); rule.resize(1); }
  const Tensor o = rule[0].reshape({-1, 64});
  const Tensor on = gated_rmsnorm_fwd(o, p[1].view({-1, 64}), f32(norm_w), eps).view({B * S, -1});
  const Tensor y = mm_nt(on, w[4], err).view({B, S, w[4].size(0)});
  if (!save) return {y};
  Tensors out = {y, p[0], p[1], p[2], p[3], qkv, gates[0], gates[1], o, on};
  out.insert(out.end(), rule.begin() + 1, rule.end());
  return out;
}

// `saved` is {x, what the forward returned after y}.  Returns {dx, d conv, dA_log, d dt_bias, d norm, dW of qkv, z, b, a, out}.
BwdResult gdn_layer_bwd(const Tensor& dy, at::TensorList saved, at::TensorList w, const Tensor& conv_w, const Tensor& A_log, const Tensor& dt_bias, const Tensor& norm_w,
                      int64_t Hk, int64_t Hv, double eps, const Tensor& err, bool want_dx, at::TensorList grads, at::IntArrayRef grad_of, at::IntArrayRef stream,
                      bool deterministic) {
  const c10::cuda::CUDAGuard guard(dy.device());
  const WeightGrads wg(grads, grad_of, stream, deterministic, err);
  const Tensor x2 = rows_of(saved[0]);
  const Tensor &qkv = saved[5], &beta = saved[6], &g = saved[7], &o = saved[8], &on = saved[9];
  const at::TensorList p = saved.slice(1, 4);
  const int64_t B = qkv.size(0), S = qkv.size(1);
  const Tensor dy2 = rows_of(dy);
  const Tensor don = mm_nn(dy2, w[4], err);
  const Tensor dw_out = wg.linear(4, dy2, on);
  auto n = gated_rmsnorm_bwd(don.view({-1, 64}), o, p[1].view({-1, 64}), f32(norm_w), eps);
  auto r = gdn_rule_bwd(qkv, g, beta, saved.slice(10), n[0].view({B, S, -1, 64}), Hk, Hv, err);
  auto gate = gdn_gates_bwd(r[2].to(at::kBFloat16), r[1], p[2], p[3], f32(A_log), f32(dt_bias));
  auto conv = conv_silu_bwd(p[0], f32(conv_w.reshape({conv_w.size(0), -1})), r[0]);
  const Tensor dp[4] = {conv[0].view({B * S, -1}), n[1].view({B * S, -1}), gate[0].view({B * S, -1}), gate[1].view({B * S, -1})};
  InputGrad in{err, {}};
  Tensor dw[4];
  for (int i = 0; i < 4; ++i) {
    const Tensor d = tma_rows(dp[i]);
    if (want_dx) in.add(d, w[i]);
    dw[i] = wg.linear(i, d, x2);
  }
  return {Tensors{in.dx, conv[1], gate[2], gate[3], n[2], dw[0], dw[1], dw[2], dw[3], dw_out}, wg.on_side};
}

// ---- attention with indexer ------------------------------------------------------------------------------------------------------
// w = {q, k, v, o} (bf16), wi = {wq, wk, ww} of the indexer (bf16; empty without one).  The indexer runs with its KL (want_kl), or, for block
// selection alone (not dense), on the first query of every block.  Returns {y, kl} or, with `save`, {y, kl, p_q, p_k, q, k, v, gate, rstd_q, rstd_k,
// o, lse, sel, go} and with the KL also {p_qi, p_ki, qi, ki, wi, blse, dblse, rstd_qi, rstd_ki}.
Tensors qsa_layer_fwd(const Tensor& x, at::TensorList w, at::TensorList wi, const Tensor& q_norm, const Tensor& k_norm, const Tensor& cos, const Tensor& sin, double q_eps,
                      double k_eps, double scale, int64_t budget, bool dense, bool want_kl, bool main_tc, const Tensor& err, bool save) {
  const c10::cuda::CUDAGuard guard(x.device());
  TORCH_CHECK(x.dim() == 3 && w.size() == 4 && (wi.empty() || wi.size() == 3), "qsa_layer_fwd: [B,S,hidden] input and four (and three) weights required");
  const int64_t B = x.size(0), S = x.size(1), nb = S / 64;
  const Tensor x2 = rows_of(x), c = f32(cos), s = f32(sin);
  auto p_q = mm_nt(x2, w[0], err).view({B, S, -1, 128}), p_k = mm_nt(x2, w[1], err).view({B, S, -1, 64});
  auto p_v = mm_nt(x2, w[2], err).view({B, S, -1, 64});
  auto hq = qsa_headprep_fwd(p_q, f32(q_norm), c, s, q_eps, true, false), hk = qsa_headprep_fwd(p_k, f32(k_norm), c, s, k_eps, false, false);
  const Tensor &q = hq[0], &gate = hq[1], &k = hk[0];
  if (!save) p_q.reset(), p_k.reset();
  Tensors idx;
  Tensor kl, lp;
  if (!wi.empty() && (want_kl || !dense)) {
    const int64_t NI = wi[2].size(0);
    const double w_scale = std::pow((double)NI, -0.5), i_scale = std::pow(64.0, -0.5);
    if (want_kl) {
      auto p_qi = mm_nt(x2, wi[0], err).view({B, S, NI, 64}), p_ki = mm_nt(x2, wi[1], err).view({B, S, 1, 64});
      auto hqi = qsa_headprep_fwd(p_qi, c10::nullopt, c, s, 0.0, false, false), hki = qsa_headprep_fwd(p_ki, c10::nullopt, c, s, 0.0, false, false);
      const Tensor ki = hki[0].select(1, 0), wt = (mm_nt(x2, wi[2], err).view({B, S, NI}).to(at::kFloat) * w_scale).contiguous();
      Tensor e = err;
      const Tensor stats = S % 128 == 0 && main_tc ? qsa_block_stats_tc(q, k, scale, e) : qsa_main_block_stats(q, k, scale);
      const Tensor blse = qsa_indexer_fwd(hqi[0], ki, wt, i_scale, err);
      auto comb = qsa_kl_combine(stats, blse, q.size(1));
      lp = comb[1];
      kl = comb[2].mean();
      if (save) idx = {p_qi, p_ki, hqi[0], ki, wt, blse, comb[3], hqi[2], hki[2]};
    } else {
      // selection looks at the first query of each block only
      const Tensor xf = rows_of(x2.view({B, S, -1}).slice(1, 0, S, 64));
      const Tensor cf = f32(cos.slice(1, 0, cos.size(1), 64)), sf = f32(sin.slice(1, 0, sin.size(1), 64));
      const Tensor qi = qsa_headprep_fwd(mm_nt(xf, wi[0], err).view({B, nb, NI, 64}), c10::nullopt, cf, sf, 0.0, false, true)[0];
      const Tensor ki = qsa_headprep_fwd(mm_nt(x2, wi[1], err).view({B, S, 1, 64}), c10::nullopt, c, s, 0.0, false, true)[0].select(1, 0);
      const Tensor wt = mm_nt(xf, wi[2], err).view({B, nb, NI}).to(at::kFloat) * w_scale;
      lp = qsa_first_query_lp(qi, ki, wt, i_scale);
    }
  }
  const Tensor v = p_v.transpose(1, 2);                                  // the kernels read it token by token
  OptTensor count, index;
  if (!dense && !wi.empty()) {
    auto sel = qsa_select(lp, budget);
    count = sel[0];
    index = sel[1];
  }
  auto a = qsa_attn_fwd(q, k, v, count, index, scale, err);
  const Tensor o = a[0].view({B, S, -1});
  const Tensor go = sigmoid_mul_fwd(o, gate).view({B * S, -1});
  const Tensor y = mm_nt(go, w[3], err).view({B, S, -1});
  if (!save) return {y, kl};
  Tensors out = {y, kl, p_q, p_k, q, k, v, gate, hq[2], hk[2], a[0], a[1], a[2], go};
  out.insert(out.end(), idx.begin(), idx.end());
  return out;
}

// dy or dkl may be absent.  `saved` is {x, cos, sin, what the forward returned after {y, kl}}.  Returns {dx, d q_norm, d k_norm, dW of q, k, v, o, wq, wk, ww}.
BwdResult qsa_layer_bwd(const OptTensor& dy, const OptTensor& dkl, at::TensorList saved, at::TensorList w, const Tensor& q_norm, const Tensor& k_norm, double scale, const Tensor& err,
                      bool want_dx, at::TensorList grads, at::IntArrayRef grad_of, at::IntArrayRef stream, bool deterministic) {
  const c10::cuda::CUDAGuard guard(saved[0].device());
  const Tensor x2 = rows_of(saved[0]), c = f32(saved[1]), s = f32(saved[2]);
  const Tensor &p_q = saved[3], &p_k = saved[4], &q = saved[5], &k = saved[6], &v = saved[7], &gate = saved[8], &o = saved[11], &go = saved[14];
  const WeightGrads wg(grads, grad_of, stream, deterministic, err);
  const int64_t B = q.size(0), S = q.size(2), T = B * S;
  Tensors out(10);
  if (dkl.has_value() && saved.size() > 15) {
    const Tensor &p_qi = saved[15], &p_ki = saved[16], &qi = saved[17], &ki = saved[18], &wt = saved[19], &blse = saved[20], &dblse = saved[21];
    const int64_t NI = qi.size(1);
    const double w_scale = std::pow((double)NI, -0.5);
    auto d = qsa_indexer_bwd(qi, ki, wt, blse, dblse, 1.0 / (double)T, std::pow(64.0, -0.5), err, f32(*dkl));
    const Tensor dqi = qsa_headprep_bwd(d[0], c10::nullopt, p_qi, c10::nullopt, c, s, saved[22])[0];
    const Tensor dki = qsa_headprep_bwd(d[1].unsqueeze(1), c10::nullopt, p_ki, c10::nullopt, c, s, saved[23])[0];
    const Tensor dwi = (d[2] * w_scale).to(at::kBFloat16);
    out[7] = wg.linear(4, dqi.view({T, -1}), x2);
    out[8] = wg.linear(5, dki.view({T, -1}), x2);
    out[9] = wg.linear(6, dwi.view({T, -1}), x2);
  }
  if (dy.has_value()) {
    const Tensor dy2 = rows_of(*dy);
    const Tensor dgo = mm_nn(dy2, w[3], err).view({B, S, -1});
    out[6] = wg.linear(3, dy2, go);
    auto sg = sigmoid_mul_bwd(dgo, o.view({B, S, -1}), gate);
    auto a = qsa_attn_bwd(q, k, v, o, sg[0].view(o.sizes()), saved[12], saved[13], scale, err);
    auto hq = qsa_headprep_bwd(a[0], sg[1], p_q, f32(q_norm), c, s, saved[9]), hk = qsa_headprep_bwd(a[1], c10::nullopt, p_k, f32(k_norm), c, s, saved[10]);
    const Tensor dp[3] = {hq[0].view({T, -1}), hk[0].view({T, -1}), a[2].transpose(1, 2).reshape({T, -1})};
    InputGrad in{err, {}};
    for (int i = 0; i < 3; ++i) {
      if (want_dx) in.add(dp[i], w[i]);
      out[3 + i] = wg.linear(i, dp[i], x2);
    }
    out[0] = in.dx;
    out[1] = hq[1];
    out[2] = hk[1];
  }
  return {out, wg.on_side};
}

// ---- experts with the shared expert -----------------------------------------------------------------------------------------------
// w = {router, shared gate, shared up, shared gate logit, shared down, experts gate_up [E,2f,h], experts down [E,h,f]} (bf16).  Returns {y, prob_sum, counts}
// or, with `save`, {.., sg, su, gate_logit, probs, top_idx, top_w, xs, gu, hmid, ys, inv, offsets, sched, mid, shared}.
Tensors moe_layer_fwd(const Tensor& x, at::TensorList w, int64_t topk, const Tensor& err_, bool save) {
  const c10::cuda::CUDAGuard guard(x.device());
  TORCH_CHECK(x.dim() == 2 && w.size() == 7, "moe_layer_fwd: [tokens,hidden] input and seven weights required");
  Tensor err = err_;
  const Tensor xc = x.contiguous();
  const int64_t T = x.size(0), h = x.size(1), E = w[5].size(0), f2 = w[5].size(1);
  Tensor p[4];
  for (int i = 0; i < 4; ++i) p[i] = mm_nt(xc, w[i], err);
  auto route = moe_route_fwd(p[0], topk);                                // top_w, top_idx, probs, counts, prob_sum
  auto sort = moe_sort(route[1], E);                                     // perm, inv, offsets, sched
  auto xs = moe_gather(xc, sort[0], topk);
  auto hmid = at::empty({T * topk, f2 / 2}, xc.options()), gu = at::empty({T * topk, f2}, xc.options());
  moe_grouped_swiglu(xs, w[5], hmid, gu, sort[3], err);
  if (!save) xs.reset(), gu.reset();
  auto ys = at::empty({T * topk, h}, xc.options());
  moe_grouped_gemm(hmid, w[6], ys, sort[3], false, err);
  if (!save) hmid.reset();
  const Tensor routed = moe_combine_fwd(ys, sort[1], route[0]);
  if (!save) ys.reset();
  const Tensor mid = swiglu_fwd(p[1], p[2]);
  const Tensor shared = mm_nt(mid, w[4], err);
  const Tensor y = gate_add_fwd(routed, shared, p[3]);
  if (!save) return {y, route[4], route[3]};
  return {y, route[4], route[3], p[1], p[2], p[3], route[2], route[1], route[0], xs, gu, hmid, ys, sort[1], sort[2], sort[3], mid, shared};
}

// dy or d_prob_sum may be absent.  `saved` is {x, what the forward returned after {y, prob_sum, counts}}.  Returns {dx, dW of w[0] .. w[6]}.
BwdResult moe_layer_bwd(const OptTensor& dy, const OptTensor& d_prob_sum, at::TensorList saved, at::TensorList w, const Tensor& err_, bool want_dx, at::TensorList grads,
                      at::IntArrayRef grad_of, at::IntArrayRef stream, bool deterministic) {
  const c10::cuda::CUDAGuard guard(saved[0].device());
  const Tensor x = saved[0].contiguous();
  const Tensor &sg = saved[1], &su = saved[2], &gl = saved[3], &probs = saved[4], &top_idx = saved[5], &top_w = saved[6], &xs = saved[7], &gu = saved[8],
               &hmid = saved[9], &ys = saved[10], &inv = saved[11], &offsets = saved[12], &sched = saved[13], &mid = saved[14], &shared = saved[15];
  Tensor err = err_;
  const WeightGrads wg(grads, grad_of, stream, deterministic, err);
  const int64_t T = x.size(0), topk = top_idx.size(1);
  Tensors out(8);
  Tensor d_top_w, dx_experts, dsg, dsu, dgl;
  if (dy.has_value()) {
    const Tensor d = dy->to(at::kBFloat16).contiguous();
    auto ga = gate_add_bwd(d, shared, gl);
    dgl = ga[1];
    const Tensor dmid = mm_nn(ga[0], w[4], err);
    out[5] = wg.linear(4, ga[0], mid);
    auto sw = swiglu_bwd(dmid, sg, su);
    dsg = sw[0];
    dsu = sw[1];
    auto comb = moe_combine_bwd(d, ys, inv, top_w);
    const Tensor& dys = comb[0];
    d_top_w = comb[1];
    auto dgu = at::empty_like(gu), dxs = at::empty_like(xs);
    moe_grouped_dswiglu(dys, w[6], gu, dgu, sched, err);
    if (want_dx) {
      moe_grouped_gemm(dgu, w[5], dxs, sched, true, err);
      dx_experts = moe_unpermute_sum(dxs, inv, T, topk);
    }
    auto grouped = [&](size_t i, const Tensor& a, const Tensor& b) -> Tensor {
      if (!wg.wanted(i)) return {};
      if (const Tensor* g = wg.buffer(i, false)) {
        Tensor dst = *g;
        wg.run([&] { moe_grouped_wgrad(a, b, dst, offsets, err); }, {a, b, offsets});
        return {};
      }
      auto fresh = at::zeros(w[i].sizes(), w[i].options().dtype(at::kFloat));
      moe_grouped_wgrad(a, b, fresh, offsets, err);
      return fresh;
    };
    out[7] = grouped(6, dys, hmid);
    out[6] = grouped(5, dgu, xs);
  } else {
    d_top_w = at::zeros_like(top_w);
  }
  const Tensor dlogits = moe_route_bwd(probs, top_idx, top_w, d_top_w.to(at::kFloat).contiguous(), d_prob_sum.has_value() ? OptTensor(f32(*d_prob_sum)) : c10::nullopt);
  InputGrad in{err, {}};
  const Tensor dp[4] = {dlogits, dsg, dsu, dgl};
  for (int i = 0; i < 4; ++i) {
    if (!dp[i].defined()) continue;
    const Tensor d = tma_rows(dp[i].view({T, -1}));
    if (want_dx) in.add(d, w[i]);
    out[1 + i] = wg.linear(i, d, x);
  }
  if (want_dx) out[0] = dx_experts.defined() ? in.dx.add_(dx_experts) : in.dx;
  return {out, wg.on_side};
}

// ---- residual streams ---------------------------------------------------------------------------------------------------------------
// X [B,S,n,h] fp32.  Returns {normalised input [T,h], coef, Lraw, z, inv, rstd}.
Tensors mhc_layer_fwd(const Tensor& X, const Tensor& A, const Tensor& Bw, const Tensor& b_pre, const Tensor& b_post, const Tensor& b_res, const Tensor& alphas,
                      const Tensor& norm_w, int64_t iters, double eps, bool out_bf16, const Tensor& err) {
  const c10::cuda::CUDAGuard guard(X.device());
  const int64_t n = X.size(2), h = X.size(3);
  const Tensor X2 = X.contiguous().view({-1, n * h}), Ac = f32(A);
  auto Lraw = at::empty({X2.size(0), Ac.size(0)}, X2.options());
  gemm_bf16_persistent(X2, Ac, Lraw, false, false, 1.0, false, err, -1);
  auto out = mhc_coef_fwd(X2.view({-1, n, h}), Lraw, f32(Bw), f32(b_pre), f32(b_post), f32(b_res), f32(alphas), f32(norm_w), iters, eps, out_bf16);
  return {out[0], out[1], Lraw, out[2], out[3], out[4]};
}

// saved = {X, coef, Lraw, z, inv, rstd}; dXo is the gradient of the sub-layer's output stream (absent: zero).  Returns {dX [T,n,h], dBw, dbias [27], d norm, dA}.
BwdResult mhc_layer_bwd(const Tensor& dxout, const OptTensor& dcoef, const OptTensor& dXo, at::TensorList saved, const Tensor& A, const Tensor& Bw, const Tensor& b_pre,
                      const Tensor& b_post, const Tensor& b_res, const Tensor& alphas, const Tensor& norm_w, int64_t iters, const Tensor& err, at::TensorList grads,
                      at::IntArrayRef grad_of, at::IntArrayRef stream, bool deterministic) {
  const c10::cuda::CUDAGuard guard(saved[0].device());
  const Tensor X = saved[0].contiguous();
  const Tensor &coef = saved[1], &Lraw = saved[2], &z = saved[3], &inv = saved[4], &rstd = saved[5];
  const WeightGrads wg(grads, grad_of, stream, deterministic, err);
  const int64_t n = X.size(2), h = X.size(3), T = X.size(0) * X.size(1);
  const Tensor X3 = X.view({T, n, h}), Ac = f32(A);
  Tensor dc = dcoef.has_value() ? dcoef->contiguous() : at::zeros_like(coef);
  auto a = mhc_pre_bwd_a(dxout.reshape({T, h}).contiguous(), X3, Lraw, f32(Bw), f32(b_pre), f32(b_post), f32(b_res), f32(alphas), f32(norm_w), coef, z, inv, rstd, dc, iters);
  const Tensor &dL = a[0], &c1 = a[1], &dxin = a[2], &Xbf = a[6];
  Tensor dA;
  if (wg.wanted(0)) {
    const Tensor l16 = dL.to(at::kBFloat16), x16 = Xbf.to(at::kBFloat16);
    const Tensor* g = wg.buffer(0, false);
    if (g != nullptr) {
      wg.run([&] { gemm_bf16_persistent(l16, x16, *g, true, true, 1.0, true, err, deterministic ? -1 : 0); }, {l16, x16});
    } else {
      dA = at::empty({dL.size(1), n * h}, dL.options());
      gemm_bf16_persistent(l16, x16, dA, true, true, 1.0, false, err, -1);
    }
  }
  // the low-rank correction of the stream gradient, kept in bf16 between the GEMM and the combine kernel; every other term of dX is fp32
  auto G = at::empty({T, n * h}, dL.options().dtype(at::kBFloat16));
  gemm_bf16_persistent(dL, Ac.t().contiguous(), G, false, false, 1.0, false, err, -1);
  const Tensor up = dXo.has_value() ? dXo->contiguous().view({T, n, h}) : at::zeros_like(X3);
  return {Tensors{mhc_pre_bwd_c(G.view({T, n, h}), up, X3, dxin, coef, c1), a[3], a[4], a[5], dA}, wg.on_side};
}

// ---- vocabulary loss -----------------------------------------------------------------------------------------------------------------
// h2 [T,hidden] and w [V,hidden] bf16.  Returns {sum of the tokens' cross-entropies, softmax - onehot [T,V] bf16}; logits of `rows` tokens at a time.
Tensors linear_ce_fwd(const Tensor& h2, const Tensor& w, const Tensor& target, int64_t rows, const Tensor& err) {
  const c10::cuda::CUDAGuard guard(h2.device());
  auto total = at::zeros({}, h2.options().dtype(at::kFloat));
  auto dlogits = at::empty({h2.size(0), w.size(0)}, h2.options());
  for (int64_t at = 0; at < h2.size(0); at += rows) {
    const int64_t n = std::min(rows, h2.size(0) - at);
    Tensor logits = dlogits.narrow(0, at, n);
    gemm_bf16_persistent(h2.narrow(0, at, n), w, logits, false, false, 1.0, false, err, -1);
    total = total + ce_inplace(logits, target.narrow(0, at, n).contiguous()).sum();
  }
  return {total, dlogits};
}

// Returns {d hidden [T,hidden] bf16, dW}; `g` is the upstream gradient (one element).
BwdResult linear_ce_bwd(const Tensor& g, const Tensor& h2, const Tensor& w, const Tensor& dlogits, const Tensor& err, at::TensorList grads, at::IntArrayRef grad_of,
                      at::IntArrayRef stream, bool deterministic) {
  const c10::cuda::CUDAGuard guard(h2.device());
  const WeightGrads wg(grads, grad_of, stream, deterministic, err);
  const Tensor gs = g.to(at::kBFloat16);
  auto scaled = [&](const Tensor& t) {
    return t.numel() % 8 == 0 && t.is_contiguous() && (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0 ? scale_bf16(t, gs) : t * gs;
  };
  const Tensor dh = scaled(mm_nn(dlogits, w, err));
  const Tensor dw = wg.wanted(0) ? wg.linear(0, dlogits, scaled(h2)) : Tensor();
  return {Tensors{dh, dw}, wg.on_side};
}

}  // namespace q38

TORCH_LIBRARY_FRAGMENT(q38, m) {
  m.def("gdn_layer_fwd(Tensor x, Tensor[] w, Tensor conv_w, Tensor A_log, Tensor dt_bias, Tensor norm_w, int Hk, int Hv, float eps, Tensor(a!) err, bool save) -> Tensor[]",
        &q38::gdn_layer_fwd);
  m.def("gdn_layer_bwd(Tensor dy, Tensor[] saved, Tensor[] w, Tensor conv_w, Tensor A_log, Tensor dt_bias, Tensor norm_w, int Hk, int Hv, float eps, Tensor(a!) err, bool want_dx, "
        "Tensor(b!)[] grads, int[] grad_of, int[] stream, bool deterministic) -> (Tensor[], bool)", &q38::gdn_layer_bwd);
  m.def("qsa_layer_fwd(Tensor x, Tensor[] w, Tensor[] wi, Tensor q_norm, Tensor k_norm, Tensor cos, Tensor sin, float q_eps, float k_eps, float scale, int budget, bool dense, "
        "bool want_kl, bool main_tc, Tensor(a!) err, bool save) -> Tensor[]", &q38::qsa_layer_fwd);
  m.def("qsa_layer_bwd(Tensor? dy, Tensor? dkl, Tensor[] saved, Tensor[] w, Tensor q_norm, Tensor k_norm, float scale, Tensor(a!) err, bool want_dx, Tensor(b!)[] grads, int[] grad_of, "
        "int[] stream, bool deterministic) -> (Tensor[], bool)", &q38::qsa_layer_bwd);
  m.def("moe_layer_fwd(Tensor x, Tensor[] w, int topk, Tensor(a!) err, bool save) -> Tensor[]", &q38::moe_layer_fwd);
  m.def("moe_layer_bwd(Tensor? dy, Tensor? d_prob_sum, Tensor[] saved, Tensor[] w, Tensor(a!) err, bool want_dx, Tensor(b!)[] grads, int[] grad_of, int[] stream, bool deterministic) "
        "-> (Tensor[], bool)", &q38::moe_layer_bwd);
  m.def("mhc_layer_fwd(Tensor X, Tensor A, Tensor Bw, Tensor b_pre, Tensor b_post, Tensor b_res, Tensor alphas, Tensor norm_w, int iters, float eps, bool out_bf16, Tensor(a!) err) "
        "-> Tensor[]", &q38::mhc_layer_fwd);
  m.def("mhc_layer_bwd(Tensor dxout, Tensor? dcoef, Tensor? dXo, Tensor[] saved, Tensor A, Tensor Bw, Tensor b_pre, Tensor b_post, Tensor b_res, Tensor alphas, Tensor norm_w, int iters, "
        "Tensor(a!) err, Tensor(b!)[] grads, int[] grad_of, int[] stream, bool deterministic) -> (Tensor[], bool)", &q38::mhc_layer_bwd);
  m.def("linear_ce_fwd(Tensor h2, Tensor w, Tensor target, int rows, Tensor(a!) err) -> Tensor[]", &q38::linear_ce_fwd);
  m.def("linear_ce_bwd(Tensor g, Tensor h2, Tensor w, Tensor dlogits, Tensor(a!) err, Tensor(b!)[] grads, int[] grad_of, int[] stream, bool deterministic) -> (Tensor[], bool)",
        &q38::linear_ce_bwd);
}
