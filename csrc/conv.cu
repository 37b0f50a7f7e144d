// Depthwise causal convolution (kernel 4, left padding 3) fused with SiLU on the [B, S, C] layout, forward and backward.
// Every thread owns two adjacent channels and a run of RUN tokens, sliding a 4-token window through registers, so x is
// read once and y written once with fully coalesced 4-byte accesses across channels.
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>

#include "common.cuh"
#include "host.h"
#include "launch.cuh"

namespace q38 {

constexpr int RUN = 32, RUN_BWD = 128, KW = 4;   // tokens per thread: the backward uses longer runs (fewer atomics per weight-gradient element)
using bf16 = __nv_bfloat16;

// Two channels at a time: packed fp32 pairs (fma.rn.f32x2 and its kin round each half like the scalar instruction).
using pair = uint64_t;
__device__ __forceinline__ pair pk(float lo, float hi) { pair d; asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi)); return d; }
__device__ __forceinline__ void unpk(pair v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ pair fma2(pair a, pair b, pair c) { pair d; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c)); return d; }
__device__ __forceinline__ pair mul2(pair a, pair b) { pair d; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ pair from_bf16x2(uint32_t v) { return pk(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u)); }
__device__ __forceinline__ uint32_t to_bf16x2(pair v) {
  float lo, hi;
  unpk(v, lo, hi);
  const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ pair sigmoid2(pair v) {
  float lo, hi;
  unpk(v, lo, hi);
  return pk(sigmoidf_(lo), sigmoidf_(hi));
}
// this thread's taps, rounded to bf16 like the activations
__device__ __forceinline__ void load_taps(const float* __restrict__ w, int c, pair (&t)[KW]) {
#pragma unroll
  for (int j = 0; j < KW; ++j) t[j] = pk(bf16_round(w[c * KW + j]), bf16_round(w[(c + 1) * KW + j]));
}
__device__ __forceinline__ uint32_t ld1(const bf16* p) { return *reinterpret_cast<const uint32_t*>(p); }

// y[b,t,c] = silu( sum_j w[c,j] * x[b,t-3+j,c] ),  x out of range = 0
// FULL: the whole run lies inside the sequence (no predicates per token).
template <bool FULL>
__device__ __forceinline__ void conv_fwd_run(const bf16* __restrict__ xb, const pair (&w)[KW], bf16* __restrict__ yb, int t0, int S, int C) {
  constexpr int GROUP = 8;                                    // loads in flight per thread
  pair win[KW];
#pragma unroll
  for (int j = 0; j < KW - 1; ++j) win[j + 1] = t0 - 3 + j >= 0 ? from_bf16x2(ld1(xb + (ptrdiff_t)(j - 3) * C)) : 0ull;
#pragma unroll 1
  for (int i0 = 0; i0 < RUN; i0 += GROUP) {
    uint32_t raw[GROUP];
#pragma unroll
    for (int u = 0; u < GROUP; ++u) raw[u] = FULL || t0 + i0 + u < S ? ld1(xb + (size_t)u * C) : 0u;
#pragma unroll
    for (int u = 0; u < GROUP; ++u) {
#pragma unroll
      for (int j = 0; j < KW - 1; ++j) win[j] = win[j + 1];
      win[KW - 1] = from_bf16x2(raw[u]);
      pair a = 0ull;
#pragma unroll
      for (int j = 0; j < KW; ++j) a = fma2(w[j], win[j], a);
      a = from_bf16x2(to_bf16x2(a));                          // the convolution output is bf16 before the activation
      if (FULL || t0 + i0 + u < S) *reinterpret_cast<uint32_t*>(yb + (size_t)u * C) = to_bf16x2(mul2(a, sigmoid2(a)));
    }
    xb += (size_t)GROUP * C;
    yb += (size_t)GROUP * C;
  }
}
__global__ void __launch_bounds__(128) conv_silu_fwd_kernel(const bf16* __restrict__ x, const float* __restrict__ w, bf16* __restrict__ y, int S, int C) {
  grid_wait();
  const int c = 2 * (blockIdx.x * 128 + threadIdx.x);
  if (c >= C) return;
  const int t0 = blockIdx.y * RUN, b = blockIdx.z;
  const size_t at = ((size_t)b * S + t0) * C + c;
  pair wt[KW];
  load_taps(w, c, wt);
  if (t0 + RUN <= S) conv_fwd_run<true>(x + at, wt, y + at, t0, S, C);
  else conv_fwd_run<false>(x + at, wt, y + at, t0, S, C);
}

// dpre[t] = dy[t] * silu'(pre[t]);  dx[t] = sum_j w[j] * dpre[t+3-j];  dw[j] += sum_t dpre[t] * x[t-3+j]
// A thread walks tokens t0 .. t0 + RUN_BWD + 2 and emits dx of token (cursor - 3).  Bound by instructions: with scalar arithmetic, a predicate and an
// address computation per access the loop took 117 per token and channel pair (66 % of the issue slots); packed pairs, running pointers
// and an interior path without predicates leave about half.  16384 x 2240: 70 us, 101 with scalar arithmetic (111 with five CTAs per SM); the
// forward, with eight loads in flight instead of one, 35 instead of 43.  The bytes need 34 and 22.
template <bool FULL>
__device__ __forceinline__ void conv_bwd_run(const bf16* __restrict__ xb, const bf16* __restrict__ gb, const pair (&w)[KW], bf16* __restrict__ dxb, pair (&g)[KW], int t0, int S, int C) {
  constexpr int GROUP = 4;
  const pair one = pk(1.f, 1.f), minus = pk(-1.f, -1.f);
  pair win[KW], dpre[KW] = {0ull, 0ull, 0ull, 0ull};          // x[t-3 .. t] and dpre[t-3 .. t]
#pragma unroll
  for (int j = 0; j < KW - 1; ++j) win[j + 1] = t0 - 3 + j >= 0 ? from_bf16x2(ld1(xb + (ptrdiff_t)(j - 3) * C)) : 0ull;
  // One token; `inside`: t < S, `own`: the token belongs to this run (weight gradient), `emit`: dx of the token three back is complete
  auto token = [&](uint32_t xr, uint32_t gr, bool inside, bool own, bool emit, bf16* out) {
#pragma unroll
    for (int j = 0; j < KW - 1; ++j) { win[j] = win[j + 1]; dpre[j] = dpre[j + 1]; }
    win[KW - 1] = from_bf16x2(xr);
    pair dp = 0ull;
    if (inside) {
      pair a = 0ull;
#pragma unroll
      for (int j = 0; j < KW; ++j) a = fma2(w[j], win[j], a);
      a = from_bf16x2(to_bf16x2(a));
      const pair s = sigmoid2(a);
      dp = mul2(mul2(from_bf16x2(gr), s), fma2(a, fma2(s, minus, one), one));
      if (own) {
#pragma unroll
        for (int j = 0; j < KW; ++j) g[j] = fma2(dp, win[j], g[j]);
      }
    }
    dpre[KW - 1] = dp;
    if (emit) {
      pair d = mul2(w[0], dpre[KW - 1]);
#pragma unroll
      for (int j = 1; j < KW; ++j) d = fma2(w[j], dpre[KW - 1 - j], d);
      *reinterpret_cast<uint32_t*>(out) = to_bf16x2(d);
    }
  };
  bf16* dst = dxb - (ptrdiff_t)3 * C;                         // dx of the cursor's token - 3
#pragma unroll 1
  for (int i0 = 0; i0 < RUN_BWD; i0 += GROUP) {
    uint32_t xs[GROUP], gs[GROUP];
#pragma unroll
    for (int u = 0; u < GROUP; ++u) {
      const bool ok = FULL || t0 + i0 + u < S;
      xs[u] = ok ? ld1(xb + (size_t)u * C) : 0u;
      gs[u] = ok ? ld1(gb + (size_t)u * C) : 0u;
    }
#pragma unroll
    for (int u = 0; u < GROUP; ++u) token(xs[u], gs[u], FULL || t0 + i0 + u < S, true, (i0 > 0 || u >= KW - 1) && (FULL || t0 + i0 + u - 3 < S), dst + (ptrdiff_t)u * C);
    xb += (size_t)GROUP * C;
    gb += (size_t)GROUP * C;
    dst += (ptrdiff_t)GROUP * C;
  }
#pragma unroll
  for (int u = 0; u < KW - 1; ++u) {                          // the three tokens behind the run that its last dx still need
    const bool ok = t0 + RUN_BWD + u < S;
    token(ok ? ld1(xb + (size_t)u * C) : 0u, ok ? ld1(gb + (size_t)u * C) : 0u, ok, false, FULL || t0 + RUN_BWD + u - 3 < S, dst + (ptrdiff_t)u * C);
  }
}
__global__ void __launch_bounds__(128, 8) conv_silu_bwd_kernel(const bf16* __restrict__ x, const float* __restrict__ w, const bf16* __restrict__ dy,
                                                               bf16* __restrict__ dx, float* __restrict__ dw, int S, int C) {
  grid_wait();
  const int c = 2 * (blockIdx.x * 128 + threadIdx.x);
  if (c >= C) return;
  const int t0 = blockIdx.y * RUN_BWD, b = blockIdx.z;
  const size_t at = ((size_t)b * S + t0) * C + c;
  pair wt[KW], g[KW] = {0ull, 0ull, 0ull, 0ull};
  load_taps(w, c, wt);
  if (t0 + RUN_BWD <= S) conv_bwd_run<true>(x + at, dy + at, wt, dx + at, g, t0, S, C);
  else conv_bwd_run<false>(x + at, dy + at, wt, dx + at, g, t0, S, C);
#pragma unroll
  for (int j = 0; j < KW; ++j) {
    float lo, hi;
    unpk(g[j], lo, hi);
    atomicAdd(&dw[c * KW + j], lo);
    atomicAdd(&dw[(c + 1) * KW + j], hi);
  }
}

at::Tensor conv_silu_fwd(const at::Tensor& x, const at::Tensor& w) {
  TORCH_CHECK(x.is_cuda() && x.scalar_type() == at::kBFloat16 && x.is_contiguous() && x.dim() == 3 && x.size(2) % 2 == 0, "conv_silu_fwd: contiguous bf16 [B,S,C] with even C required");
  TORCH_CHECK(w.scalar_type() == at::kFloat && w.is_contiguous() && w.numel() == x.size(2) * KW, "conv_silu_fwd: weight must be fp32 [C,4]");
  const c10::cuda::CUDAGuard guard(x.device());
  const int B = x.size(0), S = x.size(1), C = x.size(2);
  auto y = at::empty_like(x);
  dim3 grid((C / 2 + 127) / 128, (S + RUN - 1) / RUN, B);
  launch(conv_silu_fwd_kernel, grid, 128, 0, at::cuda::getCurrentCUDAStream(), (const bf16*)x.data_ptr(), w.data_ptr<float>(), (bf16*)y.data_ptr(), S, C);
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  count_launch();
  return y;
}

std::vector<at::Tensor> conv_silu_bwd(const at::Tensor& x, const at::Tensor& w, const at::Tensor& dy) {
  TORCH_CHECK(dy.is_cuda() && dy.scalar_type() == at::kBFloat16 && dy.is_contiguous() && x.is_contiguous(), "conv_silu_bwd: contiguous bf16 tensors required");
  const c10::cuda::CUDAGuard guard(x.device());
  const int B = x.size(0), S = x.size(1), C = x.size(2);
  auto dx = at::empty_like(x);
  auto dw = at::zeros({C, KW}, x.options().dtype(at::kFloat));
  dim3 grid((C / 2 + 127) / 128, (S + RUN_BWD - 1) / RUN_BWD, B);
  launch(conv_silu_bwd_kernel, grid, 128, 0, at::cuda::getCurrentCUDAStream(), (const bf16*)x.data_ptr(), w.data_ptr<float>(), (const bf16*)dy.data_ptr(),
                                                                           (bf16*)dx.data_ptr(), dw.data_ptr<float>(), S, C);
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  count_launch();
  return {dx, dw};
}

}  // namespace q38
