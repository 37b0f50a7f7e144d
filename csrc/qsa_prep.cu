// Head preparation for the QSA layer and its indexer: per (token, head) optional zero-centred RMSNorm over the 64 head dims,
// rotary embedding on the first 16 dims (rotate-half pairs d <-> d + 8), and the move from token-major [B,S,H,*] projection
// output to the head-major [B,H,S,64] layout of the attention kernels, in one pass.  For the query projection, whose rows hold
// q and the output gate interleaved per head ([.., H, 128]), the gate half is copied out to [B,S,H*64] in the same pass.
// The backward kernel undoes all of it and writes the gradient of the projection output (both halves) directly.
//
// Eight lanes per (b, s, h) row, 16 bytes (eight dims) each, so the rotary partner of a row's lanes 0 and 1 is the other one; a warp holds
// four rows at a time and strides over the rows with the whole grid.  Bound by memory.  With one warp and 4-byte accesses per row, 64-bit
// divisions for its position and, in the backward, 64 global atomics per eight rows, the kernels ran at a fifth of the copy bandwidth
// (projections of 16384 tokens, 22 + 2 + 4 + 1 heads: forward 124 -> 57 us, backward 250 -> 80 us; with registers for five and four CTAs
// per SM and grids of just those, 54 and 65: with 76 registers the backward ran eight CTAs per SM as three waves of three).
// cos/sin: fp32 [Bc, S, 16] with Bc in {1, B}; they are rounded to bf16 as the PyTorch path does before use.
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>

#include "common.cuh"
#include "host.h"
#include "launch.cuh"

namespace q38 {

constexpr int HP_WARPS = 8;
using bf16 = __nv_bfloat16;

__device__ __forceinline__ float bf16r(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }
__device__ __forceinline__ void unpack8(const uint4& r, float (&f)[8]) {
  const uint32_t v[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) { f[2 * i] = __uint_as_float(v[i] << 16); f[2 * i + 1] = __uint_as_float(v[i] & 0xffff0000u); }
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  uint32_t v[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) { const __nv_bfloat162 h = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]); v[i] = *reinterpret_cast<const uint32_t*>(&h); }
  return make_uint4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ uint4 shfl1(const uint4& r) {
  return make_uint4(__shfl_xor_sync(0xffffffffu, r.x, 1), __shfl_xor_sync(0xffffffffu, r.y, 1), __shfl_xor_sync(0xffffffffu, r.z, 1), __shfl_xor_sync(0xffffffffu, r.w, 1));
}
// Sum over a row's 64 values held as pair sums p[4] per lane, in the order of a butterfly over 32 lanes that hold one pair each.
__device__ __forceinline__ float row_sum(float (&p)[4]) {
#pragma unroll
  for (int o = 4; o > 0; o >>= 1)
#pragma unroll
    for (int i = 0; i < 4; ++i) p[i] += __shfl_xor_sync(0xffffffffu, p[i], o);
  return (p[0] + p[2]) + (p[1] + p[3]);
}

// `round_products` (PyTorch's bf16 rotary arithmetic): both products are rounded to bf16 before they are added.
__global__ void __launch_bounds__(32 * HP_WARPS, 5) qsa_headprep_fwd_kernel(const bf16* __restrict__ src, int src_row, const float* __restrict__ w,
                                                                         const float* __restrict__ cosv, const float* __restrict__ sinv, int Bc,
                                                                         bf16* __restrict__ out, bf16* __restrict__ gate, float* __restrict__ rstd_out,
                                                                         int S, int H, unsigned rows, float eps, bool round_products) {
  grid_wait();
  const int lane = threadIdx.x & 31, m = lane & 7;
  float wv[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) wv[e] = w != nullptr ? 1.f + w[8 * m + e] : 1.f;
  const unsigned warps = gridDim.x * HP_WARPS;
  for (unsigned base = (blockIdx.x * HP_WARPS + (threadIdx.x >> 5)) * 4u; base < rows; base += warps * 4u) {
    const unsigned row = base + (lane >> 3);
    const bool ok = row < rows;
    const unsigned tok = row / H, h = row - tok * H, b = tok / S, s = tok - b * S;
    const uint4* p = reinterpret_cast<const uint4*>(src + (size_t)row * src_row) + m;
    uint4 raw = ok ? p[0] : make_uint4(0, 0, 0, 0);
    if (ok && gate != nullptr) reinterpret_cast<uint4*>(gate + (size_t)row * 64)[m] = p[8];
    float x[8];
    unpack8(raw, x);
    if (w != nullptr) {
      float ps[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) { const float x0 = x[2 * i], x1 = x[2 * i + 1]; ps[i] = x0 * x0 + x1 * x1; }
      const float ss = row_sum(ps);
      const float rstd = rsqrtf(ss / 64.f + eps);
      if (ok && m == 0) rstd_out[row] = rstd;
#pragma unroll
      for (int e = 0; e < 8; ++e) x[e] = bf16r(x[e] * rstd * wv[e]);
      raw = pack8(x);
    }
    float o[8];
    unpack8(shfl1(raw), o);
    if (ok && m < 2) {
      const size_t at = ((size_t)(Bc == 1 ? 0 : b) * S + s) * 16 + 8 * m;
      const float sign = m == 0 ? -1.f : 1.f;
#pragma unroll
      for (int q4 = 0; q4 < 2; ++q4) {
        const float4 cv = *reinterpret_cast<const float4*>(cosv + at + 4 * q4), sv = *reinterpret_cast<const float4*>(sinv + at + 4 * q4);
        const float cc[4] = {cv.x, cv.y, cv.z, cv.w}, sc[4] = {sv.x, sv.y, sv.z, sv.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int d = 4 * q4 + e;
          const float c0 = bf16r(cc[e]), s0 = bf16r(sc[e]);
          if (round_products) x[d] = bf16r(x[d] * c0) + bf16r(sign * o[d] * s0);
          else x[d] = x[d] * c0 + sign * o[d] * s0;
        }
      }
      raw = pack8(x);
    }
    if (ok) reinterpret_cast<uint4*>(out + (((size_t)b * H + h) * S + s) * 64)[m] = raw;
  }
}

__global__ void __launch_bounds__(32 * HP_WARPS, 4) qsa_headprep_bwd_kernel(const bf16* __restrict__ dout, const bf16* __restrict__ dgate,
                                                                         const bf16* __restrict__ src, int src_row, const float* __restrict__ w,
                                                                         const float* __restrict__ cosv, const float* __restrict__ sinv, int Bc,
                                                                         const float* __restrict__ rstd_in, bf16* __restrict__ dsrc, float* __restrict__ dw,
                                                                         int S, int H, unsigned rows) {
  grid_wait();
  __shared__ float dw_s[64];
  if (threadIdx.x < 64) dw_s[threadIdx.x] = 0.f;
  __syncthreads();
  const int lane = threadIdx.x & 31, m = lane & 7;
  float wv[8], dwv[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) { wv[e] = w != nullptr ? 1.f + w[8 * m + e] : 1.f; dwv[e] = 0.f; }
  const unsigned warps = gridDim.x * HP_WARPS;
  for (unsigned base = (blockIdx.x * HP_WARPS + (threadIdx.x >> 5)) * 4u; base < rows; base += warps * 4u) {
    const unsigned row = base + (lane >> 3);
    const bool ok = row < rows;
    const unsigned tok = row / H, h = row - tok * H, b = tok / S, s = tok - b * S;
    const uint4 graw = ok ? reinterpret_cast<const uint4*>(dout + (((size_t)b * H + h) * S + s) * 64)[m] : make_uint4(0, 0, 0, 0);
    uint4* dp = reinterpret_cast<uint4*>(dsrc + (size_t)row * src_row) + m;
    if (ok && dgate != nullptr) dp[8] = reinterpret_cast<const uint4*>(dgate + (size_t)row * 64)[m];
    const uint4 xraw = ok && w != nullptr ? reinterpret_cast<const uint4*>(src + (size_t)row * src_row)[m] : make_uint4(0, 0, 0, 0);
    const float rstd = ok && w != nullptr ? rstd_in[row] : 0.f;
    float g[8], o[8];
    unpack8(graw, g);
    unpack8(shfl1(graw), o);
    // rotary backward: dx_d = dy_d c_d + dy_{d+8} s_{d+8} (d < 8),  dx_{d+8} = dy_{d+8} c_{d+8} - dy_d s_d; the tables repeat: entry d + 8 equals entry d
    if (ok && m < 2) {
      const size_t at = ((size_t)(Bc == 1 ? 0 : b) * S + s) * 16 + 8 * m;
      const float sign = m == 0 ? 1.f : -1.f;
#pragma unroll
      for (int q4 = 0; q4 < 2; ++q4) {
        const float4 cv = *reinterpret_cast<const float4*>(cosv + at + 4 * q4), sv = *reinterpret_cast<const float4*>(sinv + at + 4 * q4);
        const float cc[4] = {cv.x, cv.y, cv.z, cv.w}, sc[4] = {sv.x, sv.y, sv.z, sv.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) g[4 * q4 + e] = g[4 * q4 + e] * bf16r(cc[e]) + sign * o[4 * q4 + e] * bf16r(sc[e]);
      }
    }
    if (w != nullptr) {
      float xh[8], ps[4];
      unpack8(xraw, xh);
#pragma unroll
      for (int e = 0; e < 8; ++e) { xh[e] *= rstd; dwv[e] += g[e] * xh[e]; g[e] *= wv[e]; }
#pragma unroll
      for (int i = 0; i < 4; ++i) ps[i] = g[2 * i] * xh[2 * i] + g[2 * i + 1] * xh[2 * i + 1];
      const float dot = row_sum(ps) / 64.f;
#pragma unroll
      for (int e = 0; e < 8; ++e) g[e] = rstd * (g[e] - xh[e] * dot);
    }
    if (ok) dp[0] = pack8(g);
  }
  if (w != nullptr) {
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      dwv[e] += __shfl_xor_sync(0xffffffffu, dwv[e], 8);
      dwv[e] += __shfl_xor_sync(0xffffffffu, dwv[e], 16);
      if (lane < 8) atomicAdd(&dw_s[8 * m + e], dwv[e]);
    }
    __syncthreads();
    if (threadIdx.x < 64) atomicAdd(&dw[threadIdx.x], dw_s[threadIdx.x]);
  }
}

// As many CTAs as are resident at once, so that none waits for a second wave and a warp handles many rows (the backward adds one weight gradient per CTA).
static unsigned headprep_grid(long long rows, int resident) { return (unsigned)std::max<long long>(1, std::min<long long>((rows + 4 * HP_WARPS - 1) / (4 * HP_WARPS), kNumSMs * resident)); }

// The kernels read 16-byte pieces; a contiguous view that starts elsewhere is copied first.  Other strides go on to the checks as they are (a copy
// would make them contiguous).
static at::Tensor aligned16(const at::Tensor& t) { return (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0 || !t.is_contiguous() ? t : t.clone(); }

static void check_tables(const at::Tensor& cosv, const at::Tensor& sinv, int B, int S) {
  TORCH_CHECK(cosv.scalar_type() == at::kFloat && sinv.scalar_type() == at::kFloat && cosv.is_contiguous() && sinv.is_contiguous() && cosv.dim() == 3 &&
                  cosv.sizes() == sinv.sizes() && cosv.size(2) == 16 && cosv.size(1) == S && (cosv.size(0) == 1 || cosv.size(0) == B),
              "qsa_headprep: cos/sin must be contiguous fp32 [1 or B, S, 16]");
}

// src [B,S,H,64] or, with split_gate, [B,S,H,128] (q | gate) bf16 contiguous -> {out [B,H,S,64], gate [B,S,H*64] or empty, rstd [B,S,H] or empty}
std::vector<at::Tensor> qsa_headprep_fwd(const at::Tensor& src_in, const c10::optional<at::Tensor>& w, const at::Tensor& cos_in, const at::Tensor& sin_in, double eps,
                                         bool split_gate, bool round_products) {
  const at::Tensor src = aligned16(src_in), cosv = aligned16(cos_in), sinv = aligned16(sin_in);
  TORCH_CHECK(src.is_cuda() && src.scalar_type() == at::kBFloat16 && src.is_contiguous() && src.dim() == 4 && src.size(3) == (split_gate ? 128 : 64),
              "qsa_headprep_fwd: contiguous bf16 [B,S,H,64] (or [B,S,H,128] with the gate) required");
  TORCH_CHECK(!w.has_value() || (w->scalar_type() == at::kFloat && w->is_contiguous() && w->numel() == 64), "qsa_headprep_fwd: norm weight must be fp32 [64]");
  const c10::cuda::CUDAGuard guard(src.device());
  const int B = src.size(0), S = src.size(1), H = src.size(2);
  check_tables(cosv, sinv, B, S);
  auto out = at::empty({B, H, S, 64}, src.options());
  auto gate = at::empty({split_gate ? B : 0, S, H * 64}, src.options());
  auto rstd = at::empty({w.has_value() ? B : 0, S, H}, src.options().dtype(at::kFloat));
  const long long rows = (long long)B * S * H;
  TORCH_CHECK(rows < (1ll << 31), "qsa_headprep_fwd: too many rows");
  launch(qsa_headprep_fwd_kernel, headprep_grid(rows, 5), 32 * HP_WARPS, 0, at::cuda::getCurrentCUDAStream(), 
      (const bf16*)src.data_ptr(), (int)src.size(3), w.has_value() ? w->data_ptr<float>() : nullptr, cosv.data_ptr<float>(), sinv.data_ptr<float>(), (int)cosv.size(0),
      (bf16*)out.data_ptr(), split_gate ? (bf16*)gate.data_ptr() : nullptr, w.has_value() ? rstd.data_ptr<float>() : nullptr, S, H, (unsigned)rows, (float)eps, round_products);
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  count_launch();
  return {out, gate, rstd};
}

// dout [B,H,S,64], dgate [B,S,H*64] (with split_gate) -> {dsrc like src, dw [64] (empty without a norm)}
std::vector<at::Tensor> qsa_headprep_bwd(const at::Tensor& dout_in, const c10::optional<at::Tensor>& dgate_in, const at::Tensor& src_in, const c10::optional<at::Tensor>& w,
                                         const at::Tensor& cos_in, const at::Tensor& sin_in, const at::Tensor& rstd) {
  const at::Tensor dout = aligned16(dout_in), src = aligned16(src_in), cosv = aligned16(cos_in), sinv = aligned16(sin_in);
  c10::optional<at::Tensor> dgate;
  if (dgate_in.has_value()) dgate = aligned16(*dgate_in);
  TORCH_CHECK(dout.is_cuda() && dout.scalar_type() == at::kBFloat16 && dout.is_contiguous() && src.is_contiguous() && src.dim() == 4, "qsa_headprep_bwd: bad inputs");
  const c10::cuda::CUDAGuard guard(src.device());
  const int B = src.size(0), S = src.size(1), H = src.size(2);
  const bool split = src.size(3) == 128;
  TORCH_CHECK(dout.size(0) == B && dout.size(1) == H && dout.size(2) == S && dout.size(3) == 64 && split == dgate.has_value(), "qsa_headprep_bwd: shape mismatch");
  TORCH_CHECK(!split || (dgate->scalar_type() == at::kBFloat16 && dgate->is_contiguous() && dgate->numel() == (long long)B * S * H * 64), "qsa_headprep_bwd: bad gate gradient");
  check_tables(cosv, sinv, B, S);
  auto dsrc = at::empty_like(src);
  auto dw = w.has_value() ? at::zeros({64}, src.options().dtype(at::kFloat)) : at::empty({0}, src.options().dtype(at::kFloat));
  const long long rows = (long long)B * S * H;
  TORCH_CHECK(rows < (1ll << 31), "qsa_headprep_bwd: too many rows");
  launch(qsa_headprep_bwd_kernel, headprep_grid(rows, 4), 32 * HP_WARPS, 0, at::cuda::getCurrentCUDAStream(), 
      (const bf16*)dout.data_ptr(), split ? (const bf16*)dgate->data_ptr() : nullptr, (const bf16*)src.data_ptr(), (int)src.size(3),
      w.has_value() ? w->data_ptr<float>() : nullptr, cosv.data_ptr<float>(), sinv.data_ptr<float>(), (int)cosv.size(0),
      w.has_value() ? rstd.data_ptr<float>() : nullptr, (bf16*)dsrc.data_ptr(), dw.data_ptr<float>(), S, H, (unsigned)rows);
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  count_launch();
  return {dsrc, dw};
}

}  // namespace q38
