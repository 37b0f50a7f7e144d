// Indexer scores on the tcgen05 tensor cores, reduced to the log-sum-exp of every (query, key block):
//     I[t,s] = sum_h w_h(t) relu(bf16(q_h(t).k(s))) scale          blse[t,b] = log sum_{s in b, s <= t} exp I[t,s]
//
// One CTA per (128 queries, batch, z) walks key blocks z, z + Z, ... of 64 keys.  The scores of all heads, 128 x 64 each, fill one of two 256-column
// halves of TMEM; one thread owns a query row of a block: it rounds q.k to bf16 before the relu (the reference's matmul output dtype), sums the heads, and takes maximum and sum without a
// shuffle.  Blocks alternate between two groups of four warps, so one block's products run under the other's sums.  The order of additions is that of
// the warp-MMA kernel that stood here (heads ascending, a row's exponentials in four interleaved parts), so the results have its bits.
// Four sequences of 4096 with four heads: 100.6 -> 42.8 us; one of 8192: 103.4 -> 42.8.  Bound by the chains of instructions per score
// (rounding, widening, sums) of two row warps per scheduler: issue slots 39 % busy, tensor pipe 17 %.
// Every mbarrier wait is bounded and reports through the error word.
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>

#include "f32x2.cuh"
#include "host.h"
#include "launch.cuh"
#include "ptx.cuh"

namespace q38 {
namespace {

constexpr int IF_HEADS = 4, IF_STAGES = 4, IF_THREADS = 320;             // TMA warp, MMA warp, two groups of four row warps
constexpr int IF_Q_BYTES = 128 * 128, IF_K_BYTES = 64 * 128;
constexpr int IF_SMEM = IF_HEADS * IF_Q_BYTES + IF_STAGES * IF_K_BYTES + 256;

struct IndexFwdArgs {
  const float* wi;
  float* blse;
  int S, NI, Z;
  float scale;
  int* err;
};

__global__ void __launch_bounds__(IF_THREADS, 1) qsa_indexer_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, IndexFwdArgs p) {
  grid_wait();
  extern __shared__ __align__(1024) uint8_t smem[];
  if (ptx::smem_u32(smem) & 1023u) { if (threadIdx.x == 0) report_error(p.err, ERR_BOUNDS); return; }
  uint8_t *q_tile = smem, *ring = smem + IF_HEADS * IF_Q_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(ring + IF_STAGES * IF_K_BYTES);
  uint64_t *q_full = bars, *k_full = bars + 1, *k_empty = k_full + IF_STAGES, *s_full = k_empty + IF_STAGES, *s_empty = s_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(s_empty + 2);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nb = p.S / 64, tile = gridDim.y - 1 - blockIdx.y, b = blockIdx.x / p.Z, z = blockIdx.x % p.Z;      // the longest loops of all sequences first
  const int last = min(2 * tile + 1, nb - 1), n = z <= last ? (last - z) / p.Z + 1 : 0;
  if (n == 0) return;
  if (threadIdx.x == 0) {
    ptx::prefetch_tensormap(&tmQ);
    ptx::prefetch_tensormap(&tmK);
    ptx::mbar_init(q_full, 1);
    for (int s = 0; s < IF_STAGES; ++s) { ptx::mbar_init(&k_full[s], 1); ptx::mbar_init(&k_empty[s], 1); }
    for (int s = 0; s < 2; ++s) { ptx::mbar_init(&s_full[s], 1); ptx::mbar_init(&s_empty[s], 4); }
    ptx::fence_barrier_init();
  }
  if (warp == 1) { ptx::tmem_alloc(tmem_slot, 512); ptx::tmem_relinquish(); }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    if (ptx::elect_one()) {
      ptx::mbar_expect_tx(q_full, p.NI * IF_Q_BYTES);
      for (int h = 0; h < p.NI; ++h) ptx::tma_load_3d(q_tile + h * IF_Q_BYTES, &tmQ, q_full, 0, tile * 128, b * p.NI + h);       // rows after the sequence read as zeros
      int m = 0;
      for (; m < n; ++m) {
        const int s = m % IF_STAGES;
        if (!ptx::mbar_wait(&k_empty[s], ((m / IF_STAGES) & 1) ^ 1, 1u << 20)) { report_error(p.err, ERR_MMA_WAIT); break; }
        ptx::mbar_expect_tx(&k_full[s], IF_K_BYTES);
        ptx::tma_load_3d(ring + s * IF_K_BYTES, &tmK, &k_full[s], 0, (z + m * p.Z) * 64, b);
      }
      // copies in flight land before this thread, and with it the CTA, ends
      ptx::mbar_wait(q_full, 0, 1u << 20);
      for (int c = m > IF_STAGES ? m - IF_STAGES : 0; c < m; ++c) ptx::mbar_wait(&k_full[c % IF_STAGES], (c / IF_STAGES) & 1, 1u << 20);
    }
  } else if (warp == 1) {
    if (ptx::elect_one()) {
      const uint32_t idesc = ptx::umma_idesc_bf16(128, 64, false, false);
      bool ok = ptx::mbar_wait(q_full, 0, 1u << 20);
      if (!ok) report_error(p.err, ERR_TMA_WAIT);
      for (int m = 0; m < n && ok; ++m) {
        const int s = m % IF_STAGES, acc = m & 1;
        if (!ptx::mbar_wait(&s_empty[acc], ((m >> 1) & 1) ^ 1, 1u << 22)) { report_error(p.err, ERR_EPILOGUE_WAIT); break; }
        if (!ptx::mbar_wait(&k_full[s], (m / IF_STAGES) & 1, 1u << 20)) { report_error(p.err, ERR_TMA_WAIT); break; }
        ptx::tc_fence_after();
        const uint32_t kb = ptx::smem_u32(ring + s * IF_K_BYTES);
        for (int h = 0; h < p.NI; ++h) {
          const uint32_t qa = ptx::smem_u32(q_tile + h * IF_Q_BYTES);
#pragma unroll
          for (int k = 0; k < 4; ++k)
            ptx::umma_f16(tmem + 256 * acc + 64 * h, ptx::umma_smem_desc_sw128(qa + k * 32, 0, 1024), ptx::umma_smem_desc_sw128(kb + k * 32, 0, 1024), idesc, k != 0);
        }
        ptx::umma_commit(&k_empty[s]);
        ptx::umma_commit(&s_full[acc]);
      }
    }
  } else {
    const int group = (warp - 2) >> 2, quarter = warp & 3, r = 32 * quarter + lane, own = 2 * tile + (quarter >> 1), tin = r & 63;
    const long long t = (long long)b * p.S + tile * 128 + r;
    uint64_t w[IF_HEADS];
#pragma unroll
    for (int h = 0; h < IF_HEADS; ++h) {
      const float x = h < p.NI && own < nb ? p.wi[t * p.NI + h] * p.scale : 0.f;
      w[h] = pair2(x, x);
    }
    for (int m = group; m < n; m += 2) {
      if (!ptx::mbar_wait_warp(&s_full[group], (m >> 1) & 1, 1u << 22)) { report_error(p.err, ERR_EPILOGUE_WAIT); break; }
      const int jb = z + m * p.Z;
      if (jb <= own && own < nb) {                                       // whole warps; a block after the query's own is not causal
        ptx::tc_fence_after();
        uint64_t score[32];
#pragma unroll
        for (int e = 0; e < 32; ++e) score[e] = 0;
#pragma unroll
        for (int h = 0; h < IF_HEADS; ++h) {
          if (h < p.NI) {
#pragma unroll
            for (int half = 0; half < 2; ++half) {
              uint32_t s[32];
              ptx::tmem_ld_32x32b_x32(tmem + 256 * group + 64 * h + 32 * half + (uint32_t(32 * quarter) << 16), s);
              ptx::tmem_ld_wait();
#pragma unroll
              for (int e = 0; e < 16; ++e) {
                const __nv_bfloat162 v = __hmax2(__floats2bfloat162_rn(__uint_as_float(s[2 * e]), __uint_as_float(s[2 * e + 1])), __float2bfloat162_rn(0.f));
                score[16 * half + e] = fma2(w[h], widen_pair(*reinterpret_cast<const uint32_t*>(&v)), score[16 * half + e]);
              }
            }
          }
        }
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&s_empty[group]);
        if (jb == own) {                                                 // keys after the query's own position
#pragma unroll
          for (int e = 0; e < 32; ++e) {
            float2 f = unpair(score[e]);
            if (2 * e > tin) f.x = -INFINITY;
            if (2 * e + 1 > tin) f.y = -INFINITY;
            score[e] = pair2(f.x, f.y);
          }
        }
        float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
        for (int e = 0; e < 32; ++e) {
          const float2 f = unpair(score[e]);
          mx[0] = fmaxf(mx[0], f.x);
          mx[1] = fmaxf(mx[1], f.y);
        }
        const float mm = fmaxf(mx[0], mx[1]);
        float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int e = 0; e < 32; ++e) {
          const float2 f = unpair(score[e]);
          sum[e & 3] += __expf(f.x - mm);
          sum[e & 3] += __expf(f.y - mm);
        }
        p.blse[t * nb + jb] = mm + __logf((sum[0] + sum[1]) + (sum[2] + sum[3]));
      } else {
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&s_empty[group]);
      }
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 1) ptx::tmem_dealloc(tmem, 512);
}

}  // namespace

// qi [B,NI,S,64], ki [B,S,64], wi [B,S,NI] fp32 -> blse [B,S,nb] fp32 (non-causal entries = -1e9)
at::Tensor qsa_indexer_fwd(const at::Tensor& qi, const at::Tensor& ki, const at::Tensor& wi, double scale, const c10::optional<at::Tensor>& err) {
  for (const at::Tensor* t : {&qi, &ki})
    TORCH_CHECK(t->is_cuda() && t->scalar_type() == at::kBFloat16 && t->is_contiguous() && t->size(-1) == 64, "qsa_indexer_fwd: contiguous bf16 [...,64] required");
  const c10::cuda::CUDAGuard guard(qi.device());
  TORCH_CHECK(qi.dim() == 4 && qi.size(1) >= 1 && qi.size(1) <= IF_HEADS && qi.size(2) % 64 == 0 && wi.scalar_type() == at::kFloat && wi.is_contiguous(), "qsa_indexer_fwd: at most 4 indexer heads");
  const int B = qi.size(0), NI = qi.size(1), S = qi.size(2), nb = S / 64, tiles = (nb + 1) / 2;
  TORCH_CHECK(ki.numel() == (int64_t)B * S * 64 && wi.numel() == (int64_t)B * S * NI, "qsa_indexer_fwd: k must be [B,S,64] and w [B,S,heads]");
  auto blse = at::full({B, S, nb}, -1e9, qi.options().dtype(at::kFloat));
  // key blocks of a query tile are shared by as many CTAs as it takes to have about four per SM, at least eight blocks each, or one per SM, with fewer
  // blocks down to one (1024 tokens 12.3 -> 6.2 us, 256 tokens 8.4 -> 5.9)
  const int rows = std::max(1, B * tiles), Z = std::max({1, std::min((nb + 7) / 8, 4 * kNumSMs / rows), std::min(nb, kNumSMs / rows)});
  const CUtensorMap tq = make_tmap_box(qi.data_ptr(), 2, 64, S, (int64_t)B * NI, 64, (int64_t)S * 64, 128, 128), tk = make_tmap_box(ki.data_ptr(), 2, 64, S, B, 64, (int64_t)S * 64, 64, 128);
  IndexFwdArgs p{};
  p.wi = wi.data_ptr<float>(); p.blse = blse.data_ptr<float>(); p.S = S; p.NI = NI; p.Z = Z; p.scale = (float)scale; p.err = err.has_value() ? err->data_ptr<int>() : nullptr;
  static bool cfg = false;
  if (!cfg) { C10_CUDA_CHECK(cudaFuncSetAttribute(qsa_indexer_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, IF_SMEM)); cfg = true; }
  launch(qsa_indexer_fwd_kernel, dim3(B * Z, tiles), IF_THREADS, IF_SMEM, at::cuda::getCurrentCUDAStream(), tq, tk, p);
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  count_launch();
  return blse;
}

}  // namespace q38
