// QSA block statistics on the tcgen05 tensor cores.
//
//   stats[b, h, t, j] = (max_s x, sum_s exp(x - max)),  x = scale * q_h(t) . k(s),  s in key block j (64 keys), s <= t
//
// the raw material of the distillation target of the indexer (same contract as qsa_main_block_stats in qsa_index.cu, which
// remains the path for sequence lengths that are not a multiple of 128).
//
// One CTA per (128 query rows = two 64-token query blocks of one head, batch).  The query tile is loaded once; key tiles of 128
// keys stream through a TMA ring; each group is one 128 x 128 x 64 product (four K = 16 instructions) into one of two 128-column
// TMEM accumulators, so the row statistics of group g (four epilogue warps, one query row per thread: tcgen05.ld, running max,
// exp2, sum) overlap the MMAs of group g + 1.  The kernel is bound by the exponentials, not by the products: S^2 / 2 of them per
// head, 169 us for 22 heads of four sequences of 4096.  Two CTAs per SM (256 TMEM columns and at most 102 registers each) keep the special-function
// units busy while one of them starts, loads or takes maxima; one CTA with 256-key groups and 8-byte stores took 332 us, this 255.  A quarter
// of the exponentials of full blocks go through a polynomial on the FMA pipe: 233 us, the log-sum-exps 2 % closer to 64 bits (three eighths and
// three-operand maxima: 240).
// Every mbarrier wait is bounded and reports through the error word.
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>

#include "f32x2.cuh"
#include "host.h"
#include "launch.cuh"
#include "ptx.cuh"

namespace q38 {

constexpr int QT_ROWS = 128, QT_KEYS = 128, QT_STAGES = 3, QT_THREADS = 320;     // TMA warp, MMA warp, two epilogue warpgroups

struct QsaTcArgs {
  float2* stats;
  int S, nq, nkv, nb;
  float scale;
  int* err;
};

constexpr float EXP2_C0 = 1.f, EXP2_C1 = 0.693147004f, EXP2_C2 = 0.240222424f, EXP2_C3 = 0.0555073358f, EXP2_C4 = 0.00967151299f, EXP2_C5 = 0.00132647273f;
// 2^x for two x <= 0 on the FMA pipe.  Range reduction as in Cody and Waite, Software Manual for the Elementary Functions: x = i + f with i the nearest
// whole number, found by adding 1.5 * 2^23 (whole numbers end up in the low bits), a polynomial for 2^f on [-1/2, 1/2] (degree 5, fitted with
// Remez' exchange for the smallest largest relative error: 2e-7 in fp32, as ex2.approx), times 2^i.  Below 2^-126 the result is that.  A NaN stays one,
// as in ex2.approx: the clamp keeps it and the product carries it (adding i to the exponent bits would turn it into a number).
__device__ __forceinline__ float max_or_nan(float a, float b) { float y; asm("max.NaN.f32 %0, %1, %2;" : "=f"(y) : "f"(a), "f"(b)); return y; }
__device__ __forceinline__ float2 poly_exp2(float2 x) {
  const uint64_t magic = pair2(12582912.f, 12582912.f), v = pair2(max_or_nan(x.x, -126.f), max_or_nan(x.y, -126.f));
  const uint64_t t = add2(v, magic), f = add2(v, mul2(add2(t, pair2(-12582912.f, -12582912.f)), pair2(-1.f, -1.f)));
  uint64_t p = pair2(EXP2_C5, EXP2_C5);
  p = fma2(p, f, pair2(EXP2_C4, EXP2_C4));
  p = fma2(p, f, pair2(EXP2_C3, EXP2_C3));
  p = fma2(p, f, pair2(EXP2_C2, EXP2_C2));
  p = fma2(p, f, pair2(EXP2_C1, EXP2_C1));
  p = fma2(p, f, pair2(EXP2_C0, EXP2_C0));
  const float2 i = unpair(t);
  return unpair(mul2(p, pair2(__int_as_float((__float_as_int(i.x) << 23) + 0x3f800000), __int_as_float((__float_as_int(i.y) << 23) + 0x3f800000))));
}

__global__ void __launch_bounds__(QT_THREADS, 2) qsa_block_stats_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, QsaTcArgs p) {
  grid_wait();
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = ptx::smem_u32(smem_raw);
  uint8_t* smem = smem_raw + ((1024u - (raw & 1023u)) & 1023u);
  constexpr int Q_BYTES = QT_ROWS * 128, K_BYTES = QT_KEYS * 128;
  uint8_t* q_tile = smem;
  uint8_t* k_ring = smem + Q_BYTES;
  uint64_t* q_full = reinterpret_cast<uint64_t*>(k_ring + QT_STAGES * K_BYTES);
  uint64_t* k_full = q_full + 1;
  uint64_t* k_empty = k_full + QT_STAGES;
  uint64_t* acc_full = k_empty + QT_STAGES;      // [2]
  uint64_t* acc_empty = acc_full + 2;            // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles = p.S / QT_ROWS;
  const int tile = tiles - 1 - blockIdx.x, h = blockIdx.y, b = blockIdx.z;        // the longest key loops first
  const int row0 = tile * QT_ROWS;
  const int groups = (row0 + QT_ROWS + QT_KEYS - 1) / QT_KEYS;
  const int q_batch = b * p.nq + h, k_batch = b * p.nkv + h / (p.nq / p.nkv);

  if (threadIdx.x == 0) {
    ptx::prefetch_tensormap(&tmQ);
    ptx::prefetch_tensormap(&tmK);
    ptx::mbar_init(q_full, 1);
    for (int s = 0; s < QT_STAGES; ++s) { ptx::mbar_init(&k_full[s], 1); ptx::mbar_init(&k_empty[s], 1); }
    for (int a = 0; a < 2; ++a) { ptx::mbar_init(&acc_full[a], 1); ptx::mbar_init(&acc_empty[a], 4); }
    ptx::fence_barrier_init();
  }
  if (warp == 1) { ptx::tmem_alloc(tmem_slot, 2 * QT_KEYS); ptx::tmem_relinquish(); }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    if (ptx::elect_one()) {
      ptx::mbar_expect_tx(q_full, Q_BYTES);
      ptx::tma_load_3d(q_tile, &tmQ, q_full, 0, row0, q_batch);
      for (int g = 0; g < groups; ++g) {
        const int s = g % QT_STAGES, round = g / QT_STAGES;
        if (!ptx::mbar_wait(&k_empty[s], (round & 1) ^ 1, 1u << 20)) { report_error(p.err, ERR_MMA_WAIT); break; }
        ptx::mbar_expect_tx(&k_full[s], K_BYTES);
        ptx::tma_load_3d(k_ring + s * K_BYTES, &tmK, &k_full[s], 0, g * QT_KEYS, k_batch);     // S is a whole number of groups
      }
    }
  } else if (warp == 1) {
    if (ptx::elect_one()) {
      const uint32_t idesc = ptx::umma_idesc_bf16(QT_ROWS, QT_KEYS, false, false);
      bool ok = ptx::mbar_wait(q_full, 0, 1u << 20);
      if (!ok) report_error(p.err, ERR_TMA_WAIT);
      const uint32_t a_base = ptx::smem_u32(q_tile);
      for (int g = 0; g < groups && ok; ++g) {
        const int s = g % QT_STAGES, acc = g & 1;
        if (!ptx::mbar_wait(&acc_empty[acc], ((g >> 1) & 1) ^ 1, 1u << 22)) { report_error(p.err, ERR_EPILOGUE_WAIT); ok = false; break; }
        if (!ptx::mbar_wait(&k_full[s], (g / QT_STAGES) & 1, 1u << 20)) { report_error(p.err, ERR_TMA_WAIT); ok = false; break; }
        ptx::tc_fence_after();
        const uint32_t b_base = ptx::smem_u32(k_ring + s * K_BYTES), d_tmem = tmem_base + acc * QT_KEYS;
#pragma unroll
        for (int j = 0; j < 4; ++j)
          ptx::umma_f16(d_tmem, ptx::umma_smem_desc_sw128(a_base + j * 32, 0, 1024), ptx::umma_smem_desc_sw128(b_base + j * 32, 0, 1024), idesc, j != 0);
        ptx::umma_commit(&k_empty[s]);
        ptx::umma_commit(&acc_full[acc]);
      }
    }
  } else {
    // Two epilogue warpgroups (warps 2-5 and 6-9): group g is read out by warpgroup g & 1, which owns accumulator g & 1, so two
    // groups' exponentials are in flight per SM.  A warp may read the TMEM lanes 32 (warp % 4) .. + 31.
    const int wg = (warp - 2) >> 2, quarter = warp & 3, r = quarter * 32 + lane;
    const int t = row0 + r, own = t >> 6, tin = t & 63;
    float2* out_row = p.stats + ((long long)q_batch * p.S + t) * p.nb;
    const float c = p.scale * 1.4426950408889634f;            // scores to log2 units
    bool ok = true;
    for (int g = wg; g < groups && ok; g += 2) {
      const int acc = g & 1;
      if (!ptx::mbar_wait_warp(&acc_full[acc], (g >> 1) & 1, 1u << 22)) { report_error(p.err, ERR_EPILOGUE_WAIT); ok = false; break; }
      ptx::tc_fence_after();
      const uint32_t t_addr = tmem_base + acc * QT_KEYS + (uint32_t(quarter * 32) << 16);
      float4 pair = make_float4(0.f, 0.f, 0.f, 0.f);         // statistics of the group's two blocks
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int jb = g * 2 + half;
        if (jb > row0 / 64 + (quarter >> 1)) continue;       // a key block after this warp's query block: not causal, never read
        uint32_t lo[32], hi[32];
        ptx::tmem_ld_32x32b_x32(t_addr + half * 64, lo);
        ptx::tmem_ld_32x32b_x32(t_addr + half * 64 + 32, hi);
        ptx::tmem_ld_wait();
        auto v = [&](int e) { return __uint_as_float(e < 32 ? lo[e & 31] : hi[e & 31]); };
        float m, sum = 0.f;
        if (jb < own) {                                      // every key of the block is visible
          float m0 = v(0), m1 = v(1), m2 = v(2), m3 = v(3);
#pragma unroll
          for (int e = 4; e < 64; e += 4) { m0 = fmaxf(m0, v(e)); m1 = fmaxf(m1, v(e + 1)); m2 = fmaxf(m2, v(e + 2)); m3 = fmaxf(m3, v(e + 3)); }
          m = fmaxf(fmaxf(m0, m1), fmaxf(m2, m3));
          const float mc = m * c;
          const uint64_t c2 = pair2(c, c), minus = pair2(-mc, -mc);
          uint64_t s0 = 0, s1 = 0;
#pragma unroll
          for (int e = 0; e < 64; e += 2) {
            float2 x = unpair(fma2(pair2(v(e), v(e + 1)), c2, minus));
            if (e % 8 == 6) x = poly_exp2(x);
            else x = make_float2(exp2_approx(x.x), exp2_approx(x.y));
            if (e % 4) s1 = add2(s1, pair2(x.x, x.y));
            else s0 = add2(s0, pair2(x.x, x.y));
          }
          const float2 s = unpair(add2(s0, s1));
          sum = s.x + s.y;
        } else {                                             // the diagonal block: keys up to the query's own position
          m = -INFINITY;
#pragma unroll
          for (int e = 0; e < 64; ++e) if (e <= tin) m = fmaxf(m, v(e));
          const float mc = m * c;
#pragma unroll
          for (int e = 0; e < 64; ++e) if (e <= tin) sum += exp2_approx(v(e) * c - mc);
        }
        if (half == 0) { pair.x = m * p.scale; pair.y = sum; } else { pair.z = m * p.scale; pair.w = sum; }
      }
      *reinterpret_cast<float4*>(out_row + g * 2) = pair;    // S / 64 is even: 16-byte aligned; entries past the own block are never read
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&acc_empty[acc]);
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 1) ptx::tmem_dealloc(tmem_base, 2 * QT_KEYS);
}

// q [B, nq, S, 64], k [B, nkv, S, 64] bf16 contiguous, S a multiple of 128 -> stats [B, nq, S, S / 64] float2 (as a [.., 2] fp32 tensor).
at::Tensor qsa_block_stats_tc(const at::Tensor& q, const at::Tensor& k, double scale, at::Tensor& err) {
  TORCH_CHECK(q.is_cuda() && q.scalar_type() == at::kBFloat16 && q.is_contiguous() && k.is_contiguous() && k.scalar_type() == at::kBFloat16 && q.dim() == 4 &&
              q.size(3) == 64 && k.size(3) == 64, "qsa_block_stats_tc: contiguous bf16 [B, heads, S, 64] tensors required");
  const int B = (int)q.size(0), nq = (int)q.size(1), S = (int)q.size(2), nkv = (int)k.size(1);
  TORCH_CHECK(S % QT_ROWS == 0 && nq % nkv == 0 && k.size(2) == S && k.size(0) == B, "qsa_block_stats_tc: S must be a multiple of 128 and the shapes consistent");
  const c10::cuda::CUDAGuard guard(q.device());
  const int nb = S / 64;
  auto stats = at::empty({B, nq, S, nb, 2}, q.options().dtype(at::kFloat));
  CUtensorMap tq = make_tmap_box(q.data_ptr(), 2, 64, S, (int64_t)B * nq, 64, (int64_t)S * 64, QT_ROWS, 128);
  CUtensorMap tk = make_tmap_box(k.data_ptr(), 2, 64, S, (int64_t)B * nkv, 64, (int64_t)S * 64, QT_KEYS, 128);
  QsaTcArgs p{};
  p.stats = reinterpret_cast<float2*>(stats.data_ptr<float>()); p.S = S; p.nq = nq; p.nkv = nkv; p.nb = nb; p.scale = (float)scale; p.err = err.data_ptr<int>();
  const int smem = QT_ROWS * 128 + QT_STAGES * QT_KEYS * 128 + 1024 + 256;
  static bool configured = false;
  if (!configured) { C10_CUDA_CHECK(cudaFuncSetAttribute(qsa_block_stats_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)); configured = true; }
  launch(qsa_block_stats_tc_kernel, dim3(S / QT_ROWS, nq, B), QT_THREADS, smem, at::cuda::getCurrentCUDAStream(), tq, tk, p);
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  count_launch();
  return stats;
}

}  // namespace q38
