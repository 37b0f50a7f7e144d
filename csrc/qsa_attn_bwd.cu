// Backward of the block attention on the tcgen05 tensor cores: dQ, then dK and dV, over the query / key block pairs of the selection matrix.
//
// A tile is 128 rows = two halves of 64 query rows against one block of 64 keys.  S = Q K^T and dP = dO V^T are products of 128 x 64 x 64
// into TMEM; one thread owns 32 columns of a row, forms P = exp(S scale - lse) and dS = P (dP - D) scale in fp32 and hands bf16 on:
//
//   qsa_attn_bwd_q   one CTA per (two heads of a KV group, query block, batch).  The heads of a group attend to the same blocks, so the halves
//                    of a tile are heads and share K and V.  dS goes back to TMEM, where it is the A operand of dQ += dS K.
//   qsa_attn_bwd_kv  one CTA per (part, key block, KV head and batch): walks the (query block, head) pairs that attend to the block, two per tile.
//                    P and dS go to shared memory as the two halves of one B operand, dO and Q are the two halves of one A operand:
//                    [dO | Q]^T [P | dS] holds dV^T and dK^T in its diagonal quadrants.  That wastes the other two, but an output of 64 rows
//                    would run at half rate anyway, and it is one instruction stream with one accumulator.
//
// Both run two CTAs per SM (256 TMEM columns each): while one waits for its exponentials the other's products run; in a CTA the scores of the
// next tile are issued as soon as the threads have read the current ones.  dQ is bound by the exponentials (512 cycles of the special-function
// units per tile; a tile takes 920 where the lists are long), dK / dV by shared memory: operand reads, TMA writes and the P / dS
// tile come to 176 KB per tile, 1400 of its 1600 cycles.  Against the warp-MMA kernels in their place (16384 tokens of four sequences, 22 query heads,
// eight blocks per query): dQ 219 -> 122 us, dK / dV 290 -> 200; dense, 8192 tokens of two sequences, 16 heads: 308 -> 121 and 399 -> 213.
// Every mbarrier wait is bounded and reports through the error word.
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>

#include "f32x2.cuh"
#include "host.h"
#include "launch.cuh"
#include "ptx.cuh"
#include "qsa_blocks.cuh"

namespace q38 {
namespace {

constexpr int AB_THREADS = 320;                            // TMA warp, MMA warp, eight warps of row threads
constexpr int HALF_BYTES = 64 * 128, TILE_BYTES = 2 * HALF_BYTES;      // 64 and 128 rows of 64 bf16
constexpr uint32_t COL_S = 0, COL_DP = 64, COL_OUT = 128, COL_DS = 192;
constexpr int Q_STAGES = 3, KV_STAGES = 2;
constexpr float LOG2E = 1.4426950408889634f;

struct BwdArgs {
  const __nv_bfloat16 *o, *dout;
  const float* lse;
  float* D;
  const unsigned char* sel;
  __nv_bfloat16* dq;
  float *dk, *dv;
  int S, nq, nkv, parts, part_tiles, v_tokens;
  float scale;
  int* err;
};

// 32 scores and probability gradients of one row -> packed P and dS.  DIAG: keys after `last` (the query's own position) get zero; `key0` is
// the first of the 32.
template <bool KEEP_P, bool DIAG>
__device__ __forceinline__ void row_grads(const uint32_t (&s)[32], const uint32_t (&dp)[32], float scale2, float neg_l2, float scale, float neg_d, int key0, int last,
                                          uint32_t (&p_out)[16], uint32_t (&ds_out)[16]) {
  const uint64_t sc2 = pair2(scale2, scale2), nl2 = pair2(neg_l2, neg_l2), sc = pair2(scale, scale), nd = pair2(neg_d, neg_d);
#pragma unroll
  for (int e = 0; e < 16; ++e) {
    float2 x = unpair(fma2(pair2(__uint_as_float(s[2 * e]), __uint_as_float(s[2 * e + 1])), sc2, nl2));
    x.x = exp2_approx(x.x);
    x.y = exp2_approx(x.y);
    if (DIAG && key0 + 2 * e > last) x.x = 0.f;
    if (DIAG && key0 + 2 * e + 1 > last) x.y = 0.f;
    if (KEEP_P) p_out[e] = bf16_pair(x);
    const uint64_t g = fma2(pair2(__uint_as_float(dp[2 * e]), __uint_as_float(dp[2 * e + 1])), sc, nd);        // (dP - D) scale
    ds_out[e] = bf16_pair(unpair(mul2(pair2(x.x, x.y), g)));
  }
}

__global__ void __launch_bounds__(AB_THREADS, 2) qsa_attn_bwd_q_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                                                                       const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO, BwdArgs p) {
  grid_wait();
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (ptx::smem_u32(smem_raw) & 1023u)) & 1023u);
  uint8_t *q_tile = smem, *do_tile = smem + TILE_BYTES, *ring = smem + 2 * TILE_BYTES;              // a ring stage is {K, V}
  uint64_t* bars = reinterpret_cast<uint64_t*>(ring + Q_STAGES * TILE_BYTES);
  uint64_t *in_full = bars, *kv_full = bars + 1, *kv_empty = kv_full + Q_STAGES, *s_full = kv_empty + Q_STAGES, *s_empty = s_full + 1, *ds_full = s_empty + 1,
           *ds_empty = ds_full + 2, *out_full = ds_empty + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(out_full + 1);
  int* count = reinterpret_cast<int*>(tmem_slot + 1);
  float* dsum = reinterpret_cast<float*>(bars + 32);                     // [2][128]
  unsigned short* list = reinterpret_cast<unsigned short*>(dsum + 256);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // late query blocks (longest lists) of all sequences first, so that the last CTAs to start are short
  const int nb = p.S / 64, i = nb - 1 - blockIdx.y, rep = p.nq / p.nkv, pairs = (rep + 1) / 2, b = blockIdx.x / (p.nkv * pairs);
  const int kvh = blockIdx.x / pairs % p.nkv, first = 2 * (blockIdx.x % pairs), h0 = kvh * rep + first;
  const bool both = first + 1 < rep;                                     // an odd head has its tile to itself
  if (threadIdx.x == 0) {
    ptx::prefetch_tensormap(&tmQ);
    ptx::prefetch_tensormap(&tmK);
    ptx::prefetch_tensormap(&tmV);
    ptx::prefetch_tensormap(&tmDO);
    ptx::mbar_init(in_full, 1);
    for (int s = 0; s < Q_STAGES; ++s) { ptx::mbar_init(&kv_full[s], 1); ptx::mbar_init(&kv_empty[s], 1); }
    ptx::mbar_init(s_full, 1);
    ptx::mbar_init(s_empty, 8);
    for (int s = 0; s < 2; ++s) { ptx::mbar_init(&ds_full[s], 8); ptx::mbar_init(&ds_empty[s], 1); }
    ptx::mbar_init(out_full, 1);
    ptx::fence_barrier_init();
    ptx::mbar_expect_tx(in_full, 2 * TILE_BYTES);                        // while the list is made
    for (int x = 0; x < 2; ++x) {
      const int h = x && both ? h0 + 1 : h0;
      ptx::tma_load_3d(q_tile + x * HALF_BYTES, &tmQ, in_full, 0, (b * p.nq + h) * p.S + i * 64, 0);
      ptx::tma_load_3d(do_tile + x * HALF_BYTES, &tmDO, in_full, 0, b * p.S + i * 64, h);
    }
  }
  if (warp == 1) { ptx::tmem_alloc(tmem_slot, 256); ptx::tmem_relinquish(); }
  ptx::tc_fence_before();
  const int n = list_blocks(p.sel + ((long long)b * nb + i) * nb, 1, 0, i + 1, list, count);        // ends with a barrier
  ptx::tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    if (ptx::elect_one()) {
      const int kv_row0 = (b * p.nkv + kvh) * p.S;
      int t = 0;
      for (; t < n; ++t) {
        const int s = t % Q_STAGES;
        if (!ptx::mbar_wait(&kv_empty[s], ((t / Q_STAGES) & 1) ^ 1, 1u << 20)) { report_error(p.err, ERR_MMA_WAIT); break; }
        ptx::mbar_expect_tx(&kv_full[s], TILE_BYTES);
        ptx::tma_load_3d(ring + s * TILE_BYTES, &tmK, &kv_full[s], 0, kv_row0 + list[t] * 64, 0);
        ptx::tma_load_3d(ring + s * TILE_BYTES + HALF_BYTES, &tmV, &kv_full[s], 0, (p.v_tokens ? b * p.S : kv_row0) + list[t] * 64, p.v_tokens ? kvh : 0);
      }
      // copies in flight land before this thread, and with it the CTA, ends
      ptx::mbar_wait(in_full, 0, 1u << 20);
      for (int u = t > Q_STAGES ? t - Q_STAGES : 0; u < t; ++u) ptx::mbar_wait(&kv_full[u % Q_STAGES], (u / Q_STAGES) & 1, 1u << 20);
    }
  } else if (warp == 1) {
    if (ptx::elect_one()) {
      const uint32_t id_s = ptx::umma_idesc_bf16(128, 64, false, false), id_q = ptx::umma_idesc_bf16(128, 64, false, true);
      const uint32_t qa = ptx::smem_u32(q_tile), da = ptx::smem_u32(do_tile);
      bool ok = ptx::mbar_wait(in_full, 0, 1u << 20);
      if (!ok) report_error(p.err, ERR_TMA_WAIT);
      for (int t = 0; t <= n && ok; ++t) {
        if (t < n) {
          const uint32_t kb = ptx::smem_u32(ring + (t % Q_STAGES) * TILE_BYTES), vb = kb + HALF_BYTES;
          if (!ptx::mbar_wait(&kv_full[t % Q_STAGES], (t / Q_STAGES) & 1, 1u << 20)) { report_error(p.err, ERR_TMA_WAIT); break; }
          if (!ptx::mbar_wait(s_empty, (t & 1) ^ 1, 1u << 22)) { report_error(p.err, ERR_EPILOGUE_WAIT); break; }
          ptx::tc_fence_after();
#pragma unroll
          for (int k = 0; k < 4; ++k)
            ptx::umma_f16(tmem + COL_S, ptx::umma_smem_desc_sw128(qa + k * 32, 0, 1024), ptx::umma_smem_desc_sw128(kb + k * 32, 0, 1024), id_s, k != 0);
#pragma unroll
          for (int k = 0; k < 4; ++k)
            ptx::umma_f16(tmem + COL_DP, ptx::umma_smem_desc_sw128(da + k * 32, 0, 1024), ptx::umma_smem_desc_sw128(vb + k * 32, 0, 1024), id_s, k != 0);
          ptx::umma_commit(s_full);
        }
        if (t > 0) {
          const int u = t - 1;
          const uint32_t kb = ptx::smem_u32(ring + (u % Q_STAGES) * TILE_BYTES);
          if (!ptx::mbar_wait(&ds_full[u & 1], (u >> 1) & 1, 1u << 22)) { report_error(p.err, ERR_EPILOGUE_WAIT); break; }
          ptx::tc_fence_after();
#pragma unroll
          for (int k = 0; k < 4; ++k)
            ptx::umma_f16_ta(tmem + COL_OUT, tmem + COL_DS + 32 * (u & 1) + 8 * k, ptx::umma_smem_desc_sw128(kb + k * 2048, HALF_BYTES, 1024), id_q, (u | k) != 0);
          ptx::umma_commit(&kv_empty[u % Q_STAGES]);
          ptx::umma_commit(&ds_empty[u & 1]);
        }
      }
      ptx::umma_commit(out_full);
    }
  } else {
    const int quarter = warp & 3, half = (warp - 2) >> 2, r = 32 * quarter + lane, tin = r & 63, h = h0 + (quarter >> 1);
    const bool active = quarter < 2 || both;                             // whole warps
    const uint32_t lanes = uint32_t(32 * quarter) << 16;
    const long long row = ((long long)b * p.nq + h) * p.S + (long long)i * 64 + tin;
    const float scale2 = p.scale * LOG2E;
    float neg_l2 = 0.f, neg_d = 0.f;
    if (active) {
      const long long tok = (((long long)b * p.S + (long long)i * 64 + tin) * p.nq + h) * 64 + 32 * half;
      float part = 0.f;
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        const uint4 x = *reinterpret_cast<const uint4*>(p.dout + tok + 8 * v), y = *reinterpret_cast<const uint4*>(p.o + tok + 8 * v);
        const uint32_t xs[4] = {x.x, x.y, x.z, x.w}, ys[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
        for (int e = 0; e < 4; ++e)
          part += __uint_as_float(xs[e] << 16) * __uint_as_float(ys[e] << 16) + __uint_as_float(xs[e] & 0xffff0000u) * __uint_as_float(ys[e] & 0xffff0000u);
      }
      dsum[128 * half + r] = part;
      neg_l2 = -p.lse[row] * LOG2E;
    }
    asm volatile("bar.sync 1, 256;" ::: "memory");
    if (active) {
      const float d = dsum[r] + dsum[128 + r];
      if (half == 0) p.D[row] = d;
      neg_d = -d * p.scale;
    }
    bool ok = true;
    for (int t = 0; t < n; ++t) {
      if (!ptx::mbar_wait_warp(s_full, t & 1, 1u << 22)) { report_error(p.err, ERR_EPILOGUE_WAIT); ok = false; break; }
      uint32_t ds[16], none[16];
      if (active) {
        uint32_t s[32], dp[32];
        ptx::tc_fence_after();
        ptx::tmem_ld_32x32b_x32(tmem + COL_S + 32 * half + lanes, s);
        ptx::tmem_ld_32x32b_x32(tmem + COL_DP + 32 * half + lanes, dp);
        ptx::tmem_ld_wait();
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(s_empty);
        if (list[t] == i) row_grads<false, true>(s, dp, scale2, neg_l2, p.scale, neg_d, 32 * half, tin, none, ds);
        else row_grads<false, false>(s, dp, scale2, neg_l2, p.scale, neg_d, 0, 0, none, ds);
      } else if (lane == 0) {
        ptx::mbar_arrive(s_empty);
      }
      if (!ptx::mbar_wait_warp(&ds_empty[t & 1], ((t >> 1) & 1) ^ 1, 1u << 22)) { report_error(p.err, ERR_EPILOGUE_WAIT); ok = false; break; }
      if (active) {
        ptx::tc_fence_after();
        ptx::tmem_st_32x32b_x16(tmem + COL_DS + 32 * (t & 1) + 16 * half + lanes, ds);
        ptx::tmem_st_wait();
        ptx::tc_fence_before();
      }
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&ds_full[t & 1]);
    }
    if (ok && !ptx::mbar_wait_warp(out_full, 0, 1u << 22)) { report_error(p.err, ERR_EPILOGUE_WAIT); ok = false; }
    if (ok && active) {
      uint32_t x[32];
      ptx::tc_fence_after();
      ptx::tmem_ld_32x32b_x32(tmem + COL_OUT + 32 * half + lanes, x);
      ptx::tmem_ld_wait();
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        uint4 y = make_uint4(0, 0, 0, 0);
        auto two = [&](int e) { return bf16_pair(make_float2(__uint_as_float(x[8 * v + e]), __uint_as_float(x[8 * v + e + 1]))); };
        if (n > 0) y = make_uint4(two(0), two(2), two(4), two(6));
        *reinterpret_cast<uint4*>(p.dq + row * 64 + 32 * half + 8 * v) = y;
      }
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 1) ptx::tmem_dealloc(tmem, 256);
}

__global__ void __launch_bounds__(AB_THREADS, 2) qsa_attn_bwd_kv_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                                                                        const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO, BwdArgs p) {
  grid_wait();
  extern __shared__ __align__(1024) uint8_t smem[];                     // without slack for the alignment two CTAs fit an SM
  if (ptx::smem_u32(smem) & 1023u) { if (threadIdx.x == 0) report_error(p.err, ERR_BOUNDS); return; }
  uint8_t *kv = smem, *ring = smem + TILE_BYTES, *pds = ring + KV_STAGES * 2 * TILE_BYTES;          // {K, V}; stages of {dO, Q}; {P, dS}
  uint64_t* bars = reinterpret_cast<uint64_t*>(pds + 2 * TILE_BYTES);
  uint64_t *kv_full = bars, *in_full = bars + 1, *in_empty = in_full + KV_STAGES, *s_full = in_empty + KV_STAGES, *s_empty = s_full + 1, *p_full = s_empty + 1,
           *p_empty = p_full + 1, *out_full = p_empty + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(out_full + 1);
  int* count = reinterpret_cast<int*>(tmem_slot + 1);
  unsigned short* list = reinterpret_cast<unsigned short*>(bars + 32);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nb = p.S / 64, j = blockIdx.y, b = blockIdx.z, kvh = blockIdx.x / p.parts, part = blockIdx.x % p.parts, rep = p.nq / p.nkv;      // first key blocks (longest lists) first
  const int items = rep * list_blocks(p.sel + (long long)b * nb * nb + j, nb, j, nb, list, count);
  // The tiles of a key block are split over as many CTAs as give each `part_tiles`, at most `parts`; partial sums are added in fp32.  (Sixteen and
  // eight CTAs: 201 us; 32 and 8: 227, one wave less even; 8 and 16: 248, because CTAs without work still walk the list.  Few key blocks: see the launch.)
  const int tiles = (items + 1) / 2, parts = min(p.parts, (tiles + p.part_tiles - 1) / p.part_tiles);
  if (part >= parts) return;
  const int t0 = (int)((long long)tiles * part / parts), n = (int)((long long)tiles * (part + 1) / parts) - t0;
  if (threadIdx.x == 0) {
    ptx::prefetch_tensormap(&tmQ);
    ptx::prefetch_tensormap(&tmK);
    ptx::prefetch_tensormap(&tmV);
    ptx::prefetch_tensormap(&tmDO);
    ptx::mbar_init(kv_full, 1);
    for (int s = 0; s < KV_STAGES; ++s) { ptx::mbar_init(&in_full[s], 1); ptx::mbar_init(&in_empty[s], 1); }
    ptx::mbar_init(s_full, 1);
    ptx::mbar_init(s_empty, 8);
    ptx::mbar_init(p_full, 8);
    ptx::mbar_init(p_empty, 1);
    ptx::mbar_init(out_full, 1);
    ptx::fence_barrier_init();
  }
  if (warp == 1) { ptx::tmem_alloc(tmem_slot, 256); ptx::tmem_relinquish(); }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    if (ptx::elect_one()) {
      const int kv_row = (b * p.nkv + kvh) * p.S + j * 64;
      ptx::mbar_expect_tx(kv_full, TILE_BYTES);
      ptx::tma_load_3d(kv, &tmK, kv_full, 0, kv_row, 0);
      ptx::tma_load_3d(kv + HALF_BYTES, &tmV, kv_full, 0, p.v_tokens ? b * p.S + j * 64 : kv_row, p.v_tokens ? kvh : 0);
      int t = 0, at = 2 * t0 / rep, head = 2 * t0 % rep;
      for (; t < n; ++t) {
        const int s = t % KV_STAGES;
        if (!ptx::mbar_wait(&in_empty[s], ((t / KV_STAGES) & 1) ^ 1, 1u << 20)) { report_error(p.err, ERR_MMA_WAIT); break; }
        uint8_t* dst = ring + s * 2 * TILE_BYTES;
        ptx::mbar_expect_tx(&in_full[s], 2 * TILE_BYTES);
        for (int x = 0; x < 2; ++x) {                                    // an odd last item is loaded twice and weighs zero the second time
          if (x + t > 0 && 2 * (t0 + t) + x < items && ++head == rep) { head = 0; ++at; }
          const int i = list[at], h = kvh * rep + head;
          ptx::tma_load_3d(dst + x * HALF_BYTES, &tmDO, &in_full[s], 0, b * p.S + i * 64, h);
          ptx::tma_load_3d(dst + TILE_BYTES + x * HALF_BYTES, &tmQ, &in_full[s], 0, (b * p.nq + h) * p.S + i * 64, 0);
        }
      }
      ptx::mbar_wait(kv_full, 0, 1u << 20);
      for (int u = t > KV_STAGES ? t - KV_STAGES : 0; u < t; ++u) ptx::mbar_wait(&in_full[u % KV_STAGES], (u / KV_STAGES) & 1, 1u << 20);
    }
  } else if (warp == 1) {
    if (ptx::elect_one()) {
      const uint32_t id_s = ptx::umma_idesc_bf16(128, 64, false, false), id_o = ptx::umma_idesc_bf16(128, 128, true, true);
      const uint32_t kb = ptx::smem_u32(kv), vb = kb + HALF_BYTES, pb = ptx::smem_u32(pds);
      bool ok = ptx::mbar_wait(kv_full, 0, 1u << 20);
      if (!ok) report_error(p.err, ERR_TMA_WAIT);
      for (int t = 0; t <= n && ok; ++t) {
        if (t < n) {
          const uint32_t da = ptx::smem_u32(ring + (t % KV_STAGES) * 2 * TILE_BYTES), qa = da + TILE_BYTES;
          if (!ptx::mbar_wait(&in_full[t % KV_STAGES], (t / KV_STAGES) & 1, 1u << 20)) { report_error(p.err, ERR_TMA_WAIT); break; }
          if (!ptx::mbar_wait(s_empty, (t & 1) ^ 1, 1u << 22)) { report_error(p.err, ERR_EPILOGUE_WAIT); break; }
          ptx::tc_fence_after();
#pragma unroll
          for (int k = 0; k < 4; ++k)
            ptx::umma_f16(tmem + COL_S, ptx::umma_smem_desc_sw128(qa + k * 32, 0, 1024), ptx::umma_smem_desc_sw128(kb + k * 32, 0, 1024), id_s, k != 0);
#pragma unroll
          for (int k = 0; k < 4; ++k)
            ptx::umma_f16(tmem + COL_DP, ptx::umma_smem_desc_sw128(da + k * 32, 0, 1024), ptx::umma_smem_desc_sw128(vb + k * 32, 0, 1024), id_s, k != 0);
          ptx::umma_commit(s_full);
        }
        if (t > 0) {
          const int u = t - 1;
          const uint32_t da = ptx::smem_u32(ring + (u % KV_STAGES) * 2 * TILE_BYTES);
          if (!ptx::mbar_wait(p_full, u & 1, 1u << 22)) { report_error(p.err, ERR_EPILOGUE_WAIT); break; }
          ptx::tc_fence_after();
#pragma unroll
          for (int k = 0; k < 8; ++k)
            ptx::umma_f16(tmem + COL_OUT, ptx::umma_smem_desc_sw128(da + k * 2048, TILE_BYTES, 1024), ptx::umma_smem_desc_sw128(pb + k * 2048, TILE_BYTES, 1024), id_o,
                          (u | k) != 0);
          ptx::umma_commit(&in_empty[u % KV_STAGES]);
          ptx::umma_commit(p_empty);
        }
      }
      ptx::umma_commit(out_full);
    }
  } else {
    const int quarter = warp & 3, half = (warp - 2) >> 2, r = 32 * quarter + lane, tin = r & 63;
    const uint32_t lanes = uint32_t(32 * quarter) << 16;
    const float scale2 = p.scale * LOG2E;
    uint8_t* dst = pds + r * 128;
    // this warp's (query block, head) in the current tile, and its rows' two scalars, fetched a tile ahead
    int item = 2 * t0 + (quarter >> 1), at = item / rep, head = item % rep, own = 0;
    const long long base = ((long long)b * p.nq + kvh * rep) * p.S + tin;
    float neg_l2 = 0.f, neg_d = 0.f;
    auto fetch = [&]() {
      if (item >= items) return;
      own = list[at];
      const long long row = base + (long long)head * p.S + own * 64;
      neg_l2 = -p.lse[row] * LOG2E;
      neg_d = -p.D[row] * p.scale;
    };
    auto advance = [&]() {
      item += 2;
      for (head += 2; head >= rep; head -= rep) ++at;
      fetch();
    };
    fetch();
    bool ok = true;
    for (int t = 0; t < n; ++t) {
      if (!ptx::mbar_wait_warp(s_full, t & 1, 1u << 22)) { report_error(p.err, ERR_EPILOGUE_WAIT); ok = false; break; }
      uint32_t s[32], dp[32], pr[16], ds[16];
      ptx::tc_fence_after();
      ptx::tmem_ld_32x32b_x32(tmem + COL_S + 32 * half + lanes, s);
      ptx::tmem_ld_32x32b_x32(tmem + COL_DP + 32 * half + lanes, dp);
      ptx::tmem_ld_wait();
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(s_empty);
      if (own == j) row_grads<true, true>(s, dp, scale2, neg_l2, p.scale, neg_d, 32 * half, tin, pr, ds);
      else row_grads<true, false>(s, dp, scale2, neg_l2, p.scale, neg_d, 0, 0, pr, ds);
      if (item >= items) {
#pragma unroll
        for (int e = 0; e < 16; ++e) pr[e] = ds[e] = 0;
      }
      advance();
      if (!ptx::mbar_wait_warp(p_empty, (t & 1) ^ 1, 1u << 22)) { report_error(p.err, ERR_EPILOGUE_WAIT); ok = false; break; }
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        const int chunk = ((4 * half + v) ^ (r & 7)) << 4;               // 128-byte swizzle
        *reinterpret_cast<uint4*>(dst + chunk) = make_uint4(pr[4 * v], pr[4 * v + 1], pr[4 * v + 2], pr[4 * v + 3]);
        *reinterpret_cast<uint4*>(dst + TILE_BYTES + chunk) = make_uint4(ds[4 * v], ds[4 * v + 1], ds[4 * v + 2], ds[4 * v + 3]);
      }
      ptx::fence_proxy_async();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(p_full);
    }
    if (ok && !ptx::mbar_wait_warp(out_full, 0, 1u << 22)) { report_error(p.err, ERR_EPILOGUE_WAIT); ok = false; }
    if (ok && n > 0) {
      // lanes are dims, columns are keys: dV^T in lanes 0-63 and columns 0-63, dK^T in lanes 64-127 and columns 64-127
      uint32_t x[32];
      ptx::tc_fence_after();
      ptx::tmem_ld_32x32b_x32(tmem + COL_OUT + (quarter < 2 ? 0 : 64) + 32 * half + lanes, x);
      ptx::tmem_ld_wait();
      const int key = j * 64 + 32 * half;
      const bool tokens = quarter < 2 && p.v_tokens;                     // dV is laid out like V
      const long long step = tokens ? p.nkv * 64 : 64;
      float* out = (quarter < 2 ? p.dv : p.dk) + (tokens ? (((long long)b * p.S + key) * p.nkv + kvh) * 64 : (((long long)b * p.nkv + kvh) * p.S + key) * 64) + tin;
#pragma unroll
      for (int e = 0; e < 32; ++e) atomicAdd(out + e * step, __uint_as_float(x[e]));
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 1) ptx::tmem_dealloc(tmem, 256);
}

}  // namespace

// Returns {dq [B,nq,S,64], dk, dv [B,nkv,S,64]}
std::vector<at::Tensor> qsa_attn_bwd(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& o, const at::Tensor& dout,
                                     const at::Tensor& lse, const at::Tensor& sel, double scale, const c10::optional<at::Tensor>& err) {
  check_heads(q, "qsa_attn_bwd q"); check_heads(k, "qsa_attn_bwd k"); 
  const bool v_tokens = check_values(v, "qsa_attn_bwd v");
  const c10::cuda::CUDAGuard guard(q.device());
  const int B = q.size(0), nq = q.size(1), S = q.size(2), nkv = k.size(1), nb = S / 64;
  TORCH_CHECK(S % 64 == 0 && nkv > 0 && nq % nkv == 0 && k.sizes() == v.sizes() && k.size(0) == B && k.size(2) == S, "qsa_attn_bwd: bad shapes");
  for (const at::Tensor* t : {&dout, &o})
    TORCH_CHECK(t->is_cuda() && t->is_contiguous() && t->scalar_type() == at::kBFloat16 && t->numel() == q.numel() && (reinterpret_cast<uintptr_t>(t->data_ptr()) & 15) == 0,
                "qsa_attn_bwd: contiguous bf16 dO/o [B,S,nq,64] required");
  TORCH_CHECK(lse.scalar_type() == at::kFloat && lse.is_contiguous() && lse.numel() == (int64_t)B * nq * S && sel.scalar_type() == at::kByte && sel.is_contiguous() &&
              sel.numel() == (int64_t)B * nb * nb, "qsa_attn_bwd: lse [B,nq,S] and sel [B,nb,nb] of the forward required");
  auto dq = at::empty_like(q);
  auto dkv32 = at::zeros({2, k.numel()}, k.options().dtype(at::kFloat));
  auto D = at::empty({B, nq, S}, q.options().dtype(at::kFloat));
  auto stream = at::cuda::getCurrentCUDAStream();
  const CUtensorMap tq = make_tmap_box(q.data_ptr(), 2, 64, (int64_t)B * nq * S, 1, 64, 0, 64, 128), tk = make_tmap_box(k.data_ptr(), 2, 64, (int64_t)B * nkv * S, 1, 64, 0, 64, 128),
                    tv = value_map(v, v_tokens), tdo = make_tmap_box(dout.data_ptr(), 2, 64, (int64_t)B * S, nq, nq * 64, 64, 64, 128);
  const int rep = nq / nkv;
  BwdArgs p{};
  p.o = (const __nv_bfloat16*)o.data_ptr(); p.dout = (const __nv_bfloat16*)dout.data_ptr(); p.lse = lse.data_ptr<float>(); p.D = D.data_ptr<float>();
  p.sel = sel.data_ptr<unsigned char>(); p.dq = (__nv_bfloat16*)dq.data_ptr(); p.dk = dkv32.data_ptr<float>(); p.dv = p.dk + k.numel(); p.v_tokens = v_tokens;
  p.S = S; p.nq = nq; p.nkv = nkv; p.scale = (float)scale; p.err = err.has_value() ? err->data_ptr<int>() : nullptr;
  // Sixteen tiles a part where that makes about two CTAs per SM (as many as are resident); with fewer key blocks a part gets fewer tiles, down to one: 256 tokens, 16 heads
  // 32.7 -> 15.5 us for both kernels (19.5 before tensor memory), 1024 tokens, 22 heads 37.5 -> 33.2.  One or four CTAs per SM: 34.2 and 31.8 against 28.6 for 1024 tokens, 16 heads.
  const int most = (nb * rep + 1) / 2;                                   // tiles of the first key block when every block attends to it
  p.part_tiles = (int)std::max<int64_t>(1, std::min<int64_t>(16, ((int64_t)B * nkv * nb * most + 2 * kNumSMs - 1) / (2 * kNumSMs)));
  p.parts = p.part_tiles == 16 ? std::min(8, (most + 15) / 16) : (most + p.part_tiles - 1) / p.part_tiles;
  const int smem_q = (2 + Q_STAGES) * TILE_BYTES + 1024 + 256 + 1024 + list_bytes(nb), smem_kv = (1 + 2 * KV_STAGES + 2) * TILE_BYTES + 256 + list_bytes(nb);
  static bool cfg = false;
  if (!cfg) { allow_smem(qsa_attn_bwd_q_kernel); allow_smem(qsa_attn_bwd_kv_kernel); cfg = true; }
  launch(qsa_attn_bwd_q_kernel, dim3(B * nkv * ((rep + 1) / 2), nb), AB_THREADS, smem_q, stream, tq, tk, tv, tdo, p);
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  launch(qsa_attn_bwd_kv_kernel, dim3(p.parts * nkv, nb, B), AB_THREADS, smem_kv, stream, tq, tk, tv, tdo, p);
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  count_launch(2);
  const auto dkv = dkv32.to(at::kBFloat16);
  const auto dv = dkv.select(0, 1);
  return {dq, dkv.select(0, 0).view(k.sizes()), v_tokens ? dv.view({B, S, nkv, 64}).transpose(1, 2) : dv.view(v.sizes())};
}

}  // namespace q38
