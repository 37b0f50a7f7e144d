// Backward of the indexer scores on the tcgen05 tensor cores, one pass over the (query block, key block) pairs for all gradients.
//
//     I[t,s] = sum_h w_h(t) relu(q_h(t).k(s)) scale          dI[t,s] = dblse[t, blk(s)] exp(I[t,s] - blse[t, blk(s)])   for s <= t
//     E_h(t) = sum_s dI [S_h > 0] k(s)       dq_h(t) = w_h(t) scale E_h(t)       dw_h(t) = scale q_h(t).E_h(t)
//     dk(s)  = sum_t sum_h dI w_h(t) scale [S_h > 0] q_h(t)
//
// One CTA per (64 queries, batch, z) walks key tiles of 128 keys (z, z + Z, ...).  The 64 queries are two units of 32 queries x 4 heads = 128
// columns; a unit's scores S^T = K Q^T (128 keys x 128 columns) come into TMEM with a key per lane, so that one thread sees all heads of its
// (query, key) pairs: it rounds q.k to bf16, forms the score, one exponential, and hands on
//     dI [S_h > 0]       to shared memory, the A operand (transposed) of E += (..)^T K        (accumulated over the loop, two units), as two bf16:
//                        upper bits and what they leave, so that E, and with it dq and dw, sees dI in sixteen bits
//     dI w_h [S_h > 0]   to TMEM over its own scores, the A operand of dk += (..) Q           (over the two units, then added to memory)
// Columns are ordered (16-query half, head, query), so that each of a lane's two threads overwrites only scores it has read itself.
// E needs no weights: dq and dw are both read off it at the end, dw without a sum over lanes.  Key gradients leave through the TMA unit
// (fp32 adds of 32 x 32 boxes); query gradients are stored, or left in one slice per z that a small kernel adds in ascending order, so they have the same
// bits in every run.
//
// Bound by the instructions per element (16 compute warps; rounding, masks and packing run at half rate; issue slots 43 % busy) and the writes of E's operand (shared memory
// 46 %), not by the products (tensor pipe 26 %).  Two warp-MMA passes with the scores formed twice stood here: four
// sequences of 4096 with four heads 405 -> 120 us, one 149 -> 70, one of 1024 tokens 33 -> 22.  dk goes before the unit's next scores in the queue and E
// after them, so that compute warps wait for two products instead of four, and all sequences' longest query blocks start first.
// With dI in one bf16 it took 98, 59 and 20 us (13 us of the difference are the second operand's stores, 7 its products, 2 the ring of two stages and the single key-gradient
// boxes that make room for it), but the head weights' gradient, which the passes before summed from fp32 dI, then saw eight bits of it.  Against 64 bits (four sequences of 4096,
// 2-norm of the error over that of the gradient): dw 6.9e-4 (9.0e-4 with one bf16, 11.2e-4 in the passes before, which rounded q.k there), dq 3.17e-3 (3.49e-3, 3.49e-3), dk 3.90e-3 in all three.
//
// Roles: a warp for TMA, blse and dblse, an MMA warp, four warps for the key gradients, eight compute warps per unit.  Every mbarrier
// wait is bounded and reports through the error word.
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>

#include "f32x2.cuh"
#include "host.h"
#include "launch.cuh"
#include "ptx.cuh"

namespace q38 {
namespace {

constexpr int IB_HEADS = 4, IB_STAGES = 2, IB_WARPS = 22, IB_THREADS = 32 * IB_WARPS;
constexpr int IB_TILE = 128 * 128;                                      // bytes: 128 rows of 64 bf16
constexpr uint32_t COL_S = 0, COL_E = 256, COL_DK = 384;                // two of each: 128, 64 and 64 columns
constexpr int IB_SMEM = (2 + IB_STAGES + 8 + 1) * IB_TILE + 2 * 256 * 4 + IB_HEADS * 64 * 4 + 256;

struct IndexBwdArgs {
  const __nv_bfloat16* qi;
  const float *wi, *blse, *dblse, *upstream;
  __nv_bfloat16* dqi;                                                   // without slices
  float *dwi, *part, *dw_part;                                          // with slices: [Z,B,NI,S,64], [Z,B,S,NI]
  int B, S, NI, Z;
  float gscale, scale;
  int* err;
};

__global__ void __launch_bounds__(IB_THREADS, 1) qsa_indexer_bwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                                                                        const __grid_constant__ CUtensorMap tmDK, IndexBwdArgs p) {
  grid_wait();
  extern __shared__ __align__(1024) uint8_t smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nb = p.S / 64, i = nb - 1 - blockIdx.y, b = blockIdx.x / p.Z, z = blockIdx.x % p.Z;       // late query blocks (longest loops) of all sequences first
  const int KT = (i + 2) / 2, n = z < KT ? (KT - z + p.Z - 1) / p.Z : 0;
  if (n == 0) return;
  if (ptx::smem_u32(smem) & 1023u) { if (threadIdx.x == 0) report_error(p.err, ERR_BOUNDS); return; }
  uint8_t *q_tile = smem, *k_ring = q_tile + 2 * IB_TILE, *e_tile = k_ring + IB_STAGES * IB_TILE, *dk_out = e_tile + 8 * IB_TILE;            // e_tile: [upper, lower bits][unit][16-query half]
  float* par = reinterpret_cast<float*>(dk_out + IB_TILE);           // [2 buffers][2 key blocks][blse, dblse gscale][64 queries]
  float* w_s = par + 2 * 256;                                            // [head][64 queries], times scale
  uint64_t* bars = reinterpret_cast<uint64_t*>(w_s + IB_HEADS * 64);
  uint64_t *q_full = bars, *k_full = bars + 1, *k_empty = k_full + IB_STAGES, *s_full = k_empty + IB_STAGES, *e_free = s_full + 2, *e_full = e_free + 2,
           *dk_full = e_full + 2, *dk_empty = dk_full + 2, *par_full = dk_empty + 2, *par_empty = par_full + 2, *out_full = par_empty + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(out_full + 1);
  if (threadIdx.x == 0) {
    ptx::prefetch_tensormap(&tmQ);
    ptx::prefetch_tensormap(&tmK);
    ptx::prefetch_tensormap(&tmDK);
    ptx::mbar_init(q_full, 1);
    for (int s = 0; s < IB_STAGES; ++s) { ptx::mbar_init(&k_full[s], 1); ptx::mbar_init(&k_empty[s], 1); }
    for (int s = 0; s < 2; ++s) {
      ptx::mbar_init(&s_full[s], 1);
      ptx::mbar_init(&e_free[s], 1);
      ptx::mbar_init(&e_full[s], 8);
      ptx::mbar_init(&dk_full[s], 1);
      ptx::mbar_init(&dk_empty[s], 4);
      ptx::mbar_init(&par_full[s], 1);
      ptx::mbar_init(&par_empty[s], 16);
    }
    ptx::mbar_init(out_full, 1);
    ptx::fence_barrier_init();
  }
  for (int x = threadIdx.x; x < IB_HEADS * 64; x += IB_THREADS) {
    const int h = x >> 6, t = i * 64 + (x & 63);
    w_s[x] = h < p.NI ? p.wi[((long long)b * p.S + t) * p.NI + h] * p.scale : 0.f;
  }
  if (warp == 1) { ptx::tmem_alloc(tmem_slot, 512); ptx::tmem_relinquish(); }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    // lane 0 keeps the tiles coming, the warp brings blse and dblse of a tile's two key blocks for the 64 queries, fetched a tile ahead
    if (lane == 0) {
      ptx::mbar_expect_tx(q_full, 2 * IB_TILE);
      for (int x = 0; x < 16; ++x) {                                     // unit, 16-query half, head; heads that do not exist read as zeros
        const int h = x & 3, u = x >> 3, half = (x >> 2) & 1;
        ptx::tma_load_3d(q_tile + x * 2048, &tmQ, q_full, 0, i * 64 + 32 * u + 16 * half, h < p.NI ? b * p.NI + h : p.B * p.NI);
      }
    }
    const float gscale = p.upstream != nullptr ? p.gscale * *p.upstream : p.gscale;
    float v[8];
    auto fetch = [&](int m) {
#pragma unroll
      for (int x = 0; x < 8; ++x) {                                      // key block x >> 2, blse or dblse, queries lane and lane + 32
        const int blk = 2 * (z + m * p.Z) + (x >> 2);
        const float* src = (x & 2) ? p.dblse : p.blse;
        v[x] = blk < nb ? src[((long long)b * p.S + i * 64 + lane + 32 * (x & 1)) * nb + blk] * ((x & 2) ? gscale : 1.f) : 0.f;
      }
    };
    fetch(0);
    int m = 0;
    for (; m < n; ++m) {
      const int s = m % IB_STAGES;
      if (!ptx::mbar_wait_warp(&k_empty[s], ((m / IB_STAGES) & 1) ^ 1, 1u << 20)) { report_error(p.err, ERR_MMA_WAIT); break; }
      if (lane == 0) {
        ptx::mbar_expect_tx(&k_full[s], IB_TILE);
        ptx::tma_load_3d(k_ring + s * IB_TILE, &tmK, &k_full[s], 0, (z + m * p.Z) * 128, b);         // rows after the sequence read as zeros
      }
      if (!ptx::mbar_wait_warp(&par_empty[m & 1], ((m >> 1) & 1) ^ 1, 1u << 22)) { report_error(p.err, ERR_EPILOGUE_WAIT); ++m; break; }
#pragma unroll
      for (int x = 0; x < 8; ++x) par[(m & 1) * 256 + (x >> 1) * 64 + lane + 32 * (x & 1)] = v[x];
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&par_full[m & 1]);
      if (m + 1 < n) fetch(m + 1);
    }
    // copies in flight land before this warp, and with it the CTA, ends
    ptx::mbar_wait_warp(q_full, 0, 1u << 20);
    for (int c = m > IB_STAGES ? m - IB_STAGES : 0; c < m; ++c) ptx::mbar_wait_warp(&k_full[c % IB_STAGES], (c / IB_STAGES) & 1, 1u << 20);
  } else if (warp == 1) {
    if (ptx::elect_one()) {
      const uint32_t id_s = ptx::umma_idesc_bf16(128, 128, false, false), id_e = ptx::umma_idesc_bf16(128, 64, true, true), id_k = ptx::umma_idesc_bf16(128, 64, false, true);
      bool ok = ptx::mbar_wait(q_full, 0, 1u << 20);
      if (!ok) report_error(p.err, ERR_TMA_WAIT);
      // scores of unit (m, u); the unit before it in the same place has been read by the dk product issued earlier
      auto scores = [&](int m, int u) {
        if (u == 0 && !ptx::mbar_wait(&k_full[m % IB_STAGES], (m / IB_STAGES) & 1, 1u << 20)) { report_error(p.err, ERR_TMA_WAIT); return false; }
        ptx::tc_fence_after();
        const uint32_t kb = ptx::smem_u32(k_ring + (m % IB_STAGES) * IB_TILE), qb = ptx::smem_u32(q_tile + u * IB_TILE);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          ptx::umma_f16(tmem + COL_S + 128 * u, ptx::umma_smem_desc_sw128(kb + k * 32, 0, 1024), ptx::umma_smem_desc_sw128(qb + k * 32, 0, 1024), id_s, k != 0);
        ptx::umma_commit(&s_full[u]);
        return true;
      };
      ok = ok && scores(0, 0) && scores(0, 1);
      for (int c = 0; c < 2 * n && ok; ++c) {
        const int m = c >> 1, u = c & 1;
        if (!ptx::mbar_wait(&e_full[u], m & 1, 1u << 22)) { report_error(p.err, ERR_EPILOGUE_WAIT); break; }
        if (u == 0 && !ptx::mbar_wait(&dk_empty[m & 1], ((m >> 1) & 1) ^ 1, 1u << 22)) { report_error(p.err, ERR_EPILOGUE_WAIT); break; }
        ptx::tc_fence_after();
        const uint32_t kb = ptx::smem_u32(k_ring + (m % IB_STAGES) * IB_TILE), qb = ptx::smem_u32(q_tile + u * IB_TILE), eb = ptx::smem_u32(e_tile + 2 * u * IB_TILE);
        // dk first: the unit's next scores go where its operand was, and the compute warps wait for those
#pragma unroll
        for (int k = 0; k < 8; ++k)
          ptx::umma_f16_ta(tmem + COL_DK + 64 * (m & 1), tmem + COL_S + 128 * u + 64 * (k >> 2) + 8 * (k & 3), ptx::umma_smem_desc_sw128(qb + k * 2048, IB_TILE, 1024), id_k,
                           (u | k) != 0);
        if (u == 1) ptx::umma_commit(&dk_full[m & 1]);
        if (m + 1 < n) ok = scores(m + 1, u);
        // an even query block reaches the first half of its last tile only: zeros times a later block's keys would be NaN where those are not finite
        const int steps = z + m * p.Z == KT - 1 && (i & 1) == 0 ? 4 : 8;
        for (int low = 0; low < 2; ++low) {
          const uint32_t ab = eb + low * 4 * IB_TILE;
#pragma unroll
          for (int k = 0; k < 8; ++k)
            if (k < steps)
              ptx::umma_f16(tmem + COL_E + 64 * u, ptx::umma_smem_desc_sw128(ab + k * 2048, IB_TILE, 1024), ptx::umma_smem_desc_sw128(kb + k * 2048, IB_TILE, 1024), id_e,
                            (m | low | k) != 0);
        }
        ptx::umma_commit(&e_free[u]);
        if (u == 1) ptx::umma_commit(&k_empty[m % IB_STAGES]);
      }
      ptx::umma_commit(out_full);
    }
  } else if (warp < 6) {
    const int quarter = warp & 3;
    uint8_t* out = dk_out + (warp - 2) * 4096;                           // a box of 32 rows x 32 dims
    for (int m = 0; m < n; ++m) {
      if (!ptx::mbar_wait_warp(&dk_full[m & 1], (m >> 1) & 1, 1u << 22)) { report_error(p.err, ERR_EPILOGUE_WAIT); break; }
      ptx::tc_fence_after();
      uint32_t x[2][32];
      ptx::tmem_ld_32x32b_x32(tmem + COL_DK + 64 * (m & 1) + (uint32_t(32 * quarter) << 16), x[0]);
      ptx::tmem_ld_32x32b_x32(tmem + COL_DK + 64 * (m & 1) + 32 + (uint32_t(32 * quarter) << 16), x[1]);
      ptx::tmem_ld_wait();
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&dk_empty[m & 1]);
      const int row = (z + m * p.Z) * 128 + 32 * quarter;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        if (lane == 0) ptx::bulk_wait_read<0>();                         // the box before has been read
        __syncwarp();
#pragma unroll
        for (int v = 0; v < 8; ++v)
          *reinterpret_cast<uint4*>(out + lane * 128 + ((v ^ (lane & 7)) << 4)) = make_uint4(x[half][4 * v], x[half][4 * v + 1], x[half][4 * v + 2], x[half][4 * v + 3]);
        ptx::fence_proxy_async();
        __syncwarp();
        if (lane == 0) {
          if (row < (i + 1) * 64) ptx::tma_reduce_add_3d(&tmDK, out, 32 * half, row, b);       // later keys get nothing from this block (nor NaN from its queries)
          ptx::bulk_commit();
        }
      }
    }
    if (lane == 0) ptx::bulk_wait<0>();
  } else {
    // half: which 16 queries of the unit; r: this thread's key in the tile
    const int u = (warp - 6) >> 3, half = ((warp - 6) >> 2) & 1, quarter = warp & 3, r = 32 * quarter + lane, q0 = 32 * u + 16 * half;
    const uint32_t own = tmem + COL_S + 128 * u + 64 * half + (uint32_t(32 * quarter) << 16);
    uint8_t* e_row = e_tile + (2 * u + half) * IB_TILE + r * 128;
    const float* w = w_s + q0;
    auto two = [](const float* x, uint64_t& a, uint64_t& c) { const float4 f = *reinterpret_cast<const float4*>(x); a = pair2(f.x, f.y); c = pair2(f.z, f.w); };
    bool ok = true;
    for (int m = 0; m < n; ++m) {
      if (!ptx::mbar_wait_warp(&s_full[u], m & 1, 1u << 22)) { report_error(p.err, ERR_EPILOGUE_WAIT); ok = false; break; }
      ptx::tc_fence_after();
      uint32_t rl[32];                                                   // relu(S) in bf16, two queries each: [head][8]
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        uint32_t s[32];
        ptx::tmem_ld_32x32b_x32(own + 32 * x, s);
        ptx::tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          const __nv_bfloat162 v = __hmax2(__floats2bfloat162_rn(__uint_as_float(s[2 * e]), __uint_as_float(s[2 * e + 1])), __float2bfloat162_rn(0.f));
          rl[16 * x + e] = *reinterpret_cast<const uint32_t*>(&v);
        }
      }
      uint64_t d[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) d[e] = 0;
#pragma unroll
      for (int h = 0; h < IB_HEADS; ++h)
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          uint64_t a, c;
          two(w + 64 * h + 4 * v, a, c);
          d[2 * v] = fma2(a, widen_pair(rl[8 * h + 2 * v]), d[2 * v]);
          d[2 * v + 1] = fma2(c, widen_pair(rl[8 * h + 2 * v + 1]), d[2 * v + 1]);
        }
      if (!ptx::mbar_wait_warp(&par_full[m & 1], (m >> 1) & 1, 1u << 22)) { report_error(p.err, ERR_EPILOGUE_WAIT); ok = false; break; }
      const float* pb = par + (m & 1) * 256 + (quarter >> 1) * 128 + q0;
      const uint64_t minus = pair2(-1.f, -1.f), log2e = pair2(1.4426950408889634f, 1.4426950408889634f);
      uint32_t dI[8];
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        uint64_t bl[2], g[2];
        two(pb + 4 * v, bl[0], bl[1]);
        two(pb + 64 + 4 * v, g[0], g[1]);
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          const int e = 2 * v + x;
          float2 f = unpair(mul2(fma2(bl[x], minus, d[e]), log2e));
          d[e] = mul2(pair2(exp2_approx(f.x), exp2_approx(f.y)), g[x]);
          dI[e] = bf16_pair(unpair(d[e]));
        }
      }
      if (z + m * p.Z == KT - 1) {                                       // the tile that reaches this query block's own keys
        const int reach = (KT - 1) * 128 + r - (i * 64 + q0);            // queries q >= reach see this key
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          float2 f = unpair(d[e]);
          if (2 * e < reach) f.x = 0.f;
          if (2 * e + 1 < reach) f.y = 0.f;
          d[e] = pair2(f.x, f.y);
          dI[e] = bf16_pair(f);
        }
      }
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&par_empty[m & 1]);
      if (!ptx::mbar_wait_warp(&e_free[u], (m & 1) ^ 1, 1u << 22)) { report_error(p.err, ERR_EPILOGUE_WAIT); ok = false; break; }
      // [S > 0] as a bit mask per bf16 (the values are not negative)
      auto mask = [&](int at) { return __hgt2_mask(*reinterpret_cast<const __nv_bfloat162*>(&rl[at]), __float2bfloat162_rn(0.f)); };
      auto store = [&](int low, int h, int c) {
        *reinterpret_cast<uint4*>(e_row + low * 4 * IB_TILE + (((2 * h + c) ^ (r & 7)) << 4)) =
            make_uint4(dI[4 * c] & rl[8 * h + 4 * c], dI[4 * c + 1] & rl[8 * h + 4 * c + 1], dI[4 * c + 2] & rl[8 * h + 4 * c + 2], dI[4 * c + 3] & rl[8 * h + 4 * c + 3]);
      };
#pragma unroll
      for (int h = 0; h < IB_HEADS; ++h) {
        uint32_t ds[8];
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          uint64_t a, c;
          two(w + 64 * h + 4 * v, a, c);
          rl[8 * h + 2 * v] = mask(8 * h + 2 * v);
          rl[8 * h + 2 * v + 1] = mask(8 * h + 2 * v + 1);
          ds[2 * v] = bf16_pair(unpair(mul2(d[2 * v], a))) & rl[8 * h + 2 * v];
          ds[2 * v + 1] = bf16_pair(unpair(mul2(d[2 * v + 1], c))) & rl[8 * h + 2 * v + 1];
        }
        ptx::tmem_st_32x32b_x8(own + 8 * h, ds);
#pragma unroll
        for (int c = 0; c < 2; ++c) store(0, h, c);
      }
#pragma unroll
      for (int e = 0; e < 8; ++e) dI[e] = bf16_pair(unpair(fma2(widen_pair(dI[e]), minus, d[e])));      // what the upper bits leave
#pragma unroll
      for (int h = 0; h < IB_HEADS; ++h)
#pragma unroll
        for (int c = 0; c < 2; ++c) store(1, h, c);
      ptx::tmem_st_wait();
      ptx::tc_fence_before();
      ptx::fence_proxy_async();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&e_full[u]);
    }
    if (ok && !ptx::mbar_wait_warp(out_full, 0, 1u << 22)) { report_error(p.err, ERR_EPILOGUE_WAIT); ok = false; }
    if (ok) {
      // lanes of E are (half, head, query); this warp stores dims 32 half .. + 31, the first of a quarter's two also forms dw
      ptx::tc_fence_after();
      const int h = 2 * (quarter & 1) + (lane >> 4), tin = 32 * u + 16 * (quarter >> 1) + (lane & 15);
      const long long t = (long long)i * 64 + tin, row = ((long long)b * p.NI + h) * p.S + t;
      const float wv = w_s[64 * h + tin];
      float dw = 0.f;
      for (int x = half; x < 2; ++x) {
        __syncwarp();                                                    // the read takes whole warps; with 1 or 3 heads only half of the lanes store
        uint32_t e[32];
        ptx::tmem_ld_32x32b_x32(tmem + COL_E + 64 * u + 32 * x + (uint32_t(32 * quarter) << 16), e);
        ptx::tmem_ld_wait();
        if (half == 0 && h < p.NI) {
          const uint4* q = reinterpret_cast<const uint4*>(p.qi + row * 64 + 32 * x);
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            const uint4 y = q[v];
            const uint32_t ys[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
            for (int k = 0; k < 4; ++k)
              dw += __uint_as_float(ys[k] << 16) * __uint_as_float(e[8 * v + 2 * k]) + __uint_as_float(ys[k] & 0xffff0000u) * __uint_as_float(e[8 * v + 2 * k + 1]);
          }
        }
        const bool store = x == half && h < p.NI;
        if (store && p.part != nullptr) {
          float4* dst = reinterpret_cast<float4*>(p.part + ((long long)z * p.B * p.NI * p.S + row) * 64 + 32 * x);
#pragma unroll
          for (int v = 0; v < 8; ++v)
            dst[v] = make_float4(__uint_as_float(e[4 * v]) * wv, __uint_as_float(e[4 * v + 1]) * wv, __uint_as_float(e[4 * v + 2]) * wv, __uint_as_float(e[4 * v + 3]) * wv);
        } else if (store) {
          uint4* dst = reinterpret_cast<uint4*>(p.dqi + row * 64 + 32 * x);
          auto pk = [&](int k) { return bf16_pair(make_float2(__uint_as_float(e[k]) * wv, __uint_as_float(e[k + 1]) * wv)); };
#pragma unroll
          for (int v = 0; v < 4; ++v) dst[v] = make_uint4(pk(8 * v), pk(8 * v + 2), pk(8 * v + 4), pk(8 * v + 6));
        }
      }
      if (half == 0 && h < p.NI) {
        const long long at = ((long long)b * p.S + t) * p.NI + h;
        if (p.part != nullptr) p.dw_part[(long long)z * p.B * p.S * p.NI + at] = dw * p.scale;
        else p.dwi[at] = dw * p.scale;
      }
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 1) ptx::tmem_dealloc(tmem, 512);
}

// Partial query gradients added up: query block i has as many as key tiles, at most Z.  One thread per eight dims of a row; the
// first of a row's eight threads also takes its head weight.
__global__ void __launch_bounds__(256) qsa_indexer_sum_q_kernel(const float* __restrict__ part, const float* __restrict__ dw_part, __nv_bfloat16* __restrict__ dqi,
                                                                float* __restrict__ dwi, int B, int NI, int S, int Z) {
  grid_wait();
  const long long id = (long long)blockIdx.x * 256 + threadIdx.x, rows = (long long)B * NI * S, row = id >> 3;
  if (row >= rows) return;
  const int s = (int)(row % S), n = min((s / 64 + 2) / 2, Z);
  float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  for (int z = 0; z < n; ++z) {
    const float4* src = reinterpret_cast<const float4*>(part + (z * rows * 8 + id) * 8);
    const float4 a = src[0], c = src[1];
    v[0] += a.x; v[1] += a.y; v[2] += a.z; v[3] += a.w;
    v[4] += c.x; v[5] += c.y; v[6] += c.z; v[7] += c.w;
  }
  reinterpret_cast<uint4*>(dqi)[id] = make_uint4(bf16_pair(make_float2(v[0], v[1])), bf16_pair(make_float2(v[2], v[3])), bf16_pair(make_float2(v[4], v[5])),
                                                 bf16_pair(make_float2(v[6], v[7])));
  if ((id & 7) == 0) {
    const long long bh = row / S, at = ((bh / NI) * S + s) * NI + bh % NI;
    float w = 0.f;
    for (int z = 0; z < n; ++z) w += dw_part[z * rows + at];
    dwi[at] = w;
  }
}

void check_rows(const at::Tensor& t, const char* name) {
  TORCH_CHECK(t.is_cuda() && t.scalar_type() == at::kBFloat16 && t.is_contiguous() && t.size(-1) == 64, name, ": contiguous bf16 [...,64] required");
}

}  // namespace

// Returns {dqi [B,NI,S,64] bf16, dki [B,S,64] bf16, dwi [B,S,NI] fp32}; gscale (one over the token count) and, where given, the one-element upstream gradient multiply dblse.
std::vector<at::Tensor> qsa_indexer_bwd(const at::Tensor& qi, const at::Tensor& ki, const at::Tensor& wi, const at::Tensor& blse, const at::Tensor& dblse,
                                        double gscale, double scale, const c10::optional<at::Tensor>& err, const c10::optional<at::Tensor>& upstream) {
  check_rows(qi, "qsa_indexer_bwd q"); check_rows(ki, "qsa_indexer_bwd k");
  const c10::cuda::CUDAGuard guard(qi.device());
  TORCH_CHECK(qi.dim() == 4 && qi.size(1) <= IB_HEADS && qi.size(2) % 64 == 0, "qsa_indexer_bwd: at most 4 indexer heads and whole blocks of 64 tokens");
  const int B = qi.size(0), NI = qi.size(1), S = qi.size(2), nb = S / 64;
  TORCH_CHECK(ki.numel() == (int64_t)B * S * 64, "qsa_indexer_bwd: k must be [B,S,64]");
  auto rows = [&](const at::Tensor& t, int64_t n) { return t.is_cuda() && t.scalar_type() == at::kFloat && t.is_contiguous() && t.numel() == (int64_t)B * S * n; };
  TORCH_CHECK(rows(wi, NI) && rows(blse, nb) && rows(dblse, nb), "qsa_indexer_bwd: contiguous fp32 w [B,S,heads], blse and dblse [B,S,blocks] required");
  TORCH_CHECK(!upstream.has_value() || (upstream->is_cuda() && upstream->scalar_type() == at::kFloat && upstream->numel() == 1), "qsa_indexer_bwd: upstream gradient of one fp32 element required");
  // One CTA per query block while these fill the SMs; otherwise its key tiles are shared by up to four.
  const int Z = std::min(std::min((nb + 1) / 2, 4), std::max(1, kNumSMs / std::max(1, B * nb)));
  auto f32 = qi.options().dtype(at::kFloat);
  auto part = at::empty({Z > 1 ? Z : 0, B, NI, S, 64}, f32), dw_part = at::empty({Z > 1 ? Z : 0, B, S, NI}, f32);
  auto dqi = at::empty(qi.sizes(), qi.options()), dwi = at::empty(wi.sizes(), wi.options());
  auto dki32 = at::zeros(ki.sizes(), f32);
  IndexBwdArgs p{};
  p.qi = (const __nv_bfloat16*)qi.data_ptr(); p.wi = wi.data_ptr<float>(); p.blse = blse.data_ptr<float>(); p.dblse = dblse.data_ptr<float>();
  p.dqi = (__nv_bfloat16*)dqi.data_ptr(); p.dwi = dwi.data_ptr<float>();
  if (Z > 1) { p.part = part.data_ptr<float>(); p.dw_part = dw_part.data_ptr<float>(); }
  p.upstream = upstream.has_value() ? upstream->data_ptr<float>() : nullptr;
  p.B = B; p.S = S; p.NI = NI; p.Z = Z; p.gscale = (float)gscale; p.scale = (float)scale; p.err = err.has_value() ? err->data_ptr<int>() : nullptr;
  const CUtensorMap tq = make_tmap_box(qi.data_ptr(), 2, 64, S, (int64_t)B * NI, 64, (int64_t)S * 64, 16, 128), tk = make_tmap_box(ki.data_ptr(), 2, 64, S, B, 64, (int64_t)S * 64, 128, 128),
                    tdk = make_tmap_box(dki32.data_ptr(), 4, 64, S, B, 64, (int64_t)S * 64, 32, 128);
  static bool cfg = false;
  if (!cfg) { C10_CUDA_CHECK(cudaFuncSetAttribute(qsa_indexer_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, IB_SMEM)); cfg = true; }
  auto stream = at::cuda::getCurrentCUDAStream();
  launch(qsa_indexer_bwd_kernel, dim3(B * Z, nb), IB_THREADS, IB_SMEM, stream, tq, tk, tdk, p);
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  count_launch();
  if (Z > 1) {
    launch(qsa_indexer_sum_q_kernel, (unsigned)(((long long)B * NI * S * 8 + 255) / 256), 256, 0, stream, part.data_ptr<float>(), dw_part.data_ptr<float>(), (__nv_bfloat16*)dqi.data_ptr(),
        dwi.data_ptr<float>(), B, NI, S, Z);
    C10_CUDA_KERNEL_LAUNCH_CHECK();
    count_launch();
  }
  return {dqi, dki32.to(at::kBFloat16), dwi};
}

}  // namespace q38
