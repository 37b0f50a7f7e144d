// Block-sparse (and dense causal) GQA attention for QSA, forward pass, on 64x64 tiles.
//
// Query block i attends to the key blocks listed in index[b, i, :count[b, i]] (all <= i, own block included); inside the
// own block the mask is causal.  `dense` ignores the lists and uses every block j <= i (the warm-up phase).
//
// Online softmax over the selected key blocks; writes o token-major [B,S,nq,64] and the row log-sum-exp.
// The backward pass is in qsa_attn_bwd.cu; the [B,nb,nb] selection matrix, built on the device, serves both.
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>

#include "f32x2.cuh"
#include "host.h"
#include "launch.cuh"
#include "ptx.cuh"
#include "qsa_blocks.cuh"

namespace q38 {

void qsa_attn_fwd_small(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, bool v_tokens, const at::Tensor& sel, const at::Tensor& o, const at::Tensor& lse,
                        double scale);   // qsa_attn_small.cu

using bf16 = __nv_bfloat16;

// sel[b, i, j] = 1 iff query block i attends key block j
__global__ void qsa_selection_matrix_kernel(const int* __restrict__ count, const int* __restrict__ index, int kmax, int nb, int dense,
                                            unsigned char* __restrict__ sel) {
  grid_wait();
  const int b = blockIdx.y, i = blockIdx.x;
  unsigned char* row = sel + ((long long)b * nb + i) * nb;
  for (int j = threadIdx.x; j < nb; j += blockDim.x) row[j] = dense ? (j <= i) : 0;
  __syncthreads();
  if (!dense) {
    const int c = count[b * nb + i];
    for (int s = threadIdx.x; s < c; s += blockDim.x) {
      const int j = index[((long long)b * nb + i) * kmax + s];
      if (j >= 0 && j <= i) row[j] = 1;
    }
  }
}

// One CTA per (two heads of a KV group, query block, batch): a tile of 128 rows (64 queries of each head, which attend to the same blocks)
// against one block of 64 keys.  S = Q K^T and O += P V are tcgen05 products with their results in TMEM; one thread owns a row: maximum,
// exponentials and sum without a shuffle, P packed over the scores it came from (the A operand of the second product), O rescaled in place when the row's maximum moves.
// Four CTAs per SM (128 TMEM columns, 48 KB each) cover each other's chains: the products of a tile take 300 of its 1700 cycles, the exponentials 512
// per SM.  Every operation and its order are those of the warp-MMA kernel that stood here (scores, sums of a row in four interleaved parts, four K = 16
// steps per product), so the results have its bits.  16384 tokens of four sequences, 22 heads, eight blocks per query: 182 -> 118 us; dense, 8192 tokens
// of two sequences, 16 heads: 260 -> 143; one of 8192, 28 heads: 122 -> 77.  A grid that leaves SMs idle would pay the longer chain of a tile: it keeps the warp-MMA kernel
// (qsa_attn_small.cu).  Every mbarrier wait is bounded and reports through the error word.
constexpr int AF_THREADS = 192, AF_STAGES = 2;             // TMA warp, MMA warp, four warps of row threads
constexpr int HALF_BYTES = 64 * 128, TILE_BYTES = 2 * HALF_BYTES;
constexpr uint32_t COL_S = 0, COL_O = 64;

struct FwdArgs {
  const unsigned char* sel;
  bf16* o;
  float* lse;
  int S, nq, nkv, v_tokens;
  float scale;
  int* err;
};

__global__ void __launch_bounds__(AF_THREADS, 4) qsa_attn_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                                                                     const __grid_constant__ CUtensorMap tmV, FwdArgs p) {
  grid_wait();
  extern __shared__ __align__(1024) uint8_t smem[];
  if (ptx::smem_u32(smem) & 1023u) { if (threadIdx.x == 0) report_error(p.err, ERR_BOUNDS); return; }
  uint8_t *q_tile = smem, *ring = smem + TILE_BYTES;                     // a ring stage is {K, V}
  uint64_t* bars = reinterpret_cast<uint64_t*>(ring + AF_STAGES * TILE_BYTES);
  uint64_t *q_full = bars, *kv_full = bars + 1, *kv_empty = kv_full + AF_STAGES, *s_full = kv_empty + AF_STAGES, *p_full = s_full + 1, *o_full = p_full + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_full + 1);
  int* count = reinterpret_cast<int*>(tmem_slot + 1);
  unsigned short* list = reinterpret_cast<unsigned short*>(bars + 16);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // late query blocks (longest lists) of all sequences first, so that the last CTAs to start are short
  const int nb = p.S / 64, i = nb - 1 - blockIdx.y, rep = p.nq / p.nkv, pairs = (rep + 1) / 2, b = blockIdx.x / (p.nkv * pairs);
  const int kvh = blockIdx.x / pairs % p.nkv, first = 2 * (blockIdx.x % pairs), h0 = kvh * rep + first;
  const bool both = first + 1 < rep;                                     // an odd head has its tile to itself
  if (threadIdx.x == 0) {
    ptx::prefetch_tensormap(&tmQ);
    ptx::prefetch_tensormap(&tmK);
    ptx::prefetch_tensormap(&tmV);
    ptx::mbar_init(q_full, 1);
    for (int s = 0; s < AF_STAGES; ++s) { ptx::mbar_init(&kv_full[s], 1); ptx::mbar_init(&kv_empty[s], 1); }
    ptx::mbar_init(s_full, 1);
    ptx::mbar_init(p_full, 4);
    ptx::mbar_init(o_full, 1);
    ptx::fence_barrier_init();
    ptx::mbar_expect_tx(q_full, TILE_BYTES);                             // while the list is made
    for (int x = 0; x < 2; ++x) ptx::tma_load_3d(q_tile + x * HALF_BYTES, &tmQ, q_full, 0, (b * p.nq + (x && both ? h0 + 1 : h0)) * p.S + i * 64, 0);
  }
  if (warp == 1) { ptx::tmem_alloc(tmem_slot, 128); ptx::tmem_relinquish(); }
  ptx::tc_fence_before();
  const int n = list_blocks(p.sel + ((long long)b * nb + i) * nb, 1, 0, i + 1, list, count);        // ends with a barrier
  ptx::tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    if (ptx::elect_one()) {
      const int kv_row0 = (b * p.nkv + kvh) * p.S;
      int t = 0;
      for (; t < n; ++t) {
        const int s = t % AF_STAGES;
        if (!ptx::mbar_wait(&kv_empty[s], ((t / AF_STAGES) & 1) ^ 1, 1u << 20)) { report_error(p.err, ERR_MMA_WAIT); break; }
        ptx::mbar_expect_tx(&kv_full[s], TILE_BYTES);
        ptx::tma_load_3d(ring + s * TILE_BYTES, &tmK, &kv_full[s], 0, kv_row0 + list[t] * 64, 0);
        ptx::tma_load_3d(ring + s * TILE_BYTES + HALF_BYTES, &tmV, &kv_full[s], 0, (p.v_tokens ? b * p.S : kv_row0) + list[t] * 64, p.v_tokens ? kvh : 0);
      }
      // copies in flight land before this thread, and with it the CTA, ends
      ptx::mbar_wait(q_full, 0, 1u << 20);
      for (int u = t > AF_STAGES ? t - AF_STAGES : 0; u < t; ++u) ptx::mbar_wait(&kv_full[u % AF_STAGES], (u / AF_STAGES) & 1, 1u << 20);
    }
  } else if (warp == 1) {
    if (ptx::elect_one()) {
      const uint32_t id_s = ptx::umma_idesc_bf16(128, 64, false, false), id_o = ptx::umma_idesc_bf16(128, 64, false, true), qa = ptx::smem_u32(q_tile);
      bool ok = ptx::mbar_wait(q_full, 0, 1u << 20);
      if (!ok) report_error(p.err, ERR_TMA_WAIT);
      for (int t = 0; t < n && ok; ++t) {
        const uint32_t kb = ptx::smem_u32(ring + (t % AF_STAGES) * TILE_BYTES), vb = kb + HALF_BYTES;
        if (!ptx::mbar_wait(&kv_full[t % AF_STAGES], (t / AF_STAGES) & 1, 1u << 20)) { report_error(p.err, ERR_TMA_WAIT); break; }
        ptx::tc_fence_after();
#pragma unroll
        for (int k = 0; k < 4; ++k)                                      // over P of the block before, which the product issued last has read
          ptx::umma_f16(tmem + COL_S, ptx::umma_smem_desc_sw128(qa + k * 32, 0, 1024), ptx::umma_smem_desc_sw128(kb + k * 32, 0, 1024), id_s, k != 0);
        ptx::umma_commit(s_full);
        if (!ptx::mbar_wait(p_full, t & 1, 1u << 22)) { report_error(p.err, ERR_EPILOGUE_WAIT); break; }
        ptx::tc_fence_after();
#pragma unroll
        for (int k = 0; k < 4; ++k)
          ptx::umma_f16_ta(tmem + COL_O, tmem + COL_S + 8 * k, ptx::umma_smem_desc_sw128(vb + k * 2048, HALF_BYTES, 1024), id_o, (t | k) != 0);
        ptx::umma_commit(&kv_empty[t % AF_STAGES]);
        ptx::umma_commit(o_full);
      }
    }
  } else {
    const int quarter = warp & 3, r = 32 * quarter + lane, tin = r & 63, h = h0 + (quarter >> 1);
    const bool active = quarter < 2 || both;                             // whole warps
    const uint32_t ts = tmem + COL_S + (uint32_t(32 * quarter) << 16), to = tmem + COL_O + (uint32_t(32 * quarter) << 16);
    const uint64_t scale = pair2(p.scale, p.scale), log2e = pair2(1.4426950408889634f, 1.4426950408889634f);
    float m = -INFINITY, l = 0.f, corr = 1.f;
    // The scores of one block -> P; `diag`: keys after the query's own position are hidden.
    auto softmax = [&](auto diag) {
      uint32_t s[32];
      auto score = [&](int half, int e) {                                // keys 32 half + 2 e and the next one
        float2 f = unpair(mul2(pair2(__uint_as_float(s[2 * e]), __uint_as_float(s[2 * e + 1])), scale));
        if (diag.value && 32 * half + 2 * e > tin) f.x = -INFINITY;
        if (diag.value && 32 * half + 2 * e + 1 > tin) f.y = -INFINITY;
        return f;
      };
      float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
      for (int half = 1; half >= 0; --half) {                            // the first half stays in registers for the second pass
        ptx::tmem_ld_32x32b_x32(ts + 32 * half, s);
        ptx::tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          const float2 f = score(half, e);
          mx[0] = fmaxf(mx[0], f.x);
          mx[1] = fmaxf(mx[1], f.y);
        }
      }
      const float mn = fmaxf(m, fmaxf(mx[0], mx[1]));
      corr = __expf(m - mn);
      m = mn;
      const uint64_t minus_m = pair2(-m, -m);
      float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        if (half) { ptx::tmem_ld_32x32b_x32(ts + 32, s); ptx::tmem_ld_wait(); }
        uint32_t pk[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          const float2 f = score(half, e);
          float2 x = unpair(mul2(add2(pair2(f.x, f.y), minus_m), log2e));
          x.x = exp2_approx(x.x);
          x.y = exp2_approx(x.y);
          sum[e & 3] += x.x;
          sum[e & 3] += x.y;
          pk[e] = bf16_pair(x);
        }
        ptx::tmem_st_32x32b_x16(ts + 16 * half, pk);
      }
      l = fmaf(l, corr, (sum[0] + sum[1]) + (sum[2] + sum[3]));
    };
    bool ok = true;
    for (int t = 0; t < n; ++t) {
      if (!ptx::mbar_wait_warp(s_full, t & 1, 1u << 22)) { report_error(p.err, ERR_EPILOGUE_WAIT); ok = false; break; }
      if (active) {
        ptx::tc_fence_after();
        if (list[t] == i) softmax(std::true_type());
        else softmax(std::false_type());
      }
      if (t > 0) {
        if (!ptx::mbar_wait_warp(o_full, (t - 1) & 1, 1u << 22)) { report_error(p.err, ERR_EPILOGUE_WAIT); ok = false; break; }
        if (__any_sync(0xffffffffu, corr != 1.f)) {                      // also where corr is NaN
          ptx::tc_fence_after();
          const uint64_t c2 = pair2(corr, corr);
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            uint32_t x[32];
            ptx::tmem_ld_32x32b_x32(to + 32 * half, x);
            ptx::tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 16; ++e) {
              const float2 f = unpair(mul2(pair2(__uint_as_float(x[2 * e]), __uint_as_float(x[2 * e + 1])), c2));
              x[2 * e] = __float_as_uint(f.x);
              x[2 * e + 1] = __float_as_uint(f.y);
            }
            ptx::tmem_st_32x32b_x32(to + 32 * half, x);
          }
        }
      }
      ptx::tmem_st_wait();
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(p_full);
    }
    if (ok && n > 0 && !ptx::mbar_wait_warp(o_full, (n - 1) & 1, 1u << 22)) { report_error(p.err, ERR_EPILOGUE_WAIT); ok = false; }
    if (ok && active) {
      ptx::tc_fence_after();
      bf16* dst = p.o + (((long long)b * p.S + (long long)i * 64 + tin) * p.nq + h) * 64;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t x[32];
        ptx::tmem_ld_32x32b_x32(to + 32 * half, x);
        ptx::tmem_ld_wait();
        auto two = [&](int e) { return bf16_pair(make_float2((n ? __uint_as_float(x[e]) : 0.f) / l, (n ? __uint_as_float(x[e + 1]) : 0.f) / l)); };
#pragma unroll
        for (int v = 0; v < 4; ++v) *reinterpret_cast<uint4*>(dst + 32 * half + 8 * v) = make_uint4(two(8 * v), two(8 * v + 2), two(8 * v + 4), two(8 * v + 6));
      }
      p.lse[((long long)b * p.nq + h) * p.S + (long long)i * 64 + tin] = m + __logf(l);
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 1) ptx::tmem_dealloc(tmem, 128);
}

// ---- host ----------------------------------------------------------------------------------------------------------------------
static at::Tensor selection_matrix(const c10::optional<at::Tensor>& count, const c10::optional<at::Tensor>& index, int B, int nb, const at::TensorOptions& opts,
                                   cudaStream_t stream) {
  auto sel = at::empty({B, nb, nb}, opts.dtype(at::kByte));
  const bool dense = !count.has_value();
  if (!dense) TORCH_CHECK(count->scalar_type() == at::kInt && index->scalar_type() == at::kInt && count->is_contiguous() && index->is_contiguous(), "qsa: int32 block lists required");
  launch(qsa_selection_matrix_kernel, dim3(nb, B), 64, 0, stream, dense ? nullptr : count->data_ptr<int>(), dense ? nullptr : index->data_ptr<int>(),
                                                              dense ? 0 : (int)index->size(2), nb, dense ? 1 : 0, sel.data_ptr<unsigned char>());
  count_launch();
  return sel;
}

// Returns {o [B,S,nq,64] bf16, lse [B,nq,S] fp32, sel [B,nb,nb] uint8}
std::vector<at::Tensor> qsa_attn_fwd(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const c10::optional<at::Tensor>& count,
                                     const c10::optional<at::Tensor>& index, double scale, const c10::optional<at::Tensor>& err) {
  check_heads(q, "qsa_attn_fwd q"); check_heads(k, "qsa_attn_fwd k"); 
  const bool v_tokens = check_values(v, "qsa_attn_fwd v");
  const c10::cuda::CUDAGuard guard(q.device());
  const int B = q.size(0), nq = q.size(1), S = q.size(2), nkv = k.size(1), nb = S / 64;
  TORCH_CHECK(S % 64 == 0 && nkv > 0 && nq % nkv == 0 && k.sizes() == v.sizes() && k.size(0) == B && k.size(2) == S, "qsa_attn_fwd: bad shapes");
  auto stream = at::cuda::getCurrentCUDAStream();
  auto sel = selection_matrix(count, index, B, nb, q.options(), stream);
  auto o = at::empty({B, S, nq, 64}, q.options());
  auto lse = at::empty({B, nq, S}, q.options().dtype(at::kFloat));
  // up to one CTA per SM the shorter chain wins, above it the tensor cores (times of both: qsa_attn_small.cu)
  const int64_t ctas = (int64_t)B * nkv * ((nq / nkv + 1) / 2) * nb;
  if (ctas <= kNumSMs) {
    qsa_attn_fwd_small(q, k, v, v_tokens, sel, o, lse, scale);
    return {o, lse, sel};
  }
  const CUtensorMap tq = make_tmap_box(q.data_ptr(), 2, 64, (int64_t)B * nq * S, 1, 64, 0, 64, 128), tk = make_tmap_box(k.data_ptr(), 2, 64, (int64_t)B * nkv * S, 1, 64, 0, 64, 128),
                    tv = value_map(v, v_tokens);
  FwdArgs p{};
  p.sel = sel.data_ptr<unsigned char>(); p.o = (bf16*)o.data_ptr(); p.lse = lse.data_ptr<float>();
  p.S = S; p.nq = nq; p.nkv = nkv; p.v_tokens = v_tokens; p.scale = (float)scale; p.err = err.has_value() ? err->data_ptr<int>() : nullptr;
  const int smem = (1 + AF_STAGES) * TILE_BYTES + 128 + list_bytes(nb);
  static bool cfg = false;
  if (!cfg) { allow_smem(qsa_attn_fwd_kernel); cfg = true; }
  launch(qsa_attn_fwd_kernel, dim3((unsigned)(ctas / nb), nb), AF_THREADS, smem, stream, tq, tk, tv, p);
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  count_launch();
  return {o, lse, sel};
}

}  // namespace q38
