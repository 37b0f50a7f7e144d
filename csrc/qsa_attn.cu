// Block-sparse (and dense causal) GQA attention for QSA, forward and backward, on 64x64 tiles.
//
// Query block i attends to the key blocks listed in index[b, i, :count[b, i]] (all <= i, own block included); inside the
// own block the mask is causal.  `dense` ignores the lists and uses every block j <= i (the warm-up phase).
//
//   qsa_attn_fwd     grid (nq, nb, B): online-softmax over the selected key blocks; writes o token-major [B,S,nq,64]
//                    and the row log-sum-exp.
//   qsa_attn_bwd_q   grid (nq, nb, B): D = rowsum(dO o); dQ = sum_j (P (dP - D)) K scale.
//   qsa_attn_bwd_kv  grid (nq, nb, B): for key block j and one query head, loops over the query blocks i >= j that selected j
//                    (a [B,nb,nb] selection matrix built on the device): dV += P^T dO, dK += dS^T Q scale.
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>

#include "common.cuh"
#include "host.h"
#include "mma_tile.cuh"

namespace q38 {

// sel[b, i, j] = 1 iff query block i attends key block j
__global__ void qsa_selection_matrix_kernel(const int* __restrict__ count, const int* __restrict__ index, int kmax, int nb, int dense,
                                            unsigned char* __restrict__ sel) {
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

// The blocks that a row (column) of the selection matrix names, in ascending order, as a list in shared memory; returns its length.
// first <= j < last; stride is the distance of consecutive entries.  Executed by the whole CTA; ends with a barrier.
__device__ __forceinline__ int list_blocks(const unsigned char* __restrict__ sel, long long stride, int first, int last, unsigned short* __restrict__ list, int* __restrict__ count) {
  if (threadIdx.x < 32) {
    int n = 0;
    for (int j0 = first; j0 < last; j0 += 32) {
      const int j = j0 + (int)threadIdx.x;
      const bool on = j < last && sel[j * stride] != 0;
      const unsigned mask = __ballot_sync(0xffffffffu, on);
      if (on) list[n + __popc(mask & ((1u << threadIdx.x) - 1u))] = (unsigned short)j;
      n += __popc(mask);
    }
    if (threadIdx.x == 0) *count = n;
  }
  __syncthreads();
  return *count;
}

// The three attention kernels keep a CTA's fixed operands (queries, or keys and values) as A fragments in registers for its whole
// loop, pass probabilities and score gradients between products in registers, and fetch the next block's two tiles while the
// current one is computed: one barrier per block and no probability tile in shared memory.  They are bound by the warp MMA rate and the
// exponentials between (tensor pipe 46-57 % busy, 35 % with a shared-memory probability tile and unbuffered loads).  16384 tokens of four
// sequences, 22 query heads, eight blocks per query: forward 242 -> 183 us, backward (both kernels) 770 -> 520 us.
__global__ void __launch_bounds__(128, 4) qsa_attn_fwd_kernel(const bf16* __restrict__ q, const bf16* __restrict__ k, const bf16* __restrict__ v,
                                                              const unsigned char* __restrict__ sel, bf16* __restrict__ o, float* __restrict__ lse,
                                                              int S, int nq, int nkv, float scale) {
  extern __shared__ __align__(16) uint8_t smem_bytes[];
  bf16* KV = reinterpret_cast<bf16*>(smem_bytes);          // two buffers of {K, V}
  unsigned short* list = reinterpret_cast<unsigned short*>(KV + 4 * TILE_ELEMS);
  __shared__ int count;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // late query blocks (longest lists) first, so that the last CTAs to start are short
  const int nb = S / 64, i = nb - 1 - blockIdx.y, h = blockIdx.x, b = blockIdx.z, kvh = h / (nq / nkv);
  const bf16* kbase = k + ((long long)b * nkv + kvh) * S * 64;
  const bf16* vbase = v + ((long long)b * nkv + kvh) * S * 64;
  load_tile_async(KV + 2 * TILE_ELEMS, q + (((long long)b * nq + h) * S + (long long)i * 64) * 64, 64, tid);
  cp_async_commit();
  const int n = list_blocks(sel + ((long long)b * nb + i) * nb, 1, 0, i + 1, list, &count);
  auto fetch = [&](int t) {
    const long long off = (long long)list[t] * 4096;
    load_tile_async(KV + (t & 1) * 2 * TILE_ELEMS, kbase + off, 64, tid);
    load_tile_async(KV + ((t & 1) * 2 + 1) * TILE_ELEMS, vbase + off, 64, tid);
  };
  if (n > 0) fetch(0);
  cp_async_commit();
  cp_async_wait<1>();
  __syncthreads();
  uint32_t aq[4][4];
  load_a(KV + 2 * TILE_ELEMS, aq, warp, lane);
  const int r0 = 16 * warp + (lane >> 2), cq = 2 * (lane & 3);
  float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
  float out[8][4];
  zero_acc(out);
  for (int t = 0; t < n; ++t) {
    cp_async_wait<0>();
    __syncthreads();                                       // this block's tiles are visible; the other buffer's readers are done
    if (t + 1 < n) fetch(t + 1);
    cp_async_commit();
    const bf16* Ks = KV + (t & 1) * 2 * TILE_ELEMS;
    float s[8][4];
    zero_acc(s);
    mma_rows<true, 4, 8>(aq, Ks, s, lane);
    const bool diag = list[t] == i;
    float tm[2] = {-INFINITY, -INFINITY}, rs[2] = {0.f, 0.f}, corr[2];
#pragma unroll
    for (int nt = 0; nt < 8; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        s[nt][e] = diag && 8 * nt + cq + (e & 1) > r0 + 8 * (e >> 1) ? -INFINITY : s[nt][e] * scale;
        tm[e >> 1] = fmaxf(tm[e >> 1], s[nt][e]);
      }
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      tm[x] = fmaxf(tm[x], __shfl_xor_sync(0xffffffffu, tm[x], 1));
      tm[x] = fmaxf(tm[x], __shfl_xor_sync(0xffffffffu, tm[x], 2));
      const float mn = fmaxf(m[x], tm[x]);
      corr[x] = __expf(m[x] - mn);
      m[x] = mn;
#pragma unroll
      for (int nt = 0; nt < 8; ++nt) { out[nt][2 * x] *= corr[x]; out[nt][2 * x + 1] *= corr[x]; }
    }
#pragma unroll
    for (int nt = 0; nt < 8; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) { s[nt][e] = __expf(s[nt][e] - m[e >> 1]); rs[e >> 1] += s[nt][e]; }
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      rs[x] += __shfl_xor_sync(0xffffffffu, rs[x], 1);
      rs[x] += __shfl_xor_sync(0xffffffffu, rs[x], 2);
      l[x] = l[x] * corr[x] + rs[x];
    }
    uint32_t ap[4][4];
    pack_a<4>(s, ap);
    mma_rows<false, 4, 8>(ap, Ks + TILE_ELEMS, out, lane);
  }
  cp_async_wait<0>();
#pragma unroll
  for (int nt = 0; nt < 8; ++nt) { out[nt][0] /= l[0]; out[nt][1] /= l[0]; out[nt][2] /= l[1]; out[nt][3] /= l[1]; }
  acc_to_global(out, o + (((long long)b * S + (long long)i * 64) * nq + h) * 64, (long long)nq * 64, warp, lane);
  if ((lane & 3) == 0) {
#pragma unroll
    for (int x = 0; x < 2; ++x) lse[((long long)b * nq + h) * S + (long long)i * 64 + r0 + 8 * x] = m[x] + __logf(l[x]);
  }
}

// dO, o: token-major [B,S,nq,64].  Writes dq [B,nq,S,64] and D [B,nq,S].
__global__ void __launch_bounds__(128, 3) qsa_attn_bwd_q_kernel(const bf16* __restrict__ q, const bf16* __restrict__ k, const bf16* __restrict__ v,
                                                                const bf16* __restrict__ o, const bf16* __restrict__ dout, const float* __restrict__ lse,
                                                                const unsigned char* __restrict__ sel, bf16* __restrict__ dq, float* __restrict__ Dout,
                                                                int S, int nq, int nkv, float scale) {
  extern __shared__ __align__(16) uint8_t smem_bytes[];
  bf16* KV = reinterpret_cast<bf16*>(smem_bytes);          // two buffers of {K, V} and one tile; at the start buffer 1 holds q and dO, the tile holds o
  unsigned short* list = reinterpret_cast<unsigned short*>(KV + 5 * TILE_ELEMS);
  __shared__ int count;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nb = S / 64, i = nb - 1 - blockIdx.y, h = blockIdx.x, b = blockIdx.z, kvh = h / (nq / nkv);
  const bf16* kbase = k + ((long long)b * nkv + kvh) * S * 64;
  const bf16* vbase = v + ((long long)b * nkv + kvh) * S * 64;
  const long long tok_off = (((long long)b * S + (long long)i * 64) * nq + h) * 64, ld_tok = (long long)nq * 64;
  load_tile_async(KV + 2 * TILE_ELEMS, q + (((long long)b * nq + h) * S + (long long)i * 64) * 64, 64, tid);
  load_tile_async(KV + 3 * TILE_ELEMS, dout + tok_off, ld_tok, tid);
  load_tile_async(KV + 4 * TILE_ELEMS, o + tok_off, ld_tok, tid);
  cp_async_commit();
  const int n = list_blocks(sel + ((long long)b * nb + i) * nb, 1, 0, i + 1, list, &count);
  auto fetch = [&](int t) {
    const long long off = (long long)list[t] * 4096;
    load_tile_async(KV + (t & 1) * 2 * TILE_ELEMS, kbase + off, 64, tid);
    load_tile_async(KV + ((t & 1) * 2 + 1) * TILE_ELEMS, vbase + off, 64, tid);
  };
  if (n > 0) fetch(0);
  cp_async_commit();
  cp_async_wait<1>();
  __syncthreads();
  const int r0 = 16 * warp + (lane >> 2), cq = 2 * (lane & 3);
  uint32_t aq[4][4], ado[4][4];
  load_a(KV + 2 * TILE_ELEMS, aq, warp, lane);
  load_a(KV + 3 * TILE_ELEMS, ado, warp, lane);
  float D[2] = {0.f, 0.f}, L2[2];
  {
    uint32_t ao[4][4];
    load_a(KV + 4 * TILE_ELEMS, ao, warp, lane);
#pragma unroll
    for (int ks = 0; ks < 4; ++ks)
#pragma unroll
      for (int e = 0; e < 4; ++e) D[e & 1] += lo_f(ado[ks][e]) * lo_f(ao[ks][e]) + hi_f(ado[ks][e]) * hi_f(ao[ks][e]);
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      D[x] += __shfl_xor_sync(0xffffffffu, D[x], 1);
      D[x] += __shfl_xor_sync(0xffffffffu, D[x], 2);
      const long long idx = ((long long)b * nq + h) * S + (long long)i * 64 + r0 + 8 * x;
      L2[x] = lse[idx] * 1.4426950408889634f;
      if ((lane & 3) == 0) Dout[idx] = D[x];
    }
  }
  const float scale2 = scale * 1.4426950408889634f;
  float dQ[8][4];
  zero_acc(dQ);
  for (int t = 0; t < n; ++t) {
    cp_async_wait<0>();
    __syncthreads();
    if (t + 1 < n) fetch(t + 1);
    cp_async_commit();
    const bf16* Ks = KV + (t & 1) * 2 * TILE_ELEMS;
    const bool diag = list[t] == i;
#pragma unroll
    for (int half = 0; half < 2; ++half) {                 // 32 keys at a time: the two score fragments stay small
      float s[4][4], dp[4][4];
      zero_acc(s);
      zero_acc(dp);
      mma_rows<true, 4, 4>(aq, Ks + 32 * half * LDS, s, lane);
      mma_rows<true, 4, 4>(ado, Ks + TILE_ELEMS + 32 * half * LDS, dp, lane);
#pragma unroll
      for (int nt = 0; nt < 4; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const bool off = diag && 32 * half + 8 * nt + cq + (e & 1) > r0 + 8 * (e >> 1);
          const float p = off ? 0.f : exp2f(s[nt][e] * scale2 - L2[e >> 1]);
          s[nt][e] = p * (dp[nt][e] - D[e >> 1]) * scale;          // dS (already times the score scale)
        }
      uint32_t as[2][4];
      pack_a<2>(s, as);
      mma_rows<false, 2, 8>(as, Ks + 32 * half * LDS, dQ, lane);
    }
  }
  cp_async_wait<0>();
  acc_to_global(dQ, dq + (((long long)b * nq + h) * S + (long long)i * 64) * 64, 64, warp, lane);
}

// One CTA per (key block, query head, batch): the key blocks near the start of the sequence are selected by almost every later query
// block, so the work of a key block is spread over the heads of its group; partial dK / dV are added in fp32.  A warp owns 16 keys and
// computes the scores transposed (K Q^T), which makes P^T and dS^T the A fragments of dV += P^T dO and dK += dS^T Q.
__global__ void __launch_bounds__(128, 3) qsa_attn_bwd_kv_kernel(const bf16* __restrict__ q, const bf16* __restrict__ k, const bf16* __restrict__ v,
                                                                 const bf16* __restrict__ dout, const float* __restrict__ lse, const float* __restrict__ Din,
                                                                 const unsigned char* __restrict__ sel, float* __restrict__ dk, float* __restrict__ dv,
                                                                 int S, int nq, int nkv, float scale) {
  extern __shared__ __align__(16) uint8_t smem_bytes[];
  bf16* QD = reinterpret_cast<bf16*>(smem_bytes);          // two buffers of {Q, dO}
  float* LD = reinterpret_cast<float*>(QD + 4 * TILE_ELEMS);       // two buffers of {lse[64], D[64]}
  unsigned short* list = reinterpret_cast<unsigned short*>(LD + 256);
  __shared__ int count;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nb = S / 64, h = blockIdx.x, j = blockIdx.y, b = blockIdx.z, rep = nq / nkv, kvh = h / rep;     // first key blocks (longest lists) first
  load_tile_async(QD + 2 * TILE_ELEMS, k + (((long long)b * nkv + kvh) * S + (long long)j * 64) * 64, 64, tid);
  load_tile_async(QD + 3 * TILE_ELEMS, v + (((long long)b * nkv + kvh) * S + (long long)j * 64) * 64, 64, tid);
  cp_async_commit();
  const int n = list_blocks(sel + (long long)b * nb * nb + j, nb, j, nb, list, &count);
  const long long ld_tok = (long long)nq * 64, row_base = ((long long)b * nq + h) * S;
  auto fetch = [&](int t) {
    const int i = list[t];
    load_tile_async(QD + (t & 1) * 2 * TILE_ELEMS, q + (row_base + (long long)i * 64) * 64, 64, tid);
    load_tile_async(QD + ((t & 1) * 2 + 1) * TILE_ELEMS, dout + (((long long)b * S + (long long)i * 64) * nq + h) * 64, ld_tok, tid);
    if (tid < 32) {
      const float* src = (tid < 16 ? lse : Din) + row_base + (long long)i * 64 + 4 * (tid & 15);
      const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(LD + (t & 1) * 128 + 4 * tid));
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
    }
  };
  if (n > 0) fetch(0);
  cp_async_commit();
  cp_async_wait<1>();
  __syncthreads();
  uint32_t ak[4][4], av[4][4];
  load_a(QD + 2 * TILE_ELEMS, ak, warp, lane);
  load_a(QD + 3 * TILE_ELEMS, av, warp, lane);
  const int r0 = 16 * warp + (lane >> 2), cq = 2 * (lane & 3);
  float dK[8][4], dV[8][4];
  zero_acc(dK);
  zero_acc(dV);
  for (int t = 0; t < n; ++t) {
    cp_async_wait<0>();
    __syncthreads();
    if (t + 1 < n) fetch(t + 1);
    cp_async_commit();
    const bf16* Qs = QD + (t & 1) * 2 * TILE_ELEMS;
    const float* Ls = LD + (t & 1) * 128;
    const bool diag = list[t] == j;
#pragma unroll
    for (int half = 0; half < 2; ++half) {                 // 32 queries at a time
      float s[4][4], dp[4][4];
      zero_acc(s);
      zero_acc(dp);
      mma_rows<true, 4, 4>(ak, Qs + 32 * half * LDS, s, lane);
      mma_rows<true, 4, 4>(av, Qs + TILE_ELEMS + 32 * half * LDS, dp, lane);
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) {
        const int col = 32 * half + 8 * nt + cq;           // query
        const float2 L = *reinterpret_cast<const float2*>(Ls + col), D = *reinterpret_cast<const float2*>(Ls + 64 + col);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const bool off = diag && col + (e & 1) < r0 + 8 * (e >> 1);
          const float p = off ? 0.f : __expf(s[nt][e] * scale - (e & 1 ? L.y : L.x));
          s[nt][e] = p;
          dp[nt][e] = p * (dp[nt][e] - (e & 1 ? D.y : D.x)) * scale;
        }
      }
      uint32_t ap[2][4];
      pack_a<2>(s, ap);
      mma_rows<false, 2, 8>(ap, Qs + TILE_ELEMS + 32 * half * LDS, dV, lane);        // P^T dO
      pack_a<2>(dp, ap);
      mma_rows<false, 2, 8>(ap, Qs + 32 * half * LDS, dK, lane);                     // dS^T Q
    }
  }
  cp_async_wait<0>();
  if (n == 0) return;
  float* dkp = dk + (((long long)b * nkv + kvh) * S + (long long)j * 64) * 64;
  float* dvp = dv + (((long long)b * nkv + kvh) * S + (long long)j * 64) * 64;
#pragma unroll
  for (int nt = 0; nt < 8; ++nt)
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      const int at = (r0 + 8 * x) * 64 + 8 * nt + cq;
      atomicAdd(reinterpret_cast<float2*>(dkp + at), make_float2(dK[nt][2 * x], dK[nt][2 * x + 1]));
      atomicAdd(reinterpret_cast<float2*>(dvp + at), make_float2(dV[nt][2 * x], dV[nt][2 * x + 1]));
    }
}

// ---- host ----------------------------------------------------------------------------------------------------------------------
static int list_bytes(int nb) { return (2 * nb + 15) / 16 * 16; }

// The kernels' dynamic shared memory grows with the number of blocks in a sequence; the limit covers 58,000 blocks and is set once.
template <typename K> static void allow_smem(K kernel) { C10_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024)); }

static void check_heads(const at::Tensor& t, const char* name) {
  TORCH_CHECK(t.is_cuda() && t.scalar_type() == at::kBFloat16 && t.is_contiguous() && t.dim() == 4 && t.size(3) == 64, name, ": contiguous bf16 [B,H,S,64] required");
}

static at::Tensor selection_matrix(const c10::optional<at::Tensor>& count, const c10::optional<at::Tensor>& index, int B, int nb, const at::TensorOptions& opts,
                                   cudaStream_t stream) {
  auto sel = at::empty({B, nb, nb}, opts.dtype(at::kByte));
  const bool dense = !count.has_value();
  if (!dense) TORCH_CHECK(count->scalar_type() == at::kInt && index->scalar_type() == at::kInt && count->is_contiguous() && index->is_contiguous(), "qsa: int32 block lists required");
  qsa_selection_matrix_kernel<<<dim3(nb, B), 64, 0, stream>>>(dense ? nullptr : count->data_ptr<int>(), dense ? nullptr : index->data_ptr<int>(),
                                                              dense ? 0 : (int)index->size(2), nb, dense ? 1 : 0, sel.data_ptr<unsigned char>());
  count_launch();
  return sel;
}

// Returns {o [B,S,nq,64] bf16, lse [B,nq,S] fp32, sel [B,nb,nb] uint8}
std::vector<at::Tensor> qsa_attn_fwd(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const c10::optional<at::Tensor>& count,
                                     const c10::optional<at::Tensor>& index, double scale) {
  check_heads(q, "qsa_attn_fwd q"); check_heads(k, "qsa_attn_fwd k"); check_heads(v, "qsa_attn_fwd v");
  const c10::cuda::CUDAGuard guard(q.device());
  const int B = q.size(0), nq = q.size(1), S = q.size(2), nkv = k.size(1), nb = S / 64;
  TORCH_CHECK(S % 64 == 0 && nq % nkv == 0, "qsa_attn_fwd: bad shapes");
  auto stream = at::cuda::getCurrentCUDAStream();
  auto sel = selection_matrix(count, index, B, nb, q.options(), stream);
  auto o = at::empty({B, S, nq, 64}, q.options());
  auto lse = at::empty({B, nq, S}, q.options().dtype(at::kFloat));
  const int smem = 4 * TILE_ELEMS * 2 + list_bytes(nb);
  static bool cfg = false;
  if (!cfg) { allow_smem(qsa_attn_fwd_kernel); cfg = true; }
  qsa_attn_fwd_kernel<<<dim3(nq, nb, B), 128, smem, stream>>>((const bf16*)q.data_ptr(), (const bf16*)k.data_ptr(), (const bf16*)v.data_ptr(),
      sel.data_ptr<unsigned char>(), (bf16*)o.data_ptr(), lse.data_ptr<float>(), S, nq, nkv, (float)scale);
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  count_launch();
  return {o, lse, sel};
}

// Returns {dq [B,nq,S,64], dk, dv [B,nkv,S,64]}
std::vector<at::Tensor> qsa_attn_bwd(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& o, const at::Tensor& dout,
                                     const at::Tensor& lse, const at::Tensor& sel, double scale) {
  check_heads(q, "qsa_attn_bwd q");
  TORCH_CHECK(dout.is_contiguous() && dout.scalar_type() == at::kBFloat16 && o.is_contiguous(), "qsa_attn_bwd: contiguous bf16 dO/o [B,S,nq,64] required");
  const c10::cuda::CUDAGuard guard(q.device());
  const int B = q.size(0), nq = q.size(1), S = q.size(2), nkv = k.size(1), nb = S / 64;
  auto dq = at::empty_like(q);
  auto dk32 = at::zeros(k.sizes(), k.options().dtype(at::kFloat)), dv32 = at::zeros(v.sizes(), v.options().dtype(at::kFloat));
  auto D = at::empty({B, nq, S}, q.options().dtype(at::kFloat));
  auto stream = at::cuda::getCurrentCUDAStream();
  const int smem_q = 5 * TILE_ELEMS * 2 + list_bytes(nb), smem_kv = 4 * TILE_ELEMS * 2 + 256 * 4 + list_bytes(nb);
  static bool cfg = false;
  if (!cfg) { allow_smem(qsa_attn_bwd_q_kernel); allow_smem(qsa_attn_bwd_kv_kernel); cfg = true; }
  qsa_attn_bwd_q_kernel<<<dim3(nq, nb, B), 128, smem_q, stream>>>((const bf16*)q.data_ptr(), (const bf16*)k.data_ptr(), (const bf16*)v.data_ptr(),
      (const bf16*)o.data_ptr(), (const bf16*)dout.data_ptr(), lse.data_ptr<float>(), sel.data_ptr<unsigned char>(), (bf16*)dq.data_ptr(), D.data_ptr<float>(),
      S, nq, nkv, (float)scale);
  qsa_attn_bwd_kv_kernel<<<dim3(nq, nb, B), 128, smem_kv, stream>>>((const bf16*)q.data_ptr(), (const bf16*)k.data_ptr(), (const bf16*)v.data_ptr(),
      (const bf16*)dout.data_ptr(), lse.data_ptr<float>(), D.data_ptr<float>(), sel.data_ptr<unsigned char>(), dk32.data_ptr<float>(), dv32.data_ptr<float>(),
      S, nq, nkv, (float)scale);
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  count_launch(2);
  return {dq, dk32.to(at::kBFloat16), dv32.to(at::kBFloat16)};
}

}  // namespace q38
