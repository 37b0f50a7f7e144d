// Block-sparse (and dense causal) GQA attention for QSA, forward pass, on 64x64 tiles.
//
// Query block i attends to the key blocks listed in index[b, i, :count[b, i]] (all <= i, own block included); inside the
// own block the mask is causal.  `dense` ignores the lists and uses every block j <= i (the warm-up phase).
//
//   qsa_attn_fwd     grid (nq, nb, B): online-softmax over the selected key blocks; writes o token-major [B,S,nq,64]
//                    and the row log-sum-exp.
// The backward pass is in qsa_attn_bwd.cu; the [B,nb,nb] selection matrix, built on the device, serves both.
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>

#include "common.cuh"
#include "host.h"
#include "mma_tile.cuh"
#include "qsa_blocks.cuh"

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

// The kernel keeps a CTA's queries as A fragments in registers for its whole loop, passes probabilities between products in registers, and
// fetches the next block's two tiles while the current one is computed: one barrier per block and no probability tile in shared memory.
// It is bound by the warp MMA rate and the exponentials between (tensor pipe 46-57 % busy, 35 % with a shared-memory probability tile and
// unbuffered loads).  16384 tokens of four sequences, 22 query heads, eight blocks per query: 242 -> 183 us.
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

// ---- host ----------------------------------------------------------------------------------------------------------------------
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

}  // namespace q38
