// Forward block attention for grids that do not give every SM a CTA of qsa_attn.cu (a short prompt): one CTA per (query head, query block, batch) on warp MMAs.
//
// A CTA keeps its 64 queries as A fragments in registers for its whole loop, passes probabilities from one product to the next in registers, and fetches the next block's
// K and V while the current one is computed: one barrier per block.  Such a grid is bound by the chain of a CTA's blocks, and this chain is shorter than the one through tensor memory
// (scores, barrier, exponentials, barrier, output); beyond one CTA per SM the tensor cores' throughput counts.  Same operations in the same order, same bits.  Times of
// both, here / there: 256 tokens, 16 heads, dense 6.9 / 9.7 us; 640 tokens, 22 heads 14.7 / 17.5; 1024 tokens, 16 heads (128 CTAs there) 20.7 / 24.5; two of 640, 16 heads (160)
// 17.6 / 17.5; 2048 tokens, 16 heads (256) 51 / 47.
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAException.h>

#include "common.cuh"
#include "host.h"
#include "launch.cuh"
#include "mma_tile.cuh"
#include "qsa_blocks.cuh"

namespace q38 {

__global__ void __launch_bounds__(128, 4) qsa_attn_fwd_small_kernel(const bf16* __restrict__ q, const bf16* __restrict__ k, const bf16* __restrict__ v,
                                                                    const unsigned char* __restrict__ sel, bf16* __restrict__ o, float* __restrict__ lse,
                                                                    int S, int nq, int nkv, bool v_tokens, float scale) {
  grid_wait();
  extern __shared__ __align__(16) uint8_t smem_bytes[];
  bf16* KV = reinterpret_cast<bf16*>(smem_bytes);          // two buffers of {K, V}
  unsigned short* list = reinterpret_cast<unsigned short*>(KV + 4 * TILE_ELEMS);
  __shared__ int count;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // late query blocks (longest lists) first, so that the last CTAs to start are short
  const int nb = S / 64, i = nb - 1 - blockIdx.y, h = blockIdx.x, b = blockIdx.z, kvh = h / (nq / nkv);
  const bf16* kbase = k + ((long long)b * nkv + kvh) * S * 64;
  const bf16* vbase = v + (v_tokens ? (long long)b * S * nkv + kvh : ((long long)b * nkv + kvh) * S) * 64;
  const long long v_row = v_tokens ? (long long)nkv * 64 : 64;
  load_tile_async(KV + 2 * TILE_ELEMS, q + (((long long)b * nq + h) * S + (long long)i * 64) * 64, 64, tid);
  cp_async_commit();
  const int n = list_blocks(sel + ((long long)b * nb + i) * nb, 1, 0, i + 1, list, &count);
  auto fetch = [&](int t) {
    const long long row = (long long)list[t] * 64;
    load_tile_async(KV + (t & 1) * 2 * TILE_ELEMS, kbase + row * 64, 64, tid);
    load_tile_async(KV + ((t & 1) * 2 + 1) * TILE_ELEMS, vbase + row * v_row, v_row, tid);
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
  bf16* dst = o + (((long long)b * S + (long long)i * 64 + r0) * nq + h) * 64 + cq;
#pragma unroll
  for (int nt = 0; nt < 8; ++nt)
#pragma unroll
    for (int x = 0; x < 2; ++x)
      *reinterpret_cast<__nv_bfloat162*>(dst + (long long)8 * x * nq * 64 + 8 * nt) = __floats2bfloat162_rn(out[nt][2 * x] / l[x], out[nt][2 * x + 1] / l[x]);
  if ((lane & 3) == 0) {
#pragma unroll
    for (int x = 0; x < 2; ++x) lse[((long long)b * nq + h) * S + (long long)i * 64 + r0 + 8 * x] = m[x] + __logf(l[x]);
  }
}

// Operands as checked by qsa_attn_fwd.
void qsa_attn_fwd_small(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, bool v_tokens, const at::Tensor& sel, const at::Tensor& o, const at::Tensor& lse, double scale) {
  for (const at::Tensor* t : {&q, &k, &v}) TORCH_CHECK((reinterpret_cast<uintptr_t>(t->data_ptr()) & 15) == 0, "qsa_attn_fwd: operands that start on 16 bytes required");
  const int B = q.size(0), nq = q.size(1), S = q.size(2), nb = S / 64;
  static bool cfg = false;
  if (!cfg) { allow_smem(qsa_attn_fwd_small_kernel); cfg = true; }
  launch(qsa_attn_fwd_small_kernel, dim3(nq, nb, B), 128, 4 * TILE_ELEMS * sizeof(bf16) + list_bytes(nb), at::cuda::getCurrentCUDAStream(), (const bf16*)q.data_ptr(),
         (const bf16*)k.data_ptr(), (const bf16*)v.data_ptr(), sel.data_ptr<unsigned char>(), (bf16*)o.data_ptr(), lse.data_ptr<float>(), S, nq, (int)k.size(1), v_tokens, (float)scale);
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  count_launch();
}

}  // namespace q38
