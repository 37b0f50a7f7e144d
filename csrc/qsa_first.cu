// Indexer block log-probabilities for block selection only (evaluation, and training steps that take no KL term): selection
// looks at the first query of every 64-token block, so only those S/64 queries are scored:
//     I[s]      = sum_h w_h relu(bf16(q_h . k_s)) * scale          for the keys s <= 64 i  (causal for the query at 64 i)
//     lp_blk[j] = logsumexp_{s in block j} I[s] - logsumexp_s I[s]  for j <= i, a large negative number for j > i
// The same rounding points as the full indexer kernel (qsa_index_fwd.cu) and the PyTorch specification: q.k is rounded to bf16 before
// the relu.  (Reference: modeling_qwen3_8_moe.py:1126-1131 scores these queries with eager matmul / einsum / log_softmax /
// logsumexp calls.)
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>

#include "common.cuh"
#include "host.h"
#include "launch.cuh"

namespace q38 {

// Two kernels: scores of 256 keys against one, two or four queries per CTA, a key per thread (qsa_first_scores), then one CTA per query for the sums and the blocks.  With all keys
// of a query in one CTA the last of them had 16 rows of 128 bytes per thread to fetch one after the other: 59 us for one sequence of 8192 tokens, now
// 28 (31 with two queries per CTA, 38 with one).  Short sequences take fewer queries per CTA, which come one after the other: 256 tokens 5.7, 7.1 and 9.5 us with one, two
// and four (4.8 in one kernel), 1024 tokens 6.4, 7.9 and 10.3 (9.5), two sequences of 2048 12.2, 10.8 and 11.3.  The sum over all keys keeps the order that 128 threads give it.
constexpr int QF_THREADS = 512, QF_SUM = 128, QF_HEADS_MAX = 4, QF_KEYS = 256;
constexpr float QF_MASKED = -1e9f;

template <int QF_QUERIES>
__global__ void __launch_bounds__(QF_KEYS) qsa_first_scores_kernel(const __nv_bfloat16* __restrict__ q_first, const __nv_bfloat16* __restrict__ ki,
                                                                   const float* __restrict__ w_first, float* __restrict__ scores, int S, int NI, float scale) {
  grid_wait();
  const int nb = S / 64, i0 = (gridDim.y - 1 - blockIdx.y) * QF_QUERIES, b = blockIdx.z, n = min(QF_QUERIES, nb - i0), tid = threadIdx.x, s = blockIdx.x * QF_KEYS + tid;
  if ((int)blockIdx.x * QF_KEYS > 64 * (i0 + n - 1)) return;     // no causal key here
  __shared__ __align__(16) float qs[QF_QUERIES][QF_HEADS_MAX * 64];
  __shared__ float ws[QF_QUERIES][QF_HEADS_MAX];
  for (int e = tid; e < n * NI * 64; e += QF_KEYS) {
    const int x = e / (NI * 64), r = e % (NI * 64);
    qs[x][r] = __bfloat162float(q_first[(((long long)b * NI + (r >> 6)) * nb + i0 + x) * 64 + (r & 63)]);
  }
  if (tid < n * NI) ws[tid / NI][tid % NI] = w_first[((long long)b * nb + i0 + tid / NI) * NI + tid % NI];
  __syncthreads();
  if (s > 64 * (i0 + n - 1)) return;
  const uint4* krow = reinterpret_cast<const uint4*>(ki + ((long long)b * S + s) * 64);
  uint4 key[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) key[c] = krow[c];
  for (int x = 0; x < n; ++x) {
    if (s > 64 * (i0 + x)) continue;
    float dot[QF_HEADS_MAX] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const __nv_bfloat162* h2 = reinterpret_cast<const __nv_bfloat162*>(&key[c]);
      float kv[8];
#pragma unroll
      for (int e = 0; e < 4; ++e) { kv[2 * e] = __low2float(h2[e]); kv[2 * e + 1] = __high2float(h2[e]); }
#pragma unroll
      for (int h = 0; h < QF_HEADS_MAX; ++h) {
        if (h >= NI) break;
        const float4 qa = *reinterpret_cast<const float4*>(&qs[x][h * 64 + 8 * c]), qb = *reinterpret_cast<const float4*>(&qs[x][h * 64 + 8 * c + 4]);
        dot[h] += qa.x * kv[0] + qa.y * kv[1] + qa.z * kv[2] + qa.w * kv[3] + qb.x * kv[4] + qb.y * kv[5] + qb.z * kv[6] + qb.w * kv[7];
      }
    }
    float score = 0.f;
#pragma unroll
    for (int h = 0; h < QF_HEADS_MAX; ++h) if (h < NI) score += ws[x][h] * (fmaxf(bf16_round(dot[h]), 0.f) * scale);
    scores[((long long)b * nb + i0 + x) * S + s] = score;
  }
}

__global__ void __launch_bounds__(QF_THREADS) qsa_first_query_lp_kernel(const float* __restrict__ scored, float* __restrict__ lp_blk, int S) {
  grid_wait();
  extern __shared__ __align__(16) float qf_smem[];
  float* red = qf_smem;                      // [36]
  float* scores = red + 36;                  // [S]
  const int i = gridDim.x - 1 - blockIdx.x, b = blockIdx.y, nb = S / 64, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nkeys = 64 * i + 1;
  float m = -INFINITY;
  for (int s = tid; s < nkeys; s += QF_THREADS) {
    const float score = scored[((long long)b * nb + i) * S + s];
    scores[s] = score;
    m = fmaxf(m, score);
  }
  m = warp_max(m);
  if (lane == 0) red[warp] = m;
  __syncthreads();
  m = warp_max(lane < QF_THREADS / 32 ? red[lane] : -INFINITY);
  if (tid < QF_SUM) {
    float sum = 0.f;
    for (int s = tid; s < nkeys; s += QF_SUM) sum += __expf(scores[s] - m);
    sum = warp_sum(sum);
    if (lane == 0) red[32 + warp] = sum;
  }
  __syncthreads();
  const float lse_all = m + __logf(red[32] + red[33] + red[34] + red[35]);
  float* out = lp_blk + ((long long)b * nb + i) * nb;
  for (int j = warp; j < nb; j += QF_THREADS / 32) {
    if (j > i) { if (lane == 0) out[j] = QF_MASKED; continue; }
    const int s0 = 64 * j + lane, s1 = s0 + 32;
    const float a = s0 < nkeys ? scores[s0] : -INFINITY, c = s1 < nkeys ? scores[s1] : -INFINITY;
    const float bm = warp_max(fmaxf(a, c));
    const float bs = warp_sum((s0 < nkeys ? __expf(a - bm) : 0.f) + (s1 < nkeys ? __expf(c - bm) : 0.f));
    if (lane == 0) out[j] = bm + __logf(bs) - lse_all;
  }
}

// q_first [B, NI, S/64, 64] bf16 (the first query of every block), ki [B, S, 64] bf16, w_first [B, S/64, NI] fp32 -> lp_blk [B, S/64, S/64]
at::Tensor qsa_first_query_lp(const at::Tensor& q_first, const at::Tensor& ki, const at::Tensor& w_first, double scale) {
  TORCH_CHECK(q_first.is_cuda() && q_first.scalar_type() == at::kBFloat16 && q_first.dim() == 4 && q_first.is_contiguous() && q_first.size(3) == 64,
              "qsa_first_query_lp: contiguous bf16 queries [B,NI,nb,64] required");
  TORCH_CHECK(ki.scalar_type() == at::kBFloat16 && ki.dim() == 3 && ki.is_contiguous() && ki.size(2) == 64 && ki.size(0) == q_first.size(0),
              "qsa_first_query_lp: contiguous bf16 keys [B,S,64] required");
  const int B = q_first.size(0), NI = q_first.size(1), nb = q_first.size(2), S = ki.size(1);
  TORCH_CHECK(NI <= QF_HEADS_MAX && S == 64 * nb && S <= 8192 && w_first.scalar_type() == at::kFloat && w_first.is_contiguous() && w_first.numel() == (int64_t)B * nb * NI,
              "qsa_first_query_lp: at most 4 heads, S = 64 nb <= 8192, fp32 weights [B,nb,NI]");
  const c10::cuda::CUDAGuard guard(q_first.device());
  auto lp = at::empty({B, nb, nb}, q_first.options().dtype(at::kFloat));
  auto scores = at::empty({B, nb, S}, q_first.options().dtype(at::kFloat));       // causal entries are written and read
  auto stream = at::cuda::getCurrentCUDAStream();
  const int key_tiles = (S + QF_KEYS - 1) / QF_KEYS;
  auto score = [&](auto kernel, int queries) {
    launch(kernel, dim3(key_tiles, (nb + queries - 1) / queries, B), QF_KEYS, 0, stream, (const __nv_bfloat16*)q_first.data_ptr(), (const __nv_bfloat16*)ki.data_ptr(),
           w_first.data_ptr<float>(), scores.data_ptr<float>(), S, NI, (float)scale);
  };
  // one query per CTA up to two CTAs per SM, two up to seven (half of the pairs are not causal and end at once): see above
  const int64_t pairs = (int64_t)key_tiles * nb * B;
  if (pairs <= 2 * kNumSMs) score(qsa_first_scores_kernel<1>, 1);
  else if (pairs <= 7 * kNumSMs) score(qsa_first_scores_kernel<2>, 2);
  else score(qsa_first_scores_kernel<4>, 4);
  launch(qsa_first_query_lp_kernel, dim3(nb, B), QF_THREADS, (36 + S) * 4, stream, scores.data_ptr<float>(), lp.data_ptr<float>(), S);
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  count_launch(2);
  return lp;
}

}  // namespace q38
