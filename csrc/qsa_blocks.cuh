// Shared by the block-attention kernels: lists of selected blocks, operand checks.
#pragma once
#include <ATen/ATen.h>
#include <c10/cuda/CUDAException.h>

#include "common.cuh"
#include "host.h"

namespace q38 {

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

inline int list_bytes(int nb) { return (2 * nb + 15) / 16 * 16; }

// The kernels' dynamic shared memory grows with the number of blocks in a sequence; the limit leaves room for a few static bytes and is set once.
template <typename K> void allow_smem(K kernel) { C10_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024)); }

inline void check_heads(const at::Tensor& t, const char* name) {
  TORCH_CHECK(t.is_cuda() && t.scalar_type() == at::kBFloat16 && t.is_contiguous() && t.dim() == 4 && t.size(3) == 64, name, ": contiguous bf16 [B,H,S,64] required");
}

// Values [B,H,S,64]: contiguous, or the transposed view of a projection's output [B,S,H,64].  Returns whether it is the latter.
inline bool check_values(const at::Tensor& v, const char* name) {
  const bool tokens = v.dim() == 4 && v.size(3) == 64 && v.stride(3) == 1 && v.stride(1) == 64 && v.stride(2) == v.size(1) * 64 && v.stride(0) == v.size(2) * v.size(1) * 64;
  if (!tokens || !v.is_cuda() || v.scalar_type() != at::kBFloat16) check_heads(v, name);
  return tokens;
}
// Its tensor map: a box of 64 rows starts at {0, b S + row, head} in the transposed view, at {0, (b H + head) S + row, 0} otherwise.
inline CUtensorMap value_map(const at::Tensor& v, bool tokens) {
  const int64_t B = v.size(0), H = v.size(1), S = v.size(2);
  return tokens ? make_tmap_box(v.data_ptr(), 2, 64, B * S, H, H * 64, 64, 64, 128) : make_tmap_box(v.data_ptr(), 2, 64, B * H * S, 1, 64, 0, 64, 128);
}

}  // namespace q38
