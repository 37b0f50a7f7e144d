// Shared by the block-attention kernels: lists of selected blocks, operand checks.
#pragma once
#include <ATen/ATen.h>
#include <c10/cuda/CUDAException.h>

#include "common.cuh"

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

}  // namespace q38
