// Reverse pass of the delta-rule scan for training: only what depends on the chunk after it.
//
// With dS' the gradient of the state at a chunk's end:
//     dv_new = P^T dO + kg dS'          dS = d dS' + qg^T dO - w^T dv_new          dd = <dS', S>
// Like the forward scan (gdn_tile.cuh) this never mixes value columns, so a warp owns 16 of them, keeps dS'^T in its accumulator
// registers and needs no block barrier in the chain.  The products that sum over value columns (dw, dP, dqg, dkg) depend on the chain only
// through dS' and dv_new, which this kernel stores; the preparation backward forms them chunk-parallel over the whole chip.
// 84 pairs of 64 chunks: 130 us (1 pair 82, 156 pairs 246), where the pass that formed everything took 270.  Bound by the latency of the chain; a second warp per slice
// for the products that do not wait for it took 143 us with a whole pair per SM (the 14 KB that the two exchange per chunk cost more).
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>

#include "common.cuh"
#include "gdn_tile.cuh"
#include "host.h"
#include "launch.cuh"

namespace q38 {

template <int W>
__global__ void __launch_bounds__(32 * W) gdn_chain_bwd_kernel(const __grid_constant__ gdn::Maps4 maps, const bf16* __restrict__ dout, const bf16* __restrict__ states,
                                                               const float* __restrict__ dch, bf16* __restrict__ du, bf16* __restrict__ dstate,
                                                               float* __restrict__ dd, int NT, int H, int* __restrict__ err) {
  grid_wait();
  using namespace gdn;
  extern __shared__ __align__(1024) uint8_t scan_smem[];
  // STAGES x {w, P, qg, kg}, then per warp two pairs of slices {do, S} (a pair that has been read takes the outputs), then the barriers
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int bh = blockIdx.x, b = bh / H, hv = bh % H, slice = blockIdx.y * W + warp, col = 16 * slice;
  const uint32_t tiles = ptx::smem_u32(scan_smem), pairs = tiles + STAGES * 4 * TILE_BYTES + warp * 4 * SLICE_BYTES;
  uint64_t* full = reinterpret_cast<uint64_t*>(scan_smem + STAGES * 4 * TILE_BYTES + W * 4 * SLICE_BYTES);
  const long long base = (long long)bh * NT * 4096, tok_ld = (long long)H * 64;
  const bf16* dob = dout + ((long long)b * NT * 64 * H + hv) * 64 + col;       // token 0 of this pair's columns
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) ptx::mbar_init(&full[s], 1);
    ptx::fence_barrier_init();
  }
  __syncthreads();
  auto load_slices = [&](int c, int buf) {
    slice_load_async(pairs + buf * 2 * SLICE_BYTES, dob + (long long)c * 64 * tok_ld, tok_ld, lane);
    slice_load_async(pairs + (buf * 2 + 1) * SLICE_BYTES, states + base + (long long)c * 4096 + col, 64, lane);
  };
  // the slices are fetched one chunk ahead; three chunks ahead their lines are asked into L2
  auto prefetch_slices = [&](int c) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int row = lane + 32 * i;
      asm volatile("prefetch.global.L2 [%0];" ::"l"(dob + ((long long)c * 64 + row) * tok_ld));
      asm volatile("prefetch.global.L2 [%0];" ::"l"(states + base + (long long)c * 4096 + row * 64 + col));
    }
  };
  for (int i = 0; i < STAGES - 1 && i < NT; ++i)
    if (threadIdx.x == 0) load_stage(maps, scan_smem + i * 4 * TILE_BYTES, &full[i], (bh * NT + NT - 1 - i) * 64);
  load_slices(NT - 1, 0);
  cp_async_commit();
  float dS[8][4];
  zero_acc(dS);
  float d_next = dch[(long long)bh * NT + NT - 1];
  int stage = 0, phase = 0;
  // A chunk's tiles are waited for before the barrier that ends the chunk before it, which exchanges the verdict: a lane whose wait ran out (the
  // lanes poll for themselves) neither leaves its warp's collective instructions nor the barrier, the CTA leaves together.  It also takes the
  // wait off the start of the chain: with a vote and a branch in front of the products 84 pairs took 138 us, with each lane's own branch 133.
  bool late = !ptx::mbar_wait(&full[0], 0);
  for (int i = 0; ; ++i) {
    if (__syncthreads_or(late)) {                            // a tile never came: let the copies in flight land (bounded), then leave
      if (threadIdx.x == 0) report_error(err, ERR_TMA_WAIT);
      for (int j = 1; j < STAGES - 1 && i + j < NT; ++j) {
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
        ptx::mbar_wait(&full[stage], phase);
      }
      cp_async_wait<0>();
      return;
    }
    if (i == NT) break;
    const int c = NT - 1 - i;
    {  // refill the stage that the chunk before left
      const int n = i + STAGES - 1, ns = stage == 0 ? STAGES - 1 : stage - 1;
      if (n < NT && threadIdx.x == 0) load_stage(maps, scan_smem + ns * 4 * TILE_BYTES, &full[ns], (bh * NT + NT - 1 - n) * 64);
      if (i + 1 < NT) load_slices(c - 1, (i + 1) & 1);
      cp_async_commit();
      if (i + 3 < NT) prefetch_slices(c - 3);
    }
    const float d = d_next;
    d_next = dch[(long long)bh * NT + (c > 0 ? c - 1 : 0)];
    cp_async_wait<1>();
    __syncwarp();
    const uint32_t wt = tiles + stage * 4 * TILE_BYTES, pt = wt + TILE_BYTES, qt = pt + TILE_BYTES, kt = qt + TILE_BYTES;
    const uint32_t mine = pairs + (i & 1) * 2 * SLICE_BYTES;
    uint32_t aD[4][4], aS[4][4], av[4][4];
    float acc[8][4], part = 0.f;
    slice_read_t(mine, aD, lane);                          // dO^T
    slice_read_t(mine + SLICE_BYTES, av, lane);            // S^T, in accumulator order
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float* x = &dS[2 * ks + (e >> 1)][2 * (e & 1)];
        part += x[0] * lo_f(av[ks][e]) + x[1] * hi_f(av[ks][e]);
      }
    }
    pack_a<4>(dS, aS);
    zero_acc(acc);
    mma64<true>(aD, pt, acc, lane);                        // (P^T dO)^T
    mma64<false>(aS, kt, acc, lane);                       // + (kg dS')^T
    pack_a<4>(acc, av);
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) { dS[nt][0] *= d; dS[nt][1] *= d; dS[nt][2] *= d; dS[nt][3] *= d; }
    mma64<true>(aD, qt, dS, lane);                         // + (qg^T dO)^T
    uint32_t neg[4][4];
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
#pragma unroll
      for (int e = 0; e < 4; ++e) neg[ks][e] = av[ks][e] ^ 0x80008000u;
    }
    mma64<true>(neg, wt, dS, lane);                        // - (w^T dv_new)^T
    slice_store_t(mine, aS, dstate + base + (long long)c * 4096 + col, 64, lane);
    slice_store_t(mine + SLICE_BYTES, av, du + base + (long long)c * 4096 + col, 64, lane);
    part = warp_sum(part);
    if (lane == 0) dd[((long long)bh * NT + c) * 4 + slice] = part;
    if (++stage == STAGES) { stage = 0; phase ^= 1; }
    late = i + 1 < NT && !ptx::mbar_wait(&full[stage], phase);
  }
}

// Returns {du = dv_new [BH,NT,64,64] bf16, dstate [BH,NT,64,64] bf16 (gradient of the state at each chunk's end),
// dd [BH,NT,4] fp32 (gradient of the chunk's decay factor, one part per 16 value columns)}.
std::vector<at::Tensor> gdn_chain_bwd(const at::Tensor& w, const at::Tensor& P, const at::Tensor& qg, const at::Tensor& kg, const at::Tensor& dch,
                                      const at::Tensor& states, const at::Tensor& dout, int64_t B, int64_t H, const c10::optional<at::Tensor>& err) {
  const c10::cuda::CUDAGuard guard(w.device());
  const int64_t BH = B * H, NT = w.numel() / (BH * 64 * 64);
  for (const at::Tensor* t : {&w, &P, &qg, &kg, &states})
    TORCH_CHECK(t->is_cuda() && t->scalar_type() == at::kBFloat16 && t->is_contiguous() && t->numel() == BH * NT * 64 * 64, "gdn_chain_bwd: contiguous bf16 [BH,NT,64,64] required");
  TORCH_CHECK(dout.scalar_type() == at::kBFloat16 && dout.is_contiguous() && dout.numel() == BH * NT * 64 * 64 && (reinterpret_cast<uintptr_t>(dout.data_ptr()) & 15) == 0,
              "gdn_chain_bwd: do must be contiguous, 16-byte aligned bf16 [B,S,H,64]");
  TORCH_CHECK(dch.scalar_type() == at::kFloat && dch.is_contiguous() && dch.numel() == BH * NT, "gdn_chain_bwd: dch must be fp32 [BH,NT]");
  auto du = at::empty({BH, NT, 64, 64}, w.options()), dstate = at::empty({BH, NT, 64, 64}, w.options());
  auto dd = at::empty({BH, NT, 4}, w.options().dtype(at::kFloat));
  if (NT == 0 || BH == 0) return {du, dstate, dd};
  const at::Tensor* t[4] = {&w, &P, &qg, &kg};
  gdn::Maps4 maps;
  for (int i = 0; i < 4; ++i) maps.m[i] = make_tmap_box(t[i]->data_ptr(), 2, 64, BH * NT * 64, 1, 64, 0, 64, 128);
  auto launch = [&](auto warps) {
    constexpr int W = decltype(warps)::value;
    constexpr int smem = gdn::STAGES * 4 * gdn::TILE_BYTES + W * 4 * gdn::SLICE_BYTES + 64;
    static bool configured = false;
    if (!configured) { C10_CUDA_CHECK(cudaFuncSetAttribute(gdn_chain_bwd_kernel<W>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)); configured = true; }
    q38::launch(gdn_chain_bwd_kernel<W>, dim3((int)BH, 4 / W), 32 * W, smem, at::cuda::getCurrentCUDAStream(), 
        maps, (const bf16*)dout.data_ptr(), (const bf16*)states.data_ptr(), dch.data_ptr<float>(), (bf16*)du.data_ptr(), (bf16*)dstate.data_ptr(),
        dd.data_ptr<float>(), (int)NT, (int)H, err.has_value() ? err->data_ptr<int>() : nullptr);
  };
  if (gdn::scan_warps(BH) == 1) launch(std::integral_constant<int, 1>()); else launch(std::integral_constant<int, 2>());
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  count_launch();
  return {du, dstate, dd};
}

}  // namespace q38
