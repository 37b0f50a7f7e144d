// Gated DeltaNet: chunked gated delta rule (chunk = 64 tokens, head dims 64), forward and backward.
//
// Per (batch, value head) and chunk c, with S the [k-dim x v-dim] state at the chunk start:
//     v_new = u - w S                  o = qg S + P v_new                  S' = d S + kg^T v_new
// where (prepared per chunk, all independent of S and therefore fully parallel over chunks)
//     gc = cumsum(g) inside the chunk,  Gamma_ij = exp(gc_i - gc_j)
//     Tm = (I + tril(beta_i (k_i.k_j) Gamma_ij, -1))^-1,   w = Tm (beta e^gc k),   u = Tm (beta v)
//     P  = tril((q_i.k_j) Gamma_ij),   qg = q e^gc,   kg = k e^(gc_last - gc),   d = e^gc_last
// with q, k L2-normalised and q scaled by 64^-1/2.
//
// Kernels
//   gdn_scan_fwd   the sequential pass over chunks, one chain of warps per 16 value columns of a (batch, value head) pair (gdn_tile.cuh).
//                  The fp32 state lives in the warp's accumulator registers; the operand tiles come by TMA, several chunks ahead.
//                  The chain per chunk is latency bound (two dependent products), which is why this pass uses
//                  register-resident warp MMAs instead of the TMEM round trips of tcgen05.
//   gdn_prep_fwd   the chunk operands, gdn_prep_bwd everything of the backward that is independent between chunks (second half of this file).
//   The reverse chain of a training step is gdn_chain_bwd in gdn_chain.cu.
//   gdn_scan_bwd   a reverse pass that forms all operand gradients (dw, du, dP, dqg, dkg, dd) itself.  It serves operands that come from the
//                  PyTorch specification (Q38_GDN_HYBRID=1), which has no preparation backward to hand dS' and dv_new to.
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>

#include <array>

#include "common.cuh"
#include "host.h"
#include "launch.cuh"
#include "gdn_tile.cuh"
#include "mma_tile.cuh"

namespace q38 {

// ---------------------------------------------------------------------------------------------------------------------
// Forward scan.  Chunk operands w,u,P,qg,kg: [BH, NT, 64, 64] bf16; dch: [BH, NT] fp32.
// Outputs: o [B, S, H, 64] bf16 (token-major) and, when the backward pass will want them, vnew [BH, NT, 64, 64] bf16 and
// states [BH, NT, 64, 64] bf16 (chunk-start S).
//
// Roles: warps 0..W-1 carry the chain (v_new and the new state, two products per chunk), warps W..2W-1 turn the packed state and v_new
// that a chain warp leaves in shared memory into o and do all stores (two products), two more warps keep the operand tiles coming.
// One warp alone on its scheduler can neither hide its own latencies nor overlap its halves, and the chain is what the pass waits for (some 600
// instructions per 16 columns and chunk, six cycles each; neither memory nor the MMA rate).  84 pairs of 64 chunks: 112 us, 81 without the
// tensors saved for the backward; 142 us with one warp for both roles, 160 us with eight warps per product and three block barriers per
// chunk.  39 pairs of 128 chunks (one prompt of 8192): 123 us, before 320.
// ---------------------------------------------------------------------------------------------------------------------
constexpr int SCAN_U = 4;                                                // slices of u in flight per chain warp
template <int W> struct ScanSmem {
  static constexpr int XCHG = 2 * 4096;                                  // two slots of {S, v_new} fragments
  static constexpr int PAIR = SCAN_U * gdn::SLICE_BYTES + XCHG + gdn::SLICE_BYTES;
  static constexpr int TILES = (gdn::CHAIN_STAGES + gdn::SIDE_STAGES) * 2 * gdn::TILE_BYTES;
  static constexpr int BARS = 2 * gdn::CHAIN_STAGES + 2 * gdn::SIDE_STAGES + 4 * W;
  static constexpr int BYTES = TILES + W * PAIR + BARS * 8;
};

template <int W>
__global__ void __launch_bounds__(64 * W + 64) gdn_scan_fwd_kernel(const __grid_constant__ gdn::Maps4 maps, const bf16* __restrict__ u, const float* __restrict__ dch,
                                                                   bf16* __restrict__ o, bf16* __restrict__ vnew, bf16* __restrict__ states, int NT, int H,
                                                                   int* __restrict__ err) {
  grid_wait();
  using namespace gdn;
  using L = ScanSmem<W>;
  extern __shared__ __align__(1024) uint8_t scan_smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int bh = blockIdx.x, b = bh / H, hv = bh % H;
  uint64_t* bars = reinterpret_cast<uint64_t*>(scan_smem + L::TILES + W * L::PAIR);
  const Ring<CHAIN_STAGES> chain{scan_smem, bars, bars + CHAIN_STAGES};
  const Ring<SIDE_STAGES> side{scan_smem + CHAIN_STAGES * 2 * TILE_BYTES, bars + 2 * CHAIN_STAGES, bars + 2 * CHAIN_STAGES + SIDE_STAGES};
  uint64_t* xbars = bars + 2 * CHAIN_STAGES + 2 * SIDE_STAGES;           // per pair: two full, two empty
  if (threadIdx.x == 0) {
    chain.init(W);
    side.init(W);
    for (int i = 0; i < 4 * W; ++i) ptx::mbar_init(&xbars[i], 1);
    ptx::fence_barrier_init();
  }
  __syncthreads();
  if (warp >= 2 * W) {
    if (lane == 0) {
      const bool ok = warp == 2 * W ? chain.produce(&maps.m[0], &maps.m[1], bh * NT, NT, 1) : side.produce(&maps.m[2], &maps.m[3], bh * NT, NT, 1);
      if (!ok) report_error(err, ERR_MMA_WAIT);
    }
    return;
  }
  const int pair = warp % W, col = 16 * (blockIdx.y * W + pair);
  const uint32_t slices = ptx::smem_u32(scan_smem) + L::TILES + pair * L::PAIR, xchg = slices + SCAN_U * SLICE_BYTES, out_slice = xchg + L::XCHG;
  uint64_t *xfull = xbars + 4 * pair, *xempty = xfull + 2;
  const long long base = (long long)bh * NT * 4096;
  if (warp < W) {
    for (int c = 0; c < SCAN_U - 1; ++c) {
      if (c < NT) slice_load_async(slices + c * SLICE_BYTES, u + base + (long long)c * 4096 + col, 64, lane);
      cp_async_commit();
    }
    float S[8][4];
    zero_acc(S);
    float d_next = dch[(long long)bh * NT];
    for (int c = 0; c < NT; ++c) {
      if (c + SCAN_U - 1 < NT) slice_load_async(slices + ((c + SCAN_U - 1) % SCAN_U) * SLICE_BYTES, u + base + (long long)(c + SCAN_U - 1) * 4096 + col, 64, lane);
      cp_async_commit();
      const float d = d_next;
      d_next = dch[(long long)bh * NT + (c + 1 < NT ? c + 1 : c)];
      uint32_t aS[4][4], av[4][4];
      float acc[8][4];
      pack_a<4>(S, aS);
      bool ok = c < 2 || ptx::mbar_wait(&xempty[c & 1], ((c >> 1) & 1) ^ 1);
      frags_put(xchg + (c & 1) * 4096, aS, lane);
      cp_async_wait<SCAN_U - 1>();
      __syncwarp();
      slice_read_t(slices + (c % SCAN_U) * SLICE_BYTES, av, lane);       // u^T
      ok = ptx::mbar_wait(chain.full + c % CHAIN_STAGES, (c / CHAIN_STAGES) & 1) && ok;
      if (!__all_sync(0xffffffffu, ok)) { if (lane == 0) report_error(err, ERR_TMA_WAIT); break; }
      const uint32_t wt = chain.tile(c), kt = wt + TILE_BYTES;
      zero_acc(acc);
      mma64<false>(aS, wt, acc, lane);                                   // (w S)^T
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          float* x = &acc[2 * ks + (e >> 1)][2 * (e & 1)];
          x[0] = lo_f(av[ks][e]) - x[0];
          x[1] = hi_f(av[ks][e]) - x[1];
        }
      }
      pack_a<4>(acc, av);                                                // v_new^T
      frags_put(xchg + (c & 1) * 4096 + 2048, av, lane);
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&xfull[c & 1]);
#pragma unroll
      for (int nt = 0; nt < 8; ++nt) { S[nt][0] *= d; S[nt][1] *= d; S[nt][2] *= d; S[nt][3] *= d; }
      mma64<true>(av, kt, S, lane);                                      // + (kg^T v_new)^T
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(chain.empty + c % CHAIN_STAGES);
    }
    cp_async_wait<0>();
  } else {
    for (int c = 0; c < NT; ++c) {
      bool ok = ptx::mbar_wait(&xfull[c & 1], (c >> 1) & 1);
      ok = ptx::mbar_wait(side.full + c % SIDE_STAGES, (c / SIDE_STAGES) & 1) && ok;
      if (!__all_sync(0xffffffffu, ok)) { if (lane == 0) report_error(err, ERR_TMA_WAIT); break; }
      uint32_t aS[4][4], av[4][4];
      float acc[8][4];
      frags_get(xchg + (c & 1) * 4096, aS, lane);
      frags_get(xchg + (c & 1) * 4096 + 2048, av, lane);
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&xempty[c & 1]);
      const uint32_t qt = side.tile(c), pt = qt + TILE_BYTES;
      zero_acc(acc);
      mma64<false>(aS, qt, acc, lane);                                   // (qg S)^T
      mma64<false>(av, pt, acc, lane);                                   // + (P v_new)^T
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(side.empty + c % SIDE_STAGES);
      if (states != nullptr) {
        slice_store_t(out_slice, aS, states + base + (long long)c * 4096 + col, 64, lane);
        slice_store_t(out_slice, av, vnew + base + (long long)c * 4096 + col, 64, lane);
      }
      pack_a<4>(acc, aS);
      slice_store_t(out_slice, aS, o + (((long long)b * NT * 64 + (long long)c * 64) * H + hv) * 64 + col, (long long)H * 64, lane);
    }
  }
}

// ---------------------------------------------------------------------------------------------------------------------
// Backward scan (reverse over chunks).  Inputs: the forward operands, vnew, states, and do [B,S,H,64].
// Outputs per chunk: dw, du, dP, dqg, dkg [BH,NT,64,64] bf16 and dd [BH,NT] fp32.
// ---------------------------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) gdn_scan_bwd_kernel(const bf16* __restrict__ w, const bf16* __restrict__ P, const bf16* __restrict__ qg,
                                                           const bf16* __restrict__ kg, const float* __restrict__ dch, const bf16* __restrict__ vnew,
                                                           const bf16* __restrict__ states, const bf16* __restrict__ dout, bf16* __restrict__ dw,
                                                           bf16* __restrict__ du, bf16* __restrict__ dP, bf16* __restrict__ dqg, bf16* __restrict__ dkg,
                                                           float* __restrict__ dd, int NT, int H) {
  grid_wait();
  extern __shared__ __align__(16) uint8_t smem_bytes[];
  bf16* sm = reinterpret_cast<bf16*>(smem_bytes);
  // two buffers of seven tiles: w, P, qg, kg, vnew, state, do ; then dS (bf16) and dv_new (bf16)
  bf16* dSb = sm + 14 * TILE_ELEMS;
  bf16* dVn = dSb + TILE_ELEMS;
  __shared__ float red[8];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int bh = blockIdx.x, b = bh / H, hv = bh % H;
  const long long tile = 64 * 64, base = (long long)bh * NT * tile;
  auto prefetch = [&](int c, int buf) {
    bf16* dst = sm + buf * 7 * TILE_ELEMS;
    load_tile_async_256(dst + 0 * TILE_ELEMS, w + base + (long long)c * tile, 64, tid);
    load_tile_async_256(dst + 1 * TILE_ELEMS, P + base + (long long)c * tile, 64, tid);
    load_tile_async_256(dst + 2 * TILE_ELEMS, qg + base + (long long)c * tile, 64, tid);
    load_tile_async_256(dst + 3 * TILE_ELEMS, kg + base + (long long)c * tile, 64, tid);
    load_tile_async_256(dst + 4 * TILE_ELEMS, vnew + base + (long long)c * tile, 64, tid);
    load_tile_async_256(dst + 5 * TILE_ELEMS, states + base + (long long)c * tile, 64, tid);
    load_tile_async_256(dst + 6 * TILE_ELEMS, dout + (((long long)b * NT * 64 + (long long)c * 64) * H + hv) * 64, (long long)H * 64, tid);
    cp_async_commit();
  };
  const int r = 16 * (warp & 3) + (lane >> 2), c0 = 32 * (warp >> 2) + 2 * (lane & 3);
  float dS[4][4];
  zero_acc(dS);
  prefetch(NT - 1, (NT - 1) & 1);
  for (int c = NT - 1; c >= 0; --c) {
    const int buf = c & 1;
    if (c > 0) { prefetch(c - 1, buf ^ 1); cp_async_wait<1>(); } else { cp_async_wait<0>(); }
    acc_to_smem_h(dS, dSb, warp, lane);
    __syncthreads();
    const bf16* Wt = sm + buf * 7 * TILE_ELEMS;
    const bf16* Pt = Wt + TILE_ELEMS;
    const bf16* Qt = Pt + TILE_ELEMS;
    const bf16* Kt = Qt + TILE_ELEMS;
    const bf16* Vt = Kt + TILE_ELEMS;
    const bf16* St = Vt + TILE_ELEMS;
    const bf16* Dt = St + TILE_ELEMS;
    const long long off = base + (long long)c * tile;
    float acc[4][4];
    // dv_new = P^T dO + kg dS'
    zero_acc(acc);
    mma64h<true, false>(Pt, Dt, acc, warp, lane);
    mma64h<false, false>(Kt, dSb, acc, warp, lane);
    acc_to_smem_h(acc, dVn, warp, lane);
    acc_to_global_h(acc, du + off, 64, warp, lane);
    // dd = <dS', S>   (fragment of S read from the state tile in accumulator layout)
    {
      float part = 0.f;
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) {
        const __nv_bfloat162 s0 = *reinterpret_cast<const __nv_bfloat162*>(St + r * LDS + 8 * nt + c0);
        const __nv_bfloat162 s1 = *reinterpret_cast<const __nv_bfloat162*>(St + (r + 8) * LDS + 8 * nt + c0);
        part += dS[nt][0] * __low2float(s0) + dS[nt][1] * __high2float(s0) + dS[nt][2] * __low2float(s1) + dS[nt][3] * __high2float(s1);
      }
      part = warp_sum(part);
      if (lane == 0) red[warp] = part;
    }
    // dqg = dO S^T ;  dkg = v_new dS'^T ;  dP = tril(dO v_new^T)
    zero_acc(acc);
    mma64h<false, true>(Dt, St, acc, warp, lane);
    acc_to_global_h(acc, dqg + off, 64, warp, lane);
    zero_acc(acc);
    mma64h<false, true>(Vt, dSb, acc, warp, lane);
    acc_to_global_h(acc, dkg + off, 64, warp, lane);
    zero_acc(acc);
    mma64h<false, true>(Dt, Vt, acc, warp, lane);
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
      const int col = 8 * nt + c0;
      if (col > r) acc[nt][0] = 0.f;
      if (col + 1 > r) acc[nt][1] = 0.f;
      if (col > r + 8) acc[nt][2] = 0.f;
      if (col + 1 > r + 8) acc[nt][3] = 0.f;
    }
    acc_to_global_h(acc, dP + off, 64, warp, lane);
    __syncthreads();                                    // dVn and red[] complete
    if (tid == 0) dd[(long long)bh * NT + c] = red[0] + red[1] + red[2] + red[3] + red[4] + red[5] + red[6] + red[7];
    // dw = -dv_new S^T
    zero_acc(acc);
    mma64h<false, true>(dVn, St, acc, warp, lane);
    acc_to_global_h(acc, dw + off, 64, warp, lane, -1.f);
    // dS = d dS' + qg^T dO - w^T dv_new
    const float d = dch[(long long)bh * NT + c];
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) { dS[nt][0] *= d; dS[nt][1] *= d; dS[nt][2] *= d; dS[nt][3] *= d; }
    mma64h<true, false>(Qt, Dt, dS, warp, lane);
    zero_acc(acc);
    mma64h<true, false>(Wt, dVn, acc, warp, lane);
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) { dS[nt][0] -= acc[nt][0]; dS[nt][1] -= acc[nt][1]; dS[nt][2] -= acc[nt][2]; dS[nt][3] -= acc[nt][3]; }
    __syncthreads();
  }
}

// ---- host ----------------------------------------------------------------------------------------------------------------
static void check_tiles(const at::Tensor& t, int64_t BH, int64_t NT, const char* name) {
  TORCH_CHECK(t.is_cuda() && t.scalar_type() == at::kBFloat16 && t.is_contiguous() && t.numel() == BH * NT * 64 * 64, name, ": contiguous bf16 [BH,NT,64,64] required");
}

static gdn::Maps4 tile_maps(const at::Tensor& a, const at::Tensor& b, const at::Tensor& c, const at::Tensor& d) {
  const at::Tensor* t[4] = {&a, &b, &c, &d};
  gdn::Maps4 maps;
  for (int i = 0; i < 4; ++i) maps.m[i] = make_tmap_box(t[i]->data_ptr(), 2, 64, t[i]->numel() / 64, 1, 64, 0, 64, 128);
  return maps;
}

// Returns {o [B,S,H,64], vnew [BH,NT,64,64], states [BH,NT,64,64]}; without `save` (no backward pass will follow) the last two are empty.
std::vector<at::Tensor> gdn_scan_fwd(const at::Tensor& w, const at::Tensor& u, const at::Tensor& P, const at::Tensor& qg, const at::Tensor& kg,
                                     const at::Tensor& dch, int64_t B, int64_t H, const c10::optional<at::Tensor>& err, bool save) {
  const c10::cuda::CUDAGuard guard(w.device());
  const int64_t BH = B * H, NT = w.numel() / (BH * 64 * 64);
  check_tiles(w, BH, NT, "w"); check_tiles(u, BH, NT, "u"); check_tiles(P, BH, NT, "P"); check_tiles(qg, BH, NT, "qg"); check_tiles(kg, BH, NT, "kg");
  TORCH_CHECK(dch.scalar_type() == at::kFloat && dch.is_contiguous() && dch.numel() == BH * NT, "gdn_scan_fwd: dch must be fp32 [BH,NT]");
  auto o = at::empty({B, NT * 64, H, 64}, w.options());
  const std::vector<int64_t> kept = save ? std::vector<int64_t>{BH, NT, 64, 64} : std::vector<int64_t>{0};
  auto vnew = at::empty(kept, w.options()), states = at::empty(kept, w.options());
  if (NT == 0 || BH == 0) return {o, vnew, states};
  const auto maps = tile_maps(w, kg, qg, P);
  auto launch = [&](auto warps) {
    constexpr int W = decltype(warps)::value;
    constexpr int smem = ScanSmem<W>::BYTES;
    static bool configured = false;
    if (!configured) { C10_CUDA_CHECK(cudaFuncSetAttribute(gdn_scan_fwd_kernel<W>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)); configured = true; }
    q38::launch(gdn_scan_fwd_kernel<W>, dim3((int)BH, 4 / W), 64 * W + 64, smem, at::cuda::getCurrentCUDAStream(), 
        maps, (const bf16*)u.data_ptr(), dch.data_ptr<float>(), (bf16*)o.data_ptr(), save ? (bf16*)vnew.data_ptr() : nullptr,
        save ? (bf16*)states.data_ptr() : nullptr, (int)NT, (int)H, err.has_value() ? err->data_ptr<int>() : nullptr);
  };
  switch (gdn::scan_pairs(BH)) {
    case 1: launch(std::integral_constant<int, 1>()); break;
    case 2: launch(std::integral_constant<int, 2>()); break;
    default: launch(std::integral_constant<int, 4>());
  }
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  count_launch();
  return {o, vnew, states};
}

// Returns {dw, du, dP, dqg, dkg (bf16 tiles), dd [BH,NT] fp32}
std::vector<at::Tensor> gdn_scan_bwd(const at::Tensor& w, const at::Tensor& P, const at::Tensor& qg, const at::Tensor& kg, const at::Tensor& dch,
                                     const at::Tensor& vnew, const at::Tensor& states, const at::Tensor& dout, int64_t B, int64_t H) {
  const c10::cuda::CUDAGuard guard(w.device());
  const int64_t BH = B * H, NT = w.numel() / (BH * 64 * 64);
  check_tiles(w, BH, NT, "w"); check_tiles(P, BH, NT, "P"); check_tiles(qg, BH, NT, "qg"); check_tiles(kg, BH, NT, "kg");
  check_tiles(vnew, BH, NT, "vnew"); check_tiles(states, BH, NT, "states");
  TORCH_CHECK(dout.scalar_type() == at::kBFloat16 && dout.is_contiguous() && dout.numel() == BH * NT * 64 * 64, "gdn_scan_bwd: do must be contiguous bf16 [B,S,H,64]");
  auto opts = w.options();
  auto dw = at::empty({BH, NT, 64, 64}, opts), du = at::empty({BH, NT, 64, 64}, opts), dP = at::empty({BH, NT, 64, 64}, opts);
  auto dqg = at::empty({BH, NT, 64, 64}, opts), dkg = at::empty({BH, NT, 64, 64}, opts);
  auto dd = at::empty({BH, NT}, opts.dtype(at::kFloat));
  const int smem = 16 * TILE_ELEMS * 2;
  static bool configured = false;
  if (!configured) { C10_CUDA_CHECK(cudaFuncSetAttribute(gdn_scan_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)); configured = true; }
  launch(gdn_scan_bwd_kernel, (int)BH, 256, smem, at::cuda::getCurrentCUDAStream(), 
      (const bf16*)w.data_ptr(), (const bf16*)P.data_ptr(), (const bf16*)qg.data_ptr(), (const bf16*)kg.data_ptr(), dch.data_ptr<float>(),
      (const bf16*)vnew.data_ptr(), (const bf16*)states.data_ptr(), (const bf16*)dout.data_ptr(), (bf16*)dw.data_ptr(), (bf16*)du.data_ptr(),
      (bf16*)dP.data_ptr(), (bf16*)dqg.data_ptr(), (bf16*)dkg.data_ptr(), dd.data_ptr<float>(), (int)NT, (int)H);
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  count_launch();
  return {dw, du, dP, dqg, dkg, dd};
}

}  // namespace q38

// =====================================================================================================================
// Chunk preparation (everything that does not depend on the running state), forward and backward.
// =====================================================================================================================
namespace q38 {

// q,k: [B,S,Hk,64]; v: [B,S,Hv,64]; g fp32 / beta bf16: [B,S,Hv].  Tiles out: [B*Hv, NT, 64, 64] bf16 (Tm only for a backward pass).
// One CTA of four warps per (chunk, batch, value head), four per SM.  Every global access is a 16-byte piece of a 128-byte row.
// (I + L)^-1 is found by forward substitution in fp32, in blocks of eight rows: a warp owns blocks `warp` and `warp + 4`, one column (and from
// row 32 on a second one) per lane; the owner of a block solves it and leaves its rows in place of L's, then every warp subtracts them from
// its later blocks.  A row's dot product runs as four ascending chains (j mod 4), as it would in one pass, so the blocks do not change a bit.
// With one warp per 32 columns and all rows unrolled the other warps waited at the barrier for 2500 serial instructions that the
// instruction cache did not hold: 169 us for 5376 chunks of a 16384-token layer (207 us with one thread per column of all rows), now 146.
__global__ void __launch_bounds__(128, 4) gdn_prep_fwd_kernel(const bf16* __restrict__ q, const bf16* __restrict__ k, const bf16* __restrict__ v,
                                                              const float* __restrict__ g, const bf16* __restrict__ beta, bf16* __restrict__ w_out,
                                                              bf16* __restrict__ u_out, bf16* __restrict__ P_out, bf16* __restrict__ qg_out,
                                                              bf16* __restrict__ kg_out, bf16* __restrict__ Tm_out, float* __restrict__ carry,
                                                              float* __restrict__ gc_out, int S, int Hk, int Hv, long long qk_ld, long long v_ld) {
  grid_wait();
  extern __shared__ __align__(16) uint8_t smem_bytes[];
  bf16* sm = reinterpret_cast<bf16*>(smem_bytes);
  bf16 *Qn = sm, *Kn = sm + TILE_ELEMS, *KBG = sm + 2 * TILE_ELEMS, *VB = sm + 3 * TILE_ELEMS, *Tm = sm + 4 * TILE_ELEMS;
  constexpr int LD = 68;                                             // fp32 rows, 16-byte aligned
  float* L = reinterpret_cast<float*>(sm);                           // [64][68], over Qn and Kn once they are used up
  float *gc = reinterpret_cast<float*>(sm + 5 * TILE_ELEMS), *bet = gc + 64, *eg = bet + 64, *el = eg + 64;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int c = blockIdx.x, bh = blockIdx.y, b = bh / Hv, hv = bh % Hv, hk = hv / (Hv / Hk);
  const int NT = gridDim.x;
  const long long tok0 = (long long)b * S + (long long)c * 64;
  const long long tile_off = ((long long)bh * NT + c) * 4096;
  const int piece = 8 * (tid & 7), tok_t = tid >> 3;                 // this thread's 8 dims of tokens tok_t + 16 i
  if (tid < 32) {
    // gc = inclusive cumsum of g over the chunk, two tokens per lane
    const float g0 = g[(tok0 + 2 * tid) * Hv + hv], g1 = g[(tok0 + 2 * tid + 1) * Hv + hv];
    float run = g0 + g1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const float up = __shfl_up_sync(0xffffffffu, run, o); if (tid >= o) run += up; }
    const float last = __shfl_sync(0xffffffffu, run, 31), first = run - g1;
    gc[2 * tid] = first; gc[2 * tid + 1] = run;
    eg[2 * tid] = __expf(first); eg[2 * tid + 1] = __expf(run);
    el[2 * tid] = __expf(last - first); el[2 * tid + 1] = __expf(last - run);
    if (tid == 0) carry[(long long)bh * NT + c] = __expf(last);
  } else if (tid < 96) {
    bet[tid - 32] = __bfloat162float(beta[(tok0 + tid - 32) * Hv + hv]);
  }
  uint32_t qn[4][4], kn[4][4];
  uint4 vr[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const long long tok = tok0 + tok_t + 16 * i;
    const uint4 qr = *reinterpret_cast<const uint4*>(q + tok * qk_ld + hk * 64 + piece), kr = *reinterpret_cast<const uint4*>(k + tok * qk_ld + hk * 64 + piece);
    vr[i] = *reinterpret_cast<const uint4*>(v + tok * v_ld + hv * 64 + piece);
    qn[i][0] = qr.x; qn[i][1] = qr.y; qn[i][2] = qr.z; qn[i][3] = qr.w;
    kn[i][0] = kr.x; kn[i][1] = kr.y; kn[i][2] = kr.z; kn[i][3] = kr.w;
  }
  {
    // squared norms: each half row is one ascending chain of 32 terms, handed from lane to lane; then the two halves are added
    float sq[4] = {0.f, 0.f, 0.f, 0.f}, sk[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int step = 0; step < 4; ++step) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (step > 0) {
          const float uq = __shfl_up_sync(0xffffffffu, sq[i], 1), uk = __shfl_up_sync(0xffffffffu, sk[i], 1);
          if ((tid & 3) == step) { sq[i] = uq; sk[i] = uk; }
        }
        if ((tid & 3) == step) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            sq[i] = fmaf(lo_f(qn[i][j]), lo_f(qn[i][j]), sq[i]); sq[i] = fmaf(hi_f(qn[i][j]), hi_f(qn[i][j]), sq[i]);
            sk[i] = fmaf(lo_f(kn[i][j]), lo_f(kn[i][j]), sk[i]); sk[i] = fmaf(hi_f(kn[i][j]), hi_f(kn[i][j]), sk[i]);
          }
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float a = __shfl_sync(0xffffffffu, sq[i], (tid & 31) | 3), d = __shfl_sync(0xffffffffu, sk[i], (tid & 31) | 3);
      a += __shfl_xor_sync(0xffffffffu, a, 4);
      d += __shfl_xor_sync(0xffffffffu, d, 4);
      const float rq = rsqrtf(a + 1e-6f) * 0.125f, rk = rsqrtf(d + 1e-6f);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        qn[i][j] = pack_f2(lo_f(qn[i][j]) * rq, hi_f(qn[i][j]) * rq);
        kn[i][j] = pack_f2(lo_f(kn[i][j]) * rk, hi_f(kn[i][j]) * rk);
      }
      const int at = (tok_t + 16 * i) * LDS + piece;
      *reinterpret_cast<uint4*>(Qn + at) = make_uint4(qn[i][0], qn[i][1], qn[i][2], qn[i][3]);
      *reinterpret_cast<uint4*>(Kn + at) = make_uint4(kn[i][0], kn[i][1], kn[i][2], kn[i][3]);
    }
  }
  __syncthreads();
  auto scaled = [](const uint32_t (&x)[4], float s) {
    return make_uint4(pack_f2(lo_f(x[0]) * s, hi_f(x[0]) * s), pack_f2(lo_f(x[1]) * s, hi_f(x[1]) * s),
                      pack_f2(lo_f(x[2]) * s, hi_f(x[2]) * s), pack_f2(lo_f(x[3]) * s, hi_f(x[3]) * s));
  };
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    // qg, kg to global memory; KBG and VB to shared memory
    const int tok = tok_t + 16 * i;
    const float E = eg[tok], bt = bet[tok];
    const uint32_t vw[4] = {vr[i].x, vr[i].y, vr[i].z, vr[i].w};
    *reinterpret_cast<uint4*>(qg_out + tile_off + tok * 64 + piece) = scaled(qn[i], E);
    *reinterpret_cast<uint4*>(kg_out + tile_off + tok * 64 + piece) = scaled(kn[i], el[tok]);
    *reinterpret_cast<uint4*>(KBG + tok * LDS + piece) = scaled(kn[i], bt * E);
    *reinterpret_cast<uint4*>(VB + tok * LDS + piece) = scaled(vw, bt);
  }
  if (tid < 64) gc_out[((long long)bh * NT + c) * 64 + tid] = gc[tid];
  const int r0 = 16 * warp + (lane >> 2), cq = 2 * (lane & 3);
  float acc[8][4], kk[8][4];
  {
    const float glo = gc[r0], ghi = gc[r0 + 8], blo = bet[r0], bhi = bet[r0 + 8];
    zero_acc(kk);
    mma64<false, true>(Kn, Kn, kk, warp, lane);                        // k_i . k_j
    zero_acc(acc);
    mma64<false, true>(Qn, Kn, acc, warp, lane);                       // q_i . k_j
    __syncthreads();                                                   // Qn and Kn are used up
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
      const int cc = 8 * nt + cq;
      const float2 gj = *reinterpret_cast<const float2*>(gc + cc);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int row = r0 + 8 * (e >> 1), cl = cc + (e & 1);
        const float gam = __expf((e >> 1 ? ghi : glo) - (e & 1 ? gj.y : gj.x));
        kk[nt][e] = cl < row ? (e >> 1 ? bhi : blo) * kk[nt][e] * gam : 0.f;
        acc[nt][e] = cl <= row ? acc[nt][e] * gam : 0.f;
      }
      *reinterpret_cast<float2*>(L + r0 * LD + cc) = make_float2(kk[nt][0], kk[nt][1]);
      *reinterpret_cast<float2*>(L + (r0 + 8) * LD + cc) = make_float2(kk[nt][2], kk[nt][3]);
    }
    acc_to_smem(acc, Tm, warp, lane);                                  // P, on its way to global memory
  }
  auto store_tile = [&](const bf16* tile, bf16* dst) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int row = tok_t + 16 * i;
      *reinterpret_cast<uint4*>(dst + row * 64 + piece) = *reinterpret_cast<const uint4*>(tile + row * LDS + piece);
    }
  };
  __syncthreads();                                                     // L and P complete
  store_tile(Tm, P_out + tile_off);
  __syncthreads();                                                     // P has left Tm
  {
    // rows 8 t + r minus block s of the finished rows, for columns lane (and lane + 32)
    auto update = [&](auto& a, int t, int sblk) {
      constexpr int NC = sizeof(a) / sizeof(a[0]);
      float x[NC][8];
#pragma unroll
      for (int j = 0; j < 8; ++j)
#pragma unroll
        for (int n = 0; n < NC; ++n) x[n][j] = L[(8 * sblk + j) * LD + 32 * n + lane];
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const float4 l0 = *reinterpret_cast<const float4*>(L + (8 * t + r) * LD + 8 * sblk), l1 = *reinterpret_cast<const float4*>(L + (8 * t + r) * LD + 8 * sblk + 4);
#pragma unroll
        for (int n = 0; n < NC; ++n) {
          a[n][r][0] -= l0.x * x[n][0]; a[n][r][1] -= l0.y * x[n][1]; a[n][r][2] -= l0.z * x[n][2]; a[n][r][3] -= l0.w * x[n][3];
          a[n][r][0] -= l1.x * x[n][4]; a[n][r][1] -= l1.y * x[n][5]; a[n][r][2] -= l1.z * x[n][6]; a[n][r][3] -= l1.w * x[n][7];
        }
      }
    };
    // the block's own triangle; its rows replace L's, which nobody reads any more
    auto solve = [&](auto& a, int t) {
      constexpr int NC = sizeof(a) / sizeof(a[0]);
      float x[NC][8];
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const float4 l0 = *reinterpret_cast<const float4*>(L + (8 * t + r) * LD + 8 * t), l1 = *reinterpret_cast<const float4*>(L + (8 * t + r) * LD + 8 * t + 4);
        const float l[8] = {l0.x, l0.y, l0.z, l0.w, l1.x, l1.y, l1.z, l1.w};
#pragma unroll
        for (int n = 0; n < NC; ++n) {
#pragma unroll
          for (int j = 0; j < r; ++j) a[n][r][j & 3] -= l[j] * x[n][j];
          x[n][r] = (a[n][r][0] + a[n][r][1]) + (a[n][r][2] + a[n][r][3]);
        }
      }
      __syncwarp();                                                    // every lane has read the rows
#pragma unroll
      for (int r = 0; r < 8; ++r) {
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          if (n < NC) L[(8 * t + r) * LD + 32 * n + lane] = x[n < NC ? n : 0][r];
          Tm[(8 * t + r) * LDS + 32 * n + lane] = __float2bfloat16_rn(n < NC ? x[n < NC ? n : 0][r] : 0.f);
        }
      }
    };
    float low[1][8][4], high[2][8][4];                                 // chains of block `warp` (columns 0..31) and block `warp + 4` (both halves)
#pragma unroll
    for (int r = 0; r < 8; ++r) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        low[0][r][e] = e == 0 && 8 * warp + r == lane ? 1.f : 0.f;
        high[0][r][e] = 0.f;
        high[1][r][e] = low[0][r][e];
      }
    }
#pragma unroll 1
    for (int sblk = 0; sblk < 4; ++sblk) {
      if (warp == sblk) solve(low, sblk);
      __syncthreads();
      if (warp > sblk) update(low, warp, sblk);
      update(reinterpret_cast<float(&)[1][8][4]>(high), warp + 4, sblk);        // columns 32..63 of the first half are zero
    }
#pragma unroll 1
    for (int sblk = 4; sblk < 8; ++sblk) {
      if (warp == sblk - 4) solve(high, sblk);
      __syncthreads();
      if (warp > sblk - 4) update(high, warp + 4, sblk);
    }
  }
  __syncthreads();
  if (Tm_out != nullptr) store_tile(Tm, Tm_out + tile_off);
  zero_acc(acc);
  mma64<false, false>(Tm, KBG, acc, warp, lane);
  acc_to_smem(acc, Qn, warp, lane);
  zero_acc(acc);
  mma64<false, false>(Tm, VB, acc, warp, lane);
  acc_to_smem(acc, Kn, warp, lane);
  __syncthreads();
  store_tile(Qn, w_out + tile_off);
  store_tile(Kn, u_out + tile_off);
}

// Gradients of the chunk operands and of everything the preparation computed, chunk-parallel.  One CTA of eight warps per (chunk,
// batch, key head), looping over the value heads that share the key head so dq/dk need no atomics.
//
// From the reverse scan (dv_new = du and the state gradient dS' at the chunk's end) it forms
//     dw = -du S^T    dP = dO v_new^T    dqg = dO S^T    dkg = v_new dS'^T
// and with A = Tm^T dw = d(beta e^gc k), B = Tm^T du = d(beta v) the gradient of the triangular system is dM = -(A w^T + B u^T),
// because Tm (beta e^gc k) and Tm (beta v) are w and u themselves: two independent products instead of a chain of four.
// The gate and beta gradients are sums over rows and columns of products such as dP_ij Gamma_ij (q_i.k_j); with H = dP Gamma they equal
// q_i.(H K)_i and k_j.(H^T Q)_j, row dots of products that dq and dk need anyway, so q.k is not formed again (k.k is, for beta's own sum) and
// every row sum stays in two registers per thread until the end of the head.  H and beta dL Gamma are rounded to bf16 on the way, where dP and the
// factors of dM were; the sums cancel pairwise between rows and columns, since both sides read the same rounded tile.  Against 64 bits the
// gate gradient is 3 % closer in the mean than with fp32 sums over the tiles of the earlier pass (12 inputs; two of them 4 % further).
// Bound by the shared-memory round trips of its thirteen 64^3 products, most of them dependent (70 % of that pipe); eight warps with
// half-width accumulators and two CTAs per SM (at most 128 registers, 112 KB of tiles) hide part of them, and the next head's eight tiles load while this head's last
// products run.  5376 chunks: 230 us; the kernel that took dw, dP, dqg, dkg from the scan, four warps and sixteen row or column sums, 337.
__global__ void __launch_bounds__(256, 2) gdn_prep_bwd_kernel(const bf16* __restrict__ q, const bf16* __restrict__ k, const bf16* __restrict__ v,
                                                              const float* __restrict__ g, const bf16* __restrict__ beta, const bf16* __restrict__ Tm_in,
                                                              const bf16* __restrict__ w_in, const bf16* __restrict__ u_in, const bf16* __restrict__ vnew,
                                                              const bf16* __restrict__ states, const bf16* __restrict__ dout, const bf16* __restrict__ du,
                                                              const bf16* __restrict__ dstate, const float* __restrict__ dd,
                                                              bf16* __restrict__ dq, bf16* __restrict__ dk, bf16* __restrict__ dv,
                                                              float* __restrict__ dg, float* __restrict__ dbeta, int S, int Hk, int Hv,
                                                              long long qk_ld, long long v_ld, long long dqk_ld, long long dv_ld) {
  grid_wait();
  extern __shared__ __align__(16) uint8_t smem_bytes[];
  bf16* sm = reinterpret_cast<bf16*>(smem_bytes);
  bf16 *Qn = sm, *Kn = sm + TILE_ELEMS, *St = sm + 2 * TILE_ELEMS, *Do = sm + 3 * TILE_ELEMS, *Vn = sm + 4 * TILE_ELEMS, *Ds = sm + 5 * TILE_ELEMS;
  bf16 *Du = sm + 6 * TILE_ELEMS, *Tm = sm + 7 * TILE_ELEMS, *Wt = sm + 8 * TILE_ELEMS, *Ut = sm + 9 * TILE_ELEMS, *X1 = sm + 10 * TILE_ELEMS, *X2 = sm + 11 * TILE_ELEMS;
  float* fl = reinterpret_cast<float*>(sm + 12 * TILE_ELEMS);
  float *gc = fl, *bet = fl + 64, *eg = fl + 128, *el = fl + 192, *rqs = fl + 256, *rks = fl + 320;
  float *redg = fl + 384, *redb = fl + 512;                  // [2 column halves][64 rows]
  float* redk = fl + 640;                                    // [8 warps]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int c = blockIdx.x, NT = gridDim.x, rep = Hv / Hk;
  const int b = blockIdx.y / Hk, hk = blockIdx.y % Hk;
  const long long tok0 = (long long)b * S + (long long)c * 64;
  const int r0 = 16 * (warp & 3) + (lane >> 2), ch = warp >> 2, c0 = 32 * ch + 2 * (lane & 3);
  auto load_head = [&](int hv) {
    const long long off = ((long long)(b * Hv + hv) * NT + c) * 4096;
    load_tile_async_256(St, states + off, 64, tid);
    load_tile_async_256(Do, dout + (tok0 * Hv + hv) * 64, (long long)Hv * 64, tid);
    load_tile_async_256(Vn, vnew + off, 64, tid);
    load_tile_async_256(Ds, dstate + off, 64, tid);
    load_tile_async_256(Du, du + off, 64, tid);
    cp_async_commit();
    load_tile_async_256(Tm, Tm_in + off, 64, tid);
    load_tile_async_256(Wt, w_in + off, 64, tid);
    load_tile_async_256(Ut, u_in + off, 64, tid);
    cp_async_commit();
  };
  // gates of one head: two log decays per lane of warp 0, one beta per thread of warps 1 and 2
  float g0 = 0.f, g1 = 0.f;
  auto fetch_gates = [&](int hv) {
    if (tid < 32) { g0 = g[(tok0 + 2 * tid) * Hv + hv]; g1 = g[(tok0 + 2 * tid + 1) * Hv + hv]; }
    else if (tid < 96) g0 = __bfloat162float(beta[(tok0 + tid - 32) * Hv + hv]);
  };
  load_head(hk * rep);
  fetch_gates(hk * rep);
  {
    // normalised q and k rows: four threads per token
    const int tok = tid >> 2, part = tid & 3;
    const long long src = (tok0 + tok) * qk_ld + hk * 64 + part * 16;
    float qv[16], kv[16], sq = 0.f, sk = 0.f;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const uint4 rawq = reinterpret_cast<const uint4*>(q + src)[i], rawk = reinterpret_cast<const uint4*>(k + src)[i];
      const uint32_t wq[4] = {rawq.x, rawq.y, rawq.z, rawq.w}, wk[4] = {rawk.x, rawk.y, rawk.z, rawk.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        qv[8 * i + 2 * j] = lo_f(wq[j]); qv[8 * i + 2 * j + 1] = hi_f(wq[j]);
        kv[8 * i + 2 * j] = lo_f(wk[j]); kv[8 * i + 2 * j + 1] = hi_f(wk[j]);
      }
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) { sq += qv[i] * qv[i]; sk += kv[i] * kv[i]; }
    sq += __shfl_xor_sync(0xffffffffu, sq, 1); sq += __shfl_xor_sync(0xffffffffu, sq, 2);
    sk += __shfl_xor_sync(0xffffffffu, sk, 1); sk += __shfl_xor_sync(0xffffffffu, sk, 2);
    const float rq = rsqrtf(sq + 1e-6f), rk = rsqrtf(sk + 1e-6f);
    if (part == 0) { rqs[tok] = rq; rks[tok] = rk; }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      *reinterpret_cast<uint32_t*>(Qn + tok * LDS + part * 16 + 2 * i) = pack_f2(qv[2 * i] * (rq * 0.125f), qv[2 * i + 1] * (rq * 0.125f));
      *reinterpret_cast<uint32_t*>(Kn + tok * LDS + part * 16 + 2 * i) = pack_f2(kv[2 * i] * rk, kv[2 * i + 1] * rk);
    }
  }
  float dQn[4][4], dKn[4][4];
  zero_acc(dQn);
  zero_acc(dKn);
  // row dot of a half-width accumulator with a tile, added to the two per-row registers
  auto row_dot = [&](const float (&acc)[4][4], const bf16* tile, float& lo, float& hi) {
    lo = hi = 0.f;
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
      const uint32_t x = *reinterpret_cast<const uint32_t*>(tile + r0 * LDS + 8 * nt + c0), y = *reinterpret_cast<const uint32_t*>(tile + (r0 + 8) * LDS + 8 * nt + c0);
      lo += acc[nt][0] * lo_f(x) + acc[nt][1] * hi_f(x);
      hi += acc[nt][2] * lo_f(y) + acc[nt][3] * hi_f(y);
    }
  };
  auto add_rows = [&](float (&dst)[4][4], const float (&acc)[4][4], float slo, float shi) {
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) { dst[nt][0] += slo * acc[nt][0]; dst[nt][1] += slo * acc[nt][1]; dst[nt][2] += shi * acc[nt][2]; dst[nt][3] += shi * acc[nt][3]; }
  };
  for (int r = 0; r < rep; ++r) {
    const int hv = hk * rep + r, bh = b * Hv + hv;
    if (tid < 32) {
      float run = g0 + g1;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) { const float up = __shfl_up_sync(0xffffffffu, run, o); if (tid >= o) run += up; }
      const float last = __shfl_sync(0xffffffffu, run, 31), first = run - g1;
      gc[2 * tid] = first; gc[2 * tid + 1] = run;
      eg[2 * tid] = __expf(first); eg[2 * tid + 1] = __expf(run);
      el[2 * tid] = __expf(last - first); el[2 * tid + 1] = __expf(last - run);
    } else if (tid < 96) {
      bet[tid - 32] = g0;
    }
    uint32_t vv[4][2];                                       // this thread's fragment of v
    const bf16* vsrc = v + tok0 * v_ld + hv * 64;
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
      vv[nt][0] = *reinterpret_cast<const uint32_t*>(vsrc + (long long)r0 * v_ld + 8 * nt + c0);
      vv[nt][1] = *reinterpret_cast<const uint32_t*>(vsrc + (long long)(r0 + 8) * v_ld + 8 * nt + c0);
    }
    if (r + 1 < rep) fetch_gates(hv + 1);
    cp_async_wait<1>();
    __syncthreads();                                         // gates and the first five tiles (and, the first time, Qn and Kn)
    const float glo = gc[r0], ghi = gc[r0 + 8], blo = bet[r0], bhi = bet[r0 + 8], elo = eg[r0], ehi = eg[r0 + 8];
    float dglo = 0.f, dghi = 0.f, dblo = 0.f, dbhi = 0.f, ksum = 0.f, lo, hi;
    float acc[4][4];
    // ---- dw = -du S^T ----
    zero_acc(acc);
    mma64h<false, true>(Du, St, acc, warp, lane);
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) { acc[nt][0] = -acc[nt][0]; acc[nt][1] = -acc[nt][1]; acc[nt][2] = -acc[nt][2]; acc[nt][3] = -acc[nt][3]; }
    acc_to_smem_h(acc, X1, warp, lane);
    // ---- H = dP Gamma on and below the diagonal, dP = dO v_new^T ----
    zero_acc(acc);
    mma64h<false, true>(Do, Vn, acc, warp, lane);
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int row = r0 + 8 * (e >> 1), cc = 8 * nt + c0 + (e & 1);
        acc[nt][e] = cc <= row ? acc[nt][e] * __expf((e >> 1 ? ghi : glo) - gc[cc]) : 0.f;
      }
    }
    acc_to_smem_h(acc, X2, warp, lane);
    // ---- qg = qn e^gc ; dqg = dO S^T ----
    zero_acc(acc);
    mma64h<false, true>(Do, St, acc, warp, lane);
    add_rows(dQn, acc, elo, ehi);
    row_dot(acc, Qn, lo, hi);
    dglo += lo * elo; dghi += hi * ehi;
    // ---- kg = kn e^(gl - gc) ; dkg = v_new dS'^T ----
    zero_acc(acc);
    mma64h<false, true>(Vn, Ds, acc, warp, lane);
    {
      const float flo = el[r0], fhi = el[r0 + 8];
      add_rows(dKn, acc, flo, fhi);
      row_dot(acc, Kn, lo, hi);
      lo *= flo; hi *= fhi;
      dglo -= lo; dghi -= hi;
      ksum = lo + hi;
    }
    cp_async_wait<0>();
    __syncthreads();                                         // X1, X2 complete, Tm / w / u landed; St, Do, Vn, Ds are free
    // ---- A = Tm^T dw, the gradient of beta e^gc kn ----
    zero_acc(acc);
    mma64h<true, false>(Tm, X1, acc, warp, lane);
    acc_to_smem_h(acc, St, warp, lane);
    add_rows(dKn, acc, blo * elo, bhi * ehi);
    row_dot(acc, Kn, lo, hi);
    lo *= elo; hi *= ehi;
    dblo += lo; dbhi += hi;
    dglo += lo * blo; dghi += hi * bhi;
    // ---- B = Tm^T du, the gradient of beta v ----
    zero_acc(acc);
    mma64h<true, false>(Tm, Du, acc, warp, lane);
    acc_to_smem_h(acc, Do, warp, lane);
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
      dblo += acc[nt][0] * lo_f(vv[nt][0]) + acc[nt][1] * hi_f(vv[nt][0]);
      dbhi += acc[nt][2] * lo_f(vv[nt][1]) + acc[nt][3] * hi_f(vv[nt][1]);
      acc[nt][0] *= blo; acc[nt][1] *= blo; acc[nt][2] *= bhi; acc[nt][3] *= bhi;
    }
    acc_to_smem_h(acc, Vn, warp, lane);                      // dv, on its way to global memory
    // ---- P: dqn += H Kn, dkn += H^T Qn ----
    zero_acc(acc);
    mma64h<false, false>(X2, Kn, acc, warp, lane);
    add_rows(dQn, acc, 1.f, 1.f);
    row_dot(acc, Qn, lo, hi);
    dglo += lo; dghi += hi;
    zero_acc(acc);
    mma64h<true, false>(X2, Qn, acc, warp, lane);
    add_rows(dKn, acc, 1.f, 1.f);
    row_dot(acc, Kn, lo, hi);
    dglo -= lo; dghi -= hi;
    __syncthreads();                                         // A, B and dv complete; X1, X2 are free
    {
      bf16* dvdst = dv + tok0 * dv_ld + hv * 64;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int chunk = tid + 256 * i, row = chunk >> 3, col = (chunk & 7) * 8;
        *reinterpret_cast<uint4*>(dvdst + (long long)row * dv_ld + col) = *reinterpret_cast<const uint4*>(Vn + row * LDS + col);
      }
    }
    // ---- dM = -(A w^T + B u^T); L_ij = beta_i (kn_i.kn_j) Gamma_ij (j < i) ----
    // beta's own gradient, sum_j dL_ij (kn_i.kn_j) Gamma_ij, is taken from the fp32 fragments.  (As a row dot with the rounded tile, like the gates,
    // it would need a division by beta and came out 0.3 to 0.9 % further from the 64-bit gradient.)
    float kk[4][4];
    {
      uint32_t ak[4][4];
      load_a(Kn, ak, warp & 3, lane);
      zero_acc(kk);
      mma_rows<true, 4, 4>(ak, Kn + 32 * ch * LDS, kk, lane);
    }
    zero_acc(acc);
    mma64h<false, true>(St, Wt, acc, warp, lane);
    mma64h<false, true>(Do, Ut, acc, warp, lane);
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int row = r0 + 8 * (e >> 1), cc = 8 * nt + c0 + (e & 1);
        const float dl = cc < row ? -acc[nt][e] * __expf((e >> 1 ? ghi : glo) - gc[cc]) : 0.f;
        (e >> 1 ? dbhi : dblo) += dl * kk[nt][e];
        acc[nt][e] = dl * (e >> 1 ? bhi : blo);
      }
    }
    acc_to_smem_h(acc, X1, warp, lane);
    __syncthreads();                                         // X1 complete; every loaded tile is free
    if (r + 1 < rep) load_head(hv + 1);
    zero_acc(acc);
    mma64h<false, false>(X1, Kn, acc, warp, lane);           // dA1 Kn
    add_rows(dKn, acc, 1.f, 1.f);
    row_dot(acc, Kn, lo, hi);
    dglo += lo; dghi += hi;
    zero_acc(acc);
    mma64h<true, false>(X1, Kn, acc, warp, lane);            // dA1^T Kn
    add_rows(dKn, acc, 1.f, 1.f);
    row_dot(acc, Kn, lo, hi);
    dglo -= lo; dghi -= hi;
    // ---- gates out: dg = reverse cumsum of dgc (gc_last also collects kg's row sums and the carry term) ----
    auto quad = [](float x) { x += __shfl_xor_sync(0xffffffffu, x, 1); return x + __shfl_xor_sync(0xffffffffu, x, 2); };
    dglo = quad(dglo); dghi = quad(dghi); dblo = quad(dblo); dbhi = quad(dbhi);
    ksum = warp_sum(ksum);
    if ((lane & 3) == 0) {
      redg[64 * ch + r0] = dglo; redg[64 * ch + r0 + 8] = dghi;
      redb[64 * ch + r0] = dblo; redb[64 * ch + r0 + 8] = dbhi;
    }
    if (lane == 0) redk[warp] = ksum;
    __syncthreads();
    if (tid < 32) {
      float d0 = redg[2 * tid] + redg[64 + 2 * tid], d1 = redg[2 * tid + 1] + redg[65 + 2 * tid];
      const float4 p = reinterpret_cast<const float4*>(dd)[(long long)bh * NT + c];
      if (tid == 31) {
        float gl = ((p.x + p.y) + (p.z + p.w)) * eg[63];
        for (int i = 0; i < 8; ++i) gl += redk[i];
        d1 += gl;
      }
      float run = d0 + d1;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) { const float dn = __shfl_down_sync(0xffffffffu, run, o); if (tid + o < 32) run += dn; }
      dg[(tok0 + 2 * tid) * Hv + hv] = run;
      dg[(tok0 + 2 * tid + 1) * Hv + hv] = run - d0;
    } else if (tid < 96) {
      dbeta[(tok0 + tid - 32) * Hv + hv] = redb[tid - 32] + redb[32 + tid];
    }
    __syncthreads();                                         // the gate arrays may be replaced
  }
  // ---- L2-norm backward: qn = 0.125 rq q, kn = rk k ----
  {
    float qh[4][4], kh[4][4], dotq[2] = {0.f, 0.f}, dotk[2] = {0.f, 0.f};
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int row = r0 + 8 * half;
      const long long src = (tok0 + row) * qk_ld + hk * 64 + c0;
      const float rq = rqs[row], rk = rks[row];
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) {
        const uint32_t qq = *reinterpret_cast<const uint32_t*>(q + src + 8 * nt), kk = *reinterpret_cast<const uint32_t*>(k + src + 8 * nt);
        qh[nt][2 * half] = lo_f(qq) * rq; qh[nt][2 * half + 1] = hi_f(qq) * rq;
        kh[nt][2 * half] = lo_f(kk) * rk; kh[nt][2 * half + 1] = hi_f(kk) * rk;
        dotq[half] += 0.125f * (dQn[nt][2 * half] * qh[nt][2 * half] + dQn[nt][2 * half + 1] * qh[nt][2 * half + 1]);
        dotk[half] += dKn[nt][2 * half] * kh[nt][2 * half] + dKn[nt][2 * half + 1] * kh[nt][2 * half + 1];
      }
      dotq[half] += __shfl_xor_sync(0xffffffffu, dotq[half], 1); dotq[half] += __shfl_xor_sync(0xffffffffu, dotq[half], 2);
      dotk[half] += __shfl_xor_sync(0xffffffffu, dotk[half], 1); dotk[half] += __shfl_xor_sync(0xffffffffu, dotk[half], 2);
      if ((lane & 3) == 0) { redg[64 * ch + row] = dotq[half]; redb[64 * ch + row] = dotk[half]; }
    }
    __syncthreads();
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int row = r0 + 8 * half;
      const float rq = rqs[row], rk = rks[row], sq = redg[row] + redg[64 + row], sk = redb[row] + redb[64 + row];
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) {
        *reinterpret_cast<uint32_t*>(X1 + row * LDS + 8 * nt + c0) =
            pack_f2(rq * (0.125f * dQn[nt][2 * half] - qh[nt][2 * half] * sq), rq * (0.125f * dQn[nt][2 * half + 1] - qh[nt][2 * half + 1] * sq));
        *reinterpret_cast<uint32_t*>(X2 + row * LDS + 8 * nt + c0) =
            pack_f2(rk * (dKn[nt][2 * half] - kh[nt][2 * half] * sk), rk * (dKn[nt][2 * half + 1] - kh[nt][2 * half + 1] * sk));
      }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int chunk = tid + 256 * i, row = chunk >> 3, col = (chunk & 7) * 8;
      const long long dst = (tok0 + row) * dqk_ld + hk * 64 + col;
      *reinterpret_cast<uint4*>(dq + dst) = *reinterpret_cast<const uint4*>(X1 + row * LDS + col);
      *reinterpret_cast<uint4*>(dk + dst) = *reinterpret_cast<const uint4*>(X2 + row * LDS + col);
    }
  }
}

// ---- host ----------------------------------------------------------------------------------------------------------------
// Returns {w, u, P, qg, kg, Tm (bf16 tiles [B*Hv,NT,64,64]; Tm empty without `save`), carry [B*Hv,NT] fp32, gc [B*Hv,NT,64] fp32}
std::vector<at::Tensor> gdn_prep_fwd(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& g, const at::Tensor& beta, bool save) {
  auto token_major = [](const at::Tensor& t) {
    return t.dim() == 4 && t.size(3) == 64 && t.stride(3) == 1 && t.stride(2) == 64 && t.stride(0) == t.size(1) * t.stride(1) && t.stride(1) % 8 == 0 &&
           (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0;
  };
  TORCH_CHECK(q.is_cuda() && q.scalar_type() == at::kBFloat16 && token_major(q) && token_major(k) && token_major(v) && q.stride(1) == k.stride(1),
              "gdn_prep_fwd: bf16 [B,S,H,64] tensors with contiguous heads and a common token stride required (views of a packed qkv tensor are fine)");
  TORCH_CHECK(g.scalar_type() == at::kFloat && g.is_contiguous() && beta.scalar_type() == at::kBFloat16 && beta.is_contiguous(), "gdn_prep_fwd: g fp32 / beta bf16 [B,S,Hv]");
  const c10::cuda::CUDAGuard guard(q.device());
  const int64_t B = q.size(0), S = q.size(1), Hk = q.size(2), Hv = v.size(2);
  TORCH_CHECK(S % 64 == 0 && Hv % Hk == 0, "gdn_prep_fwd: sequence must be a multiple of 64 and value heads a multiple of key heads");
  const int64_t NT = S / 64, BH = B * Hv;
  auto opts = q.options();
  std::vector<at::Tensor> out;
  for (int i = 0; i < 5; ++i) out.push_back(at::empty({BH, NT, 64, 64}, opts));
  out.push_back(save ? at::empty({BH, NT, 64, 64}, opts) : at::empty({0}, opts));
  out.push_back(at::empty({BH, NT}, opts.dtype(at::kFloat)));
  out.push_back(at::empty({BH, NT, 64}, opts.dtype(at::kFloat)));
  constexpr int smem = 5 * TILE_ELEMS * 2 + 256 * 4;
  static bool configured = false;
  if (!configured) { C10_CUDA_CHECK(cudaFuncSetAttribute(gdn_prep_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)); configured = true; }
  launch(gdn_prep_fwd_kernel, dim3((int)NT, (int)BH), 128, smem, at::cuda::getCurrentCUDAStream(), 
      (const bf16*)q.data_ptr(), (const bf16*)k.data_ptr(), (const bf16*)v.data_ptr(), g.data_ptr<float>(), (const bf16*)beta.data_ptr(),
      (bf16*)out[0].data_ptr(), (bf16*)out[1].data_ptr(), (bf16*)out[2].data_ptr(), (bf16*)out[3].data_ptr(), (bf16*)out[4].data_ptr(),
      save ? (bf16*)out[5].data_ptr() : nullptr, out[6].data_ptr<float>(), out[7].data_ptr<float>(), (int)S, (int)Hk, (int)Hv, (long long)q.stride(1), (long long)v.stride(1));
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  count_launch();
  return out;
}

// Returns {dqkv packed bf16 [B,S,(2 Hk + Hv) 64] holding dq | dk | dv per token, dg, dbeta (fp32 [B,S,Hv])}
std::vector<at::Tensor> gdn_prep_bwd(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& g, const at::Tensor& beta,
                                     const at::Tensor& Tm, const at::Tensor& w, const at::Tensor& u, const at::Tensor& vnew, const at::Tensor& states,
                                     const at::Tensor& dout, const at::Tensor& du, const at::Tensor& dstate, const at::Tensor& dd) {
  const c10::cuda::CUDAGuard guard(q.device());
  const int64_t B = q.size(0), S = q.size(1), Hk = q.size(2), Hv = v.size(2), NT = S / 64, BH = B * Hv;
  check_tiles(Tm, BH, NT, "Tm"); check_tiles(w, BH, NT, "w"); check_tiles(u, BH, NT, "u"); check_tiles(vnew, BH, NT, "vnew");
  check_tiles(states, BH, NT, "states"); check_tiles(dout, BH, NT, "do"); check_tiles(du, BH, NT, "du"); check_tiles(dstate, BH, NT, "dstate");
  TORCH_CHECK(dd.scalar_type() == at::kFloat && dd.is_contiguous() && dd.numel() == BH * NT * 4, "gdn_prep_bwd: dd must be fp32 [BH,NT,4]");
  TORCH_CHECK(q.stride(1) == k.stride(1) && q.stride(1) % 8 == 0 && v.stride(1) % 2 == 0, "gdn_prep_bwd: q, k, v must be the strided views the forward took");
  const int64_t packed = (2 * Hk + Hv) * 64;
  auto dqkv = at::empty({B, S, packed}, q.options());
  bf16* dq_ptr = (bf16*)dqkv.data_ptr();
  bf16* dk_ptr = dq_ptr + Hk * 64;
  bf16* dv_ptr = dq_ptr + 2 * Hk * 64;
  auto dg = at::empty({B, S, Hv}, q.options().dtype(at::kFloat)), dbeta = at::empty({B, S, Hv}, q.options().dtype(at::kFloat));
  constexpr int smem = 12 * TILE_ELEMS * 2 + 648 * 4;
  static bool configured = false;
  if (!configured) { C10_CUDA_CHECK(cudaFuncSetAttribute(gdn_prep_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)); configured = true; }
  launch(gdn_prep_bwd_kernel, dim3((int)NT, (int)(B * Hk)), 256, smem, at::cuda::getCurrentCUDAStream(), 
      (const bf16*)q.data_ptr(), (const bf16*)k.data_ptr(), (const bf16*)v.data_ptr(), g.data_ptr<float>(), (const bf16*)beta.data_ptr(),
      (const bf16*)Tm.data_ptr(), (const bf16*)w.data_ptr(), (const bf16*)u.data_ptr(), (const bf16*)vnew.data_ptr(), (const bf16*)states.data_ptr(),
      (const bf16*)dout.data_ptr(), (const bf16*)du.data_ptr(), (const bf16*)dstate.data_ptr(), dd.data_ptr<float>(), dq_ptr, dk_ptr, dv_ptr,
      dg.data_ptr<float>(), dbeta.data_ptr<float>(), (int)S, (int)Hk, (int)Hv, (long long)q.stride(1), (long long)v.stride(1), (long long)packed, (long long)packed);
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  count_launch();
  return {dqkv, dg, dbeta};
}

// The whole rule on a packed ``qkv [B,S,(2 Hk + Hv) 64]`` tensor (q | k | v per token): the strided views are made here, one call per pass.
static std::array<at::Tensor, 3> split_qkv(const at::Tensor& qkv, int64_t Hk, int64_t Hv) {
  TORCH_CHECK(qkv.dim() == 3 && qkv.is_contiguous() && qkv.size(2) == (2 * Hk + Hv) * 64, "gdn_rule: contiguous [B,S,(2 Hk + Hv) 64] required");
  const int64_t B = qkv.size(0), S = qkv.size(1), C = qkv.size(2), at0 = qkv.storage_offset();
  auto heads = [&](int64_t first, int64_t n) { return qkv.as_strided({B, S, n, 64}, {S * C, C, 64, 1}, at0 + first * 64); };
  return {heads(0, Hk), heads(Hk, Hk), heads(2 * Hk, Hv)};
}

// Returns {o, w, u, P, qg, kg, Tm, carry, vnew, states}: the output and what gdn_rule_bwd takes as `saved`.
std::vector<at::Tensor> gdn_rule_fwd(const at::Tensor& qkv, const at::Tensor& g, const at::Tensor& beta, int64_t Hk, int64_t Hv, const c10::optional<at::Tensor>& err, bool save) {
  const auto x = split_qkv(qkv, Hk, Hv);
  auto p = gdn_prep_fwd(x[0], x[1], x[2], g, beta, save);
  auto s = gdn_scan_fwd(p[0], p[1], p[2], p[3], p[4], p[6], qkv.size(0), Hv, err, save);
  return {s[0], p[0], p[1], p[2], p[3], p[4], p[5], p[6], s[1], s[2]};
}

// saved = {w, u, P, qg, kg, Tm, carry, vnew, states}.  Returns {dqkv, dg, dbeta}.
std::vector<at::Tensor> gdn_rule_bwd(const at::Tensor& qkv, const at::Tensor& g, const at::Tensor& beta, at::TensorList saved, const at::Tensor& dout, int64_t Hk, int64_t Hv,
                                     const c10::optional<at::Tensor>& err) {
  TORCH_CHECK(saved.size() == 9, "gdn_rule_bwd: nine saved tensors required");
  const auto x = split_qkv(qkv, Hk, Hv);
  auto c = gdn_chain_bwd(saved[0], saved[2], saved[3], saved[4], saved[6], saved[8], dout, qkv.size(0), Hv, err);
  return gdn_prep_bwd(x[0], x[1], x[2], g, beta, saved[5], saved[0], saved[1], saved[7], saved[8], dout, c[0], c[1], c[2]);
}

}  // namespace q38
