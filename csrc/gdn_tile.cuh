// Pieces of the delta-rule scans in which every warp owns 16 value columns of the state and needs nothing from the other warps.
//
// The recurrence S' = d S + kg^T (u - w S) mixes the rows (key dims) of the state but never its columns, so a warp keeps the
// transposed slice S^T [16 v x 64 k] in its accumulator registers and computes every product transposed:
//     v_new^T = u^T - S^T w^T        o^T = S^T qg^T + v_new^T P^T        S'^T = d S^T + v_new^T kg
// An mma.sync accumulator fragment packed to bf16 is already the A fragment of the next product, so the chain of a chunk has no
// shared-memory round trip and no block barrier; only the four 64x64 operand tiles that the warps share come through shared memory.
#pragma once
#include "mma_tile.cuh"
#include "ptx.cuh"

namespace q38 {
namespace gdn {

constexpr int STAGES = 3, CHAIN_STAGES = 4, SIDE_STAGES = 3, TILE_BYTES = 64 * 128, SLICE_BYTES = 64 * 32;

// acc[16x64] += A[16x64] B[64x64] for one warp, A in registers, B a 64x64 bf16 tile of 128-byte rows with the 128-byte TMA swizzle:
// B(k,n) = TRANS ? tile[k][n] : tile[n][k].  Four warps (of one or several CTAs) make up a 64x64x64 product.
template <bool TRANS>
__device__ __forceinline__ void mma64(const uint32_t (&a)[4][4], uint32_t tile, float (&acc)[8][4], int lane) {
  const int l8 = lane & 7, m = lane >> 3;
  const uint32_t row0 = tile + (TRANS ? l8 + 8 * (m & 1) : l8 + 8 * (m >> 1)) * 128;
  const int half = TRANS ? (m >> 1) : (m & 1);
#pragma unroll
  for (int ks = 0; ks < 4; ++ks) {
#pragma unroll
    for (int np = 0; np < 4; ++np) {
      const uint32_t addr = row0 + 2048 * (TRANS ? ks : np) + (((2 * (TRANS ? np : ks) + half) ^ l8) << 4);
      uint32_t b[4];
      if (TRANS) asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(b[0]), "=r"(b[1]), "=r"(b[2]), "=r"(b[3]) : "r"(addr));
      else asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(b[0]), "=r"(b[1]), "=r"(b[2]), "=r"(b[3]) : "r"(addr));
      mma16816(acc[2 * np], a[ks], b[0], b[1]);
      mma16816(acc[2 * np + 1], a[ks], b[2], b[3]);
    }
  }
}

// A warp's slice of a 64-row operand: 64 rows x 16 columns, 32-byte rows whose two 16-byte halves change places every four rows
// (so that eight consecutive rows of one half cover all banks).
__device__ __forceinline__ uint32_t slice_at(uint32_t base, int row, int half) { return base + row * 32 + ((half ^ ((row >> 2) & 1)) << 4); }

__device__ __forceinline__ void slice_load_async(uint32_t base, const bf16* __restrict__ src, long long ld, int lane) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = (lane >> 1) + 16 * i, half = lane & 1;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(slice_at(base, row, half)), "l"(src + row * ld + 8 * half) : "memory");
  }
}
// Transposed read: A fragments of the [16 x 64] matrix whose columns are the slice's rows.
__device__ __forceinline__ void slice_read_t(uint32_t base, uint32_t (&a)[4][4], int lane) {
  const int l8 = lane & 7, m = lane >> 3;
#pragma unroll
  for (int ks = 0; ks < 4; ++ks)
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(a[ks][0]), "=r"(a[ks][1]), "=r"(a[ks][2]), "=r"(a[ks][3]) : "r"(slice_at(base, 16 * ks + l8 + 8 * (m >> 1), m & 1)) : "memory");
}
// The reverse, through the slice buffer `base` into 16 columns of a row-major matrix (row stride ld): 32 bytes per row.
__device__ __forceinline__ void slice_store_t(uint32_t base, const uint32_t (&a)[4][4], bf16* __restrict__ dst, long long ld, int lane) {
  const int l8 = lane & 7, m = lane >> 3;
  __syncwarp();
#pragma unroll
  for (int ks = 0; ks < 4; ++ks)
    asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1,%2,%3,%4};"
                 ::"r"(slice_at(base, 16 * ks + l8 + 8 * (m >> 1), m & 1)), "r"(a[ks][0]), "r"(a[ks][1]), "r"(a[ks][2]), "r"(a[ks][3]) : "memory");
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = (lane >> 1) + 16 * i, half = lane & 1;
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(slice_at(base, row, half)) : "memory");
    *reinterpret_cast<uint4*>(dst + row * ld + 8 * half) = v;
  }
}

// The four shared operand tiles of the chunk that starts at `row` into one stage.
struct Maps4 { CUtensorMap m[4]; };
__device__ __forceinline__ void load_stage(const Maps4& maps, uint8_t* stage, uint64_t* bar, int row) {
  ptx::mbar_expect_tx(bar, 4 * TILE_BYTES);
#pragma unroll
  for (int t = 0; t < 4; ++t) ptx::tma_load_3d(stage + t * TILE_BYTES, &maps.m[t], bar, 0, row, 0);
}

// Fragments handed from one warp to another through 2 KB of shared memory.
__device__ __forceinline__ void frags_put(uint32_t base, const uint32_t (&a)[4][4], int lane) {
#pragma unroll
  for (int ks = 0; ks < 4; ++ks)
    asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(base + ks * 512 + lane * 16), "r"(a[ks][0]), "r"(a[ks][1]), "r"(a[ks][2]), "r"(a[ks][3]) : "memory");
}
__device__ __forceinline__ void frags_get(uint32_t base, uint32_t (&a)[4][4], int lane) {
#pragma unroll
  for (int ks = 0; ks < 4; ++ks)
    asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(a[ks][0]), "=r"(a[ks][1]), "=r"(a[ks][2]), "=r"(a[ks][3]) : "r"(base + ks * 512 + lane * 16) : "memory");
}

// A ring of N stages of two operand tiles, filled by one thread.
template <int N> struct Ring {
  uint8_t* buf;
  uint64_t *full, *empty;
  __device__ __forceinline__ uint32_t tile(int i) const { return ptx::smem_u32(buf) + (i % N) * 2 * TILE_BYTES; }
  __device__ __forceinline__ void init(int readers) const {
    for (int i = 0; i < N; ++i) { ptx::mbar_init(&full[i], 1); ptx::mbar_init(&empty[i], readers); }
  }
  // Loads chunk `first`, `first + dir`, ... (NT of them) of two maps.  Returns false when a reader never released a stage; either way the copies
  // in flight have landed (or the bounded wait for them has run out) on return.
  __device__ __forceinline__ bool produce(const CUtensorMap* a, const CUtensorMap* b, int first, int NT, int dir) const {
    bool ok = true;
    int c = 0;
    for (; c < NT; ++c) {
      const int s = c % N;
      if (c >= N && !ptx::mbar_wait(&empty[s], ((c / N) & 1) ^ 1)) { ok = false; break; }
      ptx::mbar_expect_tx(&full[s], 2 * TILE_BYTES);
      ptx::tma_load_3d(buf + s * 2 * TILE_BYTES, a, &full[s], 0, (first + dir * c) * 64, 0);
      ptx::tma_load_3d(buf + s * 2 * TILE_BYTES + TILE_BYTES, b, &full[s], 0, (first + dir * c) * 64, 0);
    }
    for (int i = c > N ? c - N : 0; i < c; ++i) ptx::mbar_wait(&full[i % N], (i / N) & 1);
    return ok;
  }
};

// Warps per CTA of the reverse scan over BH (batch, value head) pairs, 4 / warps CTAs per pair.  One warp alone reads all four tiles of a chunk
// from L2 for 16 columns, which pays while every warp has an SM of its own (4 BH <= 148); beyond that two warps share them.
inline int scan_warps(int64_t BH) { return 4 * BH <= kNumSMs ? 1 : 2; }

// Column slices (a chain warp and its output warp each) per CTA of the forward scan: as few as keep every CTA on an SM of its own, because
// the slices of a CTA share its schedulers and MMA pipes, while every further CTA of a pair reads the four operand tiles once more.  Beyond 148
// pairs whole pairs share an SM one after the other (188 KB each): 156 pairs of 64 chunks take 218 us and 296 take 225, where
// the pass with block barriers took 302 and 306; 400 pairs 328 against 454.
inline int scan_pairs(int64_t BH) { return 4 * BH <= kNumSMs ? 1 : 2 * BH <= kNumSMs ? 2 : 4; }

}  // namespace gdn
}  // namespace q38
