// Pieces shared by the attention kernels: TMEM stores, tcgen05.mma with the A operand in TMEM, 4-D tensor maps over
// (head dim, text position, head, text) views with any strides, and the launch arguments.
#pragma once
#include <cuda.h>

#include "attn_api.h"
#include "common.cuh"

namespace mb {

// 32 lanes x 16 consecutive 32-bit TMEM columns to registers and back
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// D[tmem] (+)= A[tmem] * B[smem desc]: A (128 rows = lanes, two bf16 contraction elements per 32-bit column)
__device__ __forceinline__ void umma_bf16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(acc)
      : "memory");
}
__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* m, uint64_t* bar, int c0, int c1, int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}
// The 128-row tiles a CTA works through: every gridDim-th unit.  A unit is one tile, or (`pairs` = ceil(tiles / 2), causal
// attention with more tiles than CTAs) a long tile and the short one that makes every pair the same length: tile x from the end
// and tile x from the start.  Without the pairs a CTA's sum of lengths was left to chance, and the fullest SM had 1.6 times
// the mean (4 x 4096 causal).  Neighbouring units share K and V (or Q and dO) and meet in L2.
struct AttnWalk {
  int u, second, units, tiles, pairs;
  __device__ __forceinline__ AttnWalk(int units_, int tiles_, int pairs_) : u(blockIdx.x), second(0), units(units_), tiles(tiles_), pairs(pairs_) {}
  __device__ __forceinline__ bool valid() const { return u < units; }
  __device__ __forceinline__ int bh() const { return u / (pairs ? pairs : tiles); }
  __device__ __forceinline__ int tile() const {
    const int x = u % (pairs ? pairs : tiles);
    return second ? x : tiles - 1 - x;
  }
  __device__ __forceinline__ void next() {
    if (pairs && !second && 2 * (u % pairs) != tiles - 1) { second = 1; return; }
    second = 0;
    u += gridDim.x;
  }
};
// units, and the size of a pair list (0: single tiles), of a launch with at most `max_ctas` CTAs
inline void attn_units(long long bh, int tiles, bool causal, int max_ctas, int& units, int& pairs) {
  pairs = causal && bh * tiles > max_ctas ? (tiles + 1) / 2 : 0;
  units = (int)(bh * (pairs ? pairs : tiles));
}
// bit j: column col + j lies in [lo, hi]
__device__ __forceinline__ uint32_t seen_bits(int col, int lo, int hi) {
  const int a = lo - col, b = hi - col;                  // visible: a <= j <= b
  uint32_t m = b >= 31 ? 0xffffffffu : (b < 0 ? 0u : (2u << b) - 1u);
  return a <= 0 ? m : (a > 31 ? 0u : m & (0xffffffffu << a));
}
// 2^x on the special-function unit (arguments here are <= 8; results below 2^-126 become 0)
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

}  // namespace mb
