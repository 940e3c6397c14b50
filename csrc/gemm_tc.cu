// tcgen05 GEMM core for sm_100a: C[g] = A[g] * B[g]^T, bf16 operands, fp32 accumulation in tensor memory.
//
// One persistent CTA per SM, warp-specialised:
//   warp 0      TMA producer   (cp.async.bulk.tensor 3-D tiles -> 128B-swizzled shared-memory ring, 4 stages)
//   warp 1      MMA issuer     (one thread issues tcgen05.mma 128x256x16; accumulators double-buffered in TMEM)
//   warps 2..5  epilogue       (tcgen05.ld 32 lanes x 32 columns -> registers -> fused epilogue -> global)
// Operands may be K-major (rows x K, K contiguous) or MN-major (K x rows, rows contiguous), so transposed views of
// row-major tensors (dgrad / wgrad) need no transposing copy.  Batched ("grouped") over a leading dimension through
// 3-D tensor maps: this is how all experts of a MoE layer run in one launch.
// Epilogues: plain store (bf16 or fp32, optional += into fp32), relu^2 (also stores the pre-activation),
// relu^2 backward (acc * 2*relu(aux)), SwiGLU over column halves, per-row scale.
// Every mbarrier wait is bounded; on a timeout the kernel records a code in `status`, drains and returns.
#include <cuda.h>

#include <algorithm>
#include <cstdlib>
#include <stdexcept>
#include <string>
#include <type_traits>

#include "common.cuh"
#include "gemm_api.h"

namespace mb {

constexpr int BM = 128, BN = 256, BK = 64, STAGES = 4, UMMA_K = 16;
constexpr int A_BYTES = BM * BK * 2, B_BYTES = BN * BK * 2, STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int GEMM_THREADS = 192;
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 /*align*/ + 256 /*barriers*/;
constexpr int GROUP_M = 8;
constexpr int MAX_COUNT_G = 128;          // groups whose row tiles are counted in shared memory (more keep the plain order)

struct TmapSet { CUtensorMap m[8]; };

// tile r of a group of m_tiles row tiles, bands of row tiles first
__device__ __forceinline__ void band_coords(int r, int m_tiles, const GemmParams& p, int& mt, int& nt) {
  const int gm = p.group_m > 0 ? p.group_m : GROUP_M;
  int band = gm * p.n_tiles;
  int b = r / band;
  int first_m = b * gm;
  int gsz = min(gm, m_tiles - first_m);
  int rr = r - b * band;
  mt = first_m + rr % gsz;
  nt = rr / gsz;
}

// work item t -> group, row tile, column tile (the items of one output tile's splits are neighbours).
// `cum` (count mode 1): row tiles with rows in the groups before each.  The tiles that are computed come first and those of
// padding rows, which are only cleared, after them, so that every pair gets its share of both: dealt out by position, tiles
// of padding fell to some pairs and not to others (with 7 of 8 row tiles filled, to every second one).
// Us, the four products of 8 experts (2048 wide, hidden 4096) with some 12 000 of 8 x 2561 places filled: 1258 -> 1047.
__device__ __forceinline__ void tile_coords(int t, const GemmParams& p, int& g, int& mt, int& nt, const int* cum = nullptr) {
  if (p.splits > 1) t /= p.splits;
  if (cum != nullptr) {
    const int full = cum[p.G] * p.n_tiles;
    const bool pad = t >= full;
    if (pad) t -= full;
    auto first = [&](int i) { return pad ? i * p.m_tiles - cum[i] : cum[i]; };     // row tiles of this kind before group i
    const int row = t / p.n_tiles;
    int lo = 0, hi = p.G;                                                          // first(lo) <= row < first(hi)
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (first(mid) <= row) lo = mid; else hi = mid;
    }
    g = lo;
    const int have = cum[g + 1] - cum[g];
    band_coords(t - first(g) * p.n_tiles, pad ? p.m_tiles - have : have, p, mt, nt);
    if (pad) mt += have;
    return;
  }
  int per_g = p.m_tiles * p.n_tiles;
  g = t / per_g;
  band_coords(t - g * per_g, p.m_tiles, p, mt, nt);
}

__device__ __forceinline__ float tanh_approx(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// x * sigmoid(x) with sigmoid = (tanh(x / 2) + 1) / 2: one special-function instruction and two FMAs, no division
__device__ __forceinline__ float silu_f(float x) {
  const float h = 0.5f * x;
  return fmaf(h, tanh_approx(h), h);
}
// sigmoid to a few units of fp32's last place wherever it is: the derivative multiplies by it alone, and for a strongly negative
// gate (tanh(x / 2) + 1) / 2 leaves nothing but the rounding of the tanh
__device__ __forceinline__ float sigmoid_f(float x) { return __fdividef(1.f, 1.f + __expf(-x)); }

// Drain one accumulator tile (this warp's 32 TMEM lanes x 256 columns) through the fused epilogue to global memory.
// `row_l` = this thread's row inside M-segment `seg`; `taddr` = TMEM address of the warp's lanes, column 0 of the tile.
__device__ __forceinline__ void epilogue_tile(const GemmParams& p, int g, int seg, int row_l, int nt, uint32_t taddr) {
  const bool row_ok = row_l < p.seg_M;
  const int row = seg * p.seg_M + row_l;                                  // row of the local (M, N) problem
  // where the result goes: the local output, or the buffer of the GPU that owns this segment's tokens
  char* const obase = reinterpret_cast<char*>(p.out_seg_on ? p.out_seg[seg] : p.out);
  const long long orow = p.out_seg_on ? row_l : row;
  const long long og = g + p.out_g_off;
  if (p.epi == EPI_SWIGLU) {
    const int H = p.N >> 1;
#pragma unroll 1
    for (int c = 0; c < 4; ++c) {
      uint32_t rg[32], ru[32];
      __syncwarp();
      tmem_ld32(taddr + c * 32, rg);
      tmem_ld32(taddr + 128 + c * 32, ru);
      tmem_ld_wait();
      const int col0 = nt * 128 + c * 32;
      if (row_ok && col0 < H) {
        bf16* o = reinterpret_cast<bf16*>(obase) + og * p.out_gs + orow * p.ldo + col0;
        bf16* o2 = p.out2 ? reinterpret_cast<bf16*>(p.out2) + g * p.out2_gs + static_cast<long long>(row) * p.ldo2 + col0
                          : nullptr;
        const int nv = min(32, H - col0);
        for (int j = 0; j < nv; ++j) {
          float gg = __uint_as_float(rg[j]), uu = __uint_as_float(ru[j]);
          // operands rounded to bf16 first so forward and the recomputing backward see the same numbers
          float gr = __bfloat162float(__float2bfloat16(gg)), ur = __bfloat162float(__float2bfloat16(uu));
          o[j] = __float2bfloat16(silu_f(gr) * ur);
          if (o2) { o2[j] = __float2bfloat16(gg); o2[H + j] = __float2bfloat16(uu); }
        }
      }
    }
  } else {
#pragma unroll 1
    for (int c = 0; c < BN / 32; ++c) {
      uint32_t r[32];
      __syncwarp();                              // tcgen05.ld is warp-collective: reconverge after the stores
      tmem_ld32(taddr + c * 32, r);
      tmem_ld_wait();
      const int col0 = nt * BN + c * 32;
      if (row_ok && col0 < p.N) {
      const int nv = min(32, p.N - col0);
      float v[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
      if (p.epi == EPI_RELU2) {
        bf16* o2 = reinterpret_cast<bf16*>(p.out2) + g * p.out2_gs + static_cast<long long>(row) * p.ldo2 + col0;
        if (nv == 32) {
          uint4* d4 = reinterpret_cast<uint4*>(o2);
#pragma unroll
          for (int j = 0; j < 4; ++j)
            d4[j] = make_uint4(pack_bf16(v[8 * j], v[8 * j + 1]), pack_bf16(v[8 * j + 2], v[8 * j + 3]),
                               pack_bf16(v[8 * j + 4], v[8 * j + 5]), pack_bf16(v[8 * j + 6], v[8 * j + 7]));
        } else {
          for (int j = 0; j < nv; ++j) o2[j] = __float2bfloat16(v[j]);
        }
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          float a = __bfloat162float(__float2bfloat16(v[j]));     // activation of the stored (rounded) value
          a = fmaxf(a, 0.f);
          v[j] = a * a;
        }
      } else if (p.epi == EPI_DRELU2) {
        const bf16* ax = reinterpret_cast<const bf16*>(p.aux) + g * p.aux_gs + static_cast<long long>(row) * p.ldaux + col0;
        if (nv == 32) {
          const uint4* a4 = reinterpret_cast<const uint4*>(ax);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            uint4 u = a4[j];
            float2 f0 = unpack_bf16(u.x), f1 = unpack_bf16(u.y), f2 = unpack_bf16(u.z), f3 = unpack_bf16(u.w);
            v[8 * j + 0] *= 2.f * fmaxf(f0.x, 0.f); v[8 * j + 1] *= 2.f * fmaxf(f0.y, 0.f);
            v[8 * j + 2] *= 2.f * fmaxf(f1.x, 0.f); v[8 * j + 3] *= 2.f * fmaxf(f1.y, 0.f);
            v[8 * j + 4] *= 2.f * fmaxf(f2.x, 0.f); v[8 * j + 5] *= 2.f * fmaxf(f2.y, 0.f);
            v[8 * j + 6] *= 2.f * fmaxf(f3.x, 0.f); v[8 * j + 7] *= 2.f * fmaxf(f3.y, 0.f);
          }
        } else {
          for (int j = 0; j < nv; ++j) v[j] *= 2.f * fmaxf(__bfloat162float(ax[j]), 0.f);
        }
      } else if (p.epi == EPI_ROWSCALE) {
        const float s = reinterpret_cast<const float*>(p.aux)[g * p.aux_gs + row];
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] *= s;
      }
      if (p.out_f32) {
        float* o = reinterpret_cast<float*>(obase) + og * p.out_gs + orow * p.ldo + col0;
        if (nv == 32) {
          float4* o4 = reinterpret_cast<float4*>(o);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            float4 x = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
            if (p.accumulate) { float4 y = o4[j]; x.x += y.x; x.y += y.y; x.z += y.z; x.w += y.w; }
            o4[j] = x;
          }
        } else {
          for (int j = 0; j < nv; ++j) o[j] = p.accumulate ? o[j] + v[j] : v[j];
        }
      } else {
        bf16* o = reinterpret_cast<bf16*>(obase) + og * p.out_gs + orow * p.ldo + col0;
        if (nv == 32) {
          uint4* o4 = reinterpret_cast<uint4*>(o);
#pragma unroll
          for (int j = 0; j < 4; ++j)
            o4[j] = make_uint4(pack_bf16(v[8 * j], v[8 * j + 1]), pack_bf16(v[8 * j + 2], v[8 * j + 3]),
                               pack_bf16(v[8 * j + 4], v[8 * j + 5]), pack_bf16(v[8 * j + 6], v[8 * j + 7]));
        } else {
          for (int j = 0; j < nv; ++j) o[j] = __float2bfloat16(v[j]);
        }
      }
      }
    }
  }
}

// Width of the MMA for N tile `nt`: the full tile, or for a ragged last tile its valid columns rounded up to 16
// (rows of B past N are zero-filled by TMA; accumulator columns past the width are never stored).
__device__ __forceinline__ int tile_n_eff(const GemmParams& p, int nt) {
  if (!p.ntail || p.epi == EPI_SWIGLU) return p.bn;
  const int rem = p.N - nt * p.bn;
  return rem >= p.bn ? p.bn : ((rem + 15) & ~15);
}

template <bool A_MN, bool B_MN>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_tc_kernel(const __grid_constant__ TmapSet tmAs, const __grid_constant__ CUtensorMap tmB, const GemmParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);
  uint64_t* empty = full + STAGES;
  uint64_t* tfull = empty + STAGES;
  uint64_t* tempty = tfull + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int num_kb = (p.K + BK - 1) / BK;
  const int total = p.G * p.m_tiles * p.n_tiles;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&tfull[a], 1); mbar_init(&tempty[a], 4); }
    *abort_flag = 0;
    mbar_fence_init();
    for (int i = 0; i < p.n_seg; ++i) tma_prefetch_desc(&tmAs.m[i]);
    tma_prefetch_desc(&tmB);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
        int g, mt, nt;
        tile_coords(t, p, g, mt, nt);
        const int seg = mt / p.tiles_per_seg;
        const int m0 = (mt - seg * p.tiles_per_seg) * BM;
        const CUtensorMap* tA = &tmAs.m[seg];
        const int ga = g + p.a_g_off;
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait(&empty[stage], phase ^ 1, abort_flag)) {
            atomicCAS(p.status, 0, ST_WAIT_EMPTY); *abort_flag = 1; ok = false; break;
          }
          uint8_t* sA = smem + stage * STAGE_BYTES;
          uint8_t* sB = sA + A_BYTES;
          mbar_expect_tx(&full[stage], STAGE_BYTES);
          const int k0 = kb * BK;
          if (!A_MN) {
            tma_load_3d(sA, tA, &full[stage], k0, m0, ga);
          } else {
            tma_load_3d(sA, tA, &full[stage], m0, k0, ga);
            tma_load_3d(sA + 8192, tA, &full[stage], m0 + 64, k0, ga);
          }
          if (p.epi == EPI_SWIGLU) {
            const int H = p.N >> 1, n0 = nt * 128;
            if (!B_MN) {
              tma_load_3d(sB, &tmB, &full[stage], k0, n0, g);
              tma_load_3d(sB + 16384, &tmB, &full[stage], k0, H + n0, g);
            } else {
              tma_load_3d(sB, &tmB, &full[stage], n0, k0, g);
              tma_load_3d(sB + 8192, &tmB, &full[stage], n0 + 64, k0, g);
              tma_load_3d(sB + 16384, &tmB, &full[stage], H + n0, k0, g);
              tma_load_3d(sB + 24576, &tmB, &full[stage], H + n0 + 64, k0, g);
            }
          } else {
            const int n0 = nt * BN;
            if (!B_MN) {
              tma_load_3d(sB, &tmB, &full[stage], k0, n0, g);
            } else {
#pragma unroll
              for (int j = 0; j < 4; ++j) tma_load_3d(sB + j * 8192, &tmB, &full[stage], n0 + 64 * j, k0, g);
            }
          }
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
      if (!ok) {                                   // let copies already in flight land before the CTA leaves
        for (int i = 0; i < 2000; ++i) __nanosleep(1000);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
        int g_, mt_, nt_;
        tile_coords(t, p, g_, mt_, nt_);
        const uint32_t idesc = idesc_bf16(BM, tile_n_eff(p, nt_), A_MN ? 1u : 0u, B_MN ? 1u : 0u);
        if (!mbar_wait(&tempty[acc], acc_phase ^ 1, abort_flag)) {
          atomicCAS(p.status, 0, ST_WAIT_TMEM_EMPTY); *abort_flag = 1; ok = false; break;
        }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * BN;
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait(&full[stage], phase, abort_flag)) {
            atomicCAS(p.status, 0, ST_WAIT_FULL); *abort_flag = 1; ok = false; break;
          }
          tc_fence_after();
          const uint32_t sA = smem_u32(smem + stage * STAGE_BYTES);
          const uint32_t sB = sA + A_BYTES;
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k) {
            uint64_t ad = smem_desc_sw128(sA + k * (A_MN ? UMMA_K * 128 : UMMA_K * 2), A_MN ? BK * 128 : 0, 1024);
            uint64_t bd = smem_desc_sw128(sB + k * (B_MN ? UMMA_K * 128 : UMMA_K * 2), B_MN ? BK * 128 : 0, 1024);
            umma_bf16(d_tmem, ad, bd, idesc, (kb > 0 || k > 0) ? 1u : 0u);
          }
          umma_commit(&empty[stage]);              // the smem slot is free once these MMAs have read it
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        umma_commit(&tfull[acc]);                  // accumulator complete
        if (++acc == 2) { acc = 0; acc_phase ^= 1; }
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue (warps 2..5)
    const int q = warp & 3;                        // TMEM lane quarter this warp may read
    int acc = 0;
    uint32_t acc_phase = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
      int g, mt, nt;
      tile_coords(t, p, g, mt, nt);
      if (!mbar_wait(&tfull[acc], acc_phase, abort_flag)) {
        if (lane == 0) { atomicCAS(p.status, 0, ST_WAIT_TMEM_FULL); *abort_flag = 1; }
        ok = false; break;
      }
      tc_fence_after();
      const int seg = mt / p.tiles_per_seg;
      const int row_l = (mt - seg * p.tiles_per_seg) * BM + q * 32 + lane;     // row inside its segment
      epilogue_tile(p, g, seg, row_l, nt, tmem_base + (static_cast<uint32_t>(q * 32) << 16) + acc * BN);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty[acc]);
      if (++acc == 2) { acc = 0; acc_phase ^= 1; }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// ------------------------------------------------------------------------------------------------ CTA-pair kernel
// tcgen05.mma.cta_group::2: a cluster of two CTAs (two SMs) computes a 256x256 tile.  Each CTA stages its own 128
// rows of A and its own 128-row half of the B tile, so every SM pulls 32 KB per k-block instead of 48 KB for the
// same FLOPs; the leader CTA's single thread issues the MMAs for both, accumulators live in each CTA's own TMEM
// (128 lanes x 256 columns, double-buffered), each CTA runs its own epilogue on its rows.
// TMA loads carry no multicast: both CTAs fetch their own tiles; only the completion bytes are counted on the
// leader's barrier, and tcgen05.commit arrives on the barriers of both CTAs.
constexpr int BH_BYTES = 128 * BK * 2, STAGE2_BYTES = A_BYTES + BH_BYTES;
// The epilogue leaves through shared memory: each epilogue warp packs its 32 rows x 64 bf16 (or 32 fp32) columns
// into a 128-byte-swizzled 4 KB staging tile and one lane issues a TMA store (a TMA reduce-add for fp32
// accumulation; for peer / segmented outputs the warp writes the staged rows itself as full 128-byte lines).
// Shared-memory descriptors are built once and advanced by integer adds.  Per-group extents let padded expert rows
// cost neither loads nor MMAs.
constexpr int EPI_BUF_BYTES = 4096;
enum { DBG_NO_STORE = 2, DBG_DIRECT_STORE = 8, DBG_L2_HINTS = 16, DBG_TALL_OFF = 32, DBG_TALL_ON = 64 };   // test / measurement switches

// row `lane` of a staging tile, 16-byte piece j (the tile is 1024-byte aligned: TMA's 128B swizzle = piece ^ (row & 7))
__device__ __forceinline__ uint4* stage_piece(uint8_t* buf, int row, int j) {
  return reinterpret_cast<uint4*>(buf + row * 128 + ((j ^ (row & 7)) << 4));
}
// Warp-cooperative copy of a staged 32 x 128 B tile to global rows (4 rows x 128 B per instruction).
__device__ __forceinline__ void coop_store(const uint8_t* buf, char* gbase, long long pitch_bytes, int rows_valid,
                                           int pieces_valid, bool f32_acc, int lane) {
  const int pc = lane & 7;
#pragma unroll
  for (int it = 0; it < 8; ++it) {
    const int r = it * 4 + (lane >> 3);
    if (r < rows_valid && pc < pieces_valid) {
      uint4 v = *reinterpret_cast<const uint4*>(buf + r * 128 + ((pc ^ (r & 7)) << 4));
      uint4* dst = reinterpret_cast<uint4*>(gbase + r * pitch_bytes + pc * 16);
      if (f32_acc) {
        const float4 o = *reinterpret_cast<const float4*>(dst);
        float4 n = *reinterpret_cast<float4*>(&v);
        n.x += o.x; n.y += o.y; n.z += o.z; n.w += o.w;
        v = *reinterpret_cast<uint4*>(&n);
      }
      *dst = v;
    }
  }
}
// Warp-cooperative load of a 32 x 128 B global tile into a staging tile (zero outside the valid part).
__device__ __forceinline__ void coop_load(uint8_t* buf, const char* gbase, long long pitch_bytes, int rows_valid,
                                          int pieces_valid, int lane) {
  const int pc = lane & 7;
#pragma unroll
  for (int it = 0; it < 8; ++it) {
    const int r = it * 4 + (lane >> 3);
    uint4 v = make_uint4(0, 0, 0, 0);
    if (r < rows_valid && pc < pieces_valid) v = *reinterpret_cast<const uint4*>(gbase + r * pitch_bytes + pc * 16);
    *reinterpret_cast<uint4*>(buf + r * 128 + ((pc ^ (r & 7)) << 4)) = v;
  }
}

// Per-warp staging ring of EPI_NBUF tiles, handed out in slots of `nb` tiles (nb = staged tiles per store group of
// this launch: 1, 2 with a second output, 3 for SwiGLU with its pre-activations).  take(): wait until the slot about
// to be written is no longer read by an earlier store group, return the index of its first tile.
struct EpiRing {
  uint8_t* base;
  int next, nb, nbuf;
  bool tma;
  uint64_t store_policy;
  bool hint;
  __device__ __forceinline__ int take(int lane) {
    if (tma && lane == 0) {
      const int slots = nbuf / nb;                   // store groups that may still read their tiles: slots - 1
      if (slots >= 4) bulk_wait_read<3>();
      else if (slots == 2) bulk_wait_read<1>();
      else bulk_wait_read<0>();
    }
    __syncwarp();
    const int first = next;
    next += nb;
    if (next + nb > nbuf) next = 0;
    return first;
  }
  __device__ __forceinline__ uint8_t* buf(int i) const { return base + i * EPI_BUF_BYTES; }
};

struct EpiOut {            // where one output of the tile goes
  const CUtensorMap* tm;   // TMA path
  char* base;              // direct path: address of (first row of this warp, column 0) of the right group / segment
  long long pitch;         // bytes
};

// Send one staged tile: columns [col0, col0 + 64 bf16 | 32 fp32) of rows [row0, row0 + 32).
__device__ __forceinline__ void epi_send(const GemmParams& p, const EpiRing& ring, int bi, const EpiOut& o, int col0, int row0,
                                         int g, int rows_valid, int ncols, int esz, bool accumulate, int lane) {
  if (p.dbg & DBG_NO_STORE) return;
  if (ring.tma) {
    if (lane == 0) {
      if (accumulate) tma_reduce_add_3d(o.tm, ring.buf(bi), col0, row0, g);
      else if (ring.hint) tma_store_3d_hint(o.tm, ring.buf(bi), col0, row0, g, ring.store_policy);
      else tma_store_3d(o.tm, ring.buf(bi), col0, row0, g);
    }
  } else {
    const int per = 16 / esz;                                  // elements per 16-byte piece
    const int pieces = min(8, (ncols - col0 + per - 1) / per);
    coop_store(ring.buf(bi), o.base + static_cast<long long>(col0) * esz, o.pitch, rows_valid, pieces, accumulate, lane);
  }
}

// ---- aux prefetch.  The activation-backward epilogues (relu², SwiGLU) multiply the accumulator by a function of the
// forward's pre-activations, a second operand of the tile's own shape.  Fetching it when the accumulator is ready
// puts a global-memory round trip (microseconds while the GEMM itself loads HBM) into every 64-column chunk and
// made the epilogue the bottleneck (dgrad 0.74 ms plain, 1.37 ms with the relu² factor, 3.49 ms with SwiGLU's).  So
// each epilogue warp keeps a queue of TMA loads `slots` chunks ahead - across tile boundaries, i.e. issued while
// it waits for the next accumulator - into the very staging tiles the results are later stored from.
struct AuxPipe {
  uint64_t* bars;          // this warp's mbarriers, one per slot
  int slots, nb;           // nb staging tiles per chunk (1: relu² backward, 2: SwiGLU backward), slots = tiles / nb
  uint32_t issued, consumed, freed;   // chunks asked for, used, and whose slot may be loaded again
  int pf_t, pf_hc;         // cursor of the next chunk to fetch: tile, half * 4 + chunk (-1: the tile's place is not known yet)
  int pf_row, pf_col, pf_g;
  const CUtensorMap* tm;
  const int* cum;          // see tile_coords
  int rank, q, npairs, total, mh;
  bool on;
};

__device__ __forceinline__ void tma_load_3d_local(void* dst, const CUtensorMap* m, uint64_t* bar, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}

__device__ __forceinline__ int group_rows(const GemmParams& p, int g);
__device__ __forceinline__ int group_kblocks(const GemmParams& p, int g);

// Issue loads until `slots` chunks are in flight or the tile list ends.  Walks tiles and chunks exactly as the
// epilogue does (padding tiles and chunks past the last column are skipped).  Lane 0 only.
__device__ __forceinline__ void aux_issue(const GemmParams& p, AuxPipe& a, uint8_t* ring_base) {
  while (a.issued - a.freed < (uint32_t)a.slots && a.pf_t < a.total) {
    if (a.pf_hc < 0) {
      int g, mt, nt;
      tile_coords(a.pf_t, p, g, mt, nt, a.cum);
      const int seg = mt / p.tiles_per_seg;
      const int mseg0 = (mt - seg * p.tiles_per_seg) * 256 * a.mh;
      if (seg * p.seg_M + mseg0 >= group_rows(p, g) || group_kblocks(p, g) == 0) { a.pf_t += a.npairs; continue; }
      a.pf_row = seg * p.seg_M + mseg0 + a.rank * BM + a.q * 32;
      a.pf_col = nt * p.bn;
      a.pf_g = g;
      a.pf_hc = 0;
    }
    const int h = a.pf_hc >> 2, c = a.pf_hc & 3;
    const int col0 = a.pf_col + c * 64;
    const bool last = c == (p.bn >> 6) - 1 || col0 + 64 >= p.N;     // of this half
    const int row0 = a.pf_row + h * 256;
    const int slot = a.issued % a.slots;
    uint8_t* b = ring_base + slot * a.nb * EPI_BUF_BYTES;
    mbar_expect_tx(&a.bars[slot], a.nb * EPI_BUF_BYTES);
    tma_load_3d_local(b, a.tm, &a.bars[slot], col0, row0, a.pf_g);
    if (a.nb == 2) tma_load_3d_local(b + EPI_BUF_BYTES, a.tm, &a.bars[slot], p.N + col0, row0, a.pf_g);
    ++a.issued;
    if (!last) ++a.pf_hc;
    else if (h + 1 < a.mh) a.pf_hc = (h + 1) << 2;
    else { a.pf_t += a.npairs; a.pf_hc = -1; }
  }
}

// Drain this warp's 32 TMEM lanes x 256 columns of one accumulator through the fused epilogue.
// row0 = first row of the warp in the local (M) problem, row0_l = the same inside its M-segment.
__device__ __forceinline__ void epilogue_tile3(const GemmParams& p, const CUtensorMap* tmO, const CUtensorMap* tmO2, int g,
                                               int seg, int row0, int row0_l, int nt, uint32_t taddr, EpiRing& ring, int lane,
                                               bool zero_tile, AuxPipe* aux, volatile int* abort_flag) {
  const int rows_valid = max(0, min(32, p.seg_M - row0_l));
  const int row = row0 + lane;
  const int esz = p.out_f32 ? 4 : 2;
  EpiOut o, o2;
  o.tm = tmO; o2.tm = tmO2;
  {
    char* ob = reinterpret_cast<char*>(p.out_seg_on ? p.out_seg[seg] : p.out);
    const long long orow = p.out_seg_on ? row0_l : row0;
    o.base = ob + ((g + p.out_g_off) * p.out_gs + orow * p.ldo) * esz;
    o.pitch = static_cast<long long>(p.ldo) * esz;
    o2.base = reinterpret_cast<char*>(p.out2) + (g * p.out2_gs + static_cast<long long>(row0) * p.ldo2) * 2;
    o2.pitch = static_cast<long long>(p.ldo2) * 2;
  }
  const int og = g + p.out_g_off;

  if (zero_tile) {
    // a tile of padding rows: no accumulator was produced; the outputs are zeros (an accumulating output stays)
    if (p.accumulate) return;
    if (aux != nullptr && aux->on) {
      // the staging tiles belong to the prefetch queue: zeros go out by plain 16-byte stores
      const int wide = p.epi == EPI_DSWIGLU ? 2 : 1;
      for (int c = 0; c < p.bn / 64; ++c) {
        const int col0 = nt * p.bn + c * 64;
        if (col0 >= p.N) break;
        const int pieces = min(8, (p.N - col0 + 7) >> 3), pc = lane & 7;
        for (int w = 0; w < wide; ++w)
          for (int it = 0; it < 8; ++it) {
            const int r = it * 4 + (lane >> 3);
            if (r < rows_valid && pc < pieces)
              *reinterpret_cast<uint4*>(o.base + r * o.pitch + (static_cast<long long>(w) * p.N + col0) * 2 + pc * 16) =
                  make_uint4(0, 0, 0, 0);
          }
      }
      return;
    }
    const int bi = ring.take(lane);
    *stage_piece(ring.buf(bi), lane, 0) = make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int j = 1; j < 8; ++j) *stage_piece(ring.buf(bi), lane, j) = make_uint4(0, 0, 0, 0);
    fence_async_smem();
    __syncwarp();
    if (p.epi == EPI_SWIGLU) {
      const int H = p.N >> 1;
      for (int c = 0; c < p.bn / 128; ++c) {
        const int col0 = nt * (p.bn / 2) + c * 64;
        if (col0 >= H) break;
        epi_send(p, ring, bi, o, col0, row0, og, rows_valid, H, 2, false, lane);
        if (p.out2) {
          epi_send(p, ring, bi, o2, col0, row0, g, rows_valid, H, 2, false, lane);
          epi_send(p, ring, bi, o2, H + col0, row0, g, rows_valid, p.N, 2, false, lane);
        }
      }
    } else {
      const int cw = p.out_f32 ? 32 : 64;
      for (int c = 0; c < p.bn / cw; ++c) {
        const int col0 = nt * p.bn + c * cw;
        if (col0 >= p.N) break;
        epi_send(p, ring, bi, o, col0, row0, og, rows_valid, p.N, esz, false, lane);
        if (p.epi == EPI_RELU2) epi_send(p, ring, bi, o2, col0, row0, g, rows_valid, p.N, 2, false, lane);
        if (p.epi == EPI_DSWIGLU) {
          EpiOut oz = o;
          oz.tm = tmO2;
          oz.base = o.base + static_cast<long long>(p.N) * 2;
          epi_send(p, ring, bi, oz, col0, row0, og, rows_valid, p.N, 2, false, lane);
        }
      }
    }
    if (ring.tma && lane == 0) bulk_commit();
    return;
  }

  if (p.epi == EPI_SWIGLU) {
    const int H = p.N >> 1;
    const int nb = p.out2 ? 3 : 1;
#pragma unroll 1
    for (int c = 0; c < p.bn / 128; ++c) {
      const int col0 = nt * (p.bn / 2) + c * 64;
      if (col0 >= H) break;
      const int bi = ring.take(lane);
#pragma unroll 1
      for (int hf = 0; hf < 2; ++hf) {
        uint32_t rg[32], ru[32];
        tmem_ld32(taddr + c * 64 + hf * 32, rg);
        tmem_ld32(taddr + p.bn / 2 + c * 64 + hf * 32, ru);
        tmem_ld_wait();
        uint32_t ph[16], pg[16], pu[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const float g0 = __uint_as_float(rg[2 * j]), g1 = __uint_as_float(rg[2 * j + 1]);
          const float u0 = __uint_as_float(ru[2 * j]), u1 = __uint_as_float(ru[2 * j + 1]);
          pg[j] = pack_bf16(g0, g1);
          pu[j] = pack_bf16(u0, u1);
          // activations of the stored (rounded) values, so forward and the recomputing backward agree
          const float2 gr = unpack_bf16(pg[j]), ur = unpack_bf16(pu[j]);
          ph[j] = pack_bf16(silu_f(gr.x) * ur.x, silu_f(gr.y) * ur.y);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          *stage_piece(ring.buf(bi), lane, hf * 4 + j) = make_uint4(ph[4 * j], ph[4 * j + 1], ph[4 * j + 2], ph[4 * j + 3]);
          if (nb == 3) {
            *stage_piece(ring.buf(bi + 1), lane, hf * 4 + j) = make_uint4(pg[4 * j], pg[4 * j + 1], pg[4 * j + 2], pg[4 * j + 3]);
            *stage_piece(ring.buf(bi + 2), lane, hf * 4 + j) = make_uint4(pu[4 * j], pu[4 * j + 1], pu[4 * j + 2], pu[4 * j + 3]);
          }
        }
      }
      fence_async_smem();
      __syncwarp();
      epi_send(p, ring, bi, o, col0, row0, og, rows_valid, H, 2, false, lane);
      if (nb == 3) {
        epi_send(p, ring, bi + 1, o2, col0, row0, g, rows_valid, H, 2, false, lane);
        epi_send(p, ring, bi + 2, o2, H + col0, row0, g, rows_valid, p.N, 2, false, lane);
      }
      if (ring.tma && lane == 0) bulk_commit();
    }
    return;
  }

  if (p.out_f32) {
    // fp32 output (weight gradients): 32 columns per staged tile
#pragma unroll 1
    for (int c = 0; c < p.bn / 32; ++c) {
      const int col0 = nt * p.bn + c * 32;
      if (col0 >= p.N) break;
      uint32_t r[32];
      tmem_ld32(taddr + c * 32, r);
      tmem_ld_wait();
      float sc = 1.f;
      if (p.epi == EPI_ROWSCALE) sc = row0_l + lane < p.seg_M ? reinterpret_cast<const float*>(p.aux)[g * p.aux_gs + row] : 0.f;
      const int bi = ring.take(lane);
#pragma unroll
      for (int j = 0; j < 8; ++j)
        *stage_piece(ring.buf(bi), lane, j) =
            make_uint4(__float_as_uint(__uint_as_float(r[4 * j]) * sc), __float_as_uint(__uint_as_float(r[4 * j + 1]) * sc),
                       __float_as_uint(__uint_as_float(r[4 * j + 2]) * sc), __float_as_uint(__uint_as_float(r[4 * j + 3]) * sc));
      fence_async_smem();
      __syncwarp();
      epi_send(p, ring, bi, o, col0, row0, og, rows_valid, p.N, 4, p.accumulate != 0, lane);
      if (ring.tma && lane == 0) bulk_commit();
    }
    return;
  }

  // bf16 output, 64 columns per staged tile
  const int nb = (p.epi == EPI_RELU2 || p.epi == EPI_DSWIGLU) ? 2 : 1;
  EpiOut oh = o;                       // SwiGLU backward: second half of the output row (the `up` gradient), via tmO2
  oh.tm = tmO2;
  oh.base = o.base + static_cast<long long>(p.N) * 2;
#pragma unroll 1
  for (int c = 0; c < p.bn / 64; ++c) {
    const int col0 = nt * p.bn + c * 64;
    if (col0 >= p.N) break;
    uint32_t r[64];
    tmem_ld32(taddr + c * 64, *reinterpret_cast<uint32_t(*)[32]>(&r[0]));
    tmem_ld32(taddr + c * 64 + 32, *reinterpret_cast<uint32_t(*)[32]>(&r[32]));
    tmem_ld_wait();
    const bool piped = aux != nullptr && aux->on;
    int bi;
    if (piped) {
      // the chunk's pre-activations were fetched ahead into the slot the results will be stored from
      const int slot = aux->consumed % aux->slots;
      bi = slot * aux->nb;
      if (!mbar_wait(&aux->bars[slot], (aux->consumed / aux->slots) & 1, abort_flag)) {
        if (lane == 0) { atomicCAS(p.status, 0, ST_WAIT_FULL); *abort_flag = 1; }
        return;
      }
    } else {
      bi = ring.take(lane);
    }
    uint8_t* b0 = ring.buf(bi);
    if (p.epi == EPI_RELU2) {
      uint8_t* b1 = ring.buf(bi + 1);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        uint32_t pa[4], ph[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          pa[q] = pack_bf16(__uint_as_float(r[8 * j + 2 * q]), __uint_as_float(r[8 * j + 2 * q + 1]));
          float2 a = unpack_bf16(pa[q]);                      // activation of the stored (rounded) value
          a.x = fmaxf(a.x, 0.f); a.y = fmaxf(a.y, 0.f);
          ph[q] = pack_bf16(a.x * a.x, a.y * a.y);
        }
        *stage_piece(b0, lane, j) = make_uint4(ph[0], ph[1], ph[2], ph[3]);
        *stage_piece(b1, lane, j) = make_uint4(pa[0], pa[1], pa[2], pa[3]);
      }
    } else if (p.epi == EPI_DSWIGLU) {
      // acc = dh (columns of the hidden width H = p.N); aux = (gate | up) pre-activations, 2H columns.
      // dg = dh * u * s * (1 + g * (1 - s)), du = dh * g * s with s = sigmoid(g)
      uint8_t* b1 = ring.buf(bi + 1);
      const char* ab = reinterpret_cast<const char*>(p.aux) + (g * p.aux_gs + static_cast<long long>(row0) * p.ldaux + col0) * 2;
      const int pv = min(8, (p.N - col0 + 7) >> 3);
      if (!piped) {
        coop_load(b0, ab, static_cast<long long>(p.ldaux) * 2, rows_valid, pv, lane);
        coop_load(b1, ab + static_cast<long long>(p.N) * 2, static_cast<long long>(p.ldaux) * 2, rows_valid, pv, lane);
        __syncwarp();
      }
      // All loads of half a chunk go out before its first store: one epilogue warp per scheduler has nothing else to hide
      // the round trip to shared memory with, and a store in between holds the next load back.
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        uint4 ug[4], uu[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) { ug[j] = *stage_piece(b0, lane, 4 * hf + j); uu[j] = *stage_piece(b1, lane, 4 * hf + j); }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t wg[4] = {ug[j].x, ug[j].y, ug[j].z, ug[j].w}, wu[4] = {uu[j].x, uu[j].y, uu[j].z, uu[j].w};
          uint32_t og[4], ou[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const float2 gg = unpack_bf16(wg[q]), uv = unpack_bf16(wu[q]);
            const float d0 = __uint_as_float(r[32 * hf + 8 * j + 2 * q]), d1 = __uint_as_float(r[32 * hf + 8 * j + 2 * q + 1]);
            const float s0 = sigmoid_f(gg.x), s1 = sigmoid_f(gg.y);
            og[q] = pack_bf16(d0 * uv.x * s0 * (1.f + gg.x * (1.f - s0)), d1 * uv.y * s1 * (1.f + gg.y * (1.f - s1)));
            ou[q] = pack_bf16(d0 * gg.x * s0, d1 * gg.y * s1);
          }
          ug[j] = make_uint4(og[0], og[1], og[2], og[3]);
          uu[j] = make_uint4(ou[0], ou[1], ou[2], ou[3]);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) { *stage_piece(b0, lane, 4 * hf + j) = ug[j]; *stage_piece(b1, lane, 4 * hf + j) = uu[j]; }
      }
    } else if (p.epi == EPI_DRELU2) {
      const char* ab = reinterpret_cast<const char*>(p.aux) + (g * p.aux_gs + static_cast<long long>(row0) * p.ldaux + col0) * 2;
      if (!piped) {
        coop_load(b0, ab, static_cast<long long>(p.ldaux) * 2, rows_valid, min(8, (p.N - col0 + 7) >> 3), lane);
        __syncwarp();
      }
      uint4 u[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) u[j] = *stage_piece(b0, lane, j);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const uint32_t w[4] = {u[j].x, u[j].y, u[j].z, u[j].w};
        uint32_t o4[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float2 f = unpack_bf16(w[q]);
          o4[q] = pack_bf16(__uint_as_float(r[8 * j + 2 * q]) * 2.f * fmaxf(f.x, 0.f), __uint_as_float(r[8 * j + 2 * q + 1]) * 2.f * fmaxf(f.y, 0.f));
        }
        u[j] = make_uint4(o4[0], o4[1], o4[2], o4[3]);
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) *stage_piece(b0, lane, j) = u[j];
    } else {
      float sc = 1.f;
      if (p.epi == EPI_ROWSCALE) sc = row0_l + lane < p.seg_M ? reinterpret_cast<const float*>(p.aux)[g * p.aux_gs + row] : 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j)
        *stage_piece(b0, lane, j) = make_uint4(pack_bf16(__uint_as_float(r[8 * j]) * sc, __uint_as_float(r[8 * j + 1]) * sc),
                                               pack_bf16(__uint_as_float(r[8 * j + 2]) * sc, __uint_as_float(r[8 * j + 3]) * sc),
                                               pack_bf16(__uint_as_float(r[8 * j + 4]) * sc, __uint_as_float(r[8 * j + 5]) * sc),
                                               pack_bf16(__uint_as_float(r[8 * j + 6]) * sc, __uint_as_float(r[8 * j + 7]) * sc));
    }
    fence_async_smem();
    __syncwarp();
    epi_send(p, ring, bi, o, col0, row0, og, rows_valid, p.N, 2, false, lane);
    if (p.epi == EPI_DSWIGLU) epi_send(p, ring, bi + 1, oh, col0, row0, og, rows_valid, p.N, 2, false, lane);
    else if (nb == 2) epi_send(p, ring, bi + 1, o2, col0, row0, g, rows_valid, p.N, 2, false, lane);
    if (ring.tma && lane == 0) bulk_commit();
    if (piped) {
      ++aux->consumed;
      __syncwarp();                               // direct stores: every lane has read the slot
      if (lane == 0) {
        // A slot whose TMA stores have read it takes the next chunk.  With three slots or more that is the one before this:
        // its stores are done by now, those of this chunk would be waited for.
        if (aux->slots >= 3) { bulk_wait_read<1>(); aux->freed = aux->consumed - 1; }
        else { bulk_wait_read<0>(); aux->freed = aux->consumed; }
        fence_async_smem();
        aux_issue(p, *aux, ring.base);
      }
    }
  }
}

enum { ACT_NONE = 0, ACT_SWIGLU = 1, ACT_RELU2 = 2 };
// The activation-backward epilogues with two warps per 32 TMEM lanes, each taking 32 of a chunk's 64 columns: one warp per
// scheduler could not hide its own chain of shared-memory and special-function latencies.  Both wait for the chunk's
// pre-activations and write their results over them; the second reports on `done` (a barrier per slot), the first sends
// the tile and refills the slot before.  All waits are bounded and none is for a warp that may have given up unseen.
// Us, (M, N, K), one warp -> two, SwiGLU / relu2: (32 768, 4096, 1024) 358 -> 314 / 264 -> 237, plain product 211; (8192, 3072, 768)
// 85 -> 65 / 60 -> 47, plain 40; (4096, 2048, 512) 31 -> 25 / 23 -> 19, plain 19.  (32 768, 8192, 2048) is bound by power: 1050 / 900.
// (SwiGLU times with the sigmoid through the hardware tanh; exact, as now, they are 1 % longer: 304 -> 308 for the first size.)
template <int ACT>
__device__ __forceinline__ void epilogue_act(const GemmParams& p, const CUtensorMap* tmO, const CUtensorMap* tmO2, int og, int row0, int nt,
                                             uint32_t taddr, uint8_t* ring_base, int lane, int half, AuxPipe& aux, uint64_t* done,
                                             volatile int* abort_flag) {
#pragma unroll 1
  for (int c = 0; c < p.bn / 64; ++c) {
    const int col0 = nt * p.bn + c * 64;
    if (col0 >= p.N) break;
    uint32_t r[32];
    tmem_ld32(taddr + c * 64 + half * 32, r);
    const int slot = aux.consumed % aux.slots;
    const uint32_t phase = (aux.consumed / aux.slots) & 1;
    if (!mbar_wait(&aux.bars[slot], phase, abort_flag)) {
      if (lane == 0) { atomicCAS(p.status, 0, ST_WAIT_FULL); *abort_flag = 1; }
      tmem_ld_wait();
      return;
    }
    uint8_t* b0 = ring_base + slot * aux.nb * EPI_BUF_BYTES;
    uint8_t* b1 = b0 + EPI_BUF_BYTES;
    uint4 ug[4], uu[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      ug[j] = *stage_piece(b0, lane, 4 * half + j);
      if (ACT == ACT_SWIGLU) uu[j] = *stage_piece(b1, lane, 4 * half + j);
    }
    tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t wg[4] = {ug[j].x, ug[j].y, ug[j].z, ug[j].w};
      uint32_t o0[4], o1[4];
      if (ACT == ACT_SWIGLU) {
        // acc = dh; dg = dh * u * s * (1 + g * (1 - s)), du = dh * g * s with s = sigmoid(g)
        const uint32_t wu[4] = {uu[j].x, uu[j].y, uu[j].z, uu[j].w};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float2 gg = unpack_bf16(wg[q]), uv = unpack_bf16(wu[q]);
          const float d0 = __uint_as_float(r[8 * j + 2 * q]), d1 = __uint_as_float(r[8 * j + 2 * q + 1]);
          const float s0 = sigmoid_f(gg.x), s1 = sigmoid_f(gg.y);
          o0[q] = pack_bf16(d0 * uv.x * s0 * (1.f + gg.x * (1.f - s0)), d1 * uv.y * s1 * (1.f + gg.y * (1.f - s1)));
          o1[q] = pack_bf16(d0 * gg.x * s0, d1 * gg.y * s1);
        }
        uu[j] = make_uint4(o1[0], o1[1], o1[2], o1[3]);
      } else {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float2 f = unpack_bf16(wg[q]);
          o0[q] = pack_bf16(__uint_as_float(r[8 * j + 2 * q]) * 2.f * fmaxf(f.x, 0.f), __uint_as_float(r[8 * j + 2 * q + 1]) * 2.f * fmaxf(f.y, 0.f));
        }
      }
      ug[j] = make_uint4(o0[0], o0[1], o0[2], o0[3]);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      *stage_piece(b0, lane, 4 * half + j) = ug[j];
      if (ACT == ACT_SWIGLU) *stage_piece(b1, lane, 4 * half + j) = uu[j];
    }
    fence_async_smem();
    __syncwarp();
    ++aux.consumed;
    if (lane == 0) {
      if (half) {
        mbar_arrive(&done[slot]);
      } else if (!mbar_wait(&done[slot], phase, abort_flag)) {
        atomicCAS(p.status, 0, ST_WAIT_FULL); *abort_flag = 1;
      } else {
        if (!(p.dbg & DBG_NO_STORE)) {
          tma_store_3d(tmO, b0, col0, row0, og);
          if (ACT == ACT_SWIGLU) tma_store_3d(tmO2, b1, col0, row0, og);
        }
        bulk_commit();
        // a slot whose stores have read it takes the next chunk: the one before this, whose stores are done by now
        bulk_wait_read<1>();
        aux.freed = aux.consumed - 1;
        fence_async_smem();
        aux_issue(p, aux, ring_base);
      }
    }
    __syncwarp();
  }
}

// extent of group g under count_mode (rows for mode 1, contraction length for mode 2), else the full extent
__device__ __forceinline__ int group_rows(const GemmParams& p, int g) {
  return p.count_mode == 1 ? min(p.M, __ldg(p.counts + g)) : p.M;
}
__device__ __forceinline__ int group_kblocks(const GemmParams& p, int g) {
  const int k = p.count_mode == 2 ? min(p.K, __ldg(p.counts + g)) : p.K;
  return (k + BK - 1) / BK;
}

// first k-block of work item t; `num_kb` (the group's k-blocks) shrinks to the item's share
__device__ __forceinline__ int split_start(const GemmParams& p, int t, int& num_kb) {
  if (p.splits <= 1) return 0;
  const int kb0 = (t % p.splits) * p.kb_split;
  num_kb = min(p.kb_split, num_kb - kb0);
  return kb0;
}

// MH = 256-row MMA blocks per tile.  MH 1: 256 x 256 tile, 5 operand stages of 32 KB, accumulators double-buffered in
// TMEM (2 x 256 columns), so the epilogue of a tile runs under the MMAs of the next.  MH 2: 512 x 256 tile - every
// B k-block feeds two MMAs, so the pair pulls 96 KB per 512x256x64 of work instead of 128 KB (a quarter less L2 and
// shared-memory traffic, which on a power-capped part is clock) - 4 stages of 48 KB; the two 256-column accumulators
// fill TMEM, so the epilogue is only half hidden (the MMAs of the next tile's first block start as soon as the
// first half is drained): worth it when the contraction is long.
// ACT (256-row tiles only): the epilogues that multiply by the activation's derivative, ACT_SWIGLU and ACT_RELU2, with eight
// epilogue warps (see epilogue_act).  SwiGLU moves two tiles in and two out per 64 accumulator columns and needs three chunks
// of pre-activations in flight to keep HBM busy: one operand stage less, six staging tiles instead of four.
template <int MH, int ACT = ACT_NONE> struct PairCfg {
  static constexpr int THREADS = ACT ? 320 : GEMM_THREADS;
  static constexpr int STAGES = (MH == 2 || ACT == ACT_SWIGLU) ? 4 : 5;
  static constexpr int NBUF = MH == 2 ? 2 : (ACT == ACT_SWIGLU ? 6 : 4);
  static constexpr int STAGE_BYTES = MH * A_BYTES + BH_BYTES;
  static constexpr int SMEM = STAGES * STAGE_BYTES + 4 * NBUF * EPI_BUF_BYTES + 1024 + 384;
};

template <bool A_MN, bool B_MN, int MH, int ACT = ACT_NONE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PairCfg<MH, ACT>::THREADS, 1)
gemm_pair_kernel(const __grid_constant__ TmapSet tmAs, const __grid_constant__ CUtensorMap tmB,
                const __grid_constant__ CUtensorMap tmO, const __grid_constant__ CUtensorMap tmO2,
                const __grid_constant__ CUtensorMap tmX, const GemmParams p) {
  constexpr int STAGES3 = PairCfg<MH, ACT>::STAGES, EPI_NBUF = PairCfg<MH, ACT>::NBUF, STAGE_B = PairCfg<MH, ACT>::STAGE_BYTES;
  constexpr int TILE_M = 256 * MH;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* epi_smem = smem + STAGES3 * STAGE_B;
  uint64_t* full = reinterpret_cast<uint64_t*>(epi_smem + 4 * EPI_NBUF * EPI_BUF_BYTES);
  uint64_t* empty = full + STAGES3;
  uint64_t* tfull = empty + STAGES3;
  uint64_t* tempty = tfull + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  uint64_t* auxbars = full + 16;              // 4 lane quarters x 4 slots of the aux prefetch queue (bytes 128..255)
  uint64_t* halfbars = full + 32;             // the same slots: the second warp's half is written (bytes 256..383)

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader = rank == 0;
  const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;
  const int total = p.G * p.m_tiles * p.n_tiles * max(1, p.splits);
  __shared__ int cum_s[MAX_COUNT_G + 1];
  const int* cum = p.count_mode == 1 && p.n_seg == 1 && p.G <= MAX_COUNT_G ? cum_s : nullptr;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES3; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&tfull[a], 1); mbar_init(&tempty[a], ACT ? 16 : 8); }
    *abort_flag = 0;
    mbar_fence_init();
    for (int i = 0; i < p.n_seg; ++i) tma_prefetch_desc(&tmAs.m[i]);
    tma_prefetch_desc(&tmB);
    if (p.store_tma) { tma_prefetch_desc(&tmO); if (p.out2 || p.epi == EPI_DSWIGLU) tma_prefetch_desc(&tmO2); }
    if (p.aux_tma) {
      for (int i = 0; i < 16; ++i) { mbar_init(&auxbars[i], 1); mbar_init(&halfbars[i], 1); }
      mbar_fence_init();
      tma_prefetch_desc(&tmX);
    }
  }
  if (cum != nullptr && warp == 2) {
    // running sums of the groups' row tiles, 32 groups at a time
    int run = 0;
    for (int g0 = 0; g0 < p.G; g0 += 32) {
      int v = g0 + lane < p.G ? (max(0, group_rows(p, g0 + lane)) + TILE_M - 1) / TILE_M : 0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += u;
      }
      if (g0 + lane < p.G) cum_s[g0 + lane + 1] = run + v;
      run += __shfl_sync(0xffffffffu, v, 31);
    }
    if (lane == 0) cum_s[0] = 0;
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  cluster_sync_all();                         // both CTAs' barriers exist before anyone arrives on a peer's barrier
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  if (threadIdx.x == 0 && tmem_base != 0) atomicCAS(p.status, 0, ST_BAD_ARG);   // the pair must share one TMEM address

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer (both CTAs)
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int t = pair; t < total && ok; t += npairs) {
        int g, mt, nt;
        tile_coords(t, p, g, mt, nt, cum);
        const int seg = mt / p.tiles_per_seg;
        const int mseg0 = (mt - seg * p.tiles_per_seg) * TILE_M;
        if (seg * p.seg_M + mseg0 >= group_rows(p, g)) continue;            // a tile of padding rows
        const int m0 = mseg0 + (int)rank * BM;
        const CUtensorMap* tA = &tmAs.m[seg];
        const int ga = g + p.a_g_off;
        int num_kb = group_kblocks(p, g);
        const int kb0 = split_start(p, t, num_kb);
        const int nb = (p.epi == EPI_SWIGLU) ? (rank == 0 ? 0 : (p.N >> 1)) + nt * (p.bn >> 1)
                                             : nt * p.bn + (int)rank * (tile_n_eff(p, nt) >> 1);
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_try_wait(&empty[stage], phase ^ 1) && !mbar_wait(&empty[stage], phase ^ 1, abort_flag)) {
            atomicCAS(p.status, 0, ST_WAIT_EMPTY); *abort_flag = 1; ok = false; break;
          }
          uint8_t* sA = smem + stage * STAGE_B;
          uint8_t* sB = sA + MH * A_BYTES;
          const uint32_t lfull = mapa_shared(smem_u32(&full[stage]), 0);      // the leader's barrier
          if (leader) mbar_expect_tx(&full[stage], 2 * (MH * A_BYTES + p.bn * BK));  // bytes of both CTAs: bn / 2 rows of B each
          const int k0 = (kb0 + kb) * BK;
#pragma unroll
          for (int h = 0; h < MH; ++h) {                                       // this CTA's 128 rows of each 256-row block
            const int mh = m0 + h * 256;
            if (!A_MN) {
              tma_load_3d_pair(sA + h * A_BYTES, tA, lfull, k0, mh, ga);
            } else {
              tma_load_3d_pair(sA + h * A_BYTES, tA, lfull, mh, k0, ga);
              tma_load_3d_pair(sA + h * A_BYTES + 8192, tA, lfull, mh + 64, k0, ga);
            }
          }
          if (!B_MN) {
            tma_load_3d_pair(sB, &tmB, lfull, k0, nb, g);
          } else {
            tma_load_3d_pair(sB, &tmB, lfull, nb, k0, g);
            if (p.bn == BN) tma_load_3d_pair(sB + 8192, &tmB, lfull, nb + 64, k0, g);
          }
          if (++stage == STAGES3) { stage = 0; phase ^= 1; }
        }
      }
      if (!ok) {
        for (int i = 0; i < 2000; ++i) __nanosleep(1000);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (leader CTA only)
    // This one thread is the pacemaker of both SMs: whatever it executes between two MMAs shows up as an idle
    // tensor pipe.  So the loop holds everything in registers, looks at the next stage's barrier before it issues
    // the current stage's MMAs (the look-up's latency then overlaps their execution), and works out the next
    // tile's coordinates while the first k-block of the current one runs.
    if (lane == 0 && leader) {
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;                 // MH 1: accumulator buffer in use; MH 2: always 0 (tempty[h] = half h drained)
      uint32_t acc_phase = 0;
      bool ok = true;
      constexpr uint32_t KSTEP_A = (A_MN ? UMMA_K * 128 : UMMA_K * 2) >> 4, KSTEP_B = (B_MN ? UMMA_K * 128 : UMMA_K * 2) >> 4;
      constexpr uint32_t STAGE_STEP = STAGE_B >> 4;
      const uint64_t adesc0 = smem_desc_sw128(smem_u32(smem), A_MN ? BK * 128 : 0, 1024);
      const uint64_t bdesc0 = smem_desc_sw128(smem_u32(smem) + MH * A_BYTES, B_MN ? BK * 128 : 0, 1024);
      uint32_t soff = 0;                                                   // stage * STAGE_STEP
      // (k-blocks, instruction descriptor) of tile t; 0 k-blocks = nothing to issue (padding rows, empty contraction)
      auto tile_info = [&](int t, int& nkb, uint32_t& idesc) {
        nkb = 0; idesc = 0;
        if (t >= total) return;
        int g_, mt_, nt_;
        tile_coords(t, p, g_, mt_, nt_, cum);
        const int seg = mt_ / p.tiles_per_seg;
        if (seg * p.seg_M + (mt_ - seg * p.tiles_per_seg) * TILE_M >= group_rows(p, g_)) return;
        nkb = group_kblocks(p, g_);
        split_start(p, t, nkb);
        idesc = idesc_bf16(256, tile_n_eff(p, nt_), A_MN ? 1u : 0u, B_MN ? 1u : 0u);
      };
      int num_kb, nxt_kb = 0;
      uint32_t idesc, nxt_idesc = 0;
      tile_info(pair, num_kb, idesc);
      for (int t = pair; t < total && ok; t += npairs) {
        if (num_kb == 0) { tile_info(t + npairs, num_kb, idesc); continue; }
        if (!mbar_try_wait(&tempty[acc], acc_phase ^ 1) && !mbar_wait(&tempty[acc], acc_phase ^ 1, abort_flag)) {
          atomicCAS(p.status, 0, ST_WAIT_TMEM_EMPTY); *abort_flag = 1; ok = false; break;
        }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + (MH == 1 ? acc * BN : 0);
        bool ready = mbar_try_wait(&full[stage], phase);
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!ready && !mbar_wait(&full[stage], phase, abort_flag)) {
            atomicCAS(p.status, 0, ST_WAIT_FULL); *abort_flag = 1; ok = false; break;
          }
          tc_fence_after();
          int ns = stage + 1;
          uint32_t nph = phase, nsoff = soff + STAGE_STEP;
          if (ns == STAGES3) { ns = 0; nph ^= 1; nsoff = 0; }
          ready = mbar_try_wait(&full[ns], nph);                           // the next k-block (of this or the next tile)
          const uint64_t ad = adesc0 + soff, bd = bdesc0 + soff;
          umma_bf16_pair(d_tmem, ad, bd, idesc, kb > 0 ? 1u : 0u);
#pragma unroll
          for (int k = 1; k < BK / UMMA_K; ++k) umma_bf16_pair(d_tmem, ad + k * KSTEP_A, bd + k * KSTEP_B, idesc, 1u);
          if (MH == 2) {
            if (kb == 0) {                                                 // the second half of the last tile must be drained
              if (!mbar_try_wait(&tempty[1], acc_phase ^ 1) && !mbar_wait(&tempty[1], acc_phase ^ 1, abort_flag)) {
                atomicCAS(p.status, 0, ST_WAIT_TMEM_EMPTY); *abort_flag = 1; ok = false; break;
              }
              tc_fence_after();
            }
            const uint64_t ad2 = ad + (A_BYTES >> 4);
            umma_bf16_pair(d_tmem + BN, ad2, bd, idesc, kb > 0 ? 1u : 0u);
#pragma unroll
            for (int k = 1; k < BK / UMMA_K; ++k) umma_bf16_pair(d_tmem + BN, ad2 + k * KSTEP_A, bd + k * KSTEP_B, idesc, 1u);
          }
          umma_commit_pair(&empty[stage], 3);       // frees this stage in both CTAs
          if (kb == 0) tile_info(t + npairs, nxt_kb, nxt_idesc);
          stage = ns; phase = nph; soff = nsoff;
        }
        if (!ok) break;
        umma_commit_pair(&tfull[MH == 1 ? acc : 0], 3);           // accumulators of both CTAs complete
        if (MH == 1) { if (++acc == 2) { acc = 0; acc_phase ^= 1; } }
        else acc_phase ^= 1;
        num_kb = nxt_kb; idesc = nxt_idesc;
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue (warps 2..5 of both CTAs)
    const int q = warp & 3;
    int acc = 0;
    uint32_t acc_phase = 0;
    bool ok = true;
    EpiRing ring;
    ring.base = epi_smem + q * (EPI_NBUF * EPI_BUF_BYTES);
    ring.next = 0;
    ring.nbuf = EPI_NBUF;
    ring.hint = (p.dbg & DBG_L2_HINTS) != 0;
    ring.store_policy = l2_policy_evict_first();
    ring.nb = (p.epi == EPI_RELU2 || p.epi == EPI_DSWIGLU) ? 2 : (p.epi == EPI_SWIGLU && p.out2 ? 3 : 1);
    ring.tma = p.store_tma != 0;
    AuxPipe aux;
    aux.on = p.aux_tma != 0;
    aux.bars = auxbars + q * 4;
    aux.nb = ring.nb;
    aux.slots = EPI_NBUF / ring.nb;
    aux.issued = aux.consumed = aux.freed = 0;
    aux.pf_t = pair; aux.pf_hc = -1; aux.cum = cum;
    aux.tm = &tmX;
    aux.rank = (int)rank; aux.q = q; aux.npairs = npairs; aux.total = total; aux.mh = MH;
    [[maybe_unused]] const int half = (warp - 2) >> 2;            // ACT: which 32 of 64 columns
    if (aux.on && lane == 0 && half == 0) aux_issue(p, aux, ring.base);
    for (int t = pair; t < total && ok; t += npairs) {
      int g, mt, nt;
      tile_coords(t, p, g, mt, nt, cum);
      const int seg = mt / p.tiles_per_seg;
      const int mseg0 = (mt - seg * p.tiles_per_seg) * TILE_M;
      const bool zero_tile = seg * p.seg_M + mseg0 >= group_rows(p, g) || group_kblocks(p, g) == 0;
      if (!zero_tile) {
        if (!mbar_wait(&tfull[MH == 1 ? acc : 0], acc_phase, abort_flag)) {
          if (lane == 0) { atomicCAS(p.status, 0, ST_WAIT_TMEM_FULL); *abort_flag = 1; }
          ok = false; break;
        }
        tc_fence_after();
      }
#pragma unroll 1
      for (int h = 0; h < MH; ++h) {
        const int row0_l = mseg0 + h * 256 + (int)rank * BM + q * 32;
        const int row0 = seg * p.seg_M + row0_l;
        const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + (MH == 1 ? acc * BN : h * BN);
        bool drained = false;
        if constexpr (ACT != ACT_NONE) {
          drained = !zero_tile || half != 0;
          if (!zero_tile) epilogue_act<ACT>(p, &tmO, &tmO2, g + p.out_g_off, row0, nt, taddr, ring.base, lane, half, aux, halfbars + q * 4, abort_flag);
        }
        // a part of a cut contraction goes to its own slab
        if (!drained) epilogue_tile3(p, &tmO, &tmO2, p.splits > 1 ? t % p.splits : g, seg, row0, row0_l, nt, taddr, ring, lane, zero_tile, &aux, abort_flag);
        if (*abort_flag) { ok = false; break; }
        if (!zero_tile) {
          tc_fence_before();
          __syncwarp();
          // the leader's MMA thread waits on it (MH 2: per half, so the next tile's first MMAs start early)
          if (lane == 0) mbar_arrive_cluster(mapa_shared(smem_u32(&tempty[MH == 1 ? acc : h]), 0));
        }
      }
      if (!zero_tile) {
        if (MH == 1) { if (++acc == 2) { acc = 0; acc_phase ^= 1; } }
        else acc_phase ^= 1;
      }
    }
    if (ring.tma && lane == 0) bulk_wait_read<0>();          // staged tiles must be read before the CTA's smem goes away
    if (aux.on && lane == 0 && half == 0 && !ok) {
      // gave up with prefetches in flight: let them land (bounded) before the CTA's shared memory goes away
      for (uint32_t i = aux.consumed; i < aux.issued; ++i)
        for (uint32_t spin = 0; spin < MB_SPIN_LIMIT; ++spin)
          if (mbar_try_wait(&aux.bars[i % aux.slots], (i / aux.slots) & 1)) break;
    }
  }

  tc_fence_before();
  cluster_sync_all();                         // no CTA leaves while its pair may still touch its barriers or TMEM
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// ------------------------------------------------------------------------------------------------ host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static void check(bool ok, const char* what) {            // becomes a Python RuntimeError in the bindings
  if (!ok) throw std::runtime_error(what);
}

static EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q);
    check(e == cudaSuccess && p != nullptr, "cuTensorMapEncodeTiled entry point not found");
    fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

// 3-D tensor map: dims (inner, rows, groups), 128-byte swizzle, zero fill outside.  `esz` 1 = 8-bit, 2 = bf16, 4 = fp32.
CUtensorMap make_tmap(const void* base, int esz, uint64_t inner, uint64_t rows, uint64_t groups, uint64_t row_pitch_el,
                      uint64_t group_pitch_el, uint32_t box_inner, uint32_t box_rows, bool promote) {
  // cuTensorMapEncodeTiled is a driver call: a thread that has made no runtime call yet (an autograd worker) has no
  // current context and gets CUDA_ERROR_INVALID_CONTEXT, so bind the primary context once per thread.
  static thread_local bool ctx_bound = false;
  if (!ctx_bound) { cudaFree(nullptr); ctx_bound = true; }
  CUtensorMap m;
  cuuint64_t dims[3] = {inner, rows, groups};
  cuuint64_t strides[2] = {row_pitch_el * esz, (groups > 1 ? group_pitch_el : row_pitch_el * rows) * esz};
  cuuint32_t box[3] = {box_inner, box_rows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  check((reinterpret_cast<uintptr_t>(base) & 15) == 0, "TMA operand must be 16-byte aligned");
  check(strides[0] % 16 == 0 && strides[1] % 16 == 0, "TMA operand pitches must be multiples of 16 bytes");
  const CUtensorMapDataType dt = esz == 1 ? CU_TENSOR_MAP_DATA_TYPE_UINT8
                                : esz == 2 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
  CUresult r = encode_fn()(&m, dt, 3,
                           const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           CU_TENSOR_MAP_SWIZZLE_128B,
                           promote ? CU_TENSOR_MAP_L2_PROMOTION_L2_256B : CU_TENSOR_MAP_L2_PROMOTION_NONE,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) throw std::runtime_error("cuTensorMapEncodeTiled failed with code " + std::to_string(static_cast<int>(r)));
  return m;
}
CUtensorMap make_tmap_bf16(const void* base, uint64_t inner, uint64_t rows, uint64_t groups, uint64_t row_pitch_el,
                           uint64_t group_pitch_el, uint32_t box_inner, uint32_t box_rows) {
  return make_tmap(base, 2, inner, rows, groups, row_pitch_el, group_pitch_el, box_inner, box_rows, true);
}

int* gemm_status_word(int device) {
  static int* words[16] = {nullptr};
  check(device >= 0 && device < 16, "device index out of range");
  if (!words[device]) {
    check(cudaMalloc(&words[device], sizeof(int)) == cudaSuccess, "status word alloc failed");
    cudaMemset(words[device], 0, sizeof(int));
  }
  return words[device];
}

int gemm_status(int device) {
  int v = 0;
  cudaMemcpy(&v, gemm_status_word(device), sizeof(int), cudaMemcpyDeviceToHost);
  int z = 0;
  if (v) cudaMemcpy(gemm_status_word(device), &z, sizeof(int), cudaMemcpyHostToDevice);
  return v;
}

// The CTA-pair (cta_group::2) kernel is the default for tiles of >= 256 rows; MEMARCH_GEMM_PAIR=0 or
// gemm_set_pair(false) selects the single-CTA kernel everywhere.
static int g_pair = -1;
bool gemm_pair_on() {
  if (g_pair < 0) {
    const char* e = std::getenv("MEMARCH_GEMM_PAIR");
    g_pair = (e && e[0] == '0') ? 0 : 1;
  }
  return g_pair == 1;
}
void gemm_set_pair(bool on) { g_pair = on ? 1 : 0; }
// Test / measurement switches of the pair kernel (DBG_* bits) and the row-tile group size of its tile order.
static int g_dbg = 0, g_group_m = 0;
void gemm_set_debug(int64_t dbg, int64_t group_m) { g_dbg = (int)dbg; g_group_m = (int)group_m; }

static bool tma_stores_on() {
  static const bool off = []() { const char* e = std::getenv("MEMARCH_GEMM_TMA_STORE"); return e && e[0] == '0'; }();
  return !off && !(g_dbg & DBG_DIRECT_STORE);
}

// Raw launcher shared by the torch binding and the fused multi-GPU paths (which pass peer pointers for A).
// A_list: one base pointer per M-segment (n_seg of them, each (a_groups, seg_M, K) or MN-major (a_groups, K, seg_M)).
void launch_gemm_seg(const void* const* A_list, int n_seg, int seg_M, int a_groups, long long a_rows_pitch, long long a_gs,
                     bool a_mn, const void* B, long long b_rows_pitch, long long b_gs, bool b_mn, GemmParams p,
                     cudaStream_t stream, int max_ctas) {
  const int N = p.N, K = p.K, G = p.G;
  check(n_seg >= 1 && n_seg <= 8, "gemm: 1..8 segments");
  TmapSet tmAs;
  for (int i = 0; i < n_seg; ++i)
    tmAs.m[i] = a_mn ? make_tmap_bf16(A_list[i], seg_M, K, a_groups, a_rows_pitch, a_gs, 64, 64)
                     : make_tmap_bf16(A_list[i], K, seg_M, a_groups, a_rows_pitch, a_gs, 64, BM);
  for (int i = n_seg; i < 8; ++i) tmAs.m[i] = tmAs.m[0];
  const bool pair = gemm_pair_on() && seg_M >= 256;
  const bool sw = p.epi == EPI_SWIGLU;
  // Tiles of 128 columns where 256 would leave the CTA pairs short of work: the time of a small product is a pair's rounds of
  // tiles times the width of one (its MMAs and its epilogue); 15 % in favour of the wide tile, which reads A half as often.
  // Us, 256 -> 128 columns, (M, N, K): (2048, 256, 256) 8.8 -> 7.3; (2048, 256, 1024) 12.5 -> 11.1; (4096, 512, 512) 10.4 -> 9.3;
  // (256, 1024, 2048) 11.5 -> 10.1.
  auto tiles_of = [&](int bn) { return (long long)G * n_seg * ((seg_M + 255) / 256) * ((N + bn - 1) / bn) * std::max(1, p.splits); };
  auto rounds = [&](int bn) { const long long pairs = std::max(1, max_ctas / 2); return (tiles_of(bn) + pairs - 1) / pairs; };
  const bool narrow = pair && p.count_mode == 0 && rounds(128) * 128 * 115 < rounds(256) * 256 * 100;
  p.bn = narrow ? 128 : BN;
  const int n_tiles = (N + p.bn - 1) / p.bn;                 // SwiGLU: a tile holds bn / 2 columns of each half
  // 512-row tiles (see PairCfg) when the contraction is long enough to pay for the half-exposed epilogue and the
  // coarser tiling does not cost more in the last, partly filled wave of tiles than it saves
  bool tall = false;
  if (pair && !narrow && n_seg == 1 && p.count_mode == 0 && seg_M >= 1024 && !(sw && p.out2) && p.epi != EPI_DRELU2 &&
      p.epi != EPI_DSWIGLU) {
    auto wave_eff = [&](int tm) {
      const long long tiles = (long long)G * ((seg_M + tm - 1) / tm) * n_tiles, pairs = std::max(1, max_ctas / 2);
      return (double)tiles / (double)(((tiles + pairs - 1) / pairs) * pairs);
    };
    static const bool tall_env = []() { const char* e = std::getenv("MEMARCH_GEMM_TALL"); return !(e && e[0] == '0'); }();
    tall = tall_env && p.splits <= 1 && K >= 8192 && wave_eff(512) >= wave_eff(256) - 0.02;
    if (g_dbg & DBG_TALL_OFF) tall = false;
    if (g_dbg & DBG_TALL_ON) tall = true;
  }
  const int tile_m = pair ? (tall ? 512 : 256) : BM;
  p.n_seg = n_seg; p.seg_M = seg_M; p.tiles_per_seg = (seg_M + tile_m - 1) / tile_m;
  CUtensorMap tmB = b_mn ? make_tmap_bf16(B, N, K, G, b_rows_pitch, b_gs, 64, 64)
                         : make_tmap_bf16(B, K, N, G, b_rows_pitch, b_gs, 64, pair ? p.bn / 2 : (sw ? 128 : BN));
  p.m_tiles = n_seg * p.tiles_per_seg;
  p.n_tiles = n_tiles;
  static const bool ntail_on = []() { const char* e = std::getenv("MEMARCH_GEMM_NTAIL"); return !(e && e[0] == '0'); }();
  p.ntail = ntail_on ? 1 : 0;
  check(p.splits <= 1 || (pair && !tall && n_seg == 1 && G == 1 && p.count_mode == 0 && p.epi == EPI_NONE && p.out_f32 && !p.accumulate),
        "gemm: split contraction needs the pair kernel, a plain epilogue and fp32 slabs");
  const int total = G * p.m_tiles * p.n_tiles * std::max(1, p.splits);
  int grid = pair ? 2 * std::min(total, max_ctas / 2) : std::min(total, max_ctas);
  if (grid <= 0) return;
  const bool v3 = pair;
  check(v3 || p.count_mode == 0, "gemm: per-group extents need the pair kernel (>= 256 rows)");
  CUtensorMap tmO = tmB, tmO2 = tmB;
  if (v3) {
    p.dbg = g_dbg;
    p.group_m = g_group_m;
    const int esz = p.out_f32 ? 4 : 2;
    // TMA stores for a local, unsegmented output whose pitches keep the 16-byte rule; everything else leaves
    // through coalesced row stores (peer buffers are only ever written with plain stores)
    p.store_tma = (n_seg == 1 && !p.out_seg_on && (p.ldo * esz) % 16 == 0 && (G == 1 || (p.out_gs * esz) % 16 == 0) &&
                   (!p.out2 || ((p.ldo2 * 2) % 16 == 0 && (G == 1 || (p.out2_gs * 2) % 16 == 0)))) ? 1 : 0;
    if (!tma_stores_on()) p.store_tma = 0;
    if (p.store_tma) {
      const int No = sw ? N / 2 : N;
      tmO = make_tmap(p.out, esz, No, p.M, std::max(G, p.splits), p.ldo, p.out_gs, p.out_f32 ? 32 : 64, 32, false);
      if (p.out2) tmO2 = make_tmap(p.out2, 2, N, p.M, G, p.ldo2, p.out2_gs, 64, 32, false);
      // SwiGLU backward writes (d gate | d up) side by side: one map per half, so a ragged last chunk of the first
      // half is clipped at H instead of running into the second
      if (p.epi == EPI_DSWIGLU)
        tmO2 = make_tmap(reinterpret_cast<const char*>(p.out) + (size_t)N * 2, 2, N, p.M, G, p.ldo, p.out_gs, 64, 32, false);
    }
  }
  CUtensorMap tmX = tmB;
  p.aux_tma = 0;
  if (v3 && (p.epi == EPI_DRELU2 || p.epi == EPI_DSWIGLU)) {
    // the pre-activations are prefetched by TMA (see AuxPipe); MEMARCH_GEMM_AUX_TMA=0 keeps the warp's own loads
    static const bool aux_off = []() { const char* e = std::getenv("MEMARCH_GEMM_AUX_TMA"); return e && e[0] == '0'; }();
    const int Nx = p.epi == EPI_DSWIGLU ? 2 * N : N;
    if (!aux_off && (p.ldaux * 2) % 16 == 0 && (G == 1 || (p.aux_gs * 2) % 16 == 0) && N % 8 == 0) {
      // 256-byte L2 promotion: a row's next 128-byte piece (the next chunk of the same tile) arrives with this one
      tmX = make_tmap(p.aux, 2, Nx, (uint64_t)n_seg * seg_M, G, p.ldaux, p.aux_gs, 64, 32, true);
      p.aux_tma = 1;
    }
  }
  // eight epilogue warps where the pre-activations come and the results leave by TMA
  const int act = v3 && !tall && !a_mn && p.aux_tma && p.store_tma ? (p.epi == EPI_DSWIGLU ? ACT_SWIGLU : p.epi == EPI_DRELU2 ? ACT_RELU2 : ACT_NONE) : ACT_NONE;
  const int smem_bytes = !v3 ? SMEM_BYTES : tall ? PairCfg<2>::SMEM : act == ACT_SWIGLU ? PairCfg<1, ACT_SWIGLU>::SMEM : PairCfg<1>::SMEM;
  const int threads = act ? PairCfg<1, ACT_SWIGLU>::THREADS : GEMM_THREADS;
  auto launch = [&](auto kern, int id) {
    static bool attr_set[16][20] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (!attr_set[dev & 15][id]) {
      check(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes) == cudaSuccess,
                  "cannot raise dynamic shared memory for the GEMM kernel");
      attr_set[dev & 15][id] = true;
    }
    if constexpr (std::is_invocable_v<decltype(kern), TmapSet, CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, GemmParams>)
      kern<<<grid, threads, smem_bytes, stream>>>(tmAs, tmB, tmO, tmO2, tmX, p);
    else
      kern<<<grid, GEMM_THREADS, smem_bytes, stream>>>(tmAs, tmB, p);
  };
  const int id = (a_mn ? 2 : 0) + (b_mn ? 1 : 0);
  if (v3 && tall) {
    if (!a_mn && !b_mn) launch(gemm_pair_kernel<false, false, 2>, 12 + id);
    else if (!a_mn && b_mn) launch(gemm_pair_kernel<false, true, 2>, 12 + id);
    else if (a_mn && !b_mn) launch(gemm_pair_kernel<true, false, 2>, 12 + id);
    else launch(gemm_pair_kernel<true, true, 2>, 12 + id);
  } else if (act == ACT_SWIGLU) {
    if (!b_mn) launch(gemm_pair_kernel<false, false, 1, ACT_SWIGLU>, 4);
    else launch(gemm_pair_kernel<false, true, 1, ACT_SWIGLU>, 5);
  } else if (act == ACT_RELU2) {
    if (!b_mn) launch(gemm_pair_kernel<false, false, 1, ACT_RELU2>, 16);
    else launch(gemm_pair_kernel<false, true, 1, ACT_RELU2>, 17);
  } else if (v3) {
    if (!a_mn && !b_mn) launch(gemm_pair_kernel<false, false, 1>, 8 + id);
    else if (!a_mn && b_mn) launch(gemm_pair_kernel<false, true, 1>, 8 + id);
    else if (a_mn && !b_mn) launch(gemm_pair_kernel<true, false, 1>, 8 + id);
    else launch(gemm_pair_kernel<true, true, 1>, 8 + id);
  } else {
    if (!a_mn && !b_mn) launch(gemm_tc_kernel<false, false>, id);
    else if (!a_mn && b_mn) launch(gemm_tc_kernel<false, true>, id);
    else if (a_mn && !b_mn) launch(gemm_tc_kernel<true, false>, id);
    else launch(gemm_tc_kernel<true, true>, id);
  }
  const cudaError_t le = cudaGetLastError();
  check(le == cudaSuccess, cudaGetErrorString(le));
}

void launch_gemm(const void* A, long long a_rows_pitch, long long a_gs, bool a_mn, const void* B, long long b_rows_pitch,
                 long long b_gs, bool b_mn, GemmParams p, cudaStream_t stream, int max_ctas) {
  const void* list[1] = {A};
  launch_gemm_seg(list, 1, p.M, p.G, a_rows_pitch, a_gs, a_mn, B, b_rows_pitch, b_gs, b_mn, p, stream, max_ctas);
}

// out (+)= the sum of the slabs, always in the same order, whichever run ends first: L lanes add every L-th slab, then the lanes'
// sums are added one after the other.  The slabs were just written and are read from L2, 19 MB at most: latency.  Eight lanes from
// eight slabs on, (512, 512, K = 8192) in 18 runs 25.6 -> 23.6 us for product and sum; one lane below, (512, 1536, K = 4096) in 6
// runs 25.3 against 27.4 with four.
template <bool F32, int L>
__global__ void __launch_bounds__(256) sum_parts_kernel(const float4* __restrict__ parts, int splits, void* __restrict__ dst, int accumulate,
                                                        long long n4, int row4, int ldo) {
  constexpr int W = 256 / L;
  __shared__ float4 sh[L][W];
  const int cx = threadIdx.x % W, lane = threadIdx.x / W;
  for (long long i0 = blockIdx.x * (long long)W; i0 < n4; i0 += (long long)gridDim.x * W) {
    const long long i = i0 + cx;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i < n4) {
#pragma unroll 8
      for (int k = lane; k < splits; k += L) {
        const float4 v = parts[k * n4 + i];
        s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
      }
    }
    if (L > 1) {
      sh[lane][cx] = s;
      __syncthreads();
    }
    if (lane == 0 && i < n4) {
#pragma unroll
      for (int k = 1; k < L; ++k) { const float4 v = sh[k][cx]; s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w; }
      const long long r = i / row4, at = r * ldo + (i - r * row4) * 4;
      if (F32) {
        float4* o = reinterpret_cast<float4*>(reinterpret_cast<float*>(dst) + at);
        if (accumulate) { const float4 v = *o; s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w; }
        *o = s;
      } else {
        *reinterpret_cast<uint2*>(reinterpret_cast<bf16*>(dst) + at) = make_uint2(pack_bf16(s.x, s.y), pack_bf16(s.z, s.w));
      }
    }
    if (L > 1) __syncthreads();
  }
}
void sum_parts_launch(const float* parts, int splits, void* dst, int f32, int accumulate, long long rows, int n, int ldo, cudaStream_t stream) {
  const long long n4 = rows * (n / 4);
  const float4* src = reinterpret_cast<const float4*>(parts);
  auto go = [&](auto lanes) {
    constexpr int L = decltype(lanes)::value;
    const int grid = (int)std::min<long long>((n4 + 256 / L - 1) / (256 / L), 148 * 16);
    if (f32) sum_parts_kernel<true, L><<<grid, 256, 0, stream>>>(src, splits, dst, accumulate, n4, n / 4, ldo);
    else sum_parts_kernel<false, L><<<grid, 256, 0, stream>>>(src, splits, dst, 0, n4, n / 4, ldo);
  };
  if (splits >= 8) go(std::integral_constant<int, 8>()); else go(std::integral_constant<int, 1>());
}

// How many runs to cut the contraction of one plain product into (1: none).  A product with fewer output tiles than half of the
// 74 CTA pairs leaves the rest of the chip idle.  A cut saves each pair kb - kb_split k-blocks of 64 (0.27 us each) and costs a second
// launch and an fp32 slab per run and tile that is written and read back, 5 k-blocks and 0.31 per slab.  The line is measured
// against the whole product as launch_gemm_seg runs it, with 128-column tiles where it takes them, in runs of products back to
// back.  Us, (M, N, K), cut / whole: (256, 256, 2048) 14.5 / 17; (1024, 512, 2048) 16.5 / 18.6; (1536, 512, 2048) 17.5 / 18.6; (1024,
// 1024, 2048) 20.6 / 18.6 and 3072 20.8 / 24.3; (4096, 512, 2048) 22.6 / 20, 3072 25 / 25 and 4096 28.8 / 30.3; (1024, 256, 50304)
// 42 / 240.
int gemm_splits(int M, int N, int K, int G, int max_ctas, int& kb_split) {
  kb_split = 0;
  if (G != 1 || M < 256 || !gemm_pair_on()) return 1;
  const int tiles = ((M + 255) / 256) * ((N + BN - 1) / BN), pairs = max_ctas / 2, kb = (K + BK - 1) / BK;
  if (2 * tiles > pairs || kb < 32) return 1;
  const int want = std::min(pairs / tiles, kb / 8);
  if (want < 2) return 1;
  const int run = (kb + want - 1) / want, runs = (kb + run - 1) / run;
  if (100 * (kb - run) <= 500 + 31 * tiles * runs) return 1;
  kb_split = run;
  return runs;
}

int gemm_sm_count() {
  static int n = 0;
  if (!n) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  }
  return n;
}

}  // namespace mb
