// Causal / sliding-window attention backward on the tcgen05 tensor cores (head dim 64, bf16, fp32 accumulation).
//
// Two kernels, both persistent with two CTAs per SM (256 TMEM columns each), so that one CTA's products and copies run under
// the other's exponentials:
//   attn_dkv_kernel  item = (text, head, 128-key tile), walks the queries that see it, 64 at a time, keys in the TMEM lanes:
//       S^T = K Q^T, P^T = exp2(S^T scale - lse), dV += P^T dO;  dP^T = V dO^T, dS^T = P^T (dP^T - delta) scale, dK += dS^T Q
//   attn_dq_kernel   item = (text, head, 128-query tile), walks its keys, 64 at a time, queries in the lanes:
//       S = Q K^T, dP = dO V^T, dS as above, dQ += dS K
// P and dS go from registers to TMEM (over the scores they came from) and are the A operand of the products that follow:
// nothing is staged in shared memory, and no gradient is summed through global memory.  The scores are computed twice,
// which costs 2 of 7 products and a second set of exponentials.  The one-kernel form adds every dQ tile to fp32 sums in
// global memory (32 KB per pair of tiles) and was bound by that at about 1 TB/s, with its 448 TMEM columns leaving one
// CTA per SM: 32 texts x 32 heads x 1024 causal 1171 + 62 us against 603 + 428 now;
// 2 x 16 384 words, 16 heads, window 256: 415 + 46 + a 134 MB clear against 307 + 230 (library flash kernel 716).
// What bounds both: the special-function unit, 1024 clocks per 128 x 128 tile, with the products (1024 and 768) and the
// shared-memory reads of their operands (about 1000 and 900) close behind.
// dq and dk leave rotated back (when tables are given), all three in bf16 at the caller's strides: no pass follows.
// Every wait is bounded; on timeout the status word is set, roles stop, TMEM is freed and the kernels return.
#include <cuda.h>

#include <type_traits>

#include "attn_common.cuh"

namespace mb {

const char* attn_tmap(CUtensorMap* m, const AttnView& v, int B, int H, int T, int box_rows);

constexpr int AB_THREADS = 192;
constexpr int AB_TILE = 128 * 64 * 2;                    // 16 KB: 128 rows x 64 bf16
constexpr int AB_HALF = AB_TILE / 2;                     // 64 rows
constexpr int AB_STAT = 2 * 64 * 4;                      // lse, delta of 64 queries
constexpr int AB_STAGES = 4;                             // a copy takes longer than a step: three steps ahead
constexpr int AB_SMEM = 2 * AB_TILE + AB_STAGES * (2 * AB_HALF + AB_STAT) + 256;

struct AttnBwdParams {
  int T, window, H, half, tiles, units, pairs, nstat;
  float scale, scale_log2;
  const float* stats;
  AttnView dq, dk, dv;
  const float *cos, *sin;
  int* status;
};

__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}

// rotate a row of 64 gradients back by the angles of position t: (a, b) -> (a c + b s, b c - a s)
__device__ __forceinline__ void unrotate64(float* v, const float* cs, const float* sn, long long t, int half) {
#pragma unroll
  for (int i = 0; i < 32; i += 4) {
    const float4 c4 = *reinterpret_cast<const float4*>(cs + t * 32 + i), s4 = *reinterpret_cast<const float4*>(sn + t * 32 + i);
    const float c[4] = {c4.x, c4.y, c4.z, c4.w}, s[4] = {s4.x, s4.y, s4.z, s4.w};
    if (!half) {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float a = v[2 * (i + u)], b = v[2 * (i + u) + 1];
        v[2 * (i + u)] = a * c[u] + b * s[u];
        v[2 * (i + u) + 1] = b * c[u] - a * s[u];
      }
    } else {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float a = v[i + u], b = v[i + u + 32];
        v[i + u] = a * c[u] + b * s[u];
        v[i + u + 32] = b * c[u] - a * s[u];
      }
    }
  }
}
__device__ __forceinline__ void store_row64(bf16* dst, const float* v) {
#pragma unroll
  for (int j = 0; j < 64; j += 8)
    *reinterpret_cast<uint4*>(dst + j) = make_uint4(pack_bf16(v[j], v[j + 1]), pack_bf16(v[j + 2], v[j + 3]),
                                                    pack_bf16(v[j + 4], v[j + 5]), pack_bf16(v[j + 6], v[j + 7]));
}


// the barriers that both kernels use
struct AttnBwdBars {
  uint64_t *own_full, *own_empty;      // the item's own two 128-row tiles; empty: the item's last scores and dP are done
  uint64_t *st_full, *st_empty;        // AB_STAGES: the 64-row tiles walked over
  uint64_t *s_full, *dp_full;          // scores (2: a barrier per buffer of attn_dq_kernel), dP in TMEM
  uint64_t *p_full, *ds_full;          // P, dS in TMEM (4 warp arrivals)
  uint64_t *done;                      // all products of the item
  uint32_t* tmem_slot;
  volatile int* abort_flag;
  __device__ __forceinline__ explicit AttnBwdBars(uint8_t* at) {
    uint64_t* b = reinterpret_cast<uint64_t*>(at);
    own_full = b; own_empty = b + 1; st_full = b + 2; st_empty = st_full + AB_STAGES; s_full = st_empty + AB_STAGES;
    dp_full = s_full + 2; p_full = s_full + 3; ds_full = s_full + 4; done = s_full + 5;
    tmem_slot = reinterpret_cast<uint32_t*>(s_full + 6);
    abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  }
  __device__ __forceinline__ void init() {
    mbar_init(own_full, 1); mbar_init(own_empty, 1);
    for (int s = 0; s < AB_STAGES; ++s) { mbar_init(&st_full[s], 1); mbar_init(&st_empty[s], 1); }
    mbar_init(&s_full[0], 1); mbar_init(&s_full[1], 1); mbar_init(dp_full, 1); mbar_init(p_full, 4); mbar_init(ds_full, 4); mbar_init(done, 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
};

// ------------------------------------------------------------------------------------------------ dK, dV
__global__ void __launch_bounds__(AB_THREADS, 2)
attn_dkv_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO, const AttnBwdParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  if (threadIdx.x == 0 && (smem_u32(smem) & 1023u)) atomicCAS(p.status, 0, ST_BAD_ARG);
  uint8_t* sOwn = smem;                                   // K, V
  uint8_t* sSt = sOwn + 2 * AB_TILE;                      // stages x (Q, dO)
  uint8_t* sStat = sSt + AB_STAGES * 2 * AB_HALF;
  AttnBwdBars bar(sStat + AB_STAGES * AB_STAT);
  volatile int* abort_flag = bar.abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    bar.init();
    tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV); tma_prefetch_desc(&tmDO);
  }
  if (warp == 5) {
    tmem_alloc(bar.tmem_slot, 256);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tS = *bar.tmem_slot, tDP = tS + 64, tDV = tS + 128, tDK = tS + 192;
  auto give_up = [&](int code) { atomicCAS(p.status, 0, code); *abort_flag = 1; };
  struct Item { int k0, h, b, bh, n; };                   // n: 64-query steps from query k0 on
  auto item_at = [&](const AttnWalk& w) {
    Item it;
    it.bh = w.bh(); it.k0 = w.tile() * 128; it.h = it.bh % p.H; it.b = it.bh / p.H;
    const int last = p.window > 0 ? min(p.T - 1, it.k0 + 126 + p.window) : p.T - 1;
    it.n = ((last - it.k0) >> 6) + 1;
    return it;
  };

  if (warp == 4) {
    if (lane == 0) {
      int c = 0, n = 0;
      bool ok = true;
      for (AttnWalk w(p.units, p.tiles, p.pairs); w.valid() && ok; w.next(), ++n) {
        const Item it = item_at(w);
        if (!mbar_wait(bar.own_empty, (n & 1) ^ 1, abort_flag)) { give_up(ST_WAIT_EMPTY); break; }
        mbar_expect_tx(bar.own_full, 2 * AB_TILE);
        tma_load_4d(sOwn, &tmK, bar.own_full, 0, it.k0, it.h, it.b);
        tma_load_4d(sOwn + AB_TILE, &tmV, bar.own_full, 0, it.k0, it.h, it.b);
        for (int i = 0; i < it.n; ++i, ++c) {
          const int s = c % AB_STAGES;
          if (!mbar_wait(&bar.st_empty[s], ((c / AB_STAGES) & 1) ^ 1, abort_flag)) { give_up(ST_WAIT_EMPTY); ok = false; break; }
          const int q0 = it.k0 + i * 64;
          mbar_expect_tx(&bar.st_full[s], 2 * AB_HALF + AB_STAT);
          tma_load_4d(sSt + s * 2 * AB_HALF, &tmQ, &bar.st_full[s], 0, q0, it.h, it.b);
          bulk_load(sStat + s * AB_STAT, p.stats + ((long long)it.bh * p.nstat + (q0 >> 6)) * 128, AB_STAT, &bar.st_full[s]);
          tma_load_4d(sSt + s * 2 * AB_HALF + AB_HALF, &tmDO, &bar.st_full[s], 0, q0, it.h, it.b);
        }
      }
      if (*abort_flag) { for (int i = 0; i < 2000; ++i) __nanosleep(1000); }   // copies in flight land before the CTA leaves
    }
  } else if (warp == 5) {
    if (lane == 0) {
      const uint32_t id_kk = idesc_bf16(128, 64, 0u, 0u);        // K-major x K-major: S^T, dP^T
      const uint32_t id_ts = idesc_bf16(128, 64, 0u, 1u);        // A in TMEM, B MN-major: dV, dK
      bool ok = true;
      // scores and dP of step c (the n-th item).  They overwrite P and dS of step c - 1; the products that read those were
      // issued before, and products run in order.
      auto start = [&](int c, int n, bool first, bool last) {
        if ((first && !mbar_wait(bar.own_full, n & 1, abort_flag)) ||
            !mbar_wait(&bar.st_full[c % AB_STAGES], (c / AB_STAGES) & 1, abort_flag)) { give_up(ST_WAIT_FULL); ok = false; return; }
        tc_fence_after();
        const uint32_t aK = smem_u32(sOwn), aV = aK + AB_TILE;
        const uint32_t bQ = smem_u32(sSt + (c % AB_STAGES) * 2 * AB_HALF), bDO = bQ + AB_HALF;
#pragma unroll
        for (int k = 0; k < 4; ++k)
          umma_bf16(tS, smem_desc_sw128(aK + k * 32, 0, 1024), smem_desc_sw128(bQ + k * 32, 0, 1024), id_kk, k > 0 ? 1u : 0u);
        umma_commit(bar.s_full);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          umma_bf16(tDP, smem_desc_sw128(aV + k * 32, 0, 1024), smem_desc_sw128(bDO + k * 32, 0, 1024), id_kk, k > 0 ? 1u : 0u);
        umma_commit(bar.dp_full);
        if (last) umma_commit(bar.own_empty);
      };
      int c = 0, n = 0, steps = 0;
      {
        const AttnWalk w0(p.units, p.tiles, p.pairs);
        if (w0.valid()) { steps = item_at(w0).n; start(0, 0, true, steps == 1); }
      }
      for (AttnWalk w(p.units, p.tiles, p.pairs); w.valid() && ok; w.next(), ++n) {
        int next = 0;
        AttnWalk w1 = w;
        w1.next();
        if (w1.valid()) next = item_at(w1).n;
        for (int i = 0; i < steps && ok; ++i, ++c) {
          const uint32_t bQ = smem_u32(sSt + (c % AB_STAGES) * 2 * AB_HALF), bDO = bQ + AB_HALF;
          if (!mbar_wait(bar.p_full, c & 1, abort_flag)) { give_up(ST_WAIT_TMEM_FULL); ok = false; break; }
          tc_fence_after();
#pragma unroll
          for (int k = 0; k < 4; ++k)                            // contraction over the 64 queries, 16 per step
            umma_bf16_ts(tDV, tS + k * 8, smem_desc_sw128(bDO + k * 2048, 8192, 1024), id_ts, (i > 0 || k > 0) ? 1u : 0u);
          if (!mbar_wait(bar.ds_full, c & 1, abort_flag)) { give_up(ST_WAIT_TMEM_FULL); ok = false; break; }
          tc_fence_after();
#pragma unroll
          for (int k = 0; k < 4; ++k)
            umma_bf16_ts(tDK, tDP + k * 8, smem_desc_sw128(bQ + k * 2048, 8192, 1024), id_ts, (i > 0 || k > 0) ? 1u : 0u);
          umma_commit(&bar.st_empty[c % AB_STAGES]);
          if (i + 1 == steps) umma_commit(bar.done);
          if (i + 1 < steps) start(c + 1, n, false, i + 2 == steps);
          else if (next) start(c + 1, n + 1, true, next == 1);
        }
        steps = next;
      }
    }
  } else {
    // ------------------------------------------------------------------ P and dS (thread: one key row, 64 queries)
    const int row = warp * 32 + lane;
    const uint32_t lane_base = static_cast<uint32_t>(warp * 32) << 16;
    const float sc = p.scale_log2;
    bool ok = true;
    int c = 0, n = 0;
    for (AttnWalk w(p.units, p.tiles, p.pairs); w.valid() && ok; w.next(), ++n) {
      const Item it = item_at(w);
      const int kj = it.k0 + row;
      for (int i = 0; i < it.n; ++i, ++c) {
        const int q0 = it.k0 + i * 64, s = c % AB_STAGES;
        // the statistics came with Q: the wait makes the copy visible to this thread
        if (!mbar_wait(&bar.st_full[s], (c / AB_STAGES) & 1, abort_flag) || !mbar_wait(bar.s_full, c & 1, abort_flag)) { if (lane == 0) give_up(ST_WAIT_TMEM_FULL); ok = false; break; }
        tc_fence_after();
        __syncwarp();
        const float* lse2 = reinterpret_cast<const float*>(sStat + s * AB_STAT);
        // queries that key row 0 of the warp is seen by: columns [lo, hi], one further for each row; whole steps have straight
        // code of their own
        const int lo = it.k0 + warp * 32 - q0, hi = p.window > 0 ? lo + p.window - 1 : 1 << 20;
        auto step = [&](auto cut_) -> bool {
          constexpr bool CUT = decltype(cut_)::value;
          uint32_t r[2][32];
          float pv[64];
#pragma unroll
          for (int h = 0; h < 2; ++h)
            tmem_ld32(tS + lane_base + h * 32, r[h]);
          tmem_ld_wait();
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint32_t pk[16];
#pragma unroll
            for (int u = 0; u < 32; u += 4) {
              const float4 L = *reinterpret_cast<const float4*>(lse2 + h * 32 + u);
              pv[h * 32 + u] = ex2(fmaf(__uint_as_float(r[h][u]), sc, -L.x));
              pv[h * 32 + u + 1] = ex2(fmaf(__uint_as_float(r[h][u + 1]), sc, -L.y));
              pv[h * 32 + u + 2] = ex2(fmaf(__uint_as_float(r[h][u + 2]), sc, -L.z));
              pv[h * 32 + u + 3] = ex2(fmaf(__uint_as_float(r[h][u + 3]), sc, -L.w));
            }
            if (CUT) {
              const uint32_t bits = seen_bits(h * 32, lo + lane, hi + lane);
#pragma unroll
              for (int u = 0; u < 32; ++u)
                if (!(bits >> u & 1u)) pv[h * 32 + u] = 0.f;
            }
#pragma unroll
            for (int u = 0; u < 16; ++u) pk[u] = pack_bf16(pv[h * 32 + 2 * u], pv[h * 32 + 2 * u + 1]);
            tmem_st16(tS + lane_base + h * 16, pk);              // over scores that this warp has read
          }
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar.p_full);

          if (!mbar_wait(bar.dp_full, c & 1, abort_flag)) return false;
          tc_fence_after();
          __syncwarp();
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint32_t pk[16];
            tmem_ld32(tDP + lane_base + h * 32, r[h]);
            tmem_ld_wait();
#pragma unroll
            for (int u = 0; u < 32; u += 4) {
              const float4 D = *reinterpret_cast<const float4*>(lse2 + 64 + h * 32 + u);
              pk[u >> 1] = pack_bf16(pv[h * 32 + u] * (__uint_as_float(r[h][u]) - D.x) * p.scale, pv[h * 32 + u + 1] * (__uint_as_float(r[h][u + 1]) - D.y) * p.scale);
              pk[(u >> 1) + 1] = pack_bf16(pv[h * 32 + u + 2] * (__uint_as_float(r[h][u + 2]) - D.z) * p.scale, pv[h * 32 + u + 3] * (__uint_as_float(r[h][u + 3]) - D.w) * p.scale);
            }
            tmem_st16(tDP + lane_base + h * 16, pk);             // over columns that this warp has read
          }
          tmem_st_wait();
          return true;
        };
        const bool whole = lo + 31 <= 0 && hi >= 63;
        if (!(whole ? step(std::false_type()) : step(std::true_type()))) { if (lane == 0) give_up(ST_WAIT_TMEM_FULL); ok = false; break; }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar.ds_full);
      }
      if (ok && !mbar_wait(bar.done, n & 1, abort_flag)) { if (lane == 0) give_up(ST_WAIT_TMEM_FULL); ok = false; }
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
#pragma unroll
      for (int which = 0; which < 2; ++which) {                  // dV, then dK
        uint32_t r[2][32];
        __syncwarp();
        tmem_ld32((which ? tDK : tDV) + lane_base, r[0]);
        tmem_ld32((which ? tDK : tDV) + lane_base + 32, r[1]);
        tmem_ld_wait();
        float v[64];
#pragma unroll
        for (int u = 0; u < 64; ++u) v[u] = __uint_as_float(r[u >> 5][u & 31]);
        if (kj < p.T) {
          if (which && p.cos) unrotate64(v, p.cos, p.sin, kj, p.half);
          const AttnView& o = which ? p.dk : p.dv;
          store_row64(reinterpret_cast<bf16*>(o.p) + it.b * o.sb + (long long)kj * o.st + it.h * o.sh, v);
        }
      }
      tc_fence_before();                                         // both are read: ordered before the next item's p_full
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 5) {
    tc_fence_after();
    tmem_dealloc(tS, 256);
  }
}

// ------------------------------------------------------------------------------------------------ dQ
__global__ void __launch_bounds__(AB_THREADS, 2)
attn_dq_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
               const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO, const AttnBwdParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  if (threadIdx.x == 0 && (smem_u32(smem) & 1023u)) atomicCAS(p.status, 0, ST_BAD_ARG);
  uint8_t* sOwn = smem;                                   // Q, dO
  uint8_t* sSt = sOwn + 2 * AB_TILE;                      // stages x (K, V)
  AttnBwdBars bar(sSt + AB_STAGES * (2 * AB_HALF + AB_STAT));
  volatile int* abort_flag = bar.abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    bar.init();
    tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV); tma_prefetch_desc(&tmDO);
  }
  if (warp == 5) {
    tmem_alloc(bar.tmem_slot, 256);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tBase = *bar.tmem_slot, tDP = tBase + 128, tDQ = tBase + 192;      // scores: columns 0..63 and 64..127 in turn
  auto give_up = [&](int code) { atomicCAS(p.status, 0, code); *abort_flag = 1; };
  struct Item { int q0, h, b, bh, first, n; };            // 64-key tiles [first, first + n)
  auto item_at = [&](const AttnWalk& w) {
    Item it;
    it.bh = w.bh(); it.q0 = w.tile() * 128; it.h = it.bh % p.H; it.b = it.bh / p.H;
    it.first = p.window > 0 ? max(0, it.q0 - p.window + 1) >> 6 : 0;
    it.n = (min(p.T - 1, it.q0 + 127) >> 6) - it.first + 1;
    return it;
  };

  if (warp == 4) {
    if (lane == 0) {
      int c = 0, n = 0;
      bool ok = true;
      for (AttnWalk w(p.units, p.tiles, p.pairs); w.valid() && ok; w.next(), ++n) {
        const Item it = item_at(w);
        if (!mbar_wait(bar.own_empty, (n & 1) ^ 1, abort_flag)) { give_up(ST_WAIT_EMPTY); break; }
        mbar_expect_tx(bar.own_full, 2 * AB_TILE);
        tma_load_4d(sOwn, &tmQ, bar.own_full, 0, it.q0, it.h, it.b);
        tma_load_4d(sOwn + AB_TILE, &tmDO, bar.own_full, 0, it.q0, it.h, it.b);
        for (int i = 0; i < it.n; ++i, ++c) {
          const int s = c % AB_STAGES;
          if (!mbar_wait(&bar.st_empty[s], ((c / AB_STAGES) & 1) ^ 1, abort_flag)) { give_up(ST_WAIT_EMPTY); ok = false; break; }
          const int k0 = (it.first + i) * 64;
          mbar_expect_tx(&bar.st_full[s], 2 * AB_HALF);
          tma_load_4d(sSt + s * 2 * AB_HALF, &tmK, &bar.st_full[s], 0, k0, it.h, it.b);
          tma_load_4d(sSt + s * 2 * AB_HALF + AB_HALF, &tmV, &bar.st_full[s], 0, k0, it.h, it.b);
        }
      }
      if (*abort_flag) { for (int i = 0; i < 2000; ++i) __nanosleep(1000); }
    }
  } else if (warp == 5) {
    if (lane == 0) {
      const uint32_t id_kk = idesc_bf16(128, 64, 0u, 0u);
      const uint32_t id_ts = idesc_bf16(128, 64, 0u, 1u);
      bool ok = true;
      // Two score buffers, each with its own barrier: at the end of an item the softmax warps write dQ out and may look at the
      // scores late, when those of the step after are already done.  Buffer c & 1 was read before ds_full(c - 2).
      auto scores = [&](int c, int n, bool first) {
        if ((first && !mbar_wait(bar.own_full, n & 1, abort_flag)) ||
            !mbar_wait(&bar.st_full[c % AB_STAGES], (c / AB_STAGES) & 1, abort_flag)) { give_up(ST_WAIT_FULL); ok = false; return; }
        tc_fence_after();
        const uint32_t aQ = smem_u32(sOwn), bK = smem_u32(sSt + (c % AB_STAGES) * 2 * AB_HALF);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          umma_bf16(tBase + (c & 1) * 64, smem_desc_sw128(aQ + k * 32, 0, 1024), smem_desc_sw128(bK + k * 32, 0, 1024), id_kk, k > 0 ? 1u : 0u);
        umma_commit(&bar.s_full[c & 1]);
      };
      auto dprod = [&](int c, bool last) {                // overwrites dS of step c - 1, which dQ (issued before) reads first
        const uint32_t aDO = smem_u32(sOwn + AB_TILE), bV = smem_u32(sSt + (c % AB_STAGES) * 2 * AB_HALF + AB_HALF);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          umma_bf16(tDP, smem_desc_sw128(aDO + k * 32, 0, 1024), smem_desc_sw128(bV + k * 32, 0, 1024), id_kk, k > 0 ? 1u : 0u);
        umma_commit(bar.dp_full);
        if (last) umma_commit(bar.own_empty);
      };
      int c = 0, n = 0, steps = 0;
      {
        const AttnWalk w0(p.units, p.tiles, p.pairs);
        if (w0.valid()) { steps = item_at(w0).n; scores(0, 0, true); if (ok) dprod(0, steps == 1); }
      }
      for (AttnWalk w(p.units, p.tiles, p.pairs); w.valid() && ok; w.next(), ++n) {
        int next = 0;
        AttnWalk w1 = w;
        w1.next();
        if (w1.valid()) next = item_at(w1).n;
        for (int i = 0; i < steps && ok; ++i, ++c) {
          const bool same = i + 1 < steps;                       // the next step belongs to this item
          if (same) scores(c + 1, n, false);
          if (!ok) break;
          if (!mbar_wait(bar.ds_full, c & 1, abort_flag)) { give_up(ST_WAIT_TMEM_FULL); ok = false; break; }
          tc_fence_after();
          const uint32_t bK = smem_u32(sSt + (c % AB_STAGES) * 2 * AB_HALF);
#pragma unroll
          for (int k = 0; k < 4; ++k)                            // contraction over the 64 keys, 16 per step
            umma_bf16_ts(tDQ, tDP + k * 8, smem_desc_sw128(bK + k * 2048, 8192, 1024), id_ts, (i > 0 || k > 0) ? 1u : 0u);
          umma_commit(&bar.st_empty[c % AB_STAGES]);
          if (!same) umma_commit(bar.done);
          if (!same && next) scores(c + 1, n + 1, true);         // after dQ: the wait for the next item's Q must not hold it up
          if (ok && (same || next)) dprod(c + 1, same ? i + 2 == steps : next == 1);
        }
        steps = next;
      }
    }
  } else {
    // ------------------------------------------------------------------ dS (thread: one query row, 64 keys)
    const int row = warp * 32 + lane;
    const uint32_t lane_base = static_cast<uint32_t>(warp * 32) << 16;
    const float sc = p.scale_log2;
    bool ok = true;
    int c = 0, n = 0;
    for (AttnWalk w(p.units, p.tiles, p.pairs); w.valid() && ok; w.next(), ++n) {
      const Item it = item_at(w);
      const int qi = it.q0 + row;
      // rows past T lie in the padded part of the statistics' last 64, or past them: no weight
      const float* st = p.stats + ((long long)it.bh * p.nstat + (qi >> 6)) * 128 + (qi & 63);
      const float lse2 = qi < p.T ? st[0] : INFINITY, dlt = qi < p.T ? st[64] : 0.f;
      for (int i = 0; i < it.n; ++i, ++c) {
        const int k0 = (it.first + i) * 64;
        if (!mbar_wait(&bar.s_full[c & 1], (c >> 1) & 1, abort_flag)) { if (lane == 0) give_up(ST_WAIT_TMEM_FULL); ok = false; break; }
        tc_fence_after();
        __syncwarp();
        // keys that query row 0 of the warp sees: columns [lo, hi], one further for each row
        const int hi = it.q0 + warp * 32 - k0, lo = p.window > 0 ? hi - p.window + 1 : -(1 << 20);
        auto step = [&](auto cut_) -> bool {
          constexpr bool CUT = decltype(cut_)::value;
          uint32_t r[2][32];
          float pv[64];
#pragma unroll
          for (int h = 0; h < 2; ++h)
            tmem_ld32(tBase + (c & 1) * 64 + lane_base + h * 32, r[h]);
          tmem_ld_wait();
#pragma unroll
          for (int h = 0; h < 2; ++h) {
#pragma unroll
            for (int u = 0; u < 32; ++u) pv[h * 32 + u] = ex2(fmaf(__uint_as_float(r[h][u]), sc, -lse2));
            if (CUT) {
              const uint32_t bits = seen_bits(h * 32, lo + lane, hi + lane);
#pragma unroll
              for (int u = 0; u < 32; ++u)
                if (!(bits >> u & 1u)) pv[h * 32 + u] = 0.f;
            }
          }
          if (!mbar_wait(bar.dp_full, c & 1, abort_flag)) return false;
          tc_fence_after();
          __syncwarp();
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint32_t pk[16];
            tmem_ld32(tDP + lane_base + h * 32, r[h]);
            tmem_ld_wait();
#pragma unroll
            for (int u = 0; u < 32; u += 2)
              pk[u >> 1] = pack_bf16(pv[h * 32 + u] * (__uint_as_float(r[h][u]) - dlt) * p.scale, pv[h * 32 + u + 1] * (__uint_as_float(r[h][u + 1]) - dlt) * p.scale);
            tmem_st16(tDP + lane_base + h * 16, pk);             // over columns that this warp has read
          }
          tmem_st_wait();
          return true;
        };
        const bool whole = hi >= 63 && lo + 31 <= 0;
        if (!(whole ? step(std::false_type()) : step(std::true_type()))) { if (lane == 0) give_up(ST_WAIT_TMEM_FULL); ok = false; break; }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar.ds_full);
      }
      if (ok && !mbar_wait(bar.done, n & 1, abort_flag)) { if (lane == 0) give_up(ST_WAIT_TMEM_FULL); ok = false; }
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      uint32_t r[2][32];
      tmem_ld32(tDQ + lane_base, r[0]);
      tmem_ld32(tDQ + lane_base + 32, r[1]);
      tmem_ld_wait();
      if (qi < p.T) {
        float v[64];
#pragma unroll
        for (int u = 0; u < 64; ++u) v[u] = __uint_as_float(r[u >> 5][u & 31]);
        if (p.cos) unrotate64(v, p.cos, p.sin, qi, p.half);
        store_row64(reinterpret_cast<bf16*>(p.dq.p) + it.b * p.dq.sb + (long long)qi * p.dq.st + it.h * p.dq.sh, v);
      }
      tc_fence_before();                                         // dQ is read: ordered before the next item's ds_full
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 5) {
    tc_fence_after();
    tmem_dealloc(tBase, 256);
  }
}

// ------------------------------------------------------------------------------------------------ statistics
// stats[bh][t / 64][0][t % 64] = lse * log2(e) (+inf past T: no weight), [1] = sum_d dO * O.  One block per 128 positions, 8
// lanes per row (16 bytes of each array per lane).
__global__ void __launch_bounds__(256) attn_stats_kernel(AttnView o, AttnView dout, const float* __restrict__ lse,
                                                         float* __restrict__ stats, int T, int H, int tiles) {
  const long long bh = blockIdx.x / tiles;
  const int tile = (int)(blockIdx.x - bh * tiles), l8 = threadIdx.x & 7;
  const int h = (int)(bh % H), b = (int)(bh / H);
#pragma unroll
  for (int pass = 0; pass < 4; ++pass) {
    const int r = pass * 32 + (threadIdx.x >> 3), t = tile * 128 + r;
    float acc = 0.f;
    if (t < T) {
      const uint4 x = *reinterpret_cast<const uint4*>(reinterpret_cast<const bf16*>(o.p) + b * o.sb + (long long)t * o.st + h * o.sh + l8 * 8);
      const uint4 y = *reinterpret_cast<const uint4*>(reinterpret_cast<const bf16*>(dout.p) + b * dout.sb + (long long)t * dout.st + h * dout.sh + l8 * 8);
      const uint32_t xs[4] = {x.x, x.y, x.z, x.w}, ys[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 u = unpack_bf16(xs[j]), w = unpack_bf16(ys[j]);
        acc += u.x * w.x + u.y * w.y;
      }
    }
    acc += __shfl_xor_sync(0xffffffffu, acc, 1);
    acc += __shfl_xor_sync(0xffffffffu, acc, 2);
    acc += __shfl_xor_sync(0xffffffffu, acc, 4);
    if (l8 == 0) {
      float* out = stats + ((bh * tiles + tile) * 2 + (r >> 6)) * 128 + (r & 63);
      out[0] = t < T ? lse[bh * T + t] * 1.4426950408889634f : INFINITY;
      out[64] = acc;
    }
  }
}

const char* attn_bwd_launch(const AttnArgs& a) {
  const long long items = attn_tiles(a.T) * a.H * a.B;
  if (items > (1ll << 30)) return "attention: too many tiles";
  CUtensorMap q128, k128, v128, do128, q64, k64, v64, do64;
  struct { CUtensorMap* m; const AttnView* v; int rows; } maps[] = {{&q128, &a.q, 128}, {&do128, &a.dout, 128}, {&k64, &a.k, 64}, {&v64, &a.v, 64},
                                                                     {&k128, &a.k, 128}, {&v128, &a.v, 128}, {&q64, &a.q, 64}, {&do64, &a.dout, 64}};
  for (auto& m : maps)
    if (const char* e = attn_tmap(m.m, *m.v, a.B, a.H, a.T, m.rows)) return e;
  for (const AttnView* v : {&a.o, &a.dq, &a.dk, &a.dv})
    if ((reinterpret_cast<uintptr_t>(v->p) & 15) || v->sb % 8 || v->st % 8 || v->sh % 8) return "attention gradient rows must start on 16-byte boundaries";
  AttnBwdParams p{};
  p.T = a.T; p.H = a.H; p.half = a.rope_half;
  p.window = (a.window > 0 && a.window < a.T) ? a.window : 0;
  p.tiles = (int)attn_tiles(a.T); p.nstat = 2 * p.tiles;
  attn_units((long long)a.B * a.H, p.tiles, p.window == 0, 2 * 148, p.units, p.pairs);
  p.scale = a.scale;
  p.scale_log2 = a.scale * 1.4426950408889634f;
  p.stats = a.stats;
  p.dq = a.dq; p.dk = a.dk; p.dv = a.dv;
  p.cos = a.cos; p.sin = a.sin;
  p.status = a.status;
  if (cudaFuncSetAttribute(attn_dkv_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, AB_SMEM) != cudaSuccess ||
      cudaFuncSetAttribute(attn_dq_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, AB_SMEM) != cudaSuccess)
    return "cannot raise dynamic shared memory for the attention backward kernels";
  const int grid = p.units < 2 * 148 ? p.units : 2 * 148;
  attn_stats_kernel<<<(unsigned)items, 256, 0, a.stream>>>(a.o, a.dout, a.lse, a.stats, a.T, a.H, p.tiles);
  attn_dkv_kernel<<<grid, AB_THREADS, AB_SMEM, a.stream>>>(q64, k128, v128, do64, p);
  attn_dq_kernel<<<grid, AB_THREADS, AB_SMEM, a.stream>>>(q128, k64, v64, do128, p);
  return nullptr;
}

}  // namespace mb
