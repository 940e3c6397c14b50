// Causal / sliding-window attention forward on the tcgen05 tensor cores (head dim 64, bf16 in, fp32 softmax).
//
// Work items are (text, head, 128-query tile).  The kernel is persistent, two CTAs per SM: while one CTA's softmax runs, the
// other's products do, and within a CTA the copies and the first scores of the next item are under way before the
// current one is written out.  2 x 16 384 words, 16 heads, window 256: 141 us (library flash kernel 440, the one-item
// kernel with P in shared memory and its three copies of q, k, v 86 + 99 for a third of that work); 16 384 causal: 0.75 ms.
// Warps 0..3: softmax, thread = one query row (TMEM lane); warp 4: TMA producer (Q once, K and V tiles through
// two-stage rings of their own); warp 5: MMA issuer.  Per 128-key tile i:
//   S = Q K^T            128x128x64 into TMEM columns 0..127
//   softmax warps pull the whole row of S into registers and hand the columns back at once, so that the product
//   of tile i+1 is under way during the exponentials of tile i
//   P (bf16) goes back to TMEM columns 128..191 and is the A operand of   O += P V   (columns 192..255, V MN-major)
// P in TMEM instead of shared memory: the second product would otherwise read 48 KB of shared memory per tile (384
// clocks at 128 B/clk, against 256 clocks of multiplying) and the softmax warps would write 32 KB more.
// O stays in TMEM.  It is rescaled only when a row's maximum has grown by more than 2^8 since the reference it is
// scaled by (the quotient O / l does not depend on the reference; 2^8 leaves fp32 and bf16 far from their range).
// What bounds it: the special-function unit, 128 * 128 exponentials at 16 per clock = 1024 clocks per tile against 512
// clocks of products.  Only tiles cut by the diagonal or by the window's edge pay for the mask.
// Q, K, V are read through 4-D tensor maps over (64, T, H, B) with the caller's strides: slices of a packed qkv need no
// copies.  Every mbarrier wait is bounded; on timeout the status word is set, roles stop, TMEM is freed and the kernel
// returns.
#include <cuda.h>

#include <type_traits>

#include "attn_common.cuh"

namespace mb {

constexpr int AF_THREADS = 192;
constexpr int AF_TILE = 128 * 64 * 2;                    // 16 KB: 128 rows x 64 bf16
constexpr int AF_SMEM = 2 * AF_TILE + 2 * 2 * AF_TILE + 256;    // Q of two items, two K/V stages

struct AttnFwdParams {
  int T, window, H, tiles, units, pairs;
  float scale_log2;         // scale * log2(e)
  bf16* o;
  long long osb, ost, osh;
  float* lse;
  int* status;
};

__global__ void __launch_bounds__(AF_THREADS, 2)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                const __grid_constant__ CUtensorMap tmV, const AttnFwdParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];       // swizzle atoms are 1024 bytes: the base itself is aligned
  if (threadIdx.x == 0 && (smem_u32(smem) & 1023u)) atomicCAS(p.status, 0, ST_BAD_ARG);
  uint8_t* sQ = smem;                                     // 2 items
  uint8_t* sK = sQ + 2 * AF_TILE;                         // 2 stages
  uint8_t* sV = sK + 2 * AF_TILE;                         // 2 stages
  uint64_t* bars = reinterpret_cast<uint64_t*>(sV + 2 * AF_TILE);
  uint64_t* q_full = bars;            // 2
  uint64_t* q_empty = bars + 2;       // 2
  uint64_t* k_full = bars + 4;        // 2
  uint64_t* k_empty = bars + 6;       // 2: the scores are done
  uint64_t* v_full = bars + 8;        // 2
  uint64_t* v_empty = bars + 10;      // 2
  uint64_t* s_full = bars + 12;       // S ready in TMEM
  uint64_t* s_free = bars + 13;       // S is in registers (4 warp arrivals)
  uint64_t* p_full = bars + 14;       // P ready in TMEM, O rescaled if need be, O of the last item read (4 warp arrivals)
  uint64_t* o_full = bars + 15;       // P V of this tile added to O
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 16);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) { mbar_init(&q_full[s], 1); mbar_init(&q_empty[s], 1); mbar_init(&k_full[s], 1); mbar_init(&k_empty[s], 1); mbar_init(&v_full[s], 1); mbar_init(&v_empty[s], 1); }
    mbar_init(s_full, 1); mbar_init(s_free, 4); mbar_init(p_full, 4); mbar_init(o_full, 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV);
  }
  if (warp == 5) {
    tmem_alloc(tmem_slot, 256);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tS = tmem_base, tP = tmem_base + 128, tO = tmem_base + 192;
  auto give_up = [&](int code) { atomicCAS(p.status, 0, code); *abort_flag = 1; };
  struct Item { int q0, h, b, first_kt, n_kt; };
  auto item_at = [&](const AttnWalk& w) {
    Item it;
    const int bh = w.bh(), tile = w.tile();
    it.q0 = tile * 128; it.h = bh % p.H; it.b = bh / p.H;
    it.first_kt = p.window > 0 ? max(0, it.q0 - p.window + 1) >> 7 : 0;
    it.n_kt = tile - it.first_kt + 1;
    return it;
  };

  if (warp == 4) {
    if (lane == 0) {
      int c = 0, n = 0;                                   // key tiles, items so far
      bool ok = true;
      for (AttnWalk w(p.units, p.tiles, p.pairs); w.valid() && ok; w.next(), ++n) {
        const Item it = item_at(w);
        if (!mbar_wait(&q_empty[n & 1], ((n >> 1) & 1) ^ 1, abort_flag)) { give_up(ST_WAIT_EMPTY); break; }
        mbar_expect_tx(&q_full[n & 1], AF_TILE);
        tma_load_4d(sQ + (n & 1) * AF_TILE, &tmQ, &q_full[n & 1], 0, it.q0, it.h, it.b);
        for (int i = 0; i < it.n_kt; ++i, ++c) {
          const int s = c & 1;
          const int k0 = (it.first_kt + i) * 128;
          // K is free again as soon as its scores are, a whole tile before V
          if (!mbar_wait(&k_empty[s], ((c >> 1) & 1) ^ 1, abort_flag)) { give_up(ST_WAIT_EMPTY); ok = false; break; }
          mbar_expect_tx(&k_full[s], AF_TILE);
          tma_load_4d(sK + s * AF_TILE, &tmK, &k_full[s], 0, k0, it.h, it.b);
          if (!mbar_wait(&v_empty[s], ((c >> 1) & 1) ^ 1, abort_flag)) { give_up(ST_WAIT_EMPTY); ok = false; break; }
          mbar_expect_tx(&v_full[s], AF_TILE);
          tma_load_4d(sV + s * AF_TILE, &tmV, &v_full[s], 0, k0, it.h, it.b);
        }
      }
      if (*abort_flag) { for (int i = 0; i < 2000; ++i) __nanosleep(1000); }   // copies in flight land before the CTA leaves
    }
  } else if (warp == 5) {
    if (lane == 0) {
      const uint32_t idesc_qk = idesc_bf16(128, 128, 0u, 0u);
      const uint32_t idesc_pv = idesc_bf16(128, 64, 0u, 1u);
      bool ok = true;
      // scores of key tile c (the n-th item's Q); `last`: no later tile of the item reads Q
      auto scores = [&](int c, int n, bool first, bool last) {
        if ((first && !mbar_wait(&q_full[n & 1], (n >> 1) & 1, abort_flag)) || !mbar_wait(&k_full[c & 1], (c >> 1) & 1, abort_flag)) { give_up(ST_WAIT_FULL); ok = false; return; }
        if (c > 0 && !mbar_wait(s_free, (c - 1) & 1, abort_flag)) { give_up(ST_WAIT_TMEM_EMPTY); ok = false; return; }
        tc_fence_after();
        const uint32_t aQ = smem_u32(sQ + (n & 1) * AF_TILE), bK = smem_u32(sK + (c & 1) * AF_TILE);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          umma_bf16(tS, smem_desc_sw128(aQ + k * 32, 0, 1024), smem_desc_sw128(bK + k * 32, 0, 1024), idesc_qk, k > 0 ? 1u : 0u);
        umma_commit(s_full);
        umma_commit(&k_empty[c & 1]);
        if (last) umma_commit(&q_empty[n & 1]);
      };
      int c = 0, n = 0;
      int n_kt = 0;
      {
        const AttnWalk w0(p.units, p.tiles, p.pairs);
        if (w0.valid()) { n_kt = item_at(w0).n_kt; scores(0, 0, true, n_kt == 1); }
      }
      for (AttnWalk w(p.units, p.tiles, p.pairs); w.valid() && ok; w.next(), ++n) {
        int next_kt = 0;
        AttnWalk w1 = w;
        w1.next();
        if (w1.valid()) next_kt = item_at(w1).n_kt;
        for (int i = 0; i < n_kt && ok; ++i, ++c) {
          if (i + 1 < n_kt) scores(c + 1, n, false, i + 2 == n_kt);
          else if (next_kt) scores(c + 1, n + 1, true, next_kt == 1);
          if (!ok) break;
          if (!mbar_wait(&v_full[c & 1], (c >> 1) & 1, abort_flag)) { give_up(ST_WAIT_FULL); ok = false; break; }
          if (!mbar_wait(p_full, c & 1, abort_flag)) { give_up(ST_WAIT_TMEM_FULL); ok = false; break; }
          tc_fence_after();
          const uint32_t bV = smem_u32(sV + (c & 1) * AF_TILE);
#pragma unroll
          for (int k = 0; k < 8; ++k)                                          // contraction over the 128 keys, 16 per step
            umma_bf16_ts(tO, tP + k * 8, smem_desc_sw128(bV + k * 2048, 8192, 1024), idesc_pv, (i > 0 || k > 0) ? 1u : 0u);
          umma_commit(o_full);
          umma_commit(&v_empty[c & 1]);
        }
        n_kt = next_kt;
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax (one query row per thread)
    const int row = warp * 32 + lane;
    const uint32_t lane_base = static_cast<uint32_t>(warp * 32) << 16;
    const float sc = p.scale_log2;
    bool ok = true;
    int tc = 0;                                           // key tiles so far
    for (AttnWalk w(p.units, p.tiles, p.pairs); w.valid() && ok; w.next()) {
      const Item it = item_at(w);
      const int qi = it.q0 + row;
      float m = -INFINITY, l = 0.f;                       // m: the reference O and l are scaled by
      for (int i = 0; i < it.n_kt; ++i, ++tc) {
        const int k0 = (it.first_kt + i) * 128;
        if (!mbar_wait(s_full, tc & 1, abort_flag)) { if (lane == 0) give_up(ST_WAIT_TMEM_FULL); ok = false; break; }
        tc_fence_after();
        __syncwarp();
        // columns row 0 of the warp sees: [lo, hi]; the others one further each.  Whole tiles have
        // code of their own without the mask.  (Leaving out the 32-column chunks that a warp does not see at all cost more in
        // branches and spilled registers than it saved.)
        const int hi = it.q0 + warp * 32 - k0, lo = p.window > 0 ? hi - p.window + 1 : -(1 << 20);
        auto tile = [&](auto cut_) -> bool {
          constexpr bool CUT = decltype(cut_)::value;
          uint32_t r[4][32];
#pragma unroll
          for (int c = 0; c < 4; ++c) tmem_ld32(tS + lane_base + c * 32, r[c]);
          tmem_ld_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(s_free);
          float mc[4];
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            mc[c] = -INFINITY;
            if (CUT) {
              const uint32_t bits = seen_bits(c * 32, lo + lane, hi + lane);
#pragma unroll
              for (int jj = 0; jj < 32; ++jj)
                if (!(bits >> jj & 1u)) r[c][jj] = 0xFF800000u;                  // -infinity
            }
#pragma unroll
            for (int jj = 0; jj < 32; ++jj) mc[c] = fmaxf(mc[c], __uint_as_float(r[c][jj]));
          }
          const float mx = fmaxf(fmaxf(mc[0], mc[1]), fmaxf(mc[2], mc[3])) * sc;
          if (i == 0) {
            m = mx;
          } else {
            // the products of tile i-1 have read P and added to O by now or soon: they were issued before these maxima
            if (!mbar_wait(o_full, (tc - 1) & 1, abort_flag)) return false;
            tc_fence_after();
            if (__any_sync(0xffffffffu, mx > m + 8.f)) {
              const float m_new = fmaxf(m, mx);
              const float alpha = m_new == m ? 1.f : ex2(m - m_new);             // m = -inf: nothing seen yet, 0
              m = m_new;
              l *= alpha;
#pragma unroll 1
              for (int c = 0; c < 4; ++c) {
                uint32_t t[16];
                __syncwarp();
                tmem_ld16(tO + lane_base + c * 16, t);
                tmem_ld_wait();
#pragma unroll
                for (int jj = 0; jj < 16; ++jj) t[jj] = __float_as_uint(__uint_as_float(t[jj]) * alpha);
                tmem_st16(tO + lane_base + c * 16, t);
              }
            }
          }
          const float ref = m == -INFINITY ? 0.f : m;
          float s0 = 0.f, s1 = 0.f;
          __syncwarp();
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint32_t pk[16];
#pragma unroll
            for (int jj = 0; jj < 32; jj += 2) {
              const float e0 = ex2(fmaf(__uint_as_float(r[c][jj]), sc, -ref)), e1 = ex2(fmaf(__uint_as_float(r[c][jj + 1]), sc, -ref));
              s0 += e0; s1 += e1;
              pk[jj >> 1] = pack_bf16(e0, e1);
            }
            tmem_st16(tP + lane_base + c * 16, pk);
          }
          l += s0 + s1;
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(p_full);
          return true;
        };
        const bool whole = hi >= 127 && lo + 31 <= 0;
        if (!(whole ? tile(std::false_type()) : tile(std::true_type()))) { if (lane == 0) give_up(ST_WAIT_TMEM_FULL); ok = false; break; }
      }
      if (ok && !mbar_wait(o_full, (tc - 1) & 1, abort_flag)) { if (lane == 0) give_up(ST_WAIT_TMEM_FULL); ok = false; }
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      const float inv = l > 0.f ? 1.f / l : 0.f;
      bf16* orow = p.o + it.b * p.osb + (long long)qi * p.ost + it.h * p.osh;
      uint32_t t[2][32];
      tmem_ld32(tO + lane_base, t[0]);
      tmem_ld32(tO + lane_base + 32, t[1]);
      tmem_ld_wait();
      if (qi < p.T) {
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
          for (int jj = 0; jj < 32; jj += 8)
            *reinterpret_cast<uint4*>(orow + c * 32 + jj) =
                make_uint4(pack_bf16(__uint_as_float(t[c][jj]) * inv, __uint_as_float(t[c][jj + 1]) * inv),
                           pack_bf16(__uint_as_float(t[c][jj + 2]) * inv, __uint_as_float(t[c][jj + 3]) * inv),
                           pack_bf16(__uint_as_float(t[c][jj + 4]) * inv, __uint_as_float(t[c][jj + 5]) * inv),
                           pack_bf16(__uint_as_float(t[c][jj + 6]) * inv, __uint_as_float(t[c][jj + 7]) * inv));
        p.lse[((long long)it.b * p.H + it.h) * p.T + qi] = (l > 0.f) ? (m + log2f(l)) * 0.6931471805599453f : -INFINITY;
      }
      tc_fence_before();                                  // O is read: ordered before the next item's p_full
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 5) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 256);
  }
}

typedef CUresult (*EncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// (64, T, H, B) bf16 view, box 64 x `box_rows` positions, 128-byte swizzle, zeros past T
const char* attn_tmap(CUtensorMap* m, const AttnView& v, int B, int H, int T, int box_rows) {
  static thread_local bool ctx_bound = false;             // the encode call wants a current context on this thread
  if (!ctx_bound) { cudaFree(nullptr); ctx_bound = true; }
  static EncodeTiled fn = []() -> EncodeTiled {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult qr;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &qr) != cudaSuccess || qr != cudaDriverEntryPointSuccess) return nullptr;
    return reinterpret_cast<EncodeTiled>(f);
  }();
  if (!fn) return "cuTensorMapEncodeTiled not found";
  if ((reinterpret_cast<uintptr_t>(v.p) & 15) || v.sb % 8 || v.st % 8 || v.sh % 8) return "attention operand rows must start on 16-byte boundaries";
  // the stride of a dimension of extent 1 is never used; give it a legal value
  const long long st = T > 1 ? v.st : 64, sh = H > 1 ? v.sh : 64, sb = B > 1 ? v.sb : 64;
  if (st <= 0 || sh <= 0 || sb <= 0) return "attention operand strides must be positive";
  cuuint64_t dims[4] = {64, (cuuint64_t)T, (cuuint64_t)H, (cuuint64_t)B};
  cuuint64_t strides[3] = {(cuuint64_t)st * 2, (cuuint64_t)sh * 2, (cuuint64_t)sb * 2};
  cuuint32_t box[4] = {64, (cuuint32_t)box_rows, 1, 1}, es[4] = {1, 1, 1, 1};
  const CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, v.p, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? nullptr : "cuTensorMapEncodeTiled failed";
}

const char* attn_fwd_launch(const AttnArgs& a) {
  CUtensorMap tq, tk, tv;
  if (const char* e = attn_tmap(&tq, a.q, a.B, a.H, a.T, 128)) return e;
  if (const char* e = attn_tmap(&tk, a.k, a.B, a.H, a.T, 128)) return e;
  if (const char* e = attn_tmap(&tv, a.v, a.B, a.H, a.T, 128)) return e;
  if ((reinterpret_cast<uintptr_t>(a.o.p) & 15) || a.o.sb % 8 || a.o.st % 8 || a.o.sh % 8) return "attention output rows must start on 16-byte boundaries";
  AttnFwdParams p{};
  p.T = a.T; p.H = a.H;
  p.window = (a.window > 0 && a.window < a.T) ? a.window : 0;
  p.scale_log2 = a.scale * 1.4426950408889634f;
  p.o = reinterpret_cast<bf16*>(a.o.p);
  p.osb = a.o.sb; p.ost = a.o.st; p.osh = a.o.sh;
  p.lse = a.lse;
  p.status = a.status;
  // a per-device attribute: set whenever it is needed (the call is cheap)
  if (cudaFuncSetAttribute(attn_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, AF_SMEM) != cudaSuccess)
    return "cannot raise dynamic shared memory for the attention kernel";
  const long long items = attn_tiles(a.T) * a.H * a.B;
  if (items > (1ll << 30)) return "attention: too many query tiles";
  p.tiles = (int)attn_tiles(a.T);
  attn_units((long long)a.B * a.H, p.tiles, p.window == 0, 2 * 148, p.units, p.pairs);
  attn_fwd_kernel<<<p.units < 2 * 148 ? p.units : 2 * 148, AF_THREADS, AF_SMEM, a.stream>>>(tq, tk, tv, p);
  return nullptr;
}

// ------------------------------------------------------------------------------------------------ rotation of q and k
// q and k of qkv (B, T, 3, H, 64) rotated into slots 0 and 1 of out (B, T, slots, H, 64); with 3 slots v is copied as well unless
// out is qkv itself.  A thread takes 16 head dims of one head, in two 16-byte pieces that hold whole pairs: it reads them before
// it writes them, so that out may be qkv.
__global__ void rope_qk2_kernel(const bf16* in, bf16* out, const float* __restrict__ cs, const float* __restrict__ sn, long long n, int T, int H,
                                int half, int slots, int moved) {
  const int per_tok = moved * H * 4;                        // 16-dim groups per position
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const long long tok = i / per_tok;
    const int rem = (int)(i - tok * per_tok), gi = rem & 3, head = rem >> 2;            // head: slot * H + h
    const int t = (int)(tok % T);
    const int lo = half ? gi * 8 : gi * 16, hi = half ? lo + 32 : lo + 8;
    const bf16* src = in + (tok * 3 * H + head) * 64;
    bf16* dst = out + (tok * slots * H + head) * 64;
    uint4 u = *reinterpret_cast<const uint4*>(src + lo), w = *reinterpret_cast<const uint4*>(src + hi);
    if (head < 2 * H) {
      uint32_t *p = reinterpret_cast<uint32_t*>(&u), *q = reinterpret_cast<uint32_t*>(&w);
      const float4 c0 = *reinterpret_cast<const float4*>(cs + (long long)t * 32 + gi * 8), c1 = *reinterpret_cast<const float4*>(cs + (long long)t * 32 + gi * 8 + 4);
      const float4 s0 = *reinterpret_cast<const float4*>(sn + (long long)t * 32 + gi * 8), s1 = *reinterpret_cast<const float4*>(sn + (long long)t * 32 + gi * 8 + 4);
      const float c[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w}, s[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
      if (!half) {                                          // pairs (2i, 2i + 1)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 f = unpack_bf16(p[j]), g = unpack_bf16(q[j]);
          p[j] = pack_bf16(f.x * c[j] - f.y * s[j], f.x * s[j] + f.y * c[j]);
          q[j] = pack_bf16(g.x * c[j + 4] - g.y * s[j + 4], g.x * s[j + 4] + g.y * c[j + 4]);
        }
      } else {                                              // pairs (i, i + 32)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 a = unpack_bf16(p[j]), b = unpack_bf16(q[j]);
          p[j] = pack_bf16(a.x * c[2 * j] - b.x * s[2 * j], a.y * c[2 * j + 1] - b.y * s[2 * j + 1]);
          q[j] = pack_bf16(b.x * c[2 * j] + a.x * s[2 * j], b.y * c[2 * j + 1] + a.y * s[2 * j + 1]);
        }
      }
    }
    *reinterpret_cast<uint4*>(dst + lo) = u;
    *reinterpret_cast<uint4*>(dst + hi) = w;
  }
}
void rope_qk2_launch(const void* qkv, void* out, const float* cos, const float* sin, int B, int T, int H, int half, int slots, cudaStream_t st) {
  const int moved = qkv == out ? 2 : slots;
  const long long n = (long long)B * T * moved * H * 4;
  if (!n) return;
  const int grid = (int)((n + 255) / 256 < 148 * 16 ? (n + 255) / 256 : 148 * 16);
  rope_qk2_kernel<<<grid, 256, 0, st>>>(reinterpret_cast<const bf16*>(qkv), reinterpret_cast<bf16*>(out), cos, sin, n, T, H, half, slots, moved);
}

}  // namespace mb
