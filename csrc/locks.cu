// Keys and locks: for each position t and n-gram length n = 1..n_keys, the latest j < t whose n-gram ending at j equals
// the one ending at t; the candidate is the word after j.
//
// Scanning back from every position costs T^2 / 2 comparisons per text.  Here the n-grams are dealt out by a hash to
// warps ("shares"): every warp walks its whole text once in order, keeps the positions whose n-gram falls into its
// share, and looks each up in a small hash table in shared memory that holds the latest position of every distinct
// n-gram of the share - linear in T for each warp, and the shares of all texts and key lengths run side by side.
// 32 kept positions are looked up at a time: equal keys inside the batch find each other by match, the first of
// each group asks the table, the last of each group becomes the table's new latest position.
// The table is exact: keys are the n-gram itself (21 bits per word; a text with an id outside -2^20 .. 2^20 - 1 is scanned
// instead), chains resolve equal slots, and a share with more distinct n-grams than nodes (LK_NODES; about T / shares = 256 are expected) answers the overflowing ones by scanning
// the text back, as all positions were before.
// What bounds it: staging the text and the walk, T / 128 steps of one warp.  4 texts x 16 384 words, three key lengths: 1183 us by scanning,
// 38 by the tables.
#include <algorithm>
#include <cstdint>

#include "locks_api.h"

namespace mb {

constexpr int LK_WARPS = 8, LK_NODES = 448, LK_SLOTS = 512;
constexpr int LK_MAX_T = 30000;                      // the text is staged in shared memory (4 bytes per word + 1 for whose it is)

struct LockTable {                                   // one per warp
  unsigned long long key[LK_NODES];
  int last[LK_NODES];                                // latest position of the node's n-gram
  unsigned short next[LK_NODES];                     // chain of the slot, LK_NODES = end
  unsigned int slot[LK_SLOTS];                       // first node of the slot, LK_NODES = empty
  unsigned short pend[160];                          // kept positions not yet looked up (up to 31 + 128)
};

__device__ __forceinline__ unsigned long long ngram_key(const int* tok, int t, int n) {
  unsigned long long k = (unsigned)tok[t];
  if (n >= 2) k |= (unsigned long long)(unsigned)tok[t - 1] << 21;
  if (n >= 3) k |= (unsigned long long)(unsigned)tok[t - 2] << 42;
  return k;
}
__device__ __forceinline__ unsigned hash64(unsigned long long k) {
  k *= 0x9E3779B97F4A7C15ull;
  k ^= k >> 29;
  k *= 0xBF58476D1CE4E5B9ull;
  return (unsigned)(k >> 32);
}
__device__ __forceinline__ unsigned share_of(unsigned h, int shares) { return (unsigned)(((unsigned long long)h * (unsigned)shares) >> 32); }

// grid (share groups, n_keys, B), LK_WARPS warps.  src[b, t, n-1] = position after the latest earlier occurrence, 0 = none.
__global__ void __launch_bounds__(LK_WARPS * 32) lock_search_kernel(const long long* __restrict__ x, long long* __restrict__ src,
                                                                    int T, int n_keys, int shares) {
  extern __shared__ __align__(16) unsigned char lk_smem[];
  const int n = blockIdx.y + 1, b = blockIdx.z, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  LockTable& tab = reinterpret_cast<LockTable*>(lk_smem)[warp];
  int* tok = reinterpret_cast<int*>(lk_smem + LK_WARPS * sizeof(LockTable));
  const long long* xr = x + (long long)b * T;
  int wide = 0;
#pragma unroll 8
  for (int t = threadIdx.x; t < T; t += LK_WARPS * 32) {
    const int id = (int)xr[t];
    tok[t] = id & 0x1FFFFF;
    wide |= ((unsigned)id + (1u << 20)) >> 21;
  }
  for (int i = lane; i < LK_SLOTS; i += 32) tab.slot[i] = LK_NODES;
  if (__syncthreads_or(wide)) {
    // 21 bits do not tell this text's words apart: scan back from every position, on whole ids
    for (int t = blockIdx.x * (LK_WARPS * 32) + threadIdx.x; t < T; t += gridDim.x * (LK_WARPS * 32)) {
      int j = t >= n - 1 ? t - 1 : -1;
      for (; j >= n - 1; --j)
        if ((int)xr[j] == (int)xr[t] && (n < 2 || (int)xr[j - 1] == (int)xr[t - 1]) && (n < 3 || (int)xr[j - 2] == (int)xr[t - 2])) break;
      src[((long long)b * T + t) * n_keys + (n - 1)] = j >= n - 1 ? min(j + 1, T - 1) : 0;
    }
    return;
  }
  // which of this block's warps takes position t: hashed once for all of them (LK_WARPS = none of them, or too early for
  // an n-gram)
  unsigned char* whose = reinterpret_cast<unsigned char*>(tok + T);
  const unsigned share = blockIdx.x * LK_WARPS + warp;
#pragma unroll 4
  for (int t = threadIdx.x; t < ((T + 3) & ~3); t += LK_WARPS * 32) {
    unsigned w = LK_WARPS;
    if (t < T) {
      if (t >= n - 1) w = min(share_of(hash64(ngram_key(tok, t, n)), shares) - blockIdx.x * LK_WARPS, (unsigned)LK_WARPS);
      else if (blockIdx.x == 0) src[((long long)b * T + t) * n_keys + (n - 1)] = 0;
    }
    whose[t] = (unsigned char)w;
  }
  __syncthreads();
  if ((int)share >= shares) return;
  long long* out = src + (long long)b * T * n_keys + (n - 1);
  int n_pend = 0, n_nodes = 0;
  const unsigned below = (1u << lane) - 1u;

  auto look_up = [&](int have) {                     // the first `have` (<= 32) pending positions
    const bool mine = lane < have;
    const int t = mine ? tab.pend[lane] : 0;
    const unsigned long long key = mine ? ngram_key(tok, t, n) : ~0ull - lane;      // idle lanes match nobody
    const unsigned group = __match_any_sync(0xffffffffu, key);
    const unsigned earlier = group & below;
    // where it was last: an earlier lane of the batch, else the table
    const int near = __shfl_sync(0xffffffffu, t, earlier ? 31 - __clz(earlier) : 0);
    const unsigned s = (hash64(key) >> 3) & (LK_SLOTS - 1);
    int node = LK_NODES, last = -1;
    const bool leader = mine && !earlier;
    if (leader) {
      for (node = (int)tab.slot[s]; node != LK_NODES; node = tab.next[node])
        if (tab.key[node] == key) break;
      if (node != LK_NODES) last = tab.last[node];
    }
    __syncwarp();
    // new nodes for keys not seen before
    const unsigned fresh = __ballot_sync(0xffffffffu, leader && node == LK_NODES);
    if (leader && node == LK_NODES) {
      const int id = n_nodes + __popc(fresh & below);
      if (id < LK_NODES) {
        node = id;
        tab.key[id] = key;
        tab.next[id] = (unsigned short)atomicExch(&tab.slot[s], (unsigned)id);
      }
      if (n_nodes + __popc(fresh) > LK_NODES) {
        // more distinct n-grams than nodes: from here on a key missing in the table may still have occurred before
        for (int j = t - 1; j >= n - 1; --j)
          if (ngram_key(tok, j, n) == key) { last = j; break; }
      }
    }
    n_nodes = min(LK_NODES + 1, n_nodes + __popc(fresh));        // LK_NODES + 1: some key found no node
    // the leader's node belongs to the whole group; its last lane holds the newest position
    const int lead = __ffs(group) - 1;
    node = __shfl_sync(0xffffffffu, node, lead);
    if (mine && (group >> lane) == 1u && node != LK_NODES) tab.last[node] = t;
    if (mine) {
      const int at = earlier ? near : last;
      out[(long long)t * n_keys] = at >= 0 ? min(at + 1, T - 1) : 0;
    }
    __syncwarp();
  };

  for (int t0 = 0; t0 < T; t0 += 128) {
    // four consecutive words per lane; kept ones are appended in text order
    const int tb = t0 + lane * 4;
    const unsigned mine4 = (unsigned)warp * 0x01010101u;
    const unsigned w4 = tb < T ? *reinterpret_cast<const unsigned*>(whose + tb) : ~mine4;
    const unsigned eq = __vcmpeq4(w4, mine4);              // 0xff in the bytes that match
    const unsigned keep = (eq & 1u) | (eq >> 7 & 2u) | (eq >> 14 & 4u) | (eq >> 21 & 8u);
    const unsigned m0 = __ballot_sync(0xffffffffu, keep & 1u), m1 = __ballot_sync(0xffffffffu, keep & 2u),
                   m2 = __ballot_sync(0xffffffffu, keep & 4u), m3 = __ballot_sync(0xffffffffu, keep & 8u);
    int at = n_pend + __popc(m0 & below) + __popc(m1 & below) + __popc(m2 & below) + __popc(m3 & below);
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (keep >> u & 1u) tab.pend[at++] = (unsigned short)(tb + u);
    n_pend += __popc(m0) + __popc(m1) + __popc(m2) + __popc(m3);
    __syncwarp();
    while (n_pend >= 32) {
      look_up(32);
      // the rest moves to the front (at most 127 positions: four per lane, read before they are written)
      int v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = u * 32 + lane < n_pend - 32 ? tab.pend[32 + u * 32 + lane] : 0;
      __syncwarp();
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (u * 32 + lane < n_pend - 32) tab.pend[u * 32 + lane] = (unsigned short)v[u];
      n_pend -= 32;
      __syncwarp();
    }
  }
  if (n_pend > 0) look_up(n_pend);
}

__device__ int lock_status_word = 0;                // a word id that no entry of the trust table belongs to was met

// Trust bucket of word x: ids past the table take its last entry, negative ones count from its end.  Ids below that belong to
// nobody: the status word says so and no memory outside the table is read.
__device__ __forceinline__ long long bucket_of(const long long* bucket, long long n, long long x) {
  long long i = min(x, n - 1);
  if (i < 0) i += n;
  if (i < 0) { atomicExch(&lock_status_word, LOCK_BAD_ID); i = 0; }
  return bucket[i];
}

// candidates, firing locks (only the longest one when `longest_only`) and trust buckets from the positions
__global__ void lock_finish_kernel(LockArgs a, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const long long* xr = a.x + i / a.T * a.T;
    bool longer = false;
    for (int k = a.n_keys - 1; k >= 0; --k) {
      const long long s = a.src[i * a.n_keys + k];
      const bool found = s > 0;
      a.cand[i * a.n_keys + k] = found ? (long long)(int)xr[s] : 0;
      a.on[i * a.n_keys + k] = found && !(a.longest_only && longer);
      longer |= found;
    }
    if (a.bk) a.bk[i] = a.bucket ? bucket_of(a.bucket, a.n_bucket, a.x[i]) : 0;
  }
}

// The plain form: every position scans back until all its key lengths are found.  The text is staged in shared memory;
// grid (texts, slices): a block takes runs of blockDim positions spread evenly over the text (late positions scan
// further back, so contiguous halves would be unbalanced).
__global__ void lock_scan_kernel(const long long* __restrict__ x, long long* __restrict__ cand, bool* __restrict__ on,
                                 long long* __restrict__ src, const long long* __restrict__ bucket, long long n_bucket,
                                 long long* __restrict__ bk, int T, int n_keys, int longest_only) {
  extern __shared__ int tok[];
  const int b = blockIdx.x;
  const long long* xr = x + (long long)b * T;
  for (int t = threadIdx.x; t < T; t += blockDim.x) tok[t] = (int)xr[t];
  __syncthreads();
  for (int t = blockIdx.y * blockDim.x + threadIdx.x; t < T; t += gridDim.y * blockDim.x) {
    int last[3] = {-1, -1, -1};
    const int a0 = tok[t], a1 = t >= 1 ? tok[t - 1] : -1, a2 = t >= 2 ? tok[t - 2] : -1;
    int need = n_keys;                                   // how many key lengths are still unresolved
    for (int j = t - 1; j >= 0 && need > 0; --j) {
      if (tok[j] != a0) continue;
      if (last[0] < 0) { last[0] = j; --need; }
      if (n_keys >= 2 && t >= 1 && j >= 1 && tok[j - 1] == a1) {
        if (last[1] < 0) { last[1] = j; --need; }
        if (n_keys >= 3 && t >= 2 && j >= 2 && tok[j - 2] == a2 && last[2] < 0) { last[2] = j; --need; }
      }
      // a longer key can only match where the shorter one matches, so once the 1-gram is found we keep scanning
      // only for the longer ones; stop early when position constraints make them impossible
      if (n_keys >= 2 && t < 1 && last[0] >= 0) break;
    }
    bool ok[3];
    for (int n = 0; n < n_keys; ++n) ok[n] = last[n] >= 0;
    if (longest_only) {
      for (int n = 0; n < n_keys - 1; ++n)
        for (int q = n + 1; q < n_keys; ++q) if (ok[q]) ok[n] = false;
    }
    for (int n = 0; n < n_keys; ++n) {
      const bool found = last[n] >= 0;
      const int sp = found ? min(last[n] + 1, T - 1) : 0;
      const long long o = ((long long)b * T + t) * n_keys + n;
      cand[o] = found ? tok[sp] : 0;
      src[o] = sp;
      on[o] = ok[n];
    }
    if (bk) bk[(long long)b * T + t] = bucket ? bucket_of(bucket, n_bucket, xr[t]) : 0;
  }
}

int lock_status_read() {
  int v = 0;
  const int z = 0;
  cudaMemcpyFromSymbol(&v, lock_status_word, sizeof(int));
  if (v) cudaMemcpyToSymbol(lock_status_word, &z, sizeof(int));
  return v;
}

bool lock_find_launch(const LockArgs& a) {
  const long long n = (long long)a.B * a.T;
  if (!n) return true;
  // Words that fit 21 bits and texts that can be staged beside the tables go to the tables.  The scan serves the rest:
  // one-word texts, texts of 30 000 to 51 200 words, vocabularies above 2^20.
  if (a.vocab <= (1 << 20) && a.T >= 2 && a.T <= LK_MAX_T && a.B <= 65535) {
    // a share per 256 positions: the table then holds about 256 distinct n-grams at most, and the walk over the text,
    // not the look-ups, is what a warp spends its time on
    const int shares = a.T / 256 + 1, groups = (shares + LK_WARPS - 1) / LK_WARPS;
    const size_t smem = LK_WARPS * sizeof(LockTable) + (size_t)a.T * 5 + 4;
    if (cudaFuncSetAttribute(lock_search_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return false;
    lock_search_kernel<<<dim3(groups, a.n_keys, a.B), LK_WARPS * 32, smem, a.stream>>>(a.x, a.src, a.T, a.n_keys, shares);
    lock_finish_kernel<<<(int)((n + 255) / 256 < 148 * 8 ? (n + 255) / 256 : 148 * 8), 256, 0, a.stream>>>(a, n);
    return true;
  }
  const size_t smem = (size_t)a.T * 4;
  if (smem > 48 * 1024 && cudaFuncSetAttribute(lock_scan_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return false;
  const int threads = 256;
  const int slices = std::max(1, std::min((a.T + threads - 1) / threads, (4 * 148 + a.B - 1) / a.B));
  lock_scan_kernel<<<dim3(a.B, slices), threads, smem, a.stream>>>(a.x, a.cand, a.on, a.src, a.bucket, a.n_bucket, a.bk, a.T, a.n_keys, a.longest_only);
  return true;
}

}  // namespace mb
