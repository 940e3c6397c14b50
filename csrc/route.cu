// The router of an expert layer in two launches forward (three for more than 32 768 tokens) and three backward.
//
// Forward 1 (route_fwd_kernel): logits = x W^T in fp32 from the bf16 rows, softmax, top-k by probability (ties: smaller
// expert first), budget k_tok, renormalised weights, and per block of 32 tokens the number of choices and the sum of
// probabilities of every expert.
// Forward 2 (route_place_kernel): choices in (token, choice) order take the next free place of their expert, places beyond C
// drop; a block's first free places are the sums of the earlier blocks' numbers (taken by each block, or from ROUTE_SCAN blocks on
// by route_scan_kernel once).  Fills the slot table, its inverse,
// the combine weights of the places, and (first block) filled places, dropped share and the Switch auxiliary loss
//   aux = E * sum_e (choices of e / all choices) * (mean probability of e over the real tokens).
// Backward 1 (route_dx_kernel): gradient of the logits from the gradients of the weights, of the place weights and of aux, and
// dx = dlogits W.  Backward 2 and 3 (route_dw_kernel, route_dw_fold_kernel): dW = dlogits^T x.
// All of it is memory-bound on x (33 MB for 8192 x 2048).  A warp takes 4 or 8 tokens at a time, so that W (E x d fp32) is
// read once for them and mostly from L1 (the choice stands at route_fwd_launch).  Us for 8192 x 2048, 8 experts, 8 tokens per
// warp -> 4: route_fwd 59 -> 30, route_dx 55 -> 44; route_dw with 64 tokens per block instead of 256: 48 -> 17.
#include <algorithm>

#include "common.cuh"
#include "route_api.h"

namespace mb {

__device__ __forceinline__ void load8(const bf16* p, float (&v)[8]) {
  const uint4 u = *reinterpret_cast<const uint4*>(p);
  const uint32_t q[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) { const float2 f = unpack_bf16(q[j]); v[2 * j] = f.x; v[2 * j + 1] = f.y; }
}
__device__ __forceinline__ void load8(const float* p, float (&v)[8]) {
  const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}

template <int TOK>
__global__ void __launch_bounds__(ROUTE_TOK / TOK * 32) route_fwd_kernel(RouteArgs a) {
  constexpr int EXP = 32 / TOK;                          // experts at a time: 32 sums per lane
  __shared__ float ps_sh[ROUTE_E];
  __shared__ int cnt_sh[ROUTE_E], real_sh;
  extern __shared__ float lg_sh[];                       // (ROUTE_TOK, E) logits
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, E = a.E;
  for (int i = threadIdx.x; i < E; i += blockDim.x) { ps_sh[i] = 0.f; cnt_sh[i] = 0; }
  if (threadIdx.x == 0) real_sh = 0;
  __syncthreads();
  const int n0 = blockIdx.x * ROUTE_TOK + warp * TOK;
  const int nt = min(TOK, a.N - n0);                  // may be <= 0
  const bf16* X = reinterpret_cast<const bf16*>(a.x);
  float* lg = lg_sh + warp * TOK * E;
  // TOK tokens x EXP experts at a time: every lane sums its columns, then the 32 sums are reduced over the lanes, the lane that
  // ends up with sum v = token * EXP + expert writes it
  for (int e0 = 0; e0 < E; e0 += EXP) {
    float acc[32];
#pragma unroll
    for (int v = 0; v < 32; ++v) acc[v] = 0.f;
    if (nt > 0) {
      for (int c = lane * 8; c < a.d; c += 256) {
        float x[TOK][8];
#pragma unroll
        for (int t = 0; t < TOK; ++t) load8(X + (long long)(n0 + min(t, nt - 1)) * a.d + c, x[t]);
#pragma unroll
        for (int j = 0; j < EXP; ++j) {
          float w[8];
          load8(a.w + (long long)min(e0 + j, E - 1) * a.d + c, w);       // experts past the last are not written
#pragma unroll
          for (int t = 0; t < TOK; ++t)
#pragma unroll
            for (int u = 0; u < 8; ++u) acc[t * EXP + j] = fmaf(x[t][u], w[u], acc[t * EXP + j]);
        }
      }
    }
    // reduce-scatter: after the step with offset o a lane holds o sums, of those whose index agrees with its own bits
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const bool up = (lane & o) != 0;
#pragma unroll
      for (int v = 0; v < o; ++v) {
        const float send = up ? acc[v] : acc[v + o], keep = up ? acc[v + o] : acc[v];
        acc[v] = keep + __shfl_xor_sync(0xffffffffu, send, o);
      }
    }
    const int t = lane / EXP, e = e0 + lane % EXP;
    if (e < E) lg[t * E + e] = acc[0];
  }
  __syncwarp();
  for (int t = 0; t < nt; ++t) {
    const long long n = n0 + t;
    float v[ROUTE_E / 32];
    float mx = -INFINITY;
#pragma unroll
    for (int i = 0; i < ROUTE_E / 32; ++i) {
      const int e = lane + 32 * i;
      v[i] = e < E ? lg[t * E + e] : -INFINITY;
      mx = fmaxf(mx, v[i]);
    }
    mx = warp_max(mx);
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < ROUTE_E / 32; ++i) { v[i] = lane + 32 * i < E ? expf(v[i] - mx) : 0.f; sum += v[i]; }
    const float inv = 1.f / warp_sum(sum);
    const bool is_real = a.real[n];
    const int kt = (int)a.k_tok[n];
#pragma unroll
    for (int i = 0; i < ROUTE_E / 32; ++i) {
      const int e = lane + 32 * i;
      v[i] *= inv;
      if (e < E) {
        a.probs[n * E + e] = v[i];
        if (is_real) atomicAdd(&ps_sh[e], v[i]);
      } else {
        v[i] = -1.f;
      }
    }
    float mine_p = 0.f, kept = 0.f;                      // lane j < k ends up with choice j
    int mine_e = E;
    for (int j = 0; j < a.k; ++j) {
      float bp = -1.f;
      int be = ROUTE_E;
#pragma unroll
      for (int i = 0; i < ROUTE_E / 32; ++i)
        if (v[i] > bp) { bp = v[i]; be = lane + 32 * i; }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float op = __shfl_xor_sync(0xffffffffu, bp, o);
        const int oe = __shfl_xor_sync(0xffffffffu, be, o);
        if (op > bp || (op == bp && oe < be)) { bp = op; be = oe; }
      }
#pragma unroll
      for (int i = 0; i < ROUTE_E / 32; ++i) if (be == lane + 32 * i) v[i] = -1.f;
      if (j < kt) kept += bp;
      if (lane == j) { mine_p = bp; mine_e = be; }
    }
    if (lane < a.k) {
      const bool keep = lane < kt && mine_e < E;         // mine_e is out of range only where the logits are NaN
      mine_e = min(mine_e, E);
      a.top_e[n * a.k + lane] = mine_e;
      a.wt[n * a.k + lane] = keep ? mine_p / fmaxf(kept, 1e-9f) : 0.f;
      a.flat_idx[n * a.k + lane] = keep ? mine_e : E;    // the expert for now; route_place_kernel turns it into a place
      if (keep) atomicAdd(&cnt_sh[mine_e], 1);
    }
    if (lane == 0 && is_real) atomicAdd(&real_sh, 1);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < E; i += blockDim.x) {
    a.hist[(long long)blockIdx.x * E + i] = cnt_sh[i];
    a.psum[(long long)blockIdx.x * E + i] = ps_sh[i];
  }
  if (threadIdx.x == 0) a.n_real[blockIdx.x] = real_sh;
}

// block = one expert: its numbers of choices per block become the places taken before each block; totals beside them
__global__ void __launch_bounds__(256) route_scan_kernel(RouteArgs a, int nb) {
  __shared__ int sums[256];
  __shared__ float psums[256];
  const int e = blockIdx.x, E = a.E, tid = threadIdx.x, per = (nb + 255) / 256;
  const int b0 = min(nb, tid * per), b1 = min(nb, b0 + per);
  int s = 0;
  float p = 0.f;
  for (int b = b0; b < b1; ++b) { s += a.hist[(long long)b * E + e]; p += a.psum[(long long)b * E + e]; }
  sums[tid] = s;
  psums[tid] = p;
  __syncthreads();
  for (int o = 1; o < 256; o <<= 1) {
    const int v = tid >= o ? sums[tid - o] : 0;
    __syncthreads();
    sums[tid] += v;
    __syncthreads();
  }
  int run = sums[tid] - s;
  for (int b = b0; b < b1; ++b) {
    const int h = a.hist[(long long)b * E + e];
    a.hist[(long long)b * E + e] = run;
    run += h;
  }
  if (tid == 0) {
    float t = 0.f;
    for (int i = 0; i < 256; ++i) t += psums[i];
    a.ps[e] = t;
    a.total[e] = sums[255];
  }
}

__global__ void __launch_bounds__(256) route_place_kernel(RouteArgs a) {
  __shared__ int base[ROUTE_E], total[ROUTE_E];
  __shared__ float ps[ROUTE_E];
  __shared__ unsigned char ch[ROUTE_TOK * ROUTE_K];
  __shared__ int real_sh;
  const int E = a.E, nb = gridDim.x, tid = threadIdx.x;
  const bool first = blockIdx.x == 0;
  for (int e = tid; e < E; e += blockDim.x) { base[e] = 0; total[e] = 0; ps[e] = 0.f; }
  if (tid == 0) real_sh = 0;
  __syncthreads();
  // sums over the blocks: a thread takes one expert and every (256 / E)-th block
  const int lanes = blockDim.x / E;
  if (a.total) {
    for (int e = tid; e < E; e += blockDim.x) { base[e] = a.hist[(long long)blockIdx.x * E + e]; total[e] = a.total[e]; ps[e] = a.ps[e]; }
  } else if (tid < lanes * E) {
    const int e = tid % E;
    int before = 0, all = 0;
    float p = 0.f;
    for (int b = tid / E; b < nb; b += lanes) {
      const int h = a.hist[(long long)b * E + e];
      all += h;
      if (b < (int)blockIdx.x) before += h;
      if (first) p += a.psum[(long long)b * E + e];
    }
    atomicAdd(&base[e], before);
    atomicAdd(&total[e], all);
    if (first) atomicAdd(&ps[e], p);
  }
  if (first) {
    int r = 0;
    for (int b = tid; b < nb; b += blockDim.x) r += a.n_real[b];
    if (r) atomicAdd(&real_sh, r);
  }
  const int n0 = blockIdx.x * ROUTE_TOK, nch = min(ROUTE_TOK, a.N - n0) * a.k;
  for (int i = tid; i < nch; i += blockDim.x) ch[i] = (unsigned char)a.flat_idx[(long long)n0 * a.k + i];
  __syncthreads();
  const long long EC = (long long)E * a.C;
  for (int i = tid; i < nch; i += blockDim.x) {
    const int e = ch[i];
    long long place = EC;
    if (e < E) {
      int rank = base[e];
      for (int j = 0; j < i; ++j) rank += ch[j] == e;
      if (rank < a.C) {
        place = (long long)e * a.C + rank;
        a.table[place] = n0 + i / a.k;
        a.wtab[place] = a.wt[(long long)n0 * a.k + i];
      }
    }
    a.flat_idx[(long long)n0 * a.k + i] = place;
  }
  // the places nobody takes
  for (long long q = blockIdx.x * (long long)blockDim.x + tid; q < EC; q += (long long)nb * blockDim.x)
    if ((int)(q % a.C) >= total[q / a.C]) { a.table[q] = a.N; a.wtab[q] = 0.f; }
  if (first) {
    for (int e = tid; e < E; e += blockDim.x) a.counts[e] = min(total[e], a.C);
    if (tid == 0) {
      int kept = 0, placed = 0;
      for (int e = 0; e < E; ++e) { kept += total[e]; placed += min(total[e], a.C); }
      *a.dropped = 1.f - (float)placed / (float)max(kept, 1);
      const float scale = (float)E / ((float)max(kept, 1) * (float)max(real_sh, 1));
      float s = 0.f;
      for (int e = 0; e < E; ++e) {
        const float g = scale * (float)total[e];
        a.aux_grad[e] = g;
        s += g * ps[e];
      }
      *a.aux = s;
    }
  }
}

template <int TOK>
__global__ void __launch_bounds__(ROUTE_TOK / TOK * 32) route_dx_kernel(RouteArgs a) {
  extern __shared__ float dl_sh[];                       // (ROUTE_TOK, E)
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, E = a.E;
  const int n0 = blockIdx.x * ROUTE_TOK + warp * TOK;
  const int nt = min(TOK, a.N - n0);
  float* dl = dl_sh + warp * TOK * E;
  const float d_aux = a.d_aux ? *a.d_aux : 0.f;
  for (int t = 0; t < TOK; ++t) {
    if (t >= nt) {                                       // absent tokens of the last block
      for (int e = lane; e < E; e += 32) dl[t * E + e] = 0.f;
      continue;
    }
    const long long n = n0 + t;
    const int kt = (int)a.k_tok[n];
    const bool is_real = a.real[n];
    // lane j < k: choice j
    int te = ROUTE_E;
    float tp = 0.f, g = 0.f;
    if (lane < a.k) {
      te = (int)a.top_e[n * a.k + lane];
      if (lane < kt && te < E) {
        tp = a.probs[n * E + te];
        if (a.d_wt) g = a.d_wt[n * a.k + lane];
        if (a.d_wtab) {
          const long long place = a.flat_idx[n * a.k + lane];
          if (place < (long long)E * a.C) g += a.d_wtab[place];
        }
      }
    }
    const float s0 = warp_sum(tp), s = fmaxf(s0, 1e-9f);
    const float dot = warp_sum(g * tp) / s;
    const float dtp = lane < kt && lane < a.k ? (g - (s0 < 1e-9f ? 0.f : dot)) / s : 0.f;
    float pr[ROUTE_E / 32], dp[ROUTE_E / 32], pd = 0.f;
#pragma unroll
    for (int i = 0; i < ROUTE_E / 32; ++i) {
      const int e = lane + 32 * i;
      pr[i] = e < E ? a.probs[n * E + e] : 0.f;
      dp[i] = e < E ? (a.d_probs ? a.d_probs[n * E + e] : 0.f) + (is_real ? d_aux * a.aux_grad[e] : 0.f) : 0.f;
      for (int j = 0; j < a.k; ++j) {
        const int ej = __shfl_sync(0xffffffffu, te, j);
        const float dj = __shfl_sync(0xffffffffu, dtp, j);
        if (ej == e) dp[i] += dj;
      }
      pd += pr[i] * dp[i];
    }
    pd = warp_sum(pd);
#pragma unroll
    for (int i = 0; i < ROUTE_E / 32; ++i) {
      const int e = lane + 32 * i;
      if (e < E) {
        const float v = pr[i] * (dp[i] - pd);
        dl[t * E + e] = v;
        a.dl[n * E + e] = v;
      }
    }
  }
  __syncwarp();
  if (nt <= 0) return;
  bf16* DX = reinterpret_cast<bf16*>(a.dx);
  for (int c = lane * 8; c < a.d; c += 256) {
    float acc[TOK][8];
#pragma unroll
    for (int t = 0; t < TOK; ++t)
#pragma unroll
      for (int u = 0; u < 8; ++u) acc[t][u] = 0.f;
    for (int e = 0; e < E; ++e) {
      float w[8];
      load8(a.w + (long long)e * a.d + c, w);
#pragma unroll
      for (int t = 0; t < TOK; ++t) {
        const float v = dl[t * E + e];
#pragma unroll
        for (int u = 0; u < 8; ++u) acc[t][u] = fmaf(v, w[u], acc[t][u]);
      }
    }
#pragma unroll
    for (int t = 0; t < TOK; ++t)
      if (t < nt)
        *reinterpret_cast<uint4*>(DX + (long long)(n0 + t) * a.d + c) =
            make_uint4(pack_bf16(acc[t][0], acc[t][1]), pack_bf16(acc[t][2], acc[t][3]), pack_bf16(acc[t][4], acc[t][5]), pack_bf16(acc[t][6], acc[t][7]));
  }
}

// grid (column tiles of 512, runs of tokens, groups of 8 experts): a thread owns two columns of 8 experts and walks its run 64
// tokens at a time.  part[run] (E, d) = the run's share of dW; route_dw_fold_kernel adds the shares in order, so that the
// gradient has the same bits on every call.
constexpr int DW_RUN = 64;
__global__ void __launch_bounds__(256) route_dw_kernel(RouteArgs a) {
  __shared__ __align__(16) float g[DW_RUN][8];
  const int c = (blockIdx.x * 256 + threadIdx.x) * 2, e0 = blockIdx.z * 8;
  float acc[8][2] = {};
  const uint32_t* X = reinterpret_cast<const uint32_t*>(a.x);
  const long long pitch = a.d / 2;
  const int end = min(a.N, (int)(blockIdx.y + 1) * a.dw_run);
  for (int n0 = blockIdx.y * a.dw_run; n0 < end; n0 += DW_RUN) {
    const int n1 = min(end, n0 + DW_RUN);
    __syncthreads();
    for (int i = threadIdx.x; i < (n1 - n0) * 8; i += 256) {
      const int e = e0 + (i & 7);
      g[i >> 3][i & 7] = e < a.E ? a.dl[(long long)(n0 + (i >> 3)) * a.E + e] : 0.f;
    }
    __syncthreads();
    if (c >= a.d) continue;
#pragma unroll 8
    for (int n = n0; n < n1; ++n) {
      const float2 x = unpack_bf16(X[n * pitch + c / 2]);
      const float4 g0 = *reinterpret_cast<const float4*>(g[n - n0]), g1 = *reinterpret_cast<const float4*>(g[n - n0] + 4);
      const float ge[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
#pragma unroll
      for (int j = 0; j < 8; ++j) { acc[j][0] = fmaf(ge[j], x.x, acc[j][0]); acc[j][1] = fmaf(ge[j], x.y, acc[j][1]); }
    }
  }
  if (c >= a.d) return;
#pragma unroll
  for (int j = 0; j < 8; ++j)
    if (e0 + j < a.E)
      *reinterpret_cast<float2*>(a.dw_part + ((long long)blockIdx.y * a.E + e0 + j) * a.d + c) = make_float2(acc[j][0], acc[j][1]);
}
// block = 32 elements of dW x 8 lanes of runs
__global__ void __launch_bounds__(256) route_dw_fold_kernel(const float* __restrict__ part, float* __restrict__ dw, int runs, int n) {
  __shared__ float sh[8][33];
  const int cx = threadIdx.x & 31, ry = threadIdx.x >> 5, i = blockIdx.x * 32 + cx;
  float s = 0.f;
  if (i < n)
#pragma unroll 8
    for (int r = ry; r < runs; r += 8) s += part[(long long)r * n + i];
  sh[ry][cx] = s;
  __syncthreads();
  if (ry == 0 && i < n) {
#pragma unroll
    for (int k = 1; k < 8; ++k) s += sh[k][cx];
    dw[i] = s;
  }
}

// Runs of at least 64 tokens, and at most 32 MB of shares: with 8 experts of 2048 columns that is one run for each 64 of 32 768
// tokens.
int route_dw_runs(int N, int d, int E, int& run) {
  const long long most = std::max<long long>(1, (8ll << 20) / ((long long)E * d));
  const long long per = ((N + most - 1) / most + DW_RUN - 1) / DW_RUN * DW_RUN;
  run = (int)per;
  return (int)((N + per - 1) / per);
}

// 4 tokens per warp and 8 experts at a time keep twice the warps in flight; with many experts W no longer fits L1 and 8
// tokens per warp halve its traffic
void route_fwd_launch(const RouteArgs& a) {
  const int nb = route_blocks(a.N);
  const size_t smem = (size_t)ROUTE_TOK * a.E * 4;
  if (a.E <= 16) route_fwd_kernel<4><<<nb, ROUTE_TOK / 4 * 32, smem, a.stream>>>(a);
  else route_fwd_kernel<8><<<nb, ROUTE_TOK / 8 * 32, smem, a.stream>>>(a);
  if (a.total) route_scan_kernel<<<a.E, 256, 0, a.stream>>>(a, nb);
  route_place_kernel<<<nb, 256, 0, a.stream>>>(a);
}
void route_bwd_launch(const RouteArgs& a) {
  const int nb = route_blocks(a.N);
  const size_t smem = (size_t)ROUTE_TOK * a.E * 4;
  if (a.E <= 16) route_dx_kernel<4><<<nb, ROUTE_TOK / 4 * 32, smem, a.stream>>>(a);
  else route_dx_kernel<8><<<nb, ROUTE_TOK / 8 * 32, smem, a.stream>>>(a);
  route_dw_kernel<<<dim3((a.d + 511) / 512, a.dw_runs, (a.E + 7) / 8), 256, 0, a.stream>>>(a);
  route_dw_fold_kernel<<<(a.E * a.d + 31) / 32, 256, 0, a.stream>>>(a.dw_part, a.dw, a.dw_runs, a.E * a.d);
}

}  // namespace mb
