// RMSNorm forward (with or without the residual add in front of it) and backward.
//
// A row belongs to a team of WPR warps, NV float4 per lane, chosen so that a team covers the row exactly once: the row is
// read from memory once and stays in registers between the sum and the scaling.  A block is 8 warps = 8 / WPR teams,
// each walking its own rows; a team of one warp needs no barrier at all, a larger one has a single named barrier per
// row (the partial sums alternate between two slots).  The backward pass loads the next row before it reduces the
// current one.
// Bound by memory.  The one-block-per-row kernels this replaces spent three barriers per row with one row in flight
// and ended in n_blocks * d atomics on d addresses.
// Before / after, us: forward 32768 x 2048 fp32 -> bf16 94 / 73, with the residual add 129 / 122; backward with residual
// gradient and bf16 copy, and without, 250 each / 192 and 157 (5.6 and 3.9 TB/s); backward 2048 x 256 48 / 4.4.
#include <type_traits>

#include "common.cuh"
#include "rowops_api.h"

namespace mb {

template <typename T> struct Raw4;
template <> struct Raw4<float> { typedef float4 type; };
template <> struct Raw4<bf16> { typedef uint2 type; };
__device__ __forceinline__ float4 as_f4(const float4& v) { return v; }
__device__ __forceinline__ float4 as_f4(const uint2& u) {
  const float2 a = unpack_bf16(u.x), b = unpack_bf16(u.y);
  return make_float4(a.x, a.y, b.x, b.y);
}
template <typename T> __device__ __forceinline__ typename Raw4<T>::type ldraw(const T* p) { return *reinterpret_cast<const typename Raw4<T>::type*>(p); }
__device__ __forceinline__ void put4(float* p, const float4& v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void put4(bf16* p, const float4& v) { *reinterpret_cast<uint2*>(p) = make_uint2(pack_bf16(v.x, v.y), pack_bf16(v.z, v.w)); }

constexpr int NORM_WARPS = 8;

// Sum over a team.  `slot`: NORM_WARPS floats of shared memory, another one on each call in turn; bar.sync on barrier 1 +
// team keeps teams independent of one another.
template <int WPR>
__device__ __forceinline__ float team_sum(float v, float* slot, int team, int warp, int lane) {
  v = warp_sum(v);
  if (WPR == 1) return v;
  if (lane == 0) slot[warp] = v;
  asm volatile("bar.sync %0, %1;" ::"r"(1 + team), "n"(WPR * 32) : "memory");
  float t = 0.f;
#pragma unroll
  for (int i = 0; i < WPR; ++i) t += slot[team * WPR + i];
  return t;
}

template <typename TX, typename TY, bool ADD, int WPR, int NV>
__global__ void __launch_bounds__(NORM_WARPS * 32) rmsnorm_fwd_kernel(NormArgs a) {
  __shared__ float red[2][NORM_WARPS];
  constexpr int TEAMS = NORM_WARPS / WPR;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, team = warp / WPR;
  const int col = (threadIdx.x - team * WPR * 32) * 4;
  int turn = 0;
  for (long long row = (long long)blockIdx.x * TEAMS + team; row < a.n; row += (long long)gridDim.x * TEAMS) {
    const long long base = row * a.d;
    // all loads first: the compiler may not move a load over a store to another array
    typename Raw4<TX>::type xr[NV] = {};
    uint2 yr[ADD ? NV : 1] = {};
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c = col + i * WPR * 128;
      if (c < a.d) {
        xr[i] = ldraw(reinterpret_cast<const TX*>(a.x) + base + c);
        if (ADD) yr[i] = ldraw(reinterpret_cast<const bf16*>(a.y) + base + c);
      }
    }
    float4 v[NV];
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c = col + i * WPR * 128;
      v[i] = as_f4(xr[i]);
      if (ADD) {
        const float4 y = as_f4(yr[i]);
        v[i].x += y.x; v[i].y += y.y; v[i].z += y.z; v[i].w += y.w;
        if (c < a.d) put4(a.sum + base + c, v[i]);
      }
      ss += v[i].x * v[i].x + v[i].y * v[i].y + v[i].z * v[i].z + v[i].w * v[i].w;
    }
    ss = team_sum<WPR>(ss, red[turn], team, warp, lane);
    turn ^= 1;
    const float r = rsqrtf(ss / a.d + a.eps);
    if (col == 0) a.rstd[row] = r;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c = col + i * WPR * 128;
      if (c < a.d) {
        const float4 g = *reinterpret_cast<const float4*>(a.w + c);
        put4(reinterpret_cast<TY*>(a.out) + base + c, make_float4(v[i].x * r * g.x, v[i].y * r * g.y, v[i].z * r * g.z, v[i].w * r * g.w));
      }
    }
  }
}

// Rows of more than 8192 elements: one block per row, the row is read twice.
template <typename TX, typename TY, bool ADD>
__global__ void __launch_bounds__(256) rmsnorm_fwd_long_kernel(NormArgs a) {
  __shared__ float red[32];
  const long long base = (long long)blockIdx.x * a.d;
  auto load = [&](int c) {
    float4 v = as_f4(ldraw(reinterpret_cast<const TX*>(a.x) + base + c));
    if (ADD) {
      const float4 y = as_f4(ldraw(reinterpret_cast<const bf16*>(a.y) + base + c));
      v.x += y.x; v.y += y.y; v.z += y.z; v.w += y.w;
    }
    return v;
  };
  float ss = 0.f;
  for (int c = threadIdx.x * 4; c < a.d; c += 1024) {
    const float4 v = load(c);
    if (ADD) put4(a.sum + base + c, v);
    ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
  }
  const float r = rsqrtf(block_sum(ss, red) / a.d + a.eps);
  if (threadIdx.x == 0) a.rstd[blockIdx.x] = r;
  for (int c = threadIdx.x * 4; c < a.d; c += 1024) {
    const float4 v = load(c), g = *reinterpret_cast<const float4*>(a.w + c);
    put4(reinterpret_cast<TY*>(a.out) + base + c, make_float4(v.x * r * g.x, v.y * r * g.y, v.z * r * g.z, v.w * r * g.w));
  }
}

// dx = r (g w) - x r^3 / d * sum(g w x) (+ add);  dw_part[block] = sum over the block's rows of g x r
template <typename TX, typename TG, int WPR, int NV>
__global__ void __launch_bounds__(NORM_WARPS * 32, NV <= 2 ? 3 : 1) rmsnorm_bwd_kernel(NormArgs a) {
  __shared__ float red[2][NORM_WARPS];
  extern __shared__ float4 wsum[];                       // (TEAMS, d / 4)
  constexpr int TEAMS = NORM_WARPS / WPR;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, team = warp / WPR;
  const int col = (threadIdx.x - team * WPR * 32) * 4;
  const TX* X = reinterpret_cast<const TX*>(a.x);
  const TG* G = reinterpret_cast<const TG*>(a.y);
  float4 acc[NV], ww[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = col + i * WPR * 128;
    acc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    ww[i] = c < a.d ? *reinterpret_cast<const float4*>(a.w + c) : acc[i];
  }
  const long long step = (long long)gridDim.x * TEAMS;
  long long row = (long long)blockIdx.x * TEAMS + team;
  typename Raw4<TX>::type xn[NV] = {};
  typename Raw4<TG>::type gn[NV] = {};
  float4 qn[NV] = {};
  auto fetch = [&](long long r) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c = col + i * WPR * 128;
      if (c < a.d) {
        xn[i] = ldraw(X + r * a.d + c);
        gn[i] = ldraw(G + r * a.d + c);
        if (a.add) qn[i] = *reinterpret_cast<const float4*>(a.add + r * a.d + c);
      }
    }
  };
  if (row < a.n) fetch(row);
  int turn = 0;
  for (; row < a.n; row += step) {
    float4 x[NV], g[NV];
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {                       // columns past d hold zeros in x, g and w
      x[i] = as_f4(xn[i]); g[i] = as_f4(gn[i]);
      dot += g[i].x * ww[i].x * x[i].x + g[i].y * ww[i].y * x[i].y + g[i].z * ww[i].z * x[i].z + g[i].w * ww[i].w * x[i].w;
    }
    const float r = a.rstd[row];
    const long long base = row * a.d;
    float4 q[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) q[i] = qn[i];
    if (row + step < a.n) fetch(row + step);
    dot = team_sum<WPR>(dot, red[turn], team, warp, lane);
    turn ^= 1;
    const float k = dot * r * r * r / a.d;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c = col + i * WPR * 128;
      if (c < a.d) {
        const float4 o = make_float4(r * g[i].x * ww[i].x - x[i].x * k + q[i].x, r * g[i].y * ww[i].y - x[i].y * k + q[i].y,
                                     r * g[i].z * ww[i].z - x[i].z * k + q[i].z, r * g[i].w * ww[i].w - x[i].w * k + q[i].w);
        put4(reinterpret_cast<TX*>(a.out) + base + c, o);
        if (a.lo) put4(reinterpret_cast<bf16*>(a.lo) + base + c, o);
        acc[i].x += g[i].x * x[i].x * r; acc[i].y += g[i].y * x[i].y * r; acc[i].z += g[i].z * x[i].z * r; acc[i].w += g[i].w * x[i].w * r;
      }
    }
  }
  const int d4 = a.d >> 2;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = col + i * WPR * 128;
    if (c < a.d) wsum[team * d4 + (c >> 2)] = acc[i];
  }
  __syncthreads();
  for (int c = threadIdx.x; c < d4; c += blockDim.x) {
    float4 s = wsum[c];
#pragma unroll
    for (int t = 1; t < TEAMS; ++t) { const float4 v = wsum[t * d4 + c]; s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w; }
    reinterpret_cast<float4*>(a.dw_part + (long long)blockIdx.x * a.d)[c] = s;
  }
}

// dw[c] = sum over parts; block = 32 columns x 8 runs of parts
__global__ void __launch_bounds__(256) rmsnorm_dw_kernel(const float* __restrict__ part, float* __restrict__ dw, int parts, int d) {
  __shared__ float sh[8][33];
  const int cx = threadIdx.x & 31, ry = threadIdx.x >> 5, c = blockIdx.x * 32 + cx;
  float s = 0.f;
  if (c < d)
#pragma unroll 8
    for (int p = ry; p < parts; p += 8) s += part[(long long)p * d + c];
  sh[ry][cx] = s;
  __syncthreads();
  if (ry == 0 && c < d) {
#pragma unroll
    for (int i = 1; i < 8; ++i) s += sh[i][cx];
    dw[c] = s;
  }
}

// f(team width, float4 per lane) for a row of d elements: the smallest team with at most 4 float4 per lane (forward), 2
// (backward: three arrays in flight, the sums and the weight are all kept per lane)
template <typename F>
static void by_width_bwd(int d, F&& f) {
#define W_(wpr, nv) f(std::integral_constant<int, wpr>(), std::integral_constant<int, nv>())
  if (d <= 256) W_(1, 2); else if (d <= 512) W_(2, 2); else if (d <= 1024) W_(4, 2); else if (d <= 2048) W_(8, 2);
  else if (d <= 4096) W_(8, 4); else W_(8, 8);
#undef W_
}
template <typename F>
static void by_width(int d, F&& f) {
#define W_(wpr, nv) f(std::integral_constant<int, wpr>(), std::integral_constant<int, nv>())
  if (d <= 256) W_(1, 2); else if (d <= 512) W_(1, 4); else if (d <= 1024) W_(2, 4); else if (d <= 2048) W_(4, 4);
  else if (d <= 4096) W_(8, 4); else W_(8, 8);
#undef W_
}

template <typename F>
static void by_types(const NormArgs& a, F&& f) {
  if (a.y) f(float(), bf16(), std::true_type());
  else if (a.x_bf16 && a.out_bf16) f(bf16(), bf16(), std::false_type());
  else if (a.x_bf16) f(bf16(), float(), std::false_type());
  else if (a.out_bf16) f(float(), bf16(), std::false_type());
  else f(float(), float(), std::false_type());
}

void rmsnorm_fwd_launch(const NormArgs& a) {
  if (!a.n) return;
  by_types(a, [&](auto tx, auto ty, auto add) {
    using TX = decltype(tx);
    using TY = decltype(ty);
    constexpr bool ADD = decltype(add)::value;
    if (a.d > 8192) {
      rmsnorm_fwd_long_kernel<TX, TY, ADD><<<a.n, 256, 0, a.stream>>>(a);
      return;
    }
    by_width(a.d, [&](auto wpr, auto nv) {
      constexpr int W = decltype(wpr)::value, N = decltype(nv)::value, TEAMS = NORM_WARPS / W;
      rmsnorm_fwd_kernel<TX, TY, ADD, W, N><<<(a.n + TEAMS - 1) / TEAMS, NORM_WARPS * 32, 0, a.stream>>>(a);
    });
  });
}

// Blocks of the backward pass = rows of the dw workspace: three per SM cover the memory latency with the prefetched rows;
// fewer when a team would have less than 4 rows to spread the cost of its share of dw over.
int rmsnorm_parts(int n, int d) {
  int teams = 1;
  by_width_bwd(d, [&](auto wpr, auto) { teams = NORM_WARPS / decltype(wpr)::value; });
  const int want = (n + 4 * teams - 1) / (4 * teams);
  return want < 148 * 3 ? (want > 0 ? want : 1) : 148 * 3;
}

void rmsnorm_bwd_launch(const NormArgs& a) {
  const int grid = rmsnorm_parts(a.n, a.d);
  by_width_bwd(a.d, [&](auto wpr, auto nv) {
    constexpr int W = decltype(wpr)::value, N = decltype(nv)::value, TEAMS = NORM_WARPS / W;
    const size_t smem = (size_t)TEAMS * a.d * 4;          // at most 32 KB
#define L_(TX, TG) rmsnorm_bwd_kernel<TX, TG, W, N><<<grid, NORM_WARPS * 32, smem, a.stream>>>(a)
    if (a.x_bf16 && a.y_bf16) L_(bf16, bf16); else if (a.x_bf16) L_(bf16, float); else if (a.y_bf16) L_(float, bf16); else L_(float, float);
#undef L_
  });
  rmsnorm_dw_kernel<<<(a.d + 31) / 32, 256, 0, a.stream>>>(a.dw_part, a.dw, grid, a.d);
}

}  // namespace mb
