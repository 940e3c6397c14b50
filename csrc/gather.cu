// Slot <-> token movement of the expert layers on bf16 rows, a warp per row with 16-byte accesses, all loads of four
// 256-column pieces in flight: memory-bound copies.  Us for 8192 tokens x 2048, 16 392 places, one element at a time -> these: slots
// 35 -> 17.5, combine 30 -> 17, both gradients of the combine 57 -> 25 (100 MB: 20 at the copy rate), error probe 50 -> 22.
#include "common.cuh"
#include "gather_api.h"

namespace mb {

constexpr int GA_U = 4;                                  // 16-byte pieces per lane in flight

__device__ __forceinline__ void unpack8(const uint4& u, float (&v)[8]) {
  const uint32_t q[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) { const float2 f = unpack_bf16(q[j]); v[2 * j] = f.x; v[2 * j + 1] = f.y; }
}
__device__ __forceinline__ uint4 pack8(const float (&v)[8]) {
  return make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
}
#define GA_ROWS(r, R) for (long long r = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5; r < (R); r += ((long long)gridDim.x * blockDim.x) >> 5)

// out[s] = src[table[s]], zeros for empty places
__global__ void __launch_bounds__(256) rows_gather_kernel(const uint4* __restrict__ src, const long long* __restrict__ table, uint4* __restrict__ out,
                                                          long long S, int d8, long long n_src) {
  const int lane = threadIdx.x & 31;
  GA_ROWS(s, S) {
    const long long t = table[s];
    const bool ok = t >= 0 && t < n_src;
    for (int c0 = lane; c0 < d8; c0 += 32 * GA_U) {
      uint4 v[GA_U];
#pragma unroll
      for (int u = 0; u < GA_U; ++u) v[u] = ok && c0 + 32 * u < d8 ? src[t * d8 + c0 + 32 * u] : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int u = 0; u < GA_U; ++u)
        if (c0 + 32 * u < d8) out[s * d8 + c0 + 32 * u] = v[u];
    }
  }
}

// out[n] = sum_j (w ? w[idx[n,j]] : 1) * src[idx[n,j]] over idx < S, fp32 sums
__global__ void __launch_bounds__(256) rows_gather_sum_kernel(const uint4* __restrict__ src, const long long* __restrict__ idx, const float* __restrict__ w,
                                                              uint4* __restrict__ out, long long N, int k, int d8, long long S) {
  const int lane = threadIdx.x & 31;
  GA_ROWS(n, N) {
    for (int c0 = lane; c0 < d8; c0 += 32 * GA_U) {
      float acc[GA_U][8] = {};
      for (int j = 0; j < k; ++j) {
        const long long s = idx[n * k + j];
        if (s < 0 || s >= S) continue;
        const float ww = w ? w[s] : 1.f;
        uint4 v[GA_U];
#pragma unroll
        for (int u = 0; u < GA_U; ++u)
          if (c0 + 32 * u < d8) v[u] = src[s * d8 + c0 + 32 * u];
#pragma unroll
        for (int u = 0; u < GA_U; ++u)
          if (c0 + 32 * u < d8) {
            float f[8];
            unpack8(v[u], f);
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[u][i] += f[i] * ww;
          }
      }
#pragma unroll
      for (int u = 0; u < GA_U; ++u)
        if (c0 + 32 * u < d8) out[n * d8 + c0 + 32 * u] = pack8(acc[u]);
    }
  }
}

// backward of out[n] = sum_j w[s] ye[s]:  dye[s] = w[s] go[table[s]],  dw[s] = <go[table[s]], ye[s]>; one read of go for both
__global__ void __launch_bounds__(256) combine_bwd_kernel(const uint4* __restrict__ go, const long long* __restrict__ table, const float* __restrict__ w,
                                                          const uint4* __restrict__ ye, uint4* __restrict__ dye, float* __restrict__ dw, long long S,
                                                          int d8, long long N) {
  const int lane = threadIdx.x & 31;
  GA_ROWS(s, S) {
    const long long t = table[s];
    const bool ok = t >= 0 && t < N;
    const float ww = ok ? w[s] : 0.f;
    float dot = 0.f;
    for (int c0 = lane; c0 < d8; c0 += 32 * GA_U) {
      uint4 a[GA_U], b[GA_U];
#pragma unroll
      for (int u = 0; u < GA_U; ++u) {
        const bool in = ok && c0 + 32 * u < d8;
        a[u] = in ? go[t * d8 + c0 + 32 * u] : make_uint4(0, 0, 0, 0);
        b[u] = in ? ye[s * d8 + c0 + 32 * u] : make_uint4(0, 0, 0, 0);
      }
#pragma unroll
      for (int u = 0; u < GA_U; ++u)
        if (c0 + 32 * u < d8) {
          float f[8], g[8];
          unpack8(a[u], f);
          unpack8(b[u], g);
#pragma unroll
          for (int i = 0; i < 8; ++i) { dot += f[i] * g[i]; f[i] *= ww; }
          dye[s * d8 + c0 + 32 * u] = pack8(f);
        }
    }
    dot = warp_sum(dot);
    if (lane == 0) dw[s] = dot;
  }
}

// grid (parts, E): part[e][blockIdx.x] = sum of the norms of this block's rows of expert e
__global__ void __launch_bounds__(256) err_rows_kernel(const uint4* __restrict__ g, float* __restrict__ part, int C, int d8) {
  __shared__ float red[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long e = blockIdx.y;
  float sum = 0.f;
  for (int c = blockIdx.x * 8 + warp; c < C; c += gridDim.x * 8) {
    const uint4* row = g + (e * C + c) * d8;
    float ss = 0.f;
    for (int c0 = lane; c0 < d8; c0 += 32 * GA_U) {
      uint4 v[GA_U];
#pragma unroll
      for (int u = 0; u < GA_U; ++u) v[u] = c0 + 32 * u < d8 ? row[c0 + 32 * u] : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int u = 0; u < GA_U; ++u) {
        float f[8];
        unpack8(v[u], f);
#pragma unroll
        for (int i = 0; i < 8; ++i) ss += f[i] * f[i];
      }
    }
    sum += sqrtf(warp_sum(ss));
  }
  sum = block_sum(lane == 0 ? sum : 0.f, red);
  if (threadIdx.x == 0) part[e * gridDim.x + blockIdx.x] = sum;
}
__global__ void err_fold_kernel(const float* __restrict__ part, float* __restrict__ buf, int parts, int C) {
  float s = 0.f;
  for (int i = threadIdx.x; i < parts; i += 32) s += part[blockIdx.x * parts + i];
  s = warp_sum(s);
  if (threadIdx.x == 0) buf[blockIdx.x] = buf[blockIdx.x] * 0.9f + 0.1f * (s / (float)C);
}

static int row_grid(long long rows) { return (int)((rows + 7) / 8 < 148 * 8 ? (rows + 7) / 8 : 148 * 8); }

void rows_gather_launch(const void* src, const long long* table, void* out, long long S, int d, long long n_src, cudaStream_t st) {
  rows_gather_kernel<<<row_grid(S), 256, 0, st>>>(reinterpret_cast<const uint4*>(src), table, reinterpret_cast<uint4*>(out), S, d / 8, n_src);
}
void rows_gather_sum_launch(const void* src, const long long* idx, const float* w, void* out, long long N, int k, int d, long long S, cudaStream_t st) {
  rows_gather_sum_kernel<<<row_grid(N), 256, 0, st>>>(reinterpret_cast<const uint4*>(src), idx, w, reinterpret_cast<uint4*>(out), N, k, d / 8, S);
}
void combine_bwd_launch(const void* go, const long long* table, const float* w, const void* ye, void* dye, float* dw, long long S, int d,
                        long long N, cudaStream_t st) {
  combine_bwd_kernel<<<row_grid(S), 256, 0, st>>>(reinterpret_cast<const uint4*>(go), table, w, reinterpret_cast<const uint4*>(ye),
                                                  reinterpret_cast<uint4*>(dye), dw, S, d / 8, N);
}
int err_probe_parts(int C) { return (C + 31) / 32 < 64 ? (C + 31) / 32 : 64; }
void err_probe_launch(const void* g, float* buf, float* part, int E, int C, int d, cudaStream_t st) {
  const int parts = err_probe_parts(C);
  err_rows_kernel<<<dim3(parts, E), 256, 0, st>>>(reinterpret_cast<const uint4*>(g), part, C, d / 8);
  err_fold_kernel<<<E, 32, 0, st>>>(part, buf, parts, C);
}

}  // namespace mb
