// Data passes around the frozen expert bank: int8 tables expanded to bf16 in one pass, rows quantised to int8, whole expert
// groups moved between the full stack and the lists of learning and frozen experts.  All memory-bound, 16-byte accesses.
// Us, element-wise passes -> these, (4, 768, 1536) + (4, 768, 768) tables and 8 groups of 1025 x 768: tables 150 -> 24, rows 30 -> 24,
// groups 88 -> 26.
#include "bank_api.h"
#include "common.cuh"

namespace mb {

static int copy_grid(long long n) { return (int)((n + 255) / 256 < 148 * 16 ? (n + 255) / 256 : 148 * 16); }

__global__ void __launch_bounds__(256) dequant_i8_kernel(const uint2* __restrict__ q, const uint4* __restrict__ scale, uint4* __restrict__ out,
                                                         long long n8, long long per_f, int o8) {
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < n8; i += (long long)gridDim.x * 256) {
    const long long f = i / per_f;
    const int o = (int)((i - f * per_f) % o8);
    const uint2 v = q[i];
    const uint4 s = scale[f * o8 + o];
    const uint32_t sw[4] = {s.x, s.y, s.z, s.w};
    uint32_t r[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t w = (j < 2 ? v.x : v.y) >> (16 * (j & 1));
      const float2 k = unpack_bf16(sw[j]);
      r[j] = pack_bf16((float)(signed char)(w & 0xff) * k.x, (float)(signed char)(w >> 8 & 0xff) * k.y);
    }
    out[i] = make_uint4(r[0], r[1], r[2], r[3]);
  }
}
void dequant_i8_launch(const signed char* q, const void* scale, void* out, long long F, long long I, int O, cudaStream_t st) {
  const long long n8 = F * I * (O / 8);
  if (n8) dequant_i8_kernel<<<copy_grid(n8), 256, 0, st>>>(reinterpret_cast<const uint2*>(q), reinterpret_cast<const uint4*>(scale),
                                                           reinterpret_cast<uint4*>(out), n8, I * (O / 8), O / 8);
}

template <bool BF16> __device__ __forceinline__ void row8(const void* x, long long i, float (&v)[8]) {
  if (BF16) {
    const uint4 u = *reinterpret_cast<const uint4*>(reinterpret_cast<const bf16*>(x) + i);
    const uint32_t q[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) { const float2 f = unpack_bf16(q[j]); v[2 * j] = f.x; v[2 * j + 1] = f.y; }
  } else {
    const float4 a = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(x) + i);
    const float4 b = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(x) + i + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  }
}

// A warp per row; the second look at the row comes from L1.
template <bool BF16>
__global__ void __launch_bounds__(256) quant_rows_wide_kernel(const void* __restrict__ x, signed char* __restrict__ q, float* __restrict__ s, long long R, int K) {
  const int lane = threadIdx.x & 31;
  for (long long r = (blockIdx.x * 256ll + threadIdx.x) >> 5; r < R; r += ((long long)gridDim.x * 256) >> 5) {
    float mx = 0.f;
#pragma unroll 4
    for (int c = lane * 8; c < K; c += 256) {
      float v[8];
      row8<BF16>(x, r * K + c, v);
#pragma unroll
      for (int j = 0; j < 8; ++j) mx = fmaxf(mx, fabsf(v[j]));
    }
    mx = warp_max(mx);
    const float sc = fmaxf(mx, 1e-12f) * (1.f / 127.f);     // as the PyTorch statement computes it (division by a scalar)
#pragma unroll 4
    for (int c = lane * 8; c < K; c += 256) {
      float v[8];
      row8<BF16>(x, r * K + c, v);
      uint32_t w[2] = {0u, 0u};
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float t = rintf(__fdiv_rn(v[j], sc));          // a true division: same ties as the oracle
        w[j >> 2] |= (uint32_t)(uint8_t)(signed char)fminf(fmaxf(t, -127.f), 127.f) << (8 * (j & 3));
      }
      *reinterpret_cast<uint2*>(q + r * K + c) = make_uint2(w[0], w[1]);
    }
    if (lane == 0) s[r] = sc;
  }
}
void quant_rows_wide_launch(const void* x, int bf16_in, signed char* q, float* s, long long R, int K, cudaStream_t st) {
  const int grid = (int)((R + 7) / 8 < 148 * 8 ? (R + 7) / 8 : 148 * 8);
  if (bf16_in) quant_rows_wide_kernel<true><<<grid, 256, 0, st>>>(x, q, s, R, K);
  else quant_rows_wide_kernel<false><<<grid, 256, 0, st>>>(x, q, s, R, K);
}

// grid (blocks per group, groups)
__global__ void __launch_bounds__(256) groups_copy_kernel(const uint4* __restrict__ a, const long long* __restrict__ ia, int na, const uint4* __restrict__ b,
                                                          const long long* __restrict__ ib, uint4* __restrict__ out, long long n16, int put) {
  const int j = blockIdx.y;
  const uint4* src = a;
  long long from = j, to = j;
  if (put) {
    if (j < na) to = ia[j];
    else { src = b; from = j - na; to = ib[from]; }
  } else {
    from = ia[j];
  }
  src += from * n16;
  uint4* dst = out + to * n16;
#pragma unroll 4
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < n16; i += (long long)gridDim.x * 256) dst[i] = src[i];
}
static dim3 groups_grid(int n, long long n16) {
  const long long want = (n16 + 1023) / 1024, most = (148 * 8 + n - 1) / n;
  return dim3((unsigned)(want < most ? want : most), n);
}
void groups_take_launch(const void* src, const long long* idx, void* out, int n, long long n16, cudaStream_t st) {
  if (n && n16) groups_copy_kernel<<<groups_grid(n, n16), 256, 0, st>>>(reinterpret_cast<const uint4*>(src), idx, n, nullptr, nullptr, reinterpret_cast<uint4*>(out), n16, 0);
}
void groups_put_launch(const void* a, const long long* ia, int na, const void* b, const long long* ib, int nb, void* out, long long n16, cudaStream_t st) {
  if (na + nb && n16)
    groups_copy_kernel<<<groups_grid(na + nb, n16), 256, 0, st>>>(reinterpret_cast<const uint4*>(a), ia, na, reinterpret_cast<const uint4*>(b), ib,
                                                                  reinterpret_cast<uint4*>(out), n16, 1);
}

}  // namespace mb
