// Cross-entropy row kernel.  One block per row of bf16 logits: online max / sum -> log-sum-exp; loss; the logits are
// overwritten with d(loss)/d(logits).  With gate / hit the pointer mixture P = (1-g) p_y + g hit, loss = -log max(P, 1e-30),
// gradient w (softmax - onehot) with w = (1-g) p_y / P, dg = (p_y - hit) / P.
// The logits of a chunk (4096 x 50 304 bf16 = 412 MB) come from HBM and go back to it: 126 us at the copy rate is the
// floor, the second read of a row is served by L2.  Each thread keeps four 16-byte loads in flight (one at a time ran at
// 3.5 TB/s of the 2 x 412 MB), and the one-hot term is not compared against in the loop: the thread that holds the
// target's 16 bytes redoes that element at the end.
// 4096 x 50 304: 233 us before, 190 now; 1000 x 50 304: 66 before, 53 now.
#include "common.cuh"
#include "rowops_api.h"

namespace mb {

constexpr int CE_THREADS = 512, CE_U = 4;

__device__ __forceinline__ void unpack8(const uint4& u, float (&v)[8]) {
  const uint32_t q[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) { const float2 f = unpack_bf16(q[j]); v[2 * j] = f.x; v[2 * j + 1] = f.y; }
}

__global__ void __launch_bounds__(CE_THREADS) ce_rows_kernel(bf16* __restrict__ logits, const long long* __restrict__ y, float* __restrict__ loss,
                                                             const float* __restrict__ gate, const float* __restrict__ hit,
                                                             float* __restrict__ dg, long long stride, int V) {
  __shared__ float red[32];
  const long long row = blockIdx.x;
  bf16* p = logits + row * stride;
  uint4* p8 = reinterpret_cast<uint4*>(p);
  const int V8 = V / 8;
  const long long yy = y[row];
  float m = -INFINITY, s = 0.f;
  auto fold = [&](const float (&v)[8]) {
    float mx = v[0];
#pragma unroll
    for (int j = 1; j < 8; ++j) mx = fmaxf(mx, v[j]);
    if (mx > m) { s *= __expf(m - mx); m = mx; }                // first time: s is 0 and e^-inf is 0
    const float ref = m == -INFINITY ? 0.f : m;
    float add = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) add += __expf(v[j] - ref);
    s += add;
  };
  int i = threadIdx.x;
  for (; i + (CE_U - 1) * CE_THREADS < V8; i += CE_U * CE_THREADS) {
    uint4 u[CE_U];
#pragma unroll
    for (int k = 0; k < CE_U; ++k) u[k] = p8[i + k * CE_THREADS];
#pragma unroll
    for (int k = 0; k < CE_U; ++k) { float v[8]; unpack8(u[k], v); fold(v); }
  }
  for (; i < V8; i += CE_THREADS) { float v[8]; unpack8(p8[i], v); fold(v); }
  for (int c = V8 * 8 + threadIdx.x; c < V; c += CE_THREADS) {
    const float v = __bfloat162float(p[c]);
    if (v > m) { s *= __expf(m - v); m = v; }
    s += __expf(v - (m == -INFINITY ? 0.f : m));
  }
  const float M = block_max(m, red);
  s = (m == -INFINITY) ? 0.f : s * __expf(m - M);
  s = block_sum(s, red);
  const float lse = M + logf(s);
  const float xy = __bfloat162float(p[yy]);
  float wgt = 1.f;
  __syncthreads();                                           // every thread has read p[yy] before anyone overwrites it
  if (gate != nullptr) {
    const float g = gate[row], h = hit[row];
    const float py = __expf(xy - lse);
    const float P = fmaxf((1.f - g) * py + g * h, 1e-30f);
    wgt = (1.f - g) * py / P;
    if (threadIdx.x == 0) { loss[row] = -logf(P); dg[row] = (py - h) / P; }
  } else if (threadIdx.x == 0) {
    loss[row] = lse - xy;
  }
  auto grads = [&](int at, const uint4& u) {
    float v[8];
    unpack8(u, v);
    const int hot = (int)(yy - (long long)at * 8);           // 0..7: the target is among these
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = wgt * __expf(v[j] - lse);
    if ((unsigned)hot < 8u) {
#pragma unroll
      for (int j = 0; j < 8; ++j) if (j == hot) v[j] = wgt * (__expf(xy - lse) - 1.f);
    }
    p8[at] = make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
  };
  i = threadIdx.x;
  for (; i + (CE_U - 1) * CE_THREADS < V8; i += CE_U * CE_THREADS) {
    uint4 u[CE_U];
#pragma unroll
    for (int k = 0; k < CE_U; ++k) u[k] = p8[i + k * CE_THREADS];
#pragma unroll
    for (int k = 0; k < CE_U; ++k) grads(i + k * CE_THREADS, u[k]);
  }
  for (; i < V8; i += CE_THREADS) grads(i, p8[i]);
  for (int c = V8 * 8 + threadIdx.x; c < V; c += CE_THREADS) {
    const float v = __bfloat162float(p[c]);
    p[c] = __float2bfloat16(wgt * (__expf(v - lse) - (c == yy ? 1.f : 0.f)));
  }
}

void ce_rows_launch(void* logits, const long long* y, float* loss, const float* gate, const float* hit, float* dg, long long stride,
                    int n, int V, cudaStream_t stream) {
  ce_rows_kernel<<<n, CE_THREADS, 0, stream>>>(reinterpret_cast<bf16*>(logits), y, loss, gate, hit, dg, stride, V);
}

// out = x * *scale: the gradients of the forward pass times the one that arrives at the loss.  A plain copy in its traffic;
// four pieces of four elements per thread in flight.  (50 304 x 2064) fp32: 153 us
// (127 at the copy rate); the broadcast multiplication of PyTorch took 318.
template <bool XB, bool OB>
__global__ void __launch_bounds__(256) scale_kernel(const void* __restrict__ x, const float* __restrict__ scale, void* __restrict__ out, long long n4) {
  const float f = *scale;
  const long long step = (long long)gridDim.x * 256;
  for (long long i0 = blockIdx.x * 256ll + threadIdx.x; i0 < n4; i0 += 4 * step) {
    float4 v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const long long i = i0 + k * step;
      if (i >= n4) continue;
      if (XB) {
        const uint2 u = reinterpret_cast<const uint2*>(x)[i];
        const float2 a = unpack_bf16(u.x), b = unpack_bf16(u.y);
        v[k] = make_float4(a.x, a.y, b.x, b.y);
      } else {
        v[k] = reinterpret_cast<const float4*>(x)[i];
      }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const long long i = i0 + k * step;
      if (i >= n4) continue;
      if (OB) reinterpret_cast<uint2*>(out)[i] = make_uint2(pack_bf16(v[k].x * f, v[k].y * f), pack_bf16(v[k].z * f, v[k].w * f));
      else reinterpret_cast<float4*>(out)[i] = make_float4(v[k].x * f, v[k].y * f, v[k].z * f, v[k].w * f);
    }
  }
}
void scale_launch(const void* x, int x_bf16, const float* scale, void* out, int out_bf16, long long n, cudaStream_t stream) {
  const long long n4 = n / 4, want = (n4 + 1023) / 1024;
  const int grid = (int)(want < 148 * 8 ? want : 148 * 8);
  if (!grid) return;
  if (x_bf16 && out_bf16) scale_kernel<true, true><<<grid, 256, 0, stream>>>(x, scale, out, n4);
  else if (x_bf16) scale_kernel<true, false><<<grid, 256, 0, stream>>>(x, scale, out, n4);
  else if (out_bf16) scale_kernel<false, true><<<grid, 256, 0, stream>>>(x, scale, out, n4);
  else scale_kernel<false, false><<<grid, 256, 0, stream>>>(x, scale, out, n4);
}

}  // namespace mb
