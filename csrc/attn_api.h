// Host interface of the attention kernels (attn_fwd.cu, attn_bwd.cu): plain pointers, no torch types.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace mb {

// A (text b, position t, head h, 64) bf16 array: element strides, the 64 head dims contiguous.
struct AttnView {
  void* p;
  long long sb, st, sh;
};

struct AttnArgs {
  int B, H, T, window;      // window 0 = plain causal, else key j is visible to query i iff 0 <= i - j < window
  float scale;              // multiplies the scores
  AttnView q, k, v, o;      // q and k already rotated
  float* lse;               // (B, H, T) natural log of the softmax denominator
  // backward only
  AttnView dout, dq, dk, dv;
  const float *cos, *sin;   // (T, 32) tables: dq and dk are rotated back; null: left as they are
  int rope_half;            // 0: pairs (2i, 2i+1), 1: pairs (i, i + 32)
  float* stats;             // workspace (B*H, 2 tiles, 2, 64): lse * log2(e) and rowsum(dO * O), attn_stats_floats() floats
  int* status;
  cudaStream_t stream;
};

inline long long attn_tiles(int T) { return (T + 127) / 128; }
inline long long attn_stats_floats(int B, int H, int T) { return (long long)B * H * attn_tiles(T) * 256; }

// nullptr on success, else what went wrong (nothing was launched then)
const char* attn_fwd_launch(const AttnArgs& a);
const char* attn_bwd_launch(const AttnArgs& a);
// q and k slices of qkv (B, T, 3, H, 64) rotated into out (B, T, slots, H, 64): 2 slots, or 3 with v copied; out may be qkv (3 slots)
void rope_qk2_launch(const void* qkv, void* out, const float* cos, const float* sin, int B, int T, int H, int half, int slots, cudaStream_t st);

}  // namespace mb
