// Host interface of the row kernels in rmsnorm.cu and ce_rows.cu: plain pointers, no torch types.
#pragma once
#include <cuda_runtime.h>

namespace mb {

struct NormArgs {
  const void* x;            // (n, d): the normalised input (forward) / the same input (backward)
  int x_bf16;
  const void* y;            // forward: bf16 branch added to x first (add_rmsnorm) or null; backward: dy
  int y_bf16;
  const float* w;           // (d)
  float* rstd;              // (n)
  void* out;                // forward: normalised rows; backward: dx in the type of x
  int out_bf16;
  float* sum;               // add_rmsnorm: x + y (fp32)
  const float* add;         // backward: gradient that reached x by another path, or null
  void* lo;                 // backward: dx in bf16 as well, or null
  float* dw;                // backward: (d)
  float* dw_part;           // backward workspace: rmsnorm_parts() x d floats
  int n, d;
  float eps;
  cudaStream_t stream;
};
void rmsnorm_fwd_launch(const NormArgs& a);
int rmsnorm_parts(int n, int d);
void rmsnorm_bwd_launch(const NormArgs& a);

// logits (n, V) bf16 with row pitch `stride`: overwritten with d(loss)/d(logits); see ce_rows.cu
void ce_rows_launch(void* logits, const long long* y, float* loss, const float* gate, const float* hit, float* dg, long long stride,
                    int n, int V, cudaStream_t stream);
// out = x * *scale over n elements (n % 4 == 0, 16-byte aligned arrays), fp32 arithmetic
void scale_launch(const void* x, int x_bf16, const float* scale, void* out, int out_bf16, long long n, cudaStream_t stream);

}  // namespace mb
