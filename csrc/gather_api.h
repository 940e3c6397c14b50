// Host interface of the slot kernels (gather.cu): plain pointers, no torch types.  Rows are bf16, d % 8 == 0, 16-byte aligned.
#pragma once
#include <cuda_runtime.h>

namespace mb {

void rows_gather_launch(const void* src, const long long* table, void* out, long long S, int d, long long n_src, cudaStream_t st);
void rows_gather_sum_launch(const void* src, const long long* idx, const float* w, void* out, long long N, int k, int d, long long S, cudaStream_t st);
void combine_bwd_launch(const void* go, const long long* table, const float* w, const void* ye, void* dye, float* dw, long long S, int d,
                        long long N, cudaStream_t st);
// buf[e] <- 0.9 buf[e] + 0.1 mean_c |g[e, c]|; part: err_probe_parts(C) x E floats
int err_probe_parts(int C);
void err_probe_launch(const void* g, float* buf, float* part, int E, int C, int d, cudaStream_t st);

}  // namespace mb
