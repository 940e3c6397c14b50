// Host interface of the frozen-bank kernels (bank.cu): plain pointers, no torch types.
#pragma once
#include <cuda_runtime.h>

namespace mb {

// out[f, i, o] = bf16(q[f, i, o] * scale[f, o]); O % 8 == 0, 16-byte aligned arrays
void dequant_i8_launch(const signed char* q, const void* scale, void* out, long long F, long long I, int O, cudaStream_t st);
// q[r, :] = rint(x[r, :] / s[r]) with s[r] = max|x[r, :]| / 127; K % 8 == 0, 16-byte aligned rows
void quant_rows_wide_launch(const void* x, int bf16_in, signed char* q, float* s, long long R, int K, cudaStream_t st);
// groups of n16 16-byte words: take out[j] = src[idx[j]]; put out[ia[j]] = a[j], out[ib[j]] = b[j]
void groups_take_launch(const void* src, const long long* idx, void* out, int n, long long n16, cudaStream_t st);
void groups_put_launch(const void* a, const long long* ia, int na, const void* b, const long long* ib, int nb, void* out, long long n16, cudaStream_t st);

}  // namespace mb
