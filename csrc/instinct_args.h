// Arguments of one Instinct step (instinct_core.cuh): plain pointers, no torch types.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace mb {

struct InstinctArgs {
  void* p;                 // weight (bf16 or fp32)
  const void* g;           // gradient
  void* m;                 // momentum
  float* w;                // exact fp32 copy of a bf16 weight, or nullptr
  int p_bf16, g_bf16, m_bf16;
  const float* gain;       // device scalar: gain of this weight on the current situation card
  const float* stake;      // device scalar
  const float* lr;         // device scalar: lr * scale
  float beta, wd;
  int sr;                  // stochastic rounding of bf16 stores
  const long long* seed;   // device step counter for the rounding hash
  unsigned salt;
  const bool* frozen;      // optional mask over the leading dimension: frozen slices keep their weights
  long long frozen_stride;
  long long E, R, C;
  void* shadow;            // optional bf16 copy of an fp32 weight, refreshed by `apply` (what the GEMMs read)
};

// Scratch layout (fp32, ZEROED by the caller, 16-byte aligned base): [rowA][rowB][rowabs] of pad4(E*R) each,
// [colA][colB] of pad4(E*C) each, [rel 4]; every sub-array starts on a 16-byte boundary.
inline long long instinct_pad4(long long n) { return (n + 3) & ~3ll; }
inline long long instinct_scratch_floats(long long E, long long R, long long C) {
  return 3 * instinct_pad4(E * R) + 2 * instinct_pad4(E * C) + 4;
}

constexpr size_t INSTINCT_SMEM_MAX = 200 * 1024;     // dynamic shared memory the row-staging kernels may ask for

// instinct_launch() of instinct_core.cuh, compiled once (instinct.cu)
int64_t instinct_run(const InstinctArgs& a, int kind, float* scratch, float* rel_out, cudaStream_t st, float* cs, int* cs_ok, int phase,
                     long long col_rows);

}  // namespace mb
