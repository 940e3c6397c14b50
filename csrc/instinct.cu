// Instinct optimizer step on the device: momentum, homeostasis normalisation (row -> column -> row, or the
// transposed order for experts), weight decay, step scaled by the situation card's gain and stake, fp32 master copy
// or counter-hash stochastic rounding for bf16 weights.  No scalar ever visits the host: gain, stake and the learning
// rate are read from device memory.
//
// A weight is viewed as (E, R, C) with C contiguous; the kernels and their launch order are in instinct_core.cuh:
//   hs   (2-D)  : rows -> cols(rows) -> apply with the last row norm fused (row staged in shared memory)
//   hs3  (E,K,N): cols -> rows(cols) -> cols(cols, rows) -> apply
//   vocab       : rows (+|g|) -> apply, rows without gradient stay put, no weight decay
//   row / row3 / tensor : one stat -> apply
//   lagged hs   : one pass (column norm of the previous step); lagged hs3: the exact sequence with the row norm
//                 taken from the previous step
// Scratch statistics live in a caller-owned arena (zeroed here with one cudaMemsetAsync), not in memory allocated per
// call.
#include "instinct_core.cuh"

namespace mb {

int64_t instinct_run(const InstinctArgs& a, int kind, float* scratch, float* rel_out, cudaStream_t st, float* cs, int* cs_ok, int phase,
                     long long col_rows) {
  return instinct_launch(a, kind, scratch, rel_out, st, cs, cs_ok, phase, col_rows);
}

}  // namespace mb
