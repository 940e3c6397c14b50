// Host interface of the tcgen05 GEMM (gemm_tc.cu): plain pointers, no torch types.  Failures are std::runtime_error.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace mb {

enum { EPI_NONE = 0, EPI_RELU2 = 1, EPI_DRELU2 = 2, EPI_SWIGLU = 3, EPI_ROWSCALE = 4, EPI_DSWIGLU = 5 };

struct GemmParams {
  int M, N, K, G;                 // logical per-group problem; for EPI_SWIGLU N = 2H (B rows), out has H columns
  void* out;
  void* out2;
  const void* aux;
  long long out_gs, out2_gs, aux_gs;   // group strides in elements
  int ldo, ldo2, ldaux;                // row pitches in elements
  int epi, out_f32, accumulate;
  int m_tiles, n_tiles, bn;  // bn: columns of a tile (pair kernel: 256 or 128, else 256)
  int ntail;                 // 1: the last N tile issues MMAs only as wide as its valid columns (rounded up to 16)
  int* status;
  // M may be cut into `n_seg` segments of `seg_M` rows, each read through its own A tensor map (a peer GPU's
  // buffer) and, when `out_seg_on`, written to its own output base (the owner GPU's buffer).  Tiles never straddle
  // segments.  Plain GEMM: n_seg = 1, seg_M = M.
  int n_seg, seg_M, tiles_per_seg, a_g_off, out_g_off, out_seg_on;
  void* out_seg[8];
  // Pair kernel v3 only.  store_tma: the epilogue leaves through TMA stores (local output, one segment); otherwise
  // through coalesced row stores from the staged tile (peer buffers, segmented output).
  // counts: valid extent per group (device ints) - count_mode 1: rows of A/out (tiles wholly past it are not
  // computed and are written as zeros), 2: length of the contraction (k-blocks past it are not read).
  int store_tma, count_mode, dbg, group_m;
  int aux_tma;             // the aux operand of an epilogue (pre-activations) is prefetched by TMA into the staging tiles
  const int* counts;
  // Pair kernel, plain epilogue, one group: the contraction is cut into `splits` runs of `kb_split` k-blocks, each a work item
  // of its own whose fp32 partial result goes to its own slab out + run * out_gs (0 or 1: not cut).
  int splits, kb_split;
};

void launch_gemm_seg(const void* const* A_list, int n_seg, int seg_M, int a_groups, long long a_rows_pitch, long long a_gs,
                     bool a_mn, const void* B, long long b_rows_pitch, long long b_gs, bool b_mn, GemmParams p,
                     cudaStream_t stream, int max_ctas);
void launch_gemm(const void* A, long long a_rows_pitch, long long a_gs, bool a_mn, const void* B, long long b_rows_pitch,
                 long long b_gs, bool b_mn, GemmParams p, cudaStream_t stream, int max_ctas);
int gemm_splits(int M, int N, int K, int G, int max_ctas, int& kb_split);
// dst (rows, n) of pitch ldo (+)= the sum of `splits` fp32 slabs (rows, n), always in the same order; n % 4 == 0, 16-byte rows
void sum_parts_launch(const float* parts, int splits, void* dst, int f32, int accumulate, long long rows, int n, int ldo, cudaStream_t stream);
int gemm_sm_count();
int* gemm_status_word(int device);
bool gemm_pair_on();

}  // namespace mb
