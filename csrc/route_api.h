// Host interface of the fused MoE router (route.cu): plain pointers, no torch types.
#pragma once
#include <cuda_runtime.h>

namespace mb {

constexpr int ROUTE_E = 128, ROUTE_K = 8, ROUTE_TOK = 32;     // experts, choices per token, tokens per block

struct RouteArgs {
  const void* x;               // (N, d) bf16
  const float* w;              // (E, d)
  const bool* real;            // (N)
  const long long* k_tok;      // (N)
  int N, d, E, k, C;           // k choices per token, C places per expert
  // forward results
  float* probs;                // (N, E)
  long long* top_e;            // (N, k)
  float* wt;                   // (N, k)
  float* wtab;                 // (E * C)
  long long* table;            // (E * C): token of every place, N = empty
  long long* flat_idx;         // (N, k): place of every choice, E * C = none
  float* dropped;              // scalar
  float* aux;                  // scalar
  float* aux_grad;             // (E): d aux / d (sum of probs of expert e over the real tokens)
  int* counts;                 // (E): filled places
  int* hist;                   // workspace (blocks, E)
  float* psum;                 // workspace (blocks, E)
  int* n_real;                 // workspace (blocks)
  int* total;                  // workspace (E), or null: every block of route_place_kernel adds up the blocks' numbers itself
  float* ps;                   // workspace (E) beside it
  // backward (null: no gradient arrives there)
  const float *d_wt, *d_wtab, *d_aux, *d_probs;
  float* dl;                   // workspace (N, E): gradient of the logits
  void* dx;                    // (N, d) bf16
  float* dw;                   // (E, d)
  float* dw_part;              // workspace (dw_runs, E, d)
  int dw_runs, dw_run;         // runs of tokens and their length: route_dw_runs()
  cudaStream_t stream;
};
// Blocks from which on their numbers are added up once, in a kernel of their own, instead of by every block: the latter is quadratic
// in the tokens.
constexpr int ROUTE_SCAN = 1024;
inline int route_blocks(int N) { return (N + ROUTE_TOK - 1) / ROUTE_TOK; }
void route_fwd_launch(const RouteArgs& a);
int route_dw_runs(int N, int d, int E, int& run);
void route_bwd_launch(const RouteArgs& a);

}  // namespace mb
