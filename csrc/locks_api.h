// Host interface of the keys-and-locks search (locks.cu): plain pointers, no torch types.
#pragma once
#include <cuda_runtime.h>

namespace mb {

struct LockArgs {
  const long long* x;            // (B, T) word ids
  long long *cand, *src;         // (B, T, n_keys)
  bool* on;                      // (B, T, n_keys)
  const long long* bucket;       // optional table of n_bucket entries: bk[b, t] = bucket[min(x, n_bucket - 1)]
  long long* bk;                 // (B, T), zeros without a table; null: not wanted
  long long n_bucket;
  long long vocab;
  int B, T, n_keys, longest_only;
  cudaStream_t stream;
};
// false: the shared memory could not be had (nothing was launched)
bool lock_find_launch(const LockArgs& a);

}  // namespace mb
