// Host interface of the keys-and-locks search (locks.cu): plain pointers, no torch types.
#pragma once
#include <cuda_runtime.h>

namespace mb {

struct LockArgs {
  const long long* x;            // (B, T) word ids
  long long *cand, *src;         // (B, T, n_keys)
  bool* on;                      // (B, T, n_keys)
  const long long* bucket;       // optional table of n_bucket entries: bk[b, t] = bucket[min(x, n_bucket - 1)], x < 0 from the end
  long long* bk;                 // (B, T), zeros without a table; null: not wanted
  long long n_bucket;
  long long vocab;
  int B, T, n_keys, longest_only;
  cudaStream_t stream;
};
// false: the shared memory could not be had (nothing was launched)
bool lock_find_launch(const LockArgs& a);
enum { LOCK_BAD_ID = 1 };
// status word of the current device, cleared: LOCK_BAD_ID when a word id below -n_bucket was looked up (host sync)
int lock_status_read();

}  // namespace mb
