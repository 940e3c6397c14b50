// Torch side of the keys-and-locks search (locks.cu).
#include <torch/extension.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>

#include "locks_api.h"

namespace mb {

static std::vector<torch::Tensor> find(torch::Tensor x, int64_t vocab, int64_t n_keys, bool longest_only,
                                       c10::optional<torch::Tensor> bucket, bool want_bk) {
  const c10::cuda::CUDAGuard guard(x.device());
  TORCH_CHECK(x.dim() == 2 && x.is_contiguous() && x.scalar_type() == torch::kInt64, "lock_find: (B,T) int64");
  TORCH_CHECK(n_keys >= 1 && n_keys <= 3, "lock_find: 1..3 key lengths");
  const int64_t B = x.size(0), T = x.size(1);
  TORCH_CHECK((size_t)T * 4 <= 200 * 1024, "lock_find: text too long for shared memory staging");
  auto cand = torch::empty({B, T, n_keys}, x.options());
  auto src = torch::empty({B, T, n_keys}, x.options());
  auto on = torch::empty({B, T, n_keys}, x.options().dtype(torch::kBool));
  torch::Tensor bk;
  LockArgs a{};
  if (want_bk) {
    bk = torch::empty({B, T}, x.options());
    a.bk = reinterpret_cast<long long*>(bk.data_ptr<int64_t>());
    if (bucket.has_value() && bucket->defined()) {
      TORCH_CHECK(bucket->dim() == 1 && bucket->is_contiguous() && bucket->scalar_type() == torch::kInt64 && bucket->numel() > 0 &&
                  bucket->device() == x.device(), "lock_find: bucket table int64 on the device of x");
      a.bucket = reinterpret_cast<const long long*>(bucket->data_ptr<int64_t>());
      a.n_bucket = bucket->numel();
    }
  }
  a.x = reinterpret_cast<const long long*>(x.data_ptr<int64_t>());
  a.cand = reinterpret_cast<long long*>(cand.data_ptr<int64_t>());
  a.src = reinterpret_cast<long long*>(src.data_ptr<int64_t>());
  a.on = on.data_ptr<bool>();
  a.vocab = vocab;
  a.B = (int)B; a.T = (int)T; a.n_keys = (int)n_keys; a.longest_only = longest_only ? 1 : 0;
  a.stream = at::cuda::getCurrentCUDAStream();
  TORCH_CHECK(lock_find_launch(a), "lock_find: cannot raise dynamic shared memory");
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  if (want_bk) return {cand, on, src, bk};
  return {cand, on, src};
}

std::vector<torch::Tensor> lock_find(torch::Tensor x, int64_t vocab, int64_t n_keys, bool longest_only) {
  return find(x, vocab, n_keys, longest_only, c10::nullopt, false);
}
// the same with the trust bucket of every word (zeros without a table); a table means only the longest lock fires
std::vector<torch::Tensor> lock_find_bucket(torch::Tensor x, int64_t vocab, int64_t n_keys, c10::optional<torch::Tensor> bucket) {
  return find(x, vocab, n_keys, bucket.has_value() && bucket->defined(), bucket, true);
}

int64_t lock_status(int64_t device) {
  const c10::cuda::CUDAGuard guard((c10::DeviceIndex)device);
  return lock_status_read();
}

}  // namespace mb
