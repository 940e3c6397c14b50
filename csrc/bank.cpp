// Torch side of the frozen-bank kernels (bank.cu).
#include <torch/extension.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>

#include "bank_api.h"

namespace mb {

static bool aligned(const torch::Tensor& t) { return t.is_contiguous() && (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0; }
static const long long* i64(const torch::Tensor& t) {
  TORCH_CHECK(t.is_contiguous() && t.scalar_type() == torch::kInt64 && t.dim() == 1, "group list: contiguous int64");
  return reinterpret_cast<const long long*>(t.data_ptr<int64_t>());
}

// q (F, I, O) int8, scale (F, 1, O) bf16 -> (F, I, O) bf16
torch::Tensor dequant_i8(torch::Tensor q, torch::Tensor scale) {
  const c10::cuda::CUDAGuard guard(q.device());
  TORCH_CHECK(q.dim() == 3 && q.scalar_type() == torch::kInt8 && scale.scalar_type() == torch::kBFloat16 && q.size(2) % 8 == 0 &&
              scale.numel() == q.size(0) * q.size(2) && aligned(q) && aligned(scale), "dequant_i8: (F, I, O) int8, (F, 1, O) bf16, O % 8 == 0");
  auto out = torch::empty(q.sizes(), scale.options());
  dequant_i8_launch(reinterpret_cast<const signed char*>(q.data_ptr()), scale.data_ptr(), out.data_ptr(), q.size(0), q.size(1), (int)q.size(2),
                    at::cuda::getCurrentCUDAStream());
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  return out;
}

// x (..., K) bf16 or fp32 -> int8 rows and their scales
std::vector<torch::Tensor> quant_rows_wide(torch::Tensor x) {
  const c10::cuda::CUDAGuard guard(x.device());
  const int64_t K = x.size(-1);
  TORCH_CHECK((x.scalar_type() == torch::kBFloat16 || x.scalar_type() == torch::kFloat32) && K % 8 == 0 && K > 0 && aligned(x),
              "quant_rows_wide: aligned bf16 or fp32 rows, K % 8 == 0");
  auto q = torch::empty(x.sizes(), x.options().dtype(torch::kInt8));
  auto s = torch::empty(x.sizes().slice(0, x.dim() - 1), x.options().dtype(torch::kFloat32));
  if (x.numel())
    quant_rows_wide_launch(x.data_ptr(), x.scalar_type() == torch::kBFloat16, reinterpret_cast<signed char*>(q.data_ptr()), s.data_ptr<float>(),
                           x.numel() / K, (int)K, at::cuda::getCurrentCUDAStream());
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  return {q, s};
}

static int64_t group_words(const torch::Tensor& t) {
  const int64_t bytes = t.numel() / std::max<int64_t>(1, t.size(0)) * t.element_size();
  TORCH_CHECK(aligned(t) && bytes % 16 == 0, "groups: 16-byte groups");
  return bytes / 16;
}
// src (E, ...) -> (n, ...): the groups named by idx
torch::Tensor groups_take(torch::Tensor src, torch::Tensor idx) {
  const c10::cuda::CUDAGuard guard(src.device());
  auto shape = src.sizes().vec();
  shape[0] = idx.numel();
  auto out = torch::empty(shape, src.options());
  groups_take_launch(src.data_ptr(), i64(idx), out.data_ptr(), (int)idx.numel(), group_words(src), at::cuda::getCurrentCUDAStream());
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  return out;
}
// a (na, ...), b (nb, ...) -> (na + nb, ...) with a[j] at ia[j], b[j] at ib[j]; the lists together name every group once
torch::Tensor groups_put(torch::Tensor a, torch::Tensor ia, torch::Tensor b, torch::Tensor ib) {
  const c10::cuda::CUDAGuard guard(a.device());
  TORCH_CHECK(a.scalar_type() == b.scalar_type() && a.sizes().slice(1) == b.sizes().slice(1) && a.size(0) == ia.numel() && b.size(0) == ib.numel() &&
              a.size(0) > 0 && group_words(a) == group_words(b), "groups_put: two lists of equal groups");
  auto shape = a.sizes().vec();
  shape[0] = ia.numel() + ib.numel();
  auto out = torch::empty(shape, a.options());
  groups_put_launch(a.data_ptr(), i64(ia), (int)ia.numel(), b.data_ptr(), i64(ib), (int)ib.numel(), out.data_ptr(), group_words(a),
                    at::cuda::getCurrentCUDAStream());
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  return out;
}

}  // namespace mb
