// Torch side of the slot kernels (gather.cu).
#include <torch/extension.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>

#include "gather_api.h"

namespace mb {

static void check_rows(const torch::Tensor& t, int64_t d, const char* what) {
  TORCH_CHECK(t.is_contiguous() && t.scalar_type() == torch::kBFloat16 && t.size(-1) == d && d > 0 && d % 8 == 0 &&
              (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0, what, ": contiguous 16-byte aligned bf16 rows, d % 8 == 0");
}
static const long long* i64(const torch::Tensor& t) {
  TORCH_CHECK(t.is_contiguous() && t.scalar_type() == torch::kInt64, "slot index: contiguous int64");
  return reinterpret_cast<const long long*>(t.data_ptr<int64_t>());
}
static const float* f32(const torch::Tensor& t, int64_t n) {
  TORCH_CHECK(t.is_contiguous() && t.scalar_type() == torch::kFloat32 && t.numel() == n, "slot weight: contiguous fp32");
  return t.data_ptr<float>();
}

torch::Tensor rows_gather(torch::Tensor src, torch::Tensor table) {
  const c10::cuda::CUDAGuard guard(src.device());
  const int64_t d = src.size(-1), S = table.numel();
  check_rows(src, d, "rows_gather");
  auto out = torch::empty({S, d}, src.options());
  if (S) rows_gather_launch(src.data_ptr(), i64(table), out.data_ptr(), S, (int)d, src.numel() / d, at::cuda::getCurrentCUDAStream());
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  return out;
}

torch::Tensor rows_gather_sum(torch::Tensor src, torch::Tensor idx, c10::optional<torch::Tensor> w) {
  const c10::cuda::CUDAGuard guard(src.device());
  const int64_t d = src.size(-1), N = idx.size(0);
  check_rows(src, d, "rows_gather_sum");
  const int64_t S = src.numel() / d;
  auto out = torch::empty({N, d}, src.options());
  if (N) rows_gather_sum_launch(src.data_ptr(), i64(idx), w.has_value() && w->defined() ? f32(*w, S) : nullptr, out.data_ptr(), N, (int)idx.size(1),
                                (int)d, S, at::cuda::getCurrentCUDAStream());
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  return out;
}

// -> dye (S, d), dw (S)
std::vector<torch::Tensor> combine_bwd(torch::Tensor go, torch::Tensor table, torch::Tensor w, torch::Tensor ye) {
  const c10::cuda::CUDAGuard guard(go.device());
  const int64_t d = go.size(-1), S = table.numel();
  check_rows(go, d, "combine_bwd");
  check_rows(ye, d, "combine_bwd");
  TORCH_CHECK(ye.numel() == S * d, "combine_bwd: one row of ye per place");
  auto dye = torch::empty_like(ye);
  auto dw = torch::empty({S}, w.options());
  if (S) combine_bwd_launch(go.data_ptr(), i64(table), f32(w, S), ye.data_ptr(), dye.data_ptr(), dw.data_ptr<float>(), S, (int)d, go.numel() / d,
                            at::cuda::getCurrentCUDAStream());
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  return {dye, dw};
}

// buf (E) fp32 <- 0.9 buf + 0.1 mean over the places of the gradient's norm; g (E, C, d)
void err_probe(torch::Tensor g, torch::Tensor buf) {
  const c10::cuda::CUDAGuard guard(g.device());
  TORCH_CHECK(g.dim() == 3, "err_probe: (E, C, d)");
  check_rows(g, g.size(2), "err_probe");
  const int E = g.size(0), C = g.size(1);
  f32(buf, E);
  auto part = torch::empty({(int64_t)err_probe_parts(C) * E}, buf.options());
  if (E && C) err_probe_launch(g.data_ptr(), buf.data_ptr<float>(), part.data_ptr<float>(), E, C, (int)g.size(2), at::cuda::getCurrentCUDAStream());
  C10_CUDA_KERNEL_LAUNCH_CHECK();
}

}  // namespace mb
