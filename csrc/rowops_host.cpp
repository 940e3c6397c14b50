// Torch side of rmsnorm.cu and ce_rows.cu.
#include <torch/extension.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>

#include "rowops_api.h"

namespace mb {

static bool on16(const torch::Tensor& t) { return (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0; }
// the norm weight as the kernels read it: d consecutive fp32 values from a 16-byte boundary on
static torch::Tensor norm_weight(const torch::Tensor& w, int64_t d) {
  TORCH_CHECK(w.numel() == d, "rmsnorm: one weight per column");
  const torch::Tensor f = w.to(torch::kFloat32).contiguous();
  return on16(f) ? f : f.clone();
}
static bool is_bf16(const torch::Tensor& t) { return t.scalar_type() == torch::kBFloat16; }
static bool float_or_bf16(const torch::Tensor& t) { return is_bf16(t) || t.scalar_type() == torch::kFloat32; }

// h = x (fp32) + y (bf16); n = rmsnorm(h) * w in bf16: the residual add and the next normalisation in one pass.
std::vector<torch::Tensor> add_rmsnorm_fwd(torch::Tensor x, torch::Tensor y, torch::Tensor w, double eps) {
  const c10::cuda::CUDAGuard guard(x.device());
  TORCH_CHECK(x.dim() == 2 && x.is_contiguous() && y.is_contiguous() && x.scalar_type() == torch::kFloat32 &&
              is_bf16(y) && x.numel() == y.numel() && x.size(1) % 4 == 0 && on16(x) && on16(y), "add_rmsnorm: fp32 + bf16, 16-byte aligned");
  const int n = x.size(0), d = x.size(1);
  const torch::Tensor wf = norm_weight(w, d);
  auto h = torch::empty_like(x);
  auto nn = torch::empty({n, d}, x.options().dtype(torch::kBFloat16));
  auto rstd = torch::empty({n}, x.options());
  NormArgs a{};
  a.x = x.data_ptr(); a.y = y.data_ptr(); a.y_bf16 = 1; a.w = wf.data_ptr<float>(); a.rstd = rstd.data_ptr<float>();
  a.out = nn.data_ptr(); a.out_bf16 = 1; a.sum = h.data_ptr<float>(); a.n = n; a.d = d; a.eps = (float)eps;
  a.stream = at::cuda::getCurrentCUDAStream();
  rmsnorm_fwd_launch(a);
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  return {h, nn, rstd};
}

std::vector<torch::Tensor> rmsnorm_fwd(torch::Tensor x, torch::Tensor w, double eps, bool out_bf16) {
  const c10::cuda::CUDAGuard guard(x.device());
  TORCH_CHECK(x.dim() == 2 && x.is_contiguous() && x.size(1) % 4 == 0 && on16(x), "rmsnorm: (N,d) contiguous and 16-byte aligned, d % 4 == 0");
  const int n = x.size(0), d = x.size(1);
  const torch::Tensor wf = norm_weight(w, d);
  auto y = torch::empty({n, d}, x.options().dtype(out_bf16 ? torch::kBFloat16 : torch::kFloat32));
  auto rstd = torch::empty({n}, x.options().dtype(torch::kFloat32));
  if (n == 0) return {y, rstd};
  NormArgs a{};
  a.x = x.data_ptr(); a.x_bf16 = is_bf16(x); a.w = wf.data_ptr<float>(); a.rstd = rstd.data_ptr<float>();
  a.out = y.data_ptr(); a.out_bf16 = out_bf16; a.n = n; a.d = d; a.eps = (float)eps;
  a.stream = at::cuda::getCurrentCUDAStream();
  rmsnorm_fwd_launch(a);
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  return {y, rstd};
}

// dy, x (N,d); optional `add` (fp32): a gradient that reached x by another path is summed in the same pass; `want_lo`: dx is
// also returned in bf16 (the branch that produced part of x wants it).
std::vector<torch::Tensor> rmsnorm_bwd(torch::Tensor dy, torch::Tensor x, torch::Tensor w, torch::Tensor rstd,
                                       c10::optional<torch::Tensor> add_, bool want_lo) {
  const c10::cuda::CUDAGuard guard(x.device());
  NormArgs a{};
  if (add_.has_value() && add_->defined()) {
    TORCH_CHECK(add_->scalar_type() == torch::kFloat32 && add_->is_contiguous() && add_->numel() == x.numel() && on16(*add_), "rmsnorm_bwd: add");
    a.add = add_->data_ptr<float>();
  }
  const int n = x.size(0), d = x.size(1);
  TORCH_CHECK(d <= 8 * 4 * 256 && d % 4 == 0, "rmsnorm_bwd: d <= 8192");
  TORCH_CHECK(float_or_bf16(x) && float_or_bf16(dy) && x.is_contiguous() && dy.is_contiguous() && dy.numel() == x.numel() && on16(x) && on16(dy),
              "rmsnorm_bwd: fp32 or bf16 rows, contiguous and 16-byte aligned");
  const torch::Tensor wf = norm_weight(w, d);
  auto dx = torch::empty_like(x);
  torch::Tensor lo = want_lo ? torch::empty({n, d}, x.options().dtype(torch::kBFloat16)) : torch::Tensor();
  auto f = x.options().dtype(torch::kFloat32);
  if (n == 0) return {dx, torch::zeros({d}, f), lo};
  auto dw = torch::empty({d}, f);
  auto part = torch::empty({rmsnorm_parts(n, d), d}, f);
  a.x = x.data_ptr(); a.x_bf16 = is_bf16(x); a.y = dy.data_ptr(); a.y_bf16 = is_bf16(dy);
  a.w = wf.data_ptr<float>(); a.rstd = rstd.data_ptr<float>(); a.out = dx.data_ptr();
  a.lo = want_lo ? lo.data_ptr() : nullptr;
  a.dw = dw.data_ptr<float>(); a.dw_part = part.data_ptr<float>(); a.n = n; a.d = d;
  a.stream = at::cuda::getCurrentCUDAStream();
  rmsnorm_bwd_launch(a);
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  return {dx, dw, lo};
}

void ce_rows(torch::Tensor logits, torch::Tensor y, torch::Tensor loss, c10::optional<torch::Tensor> gate,
             c10::optional<torch::Tensor> hit, c10::optional<torch::Tensor> dg) {
  const c10::cuda::CUDAGuard guard(logits.device());
  TORCH_CHECK(logits.dim() == 2 && logits.stride(1) == 1 && is_bf16(logits), "ce_rows: bf16 (n,V)");
  TORCH_CHECK(y.scalar_type() == torch::kInt64 && y.is_contiguous() && loss.is_contiguous(), "ce_rows: y int64");
  TORCH_CHECK(logits.stride(0) % 8 == 0 && (reinterpret_cast<uintptr_t>(logits.data_ptr()) & 15) == 0, "ce_rows: row alignment");
  const int n = logits.size(0), V = logits.size(1);
  if (!n) return;
  const bool mix = gate.has_value() && gate->defined();
  ce_rows_launch(logits.data_ptr(), reinterpret_cast<const long long*>(y.data_ptr<int64_t>()), loss.data_ptr<float>(),
                 mix ? gate->data_ptr<float>() : nullptr, mix ? hit->data_ptr<float>() : nullptr, mix ? dg->data_ptr<float>() : nullptr,
                 logits.stride(0), n, V, at::cuda::getCurrentCUDAStream());
  C10_CUDA_KERNEL_LAUNCH_CHECK();
}

// x * scale (one fp32 element on the device) in bf16 or fp32
torch::Tensor scale_by(torch::Tensor x, torch::Tensor scale, bool out_bf16) {
  const c10::cuda::CUDAGuard guard(x.device());
  TORCH_CHECK(x.is_contiguous() && float_or_bf16(x) && x.numel() % 4 == 0 && (reinterpret_cast<uintptr_t>(x.data_ptr()) & 15) == 0 &&
              scale.scalar_type() == torch::kFloat32 && scale.numel() == 1 && scale.device() == x.device(), "scale_by: bf16 or fp32 by one fp32 element");
  auto out = torch::empty(x.sizes(), x.options().dtype(out_bf16 ? torch::kBFloat16 : torch::kFloat32));
  scale_launch(x.data_ptr(), is_bf16(x), scale.data_ptr<float>(), out.data_ptr(), out_bf16, x.numel(), at::cuda::getCurrentCUDAStream());
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  return out;
}

}  // namespace mb
