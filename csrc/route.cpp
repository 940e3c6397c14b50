// Torch side of the fused MoE router (route.cu).
#include <torch/extension.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>

#include "route_api.h"

namespace mb {

static void fill_inputs(RouteArgs& a, const torch::Tensor& x, const torch::Tensor& w, const torch::Tensor& real, const torch::Tensor& k_tok,
                        int64_t k, int64_t C) {
  TORCH_CHECK(x.dim() == 2 && x.is_contiguous() && x.scalar_type() == torch::kBFloat16 && x.size(1) % 8 == 0 &&
              (reinterpret_cast<uintptr_t>(x.data_ptr()) & 15) == 0, "route: x (N, d) bf16, d % 8 == 0");
  TORCH_CHECK(w.dim() == 2 && w.is_contiguous() && w.scalar_type() == torch::kFloat32 && w.size(1) == x.size(1) &&
              (reinterpret_cast<uintptr_t>(w.data_ptr()) & 15) == 0, "route: router weight (E, d) fp32");
  a.N = x.size(0); a.d = x.size(1); a.E = w.size(0); a.k = (int)k; a.C = (int)C;
  TORCH_CHECK(a.E >= 1 && a.E <= ROUTE_E && k >= 1 && k <= ROUTE_K && k <= a.E && C >= 1, "route: E <= 128, k <= 8");
  TORCH_CHECK(real.scalar_type() == torch::kBool && real.is_contiguous() && real.numel() == a.N && k_tok.scalar_type() == torch::kInt64 &&
              k_tok.is_contiguous() && k_tok.numel() == a.N, "route: real bool, k_tok int64");
  a.x = x.data_ptr(); a.w = w.data_ptr<float>(); a.real = real.data_ptr<bool>();
  a.k_tok = reinterpret_cast<const long long*>(k_tok.data_ptr<int64_t>());
  a.stream = at::cuda::getCurrentCUDAStream();
}
static long long* i64(const torch::Tensor& t) { return reinterpret_cast<long long*>(t.data_ptr<int64_t>()); }

// -> weights (N,k), place weights (E C), aux, probs (N,E), table (E C), places (N,k), dropped, counts (E), chosen experts (N,k), d aux / d psum (E)
std::vector<torch::Tensor> route_fwd(torch::Tensor x, torch::Tensor w, torch::Tensor real, torch::Tensor k_tok, int64_t k, int64_t C) {
  const c10::cuda::CUDAGuard guard(x.device());
  RouteArgs a{};
  fill_inputs(a, x, w, real, k_tok, k, C);
  const int64_t N = a.N, E = a.E;
  auto f = w.options(), l = k_tok.options(), i = x.options().dtype(torch::kInt32);
  auto wt = torch::empty({N, k}, f), wtab = torch::empty({E * C}, f), probs = torch::empty({N, E}, f), aux = torch::empty({}, f),
       dropped = torch::empty({}, f), aux_grad = torch::empty({E}, f);
  auto table = torch::empty({E * C}, l), flat_idx = torch::empty({N, k}, l), top_e = torch::empty({N, k}, l);
  auto counts = torch::empty({E}, i);
  const int64_t nb = route_blocks(a.N);
  TORCH_CHECK(N > 0, "route: no tokens");
  auto work_i = torch::empty({(nb + 1) * (E + 1)}, i), psum = torch::empty({(nb + 1) * E}, f);
  a.wt = wt.data_ptr<float>(); a.wtab = wtab.data_ptr<float>(); a.probs = probs.data_ptr<float>(); a.aux = aux.data_ptr<float>();
  a.dropped = dropped.data_ptr<float>(); a.aux_grad = aux_grad.data_ptr<float>(); a.table = i64(table); a.flat_idx = i64(flat_idx);
  a.top_e = i64(top_e); a.counts = counts.data_ptr<int>(); a.hist = work_i.data_ptr<int>(); a.n_real = a.hist + nb * E; a.psum = psum.data_ptr<float>();
  if (nb > ROUTE_SCAN) { a.total = a.n_real + nb; a.ps = a.psum + nb * E; }
  route_fwd_launch(a);
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  return {wt, wtab, aux, probs, table, flat_idx, dropped, counts, top_e, aux_grad};
}

static const float* grad_ptr(const c10::optional<torch::Tensor>& t, int64_t numel) {
  if (!t.has_value() || !t->defined()) return nullptr;
  TORCH_CHECK(t->is_contiguous() && t->scalar_type() == torch::kFloat32 && t->numel() == numel, "route: gradient fp32 contiguous");
  return t->data_ptr<float>();
}

std::vector<torch::Tensor> route_bwd(torch::Tensor x, torch::Tensor w, torch::Tensor real, torch::Tensor k_tok, torch::Tensor probs,
                                     torch::Tensor top_e, torch::Tensor flat_idx, torch::Tensor aux_grad, int64_t C,
                                     c10::optional<torch::Tensor> d_wt, c10::optional<torch::Tensor> d_wtab,
                                     c10::optional<torch::Tensor> d_aux, c10::optional<torch::Tensor> d_probs) {
  const c10::cuda::CUDAGuard guard(x.device());
  RouteArgs a{};
  fill_inputs(a, x, w, real, k_tok, top_e.size(1), C);
  auto dx = torch::empty_like(x), dw = torch::empty_like(w), dl = torch::empty_like(probs);
  a.probs = probs.data_ptr<float>(); a.top_e = i64(top_e); a.flat_idx = i64(flat_idx); a.aux_grad = aux_grad.data_ptr<float>();
  a.d_wt = grad_ptr(d_wt, (int64_t)a.N * a.k); a.d_wtab = grad_ptr(d_wtab, (int64_t)a.E * C); a.d_aux = grad_ptr(d_aux, 1);
  a.d_probs = grad_ptr(d_probs, probs.numel());
  a.dw_runs = route_dw_runs(a.N, a.d, a.E, a.dw_run);
  auto part = torch::empty({a.dw_runs, a.E, a.d}, dw.options());
  a.dw_part = part.data_ptr<float>();
  a.dl = dl.data_ptr<float>(); a.dx = dx.data_ptr(); a.dw = dw.data_ptr<float>();
  route_bwd_launch(a);
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  return {dx, dw};
}

}  // namespace mb
