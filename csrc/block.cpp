// The two halves of a light layer as one call each way: the launches follow one another without the interpreter and the
// autograd engine in between (a layer of the smallest model spent 0.95 ms on the host for 0.25 ms of kernels).
//   attention half:    h = x (+ pending), n = rmsnorm(h), qkv = n Wqkv^T, o = attention(qkv), a = o Wo^T
//   feed-forward half: x2 = h + a, n2 = rmsnorm(x2), y = act(n2 Wup^T) Wdown^T (, out = x2 + y)
// Backward sums the gradient that reaches the residual stream past the half inside the norm's own pass.  Weight gradients leave
// in fp32 (`grad_f32`: what an fp32 weight's .grad wants) or in bf16 (what the optimizer takes inside backward: `offer(i, gradient)`,
// i counting the weights in argument order, is called for each as soon as it and the last product that reads the weight are
// enqueued, so that its exchange or step runs under what follows).
#include <torch/extension.h>
#include <c10/cuda/CUDAGuard.h>

namespace mb {

torch::Tensor gemm(torch::Tensor a, torch::Tensor b, c10::optional<torch::Tensor> out, c10::optional<torch::Tensor> out2,
                   c10::optional<torch::Tensor> aux, bool a_mn, bool b_mn, bool accumulate, int64_t epi, bool out_f32,
                   int64_t groups, c10::optional<torch::Tensor> counts, int64_t count_mode);
std::vector<torch::Tensor> rmsnorm_fwd(torch::Tensor x, torch::Tensor w, double eps, bool out_bf16);
std::vector<torch::Tensor> rmsnorm_bwd(torch::Tensor dy, torch::Tensor x, torch::Tensor w, torch::Tensor rstd,
                                       c10::optional<torch::Tensor> add, bool want_lo);
std::vector<torch::Tensor> add_rmsnorm_fwd(torch::Tensor x, torch::Tensor y, torch::Tensor w, double eps);
torch::Tensor resid_add(torch::Tensor x, torch::Tensor y);
std::vector<torch::Tensor> attn_qkv_fwd(torch::Tensor qkv, torch::Tensor cos, torch::Tensor sin, bool half, int64_t window, bool keep, bool in_place);
torch::Tensor attn_qkv_bwd(torch::Tensor dout, torch::Tensor o, torch::Tensor lse, torch::Tensor qkv, torch::Tensor cos, torch::Tensor sin, bool half,
                           int64_t window);

typedef c10::optional<torch::Tensor> Opt;
static bool has(const Opt& t) { return t.has_value() && t->defined(); }
// hands a gradient to `offer`, which takes it, or returns it
static torch::Tensor handed(const pybind11::object& offer, int i, torch::Tensor g) {
  if (offer.is_none()) return g;
  offer(i, g);
  return torch::Tensor();
}
enum { EPI_NONE = 0, EPI_RELU2 = 1, EPI_DRELU2 = 2, EPI_SWIGLU = 3, EPI_DSWIGLU = 5 };

static torch::Tensor project(const torch::Tensor& a, const torch::Tensor& b) {                     // a b^T
  return gemm(a, b, c10::nullopt, c10::nullopt, c10::nullopt, false, false, false, EPI_NONE, false, 1, c10::nullopt, 0);
}
static torch::Tensor dgrad(const torch::Tensor& dy, const torch::Tensor& w) {                 // dy W
  return gemm(dy, w, c10::nullopt, c10::nullopt, c10::nullopt, false, true, false, EPI_NONE, false, 1, c10::nullopt, 0);
}
static torch::Tensor wgrad(const torch::Tensor& dy, const torch::Tensor& x, bool f32) {       // dy^T x
  return gemm(dy, x, c10::nullopt, c10::nullopt, c10::nullopt, true, true, false, EPI_NONE, f32, 1, c10::nullopt, 0);
}
// (rows, width), contiguous and on a 16-byte boundary
static torch::Tensor rows(const torch::Tensor& t) {
  torch::Tensor r = t.reshape({-1, t.size(-1)}).contiguous();
  return (reinterpret_cast<uintptr_t>(r.data_ptr()) & 15) == 0 ? r : r.clone();
}

// x (B,T,d) fp32; pending (B,T,d) bf16 or none.  -> h (M,d), a (M,d) | n, rstd, qkv (q and k rotated), o, lse
std::vector<torch::Tensor> attn_half_fwd(torch::Tensor x, Opt pending, torch::Tensor nw, double eps, torch::Tensor wqkv, torch::Tensor wo,
                                         torch::Tensor cos, torch::Tensor sin, bool half, int64_t window) {
  const c10::cuda::CUDAGuard guard(x.device());
  TORCH_CHECK(x.dim() == 3 && x.scalar_type() == torch::kFloat32, "attn_half: x (B,T,d) fp32");
  const int64_t B = x.size(0), T = x.size(1), d = x.size(2);
  torch::Tensor h, n, rstd;
  if (has(pending)) {
    auto r = add_rmsnorm_fwd(rows(x), rows(*pending), nw, eps);
    h = r[0]; n = r[1]; rstd = r[2];
  } else {
    h = rows(x);
    auto r = rmsnorm_fwd(h, nw, eps, true);
    n = r[0]; rstd = r[1];
  }
  auto qkv = project(n, wqkv).view({B, T, 3, d / 64, 64});
  auto at = attn_qkv_fwd(qkv, cos, sin, half, window, true, true);
  auto a = project(at[0].view({B * T, d}), wo);
  return {h, a, n, rstd, qkv, at[0], at[1]};
}

// da (B,T,d) bf16; dh (B,T,d) fp32 or none.  -> dx (M,d), dx in bf16 (or undefined), d nw, d wqkv, d wo
std::vector<torch::Tensor> attn_half_bwd(torch::Tensor da, Opt dh, torch::Tensor h, torch::Tensor n, torch::Tensor rstd, torch::Tensor qkv,
                                         torch::Tensor o, torch::Tensor lse, torch::Tensor nw, torch::Tensor wqkv,
                                         torch::Tensor wo, torch::Tensor cos, torch::Tensor sin, bool half, int64_t window, bool want_lo,
                                         bool grad_f32, pybind11::object offer) {
  const c10::cuda::CUDAGuard guard(da.device());
  const int64_t M = h.size(0), d = h.size(1);
  const torch::Tensor g = rows(da);
  auto dout = dgrad(g, wo);
  auto dwo = handed(offer, 1, wgrad(g, o.view({M, d}), grad_f32));
  auto dqkv = attn_qkv_bwd(dout, o, lse, qkv, cos, sin, half, window).view({M, 3 * d});
  auto dn = dgrad(dqkv, wqkv);
  auto dwqkv = handed(offer, 0, wgrad(dqkv, n, grad_f32));
  auto r = rmsnorm_bwd(dn, h, nw, rstd, has(dh) ? Opt(rows(*dh)) : Opt(), want_lo);
  return {r[0], r[2], r[1], dwqkv, dwo};
}

// h (B,T,d) fp32, a (B,T,d) bf16.  -> x2, y (`add_out`: x2 + y instead) | x2, n, rstd, pre, hid
std::vector<torch::Tensor> ffn_half_fwd(torch::Tensor h, torch::Tensor a, torch::Tensor nw, double eps, torch::Tensor wup, torch::Tensor wdown,
                                        bool swiglu, bool add_out) {
  const c10::cuda::CUDAGuard guard(h.device());
  auto r = add_rmsnorm_fwd(rows(h), rows(a), nw, eps);
  const int64_t M = r[0].size(0), N = wup.size(0);
  auto pre = torch::empty({M, N}, r[1].options()), hid = torch::empty({M, swiglu ? N / 2 : N}, r[1].options());
  gemm(r[1], wup, hid, pre, c10::nullopt, false, false, false, swiglu ? EPI_SWIGLU : EPI_RELU2, false, 1, c10::nullopt, 0);
  auto y = project(hid, wdown);
  if (add_out) y = resid_add(r[0], y);
  return {r[0], y, r[1], r[2], pre, hid};
}

// dy (B,T,d) bf16 (or, with `add_out`, the fp32 gradient of x2 + y); dx2 (B,T,d) fp32 or none.  -> dh (M,d), da (M,d) bf16, d nw, d wup, d wdown
std::vector<torch::Tensor> ffn_half_bwd(torch::Tensor dy, Opt dx2, torch::Tensor x2, torch::Tensor n, torch::Tensor rstd, torch::Tensor pre,
                                        torch::Tensor hid, torch::Tensor nw, torch::Tensor wup, torch::Tensor wdown, bool swiglu, bool grad_f32,
                                        pybind11::object offer) {
  const c10::cuda::CUDAGuard guard(dy.device());
  torch::Tensor g = rows(dy);
  Opt through = has(dx2) ? Opt(rows(*dx2)) : Opt();
  if (g.scalar_type() == torch::kFloat32) {
    TORCH_CHECK(!has(through), "ffn_half: one gradient of the summed output");
    through = g;
    g = g.to(torch::kBFloat16);
  }
  auto dpre = gemm(g, wdown, c10::nullopt, c10::nullopt, pre, false, true, false, swiglu ? EPI_DSWIGLU : EPI_DRELU2, false, 1, c10::nullopt, 0);
  auto dwd = handed(offer, 1, wgrad(g, hid, grad_f32));
  auto dn = dgrad(dpre, wup);
  auto dwu = handed(offer, 0, wgrad(dpre, n, grad_f32));
  auto r = rmsnorm_bwd(dn, x2, nw, rstd, through, true);
  return {r[0], r[2], r[1], dwu, dwd};
}

}  // namespace mb
