// Torch side of the attention kernels (attn_fwd.cu, attn_bwd.cu): checks, outputs and workspaces.
#include <torch/extension.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>

#include <mutex>

#include "attn_api.h"

namespace mb {

// One status word per device and direction (forward, backward): a bounded wait that ran out leaves its code there.
static int* attn_word(int device, int which) {
  static int* words[16][2] = {};
  static std::mutex mu;
  TORCH_CHECK(device >= 0 && device < 16, "device index out of range");
  std::lock_guard<std::mutex> lock(mu);
  int*& w = words[device][which];
  if (!w) {
    TORCH_CHECK(cudaMalloc(&w, sizeof(int)) == cudaSuccess, "status word alloc failed");
    cudaMemset(w, 0, sizeof(int));
  }
  return w;
}
static int64_t read_word(int64_t device, int which) {        // device -1: the current one
  c10::cuda::OptionalCUDAGuard guard;
  if (device >= 0) guard.set_index((c10::DeviceIndex)device);
  int dev = 0;
  cudaGetDevice(&dev);
  int v = 0;
  const int z = 0;
  cudaMemcpy(&v, attn_word(dev, which), sizeof(int), cudaMemcpyDeviceToHost);
  if (v) cudaMemcpy(attn_word(dev, which), &z, sizeof(int), cudaMemcpyHostToDevice);
  return v;
}
int64_t attn_status_read(int64_t device) { return read_word(device, 0); }
int64_t attn_bwd_status_read(int64_t device) { return read_word(device, 1); }

// t (B, H, T, 64) contiguous
static AttnView view_bhtd(const torch::Tensor& t) { return {t.data_ptr(), t.stride(0), t.stride(2), t.stride(1)}; }
// slot `s` of a packed (B, T, n, H, 64) array
static AttnView view_packed(const torch::Tensor& t, int64_t s) {
  return {static_cast<char*>(t.data_ptr()) + s * t.stride(2) * 2, t.stride(0), t.stride(1), t.stride(3)};
}
// o (B, T, H, 64) contiguous
static AttnView view_bthd(const torch::Tensor& t) { return {t.data_ptr(), t.stride(0), t.stride(1), t.stride(2)}; }

static AttnArgs common_args(const torch::Tensor& like, int64_t B, int64_t H, int64_t T, int64_t window, double scale, int which) {
  AttnArgs a{};
  a.B = (int)B; a.H = (int)H; a.T = (int)T; a.window = (int)window; a.scale = (float)scale;
  a.status = attn_word(like.device().index(), which);
  a.stream = at::cuda::getCurrentCUDAStream();
  return a;
}
static void set_tables(AttnArgs& a, const torch::Tensor& cos, const torch::Tensor& sin, bool half) {
  TORCH_CHECK(cos.is_contiguous() && sin.is_contiguous() && cos.scalar_type() == torch::kFloat32 && cos.size(0) >= a.T &&
              cos.size(1) == 32 && sin.sizes() == cos.sizes(), "attention: cos/sin tables (T, 32) fp32");
  a.cos = cos.data_ptr<float>(); a.sin = sin.data_ptr<float>(); a.rope_half = half ? 1 : 0;
}
static void run_fwd(const AttnArgs& a) {
  if (const char* e = attn_fwd_launch(a)) TORCH_CHECK(false, e);
  C10_CUDA_KERNEL_LAUNCH_CHECK();
}
static void run_bwd(AttnArgs& a, const torch::Tensor& like) {
  auto f = like.options().dtype(torch::kFloat32);
  auto stats = torch::empty({(int64_t)attn_stats_floats(a.B, a.H, a.T)}, f);
  a.stats = stats.data_ptr<float>();
  if (const char* e = attn_bwd_launch(a)) TORCH_CHECK(false, e);
  C10_CUDA_KERNEL_LAUNCH_CHECK();
}

// q, k, v: (B, H, T, 64) bf16 contiguous (RoPE already applied).  Returns o (B, H, T, 64) bf16 and lse (B, H, T) fp32.
std::vector<torch::Tensor> attn_fwd_tc(torch::Tensor q, torch::Tensor k, torch::Tensor v, int64_t window, double scale) {
  const c10::cuda::CUDAGuard guard(q.device());
  TORCH_CHECK(q.dim() == 4 && q.size(3) == 64 && q.scalar_type() == torch::kBFloat16 && q.is_contiguous() &&
              k.is_contiguous() && v.is_contiguous() && k.sizes() == q.sizes() && v.sizes() == q.sizes() &&
              k.scalar_type() == torch::kBFloat16 && v.scalar_type() == torch::kBFloat16,
              "attn_fwd_tc: q, k, v (B, H, T, 64) bf16 contiguous");
  const int64_t B = q.size(0), H = q.size(1), T = q.size(2);
  auto o = torch::empty_like(q);
  auto lse = torch::empty({B, H, T}, q.options().dtype(torch::kFloat32));
  if (B * H * T == 0) return {o, lse};
  AttnArgs a = common_args(q, B, H, T, window, scale, 0);
  a.q = view_bhtd(q); a.k = view_bhtd(k); a.v = view_bhtd(v); a.o = view_bhtd(o);
  a.lse = lse.data_ptr<float>();
  run_fwd(a);
  return {o, lse};
}

// q, k, v, o, dout: (B, H, T, 64) bf16 contiguous; lse (B, H, T) fp32.  Returns dq, dk, dv (bf16).
std::vector<torch::Tensor> attn_bwd_tc(torch::Tensor q, torch::Tensor k, torch::Tensor v, torch::Tensor o, torch::Tensor dout,
                                       torch::Tensor lse, int64_t window, double scale) {
  const c10::cuda::CUDAGuard guard(q.device());
  for (const torch::Tensor& t : {q, k, v, o, dout})
    TORCH_CHECK(t.dim() == 4 && t.size(3) == 64 && t.scalar_type() == torch::kBFloat16 && t.is_contiguous() && t.sizes() == q.sizes(),
                "attn_bwd_tc: q, k, v, o, dout (B, H, T, 64) bf16 contiguous");
  const int64_t B = q.size(0), H = q.size(1), T = q.size(2);
  TORCH_CHECK(lse.is_contiguous() && lse.scalar_type() == torch::kFloat32 && lse.numel() == B * H * T, "attn_bwd_tc: lse fp32 contiguous");
  auto dq = torch::empty_like(q), dk = torch::empty_like(q), dv = torch::empty_like(q);
  if (B * H * T == 0) return {dq, dk, dv};
  AttnArgs a = common_args(q, B, H, T, window, scale, 1);
  a.q = view_bhtd(q); a.k = view_bhtd(k); a.v = view_bhtd(v); a.o = view_bhtd(o); a.dout = view_bhtd(dout);
  a.dq = view_bhtd(dq); a.dk = view_bhtd(dk); a.dv = view_bhtd(dv);
  a.lse = lse.data_ptr<float>();
  run_bwd(a, q);
  return {dq, dk, dv};
}

static void check_qkv(const torch::Tensor& qkv) {
  TORCH_CHECK(qkv.dim() == 5 && qkv.size(2) == 3 && qkv.size(4) == 64 && qkv.is_contiguous() && qkv.scalar_type() == torch::kBFloat16 &&
              (reinterpret_cast<uintptr_t>(qkv.data_ptr()) & 15) == 0, "attn_qkv: (B, T, 3, H, 64) bf16 contiguous");
}

// The attention of a light layer on packed projections: qkv (B, T, 3, H, 64) -> o (B, T, H, 64), lse (B, H, T) and, with
// `keep`, the packed array with q and k rotated, all that the backward pass reads of them.  `in_place`: qkv is the caller's own
// and is rotated where it lies.
std::vector<torch::Tensor> attn_qkv_fwd(torch::Tensor qkv, torch::Tensor cos, torch::Tensor sin, bool half, int64_t window, bool keep, bool in_place) {
  const c10::cuda::CUDAGuard guard(qkv.device());
  check_qkv(qkv);
  const int64_t B = qkv.size(0), T = qkv.size(1), H = qkv.size(3), slots = keep || in_place ? 3 : 2;
  auto rot = in_place ? qkv : torch::empty({B, T, slots, H, 64}, qkv.options());
  auto o = torch::empty({B, T, H, 64}, qkv.options());
  auto lse = torch::empty({B, H, T}, qkv.options().dtype(torch::kFloat32));
  if (B * H * T == 0) return {o, lse, rot};
  AttnArgs a = common_args(qkv, B, H, T, window, 0.125, 0);
  set_tables(a, cos, sin, half);
  rope_qk2_launch(qkv.data_ptr(), rot.data_ptr(), a.cos, a.sin, a.B, a.T, a.H, a.rope_half, (int)slots, a.stream);
  a.q = view_packed(rot, 0); a.k = view_packed(rot, 1); a.v = slots == 3 ? view_packed(rot, 2) : view_packed(qkv, 2); a.o = view_bthd(o);
  a.lse = lse.data_ptr<float>();
  run_fwd(a);
  return {o, lse, rot};
}

// dout (B, T, H, 64) contiguous -> gradient of the packed projections (B, T, 3, H, 64); qkv with q and k rotated
torch::Tensor attn_qkv_bwd(torch::Tensor dout, torch::Tensor o, torch::Tensor lse, torch::Tensor qkv, torch::Tensor cos, torch::Tensor sin, bool half,
                           int64_t window) {
  const c10::cuda::CUDAGuard guard(qkv.device());
  check_qkv(qkv);
  const int64_t B = qkv.size(0), T = qkv.size(1), H = qkv.size(3);
  TORCH_CHECK(dout.is_contiguous() && dout.scalar_type() == torch::kBFloat16 && dout.numel() == B * T * H * 64 &&
              (reinterpret_cast<uintptr_t>(dout.data_ptr()) & 15) == 0, "attn_qkv_bwd: dout (B, T, H, 64) bf16 contiguous");
  auto dqkv = torch::empty_like(qkv);
  if (B * H * T == 0) return dqkv;
  AttnArgs a = common_args(qkv, B, H, T, window, 0.125, 1);
  set_tables(a, cos, sin, half);
  a.q = view_packed(qkv, 0); a.k = view_packed(qkv, 1); a.v = view_packed(qkv, 2); a.o = view_bthd(o);
  a.dout = {dout.data_ptr(), T * H * 64, H * 64, 64};
  a.dq = view_packed(dqkv, 0); a.dk = view_packed(dqkv, 1); a.dv = view_packed(dqkv, 2);
  a.lse = lse.data_ptr<float>();
  run_bwd(a, qkv);
  return dqkv;
}

}  // namespace mb
