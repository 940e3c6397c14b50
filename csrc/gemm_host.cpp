// Torch side of the tcgen05 GEMM (gemm_tc.cu): checks and outputs.
#include <torch/extension.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>

#include <atomic>

#include "gemm_api.h"

namespace mb {

// kernels that added the parts of cut contractions, since the library was loaded
static std::atomic<int64_t> sum_launches{0};
int64_t gemm_sum_launches() { return sum_launches.load(); }

// torch binding.  a: (G?, M, K) or MN-major (G?, K, M); b: (G?, N, K) or MN-major (G?, K, N).
torch::Tensor gemm(torch::Tensor a, torch::Tensor b, c10::optional<torch::Tensor> out_,
                   c10::optional<torch::Tensor> out2_, c10::optional<torch::Tensor> aux_, bool a_mn, bool b_mn,
                   bool accumulate, int64_t epi, bool out_f32, int64_t groups, c10::optional<torch::Tensor> counts_,
                   int64_t count_mode) {
  TORCH_CHECK(a.is_cuda() && b.is_cuda(), "gemm: CUDA tensors expected");
  TORCH_CHECK(a.scalar_type() == torch::kBFloat16 && b.scalar_type() == torch::kBFloat16, "gemm: bf16 operands");
  const c10::cuda::CUDAGuard guard(a.device());
  const int G = (int)groups;
  auto as3 = [&](torch::Tensor t) { return t.dim() == 2 ? t.unsqueeze(0) : t; };
  torch::Tensor A = as3(a), B = as3(b);
  TORCH_CHECK(A.dim() == 3 && B.dim() == 3 && A.size(0) == G && B.size(0) == G, "gemm: group dimension mismatch");
  TORCH_CHECK(A.stride(2) == 1 && B.stride(2) == 1, "gemm: innermost dimension must be contiguous");
  const int M = a_mn ? A.size(2) : A.size(1), K = a_mn ? A.size(1) : A.size(2);
  const int N = b_mn ? B.size(2) : B.size(1), Kb = b_mn ? B.size(1) : B.size(2);
  TORCH_CHECK(K == Kb, "gemm: K mismatch ", K, " vs ", Kb);
  const int Nout = epi == EPI_SWIGLU ? N / 2 : (epi == EPI_DSWIGLU ? 2 * N : N);
  torch::Tensor out;
  if (out_.has_value() && out_->defined()) {
    out = *out_;
  } else {
    auto opt = a.options().dtype(out_f32 ? torch::kFloat32 : torch::kBFloat16);
    out = (a.dim() == 2 && G == 1) ? torch::empty({M, Nout}, opt) : torch::empty({G, M, Nout}, opt);
  }
  TORCH_CHECK(out.scalar_type() == (out_f32 ? torch::kFloat32 : torch::kBFloat16), "gemm: out dtype");
  torch::Tensor O = as3(out);
  TORCH_CHECK(O.size(0) == G && O.size(1) == M && O.size(2) == Nout && O.stride(2) == 1, "gemm: out shape");
  GemmParams p{};
  p.M = M; p.N = N; p.K = K; p.G = G;
  p.out = O.data_ptr(); p.ldo = (int)O.stride(1); p.out_gs = G > 1 ? O.stride(0) : 0;
  p.epi = (int)epi; p.out_f32 = out_f32; p.accumulate = accumulate;
  TORCH_CHECK(!accumulate || out_f32, "gemm: accumulate needs an fp32 output");
  const int vec = out_f32 ? 4 : 8;
  TORCH_CHECK(p.ldo % vec == 0 && (reinterpret_cast<uintptr_t>(p.out) & 15) == 0 && (p.out_gs % vec) == 0,
              "gemm: output must allow 16-byte row stores");
  if (out2_.has_value() && out2_->defined()) {
    torch::Tensor O2 = as3(*out2_);
    TORCH_CHECK(O2.scalar_type() == torch::kBFloat16 && O2.stride(2) == 1 && O2.size(1) == M, "gemm: out2");
    p.out2 = O2.data_ptr(); p.ldo2 = (int)O2.stride(1); p.out2_gs = G > 1 ? O2.stride(0) : 0;
    TORCH_CHECK(p.ldo2 % 8 == 0 && (reinterpret_cast<uintptr_t>(p.out2) & 15) == 0, "gemm: out2 alignment");
  }
  TORCH_CHECK(epi != EPI_RELU2 || p.out2 != nullptr, "gemm: relu2 epilogue needs out2 for the pre-activation");
  if (aux_.has_value() && aux_->defined()) {
    if (epi == EPI_ROWSCALE) {
      TORCH_CHECK(aux_->scalar_type() == torch::kFloat32 && aux_->is_contiguous(), "gemm: row scale must be fp32");
      p.aux = aux_->data_ptr(); p.aux_gs = G > 1 ? M : 0;
    } else {
      torch::Tensor X = as3(*aux_);
      TORCH_CHECK(X.scalar_type() == torch::kBFloat16 && X.stride(2) == 1 && X.size(1) == M &&
                  X.size(2) == (epi == EPI_DSWIGLU ? 2 * N : N), "gemm: aux");
      p.aux = X.data_ptr(); p.ldaux = (int)X.stride(1); p.aux_gs = G > 1 ? X.stride(0) : 0;
      TORCH_CHECK(p.ldaux % 8 == 0 && (reinterpret_cast<uintptr_t>(p.aux) & 15) == 0, "gemm: aux alignment");
    }
  }
  TORCH_CHECK((epi != EPI_DRELU2 && epi != EPI_ROWSCALE && epi != EPI_DSWIGLU) || p.aux != nullptr, "gemm: epilogue needs aux");
  TORCH_CHECK(epi != EPI_DSWIGLU || (!out_f32 && N % 8 == 0 && M >= 256 && gemm_pair_on()),
              "gemm: the SwiGLU-backward epilogue writes bf16, needs a hidden width that is a multiple of 8 and the pair kernel (>= 256 rows)");
  if (counts_.has_value() && counts_->defined() && count_mode != 0) {
    TORCH_CHECK(counts_->is_cuda() && counts_->scalar_type() == torch::kInt32 && counts_->is_contiguous() &&
                counts_->numel() >= G, "gemm: counts must be a contiguous int32 CUDA tensor with one entry per group");
    TORCH_CHECK(count_mode == 1 || count_mode == 2, "gemm: count_mode 1 (rows) or 2 (contraction length)");
    p.counts = counts_->data_ptr<int>(); p.count_mode = (int)count_mode;
  }
  TORCH_CHECK(epi != EPI_SWIGLU || (!out_f32 && N % 16 == 0),
              "gemm: the SwiGLU epilogue writes bf16 and needs column halves of a multiple of 8 (16-byte TMA coordinates)");
  p.status = gemm_status_word(a.get_device());
  // few output tiles and a long contraction: split it.  Every part is kept in fp32 and they are added in a fixed order: the
  // same bits on every call.
  torch::Tensor parts;
  const cudaStream_t stream = at::cuda::getCurrentCUDAStream();
  if (p.epi == EPI_NONE && p.count_mode == 0 && N % 4 == 0) {
    int kb_split = 0;
    const int splits = gemm_splits(M, N, K, G, gemm_sm_count(), kb_split);
    if (splits > 1) {
      parts = torch::empty({splits, M, N}, a.options().dtype(torch::kFloat32));
      p.out = parts.data_ptr(); p.ldo = N; p.out_gs = (long long)M * N; p.out_f32 = 1; p.accumulate = 0;
      p.splits = splits; p.kb_split = kb_split;
    }
  }
  launch_gemm(A.data_ptr(), A.stride(1), G > 1 ? A.stride(0) : 0, a_mn, B.data_ptr(), B.stride(1), G > 1 ? B.stride(0) : 0,
              b_mn, p, stream, gemm_sm_count());
  if (parts.defined()) {
    sum_parts_launch(parts.data_ptr<float>(), p.splits, O.data_ptr(), out_f32, accumulate, M, N, (int)O.stride(1), stream);
    C10_CUDA_KERNEL_LAUNCH_CHECK();
    ++sum_launches;
  }
  return out;
}

// Segmented GEMM over peer buffers (expert parallelism without a separate all-to-all):
//   A rows of segment s come from `a_ptrs[s]`, a (a_groups, seg_M, K) bf16 buffer (a peer GPU's dispatch buffer);
//   group g of this launch reads A group `a_g_off + g`;
//   the result goes to `out_local` (G, n_seg*seg_M, N) or, when `out_ptrs` is given, rows of segment s go to
//   `out_ptrs[s]`, a (.., seg_M, N) buffer with row pitch `out_ld` and group pitch `out_gs` at group `out_g_off + g`.
torch::Tensor gemm_peer(std::vector<int64_t> a_ptrs, int64_t seg_M, int64_t K, int64_t a_groups, int64_t a_pitch,
                        int64_t a_gs, int64_t a_g_off, torch::Tensor b, bool b_mn, c10::optional<torch::Tensor> out_local,
                        std::vector<int64_t> out_ptrs, int64_t out_ld, int64_t out_gs, int64_t out_g_off,
                        c10::optional<torch::Tensor> out2_, c10::optional<torch::Tensor> aux_, int64_t epi, int64_t groups) {
  TORCH_CHECK(b.is_cuda() && b.scalar_type() == torch::kBFloat16, "gemm_peer: bf16 B");
  const c10::cuda::CUDAGuard guard(b.device());
  const int G = (int)groups, n_seg = (int)a_ptrs.size();
  torch::Tensor B = b.dim() == 2 ? b.unsqueeze(0) : b;
  TORCH_CHECK(B.size(0) == G && B.stride(2) == 1, "gemm_peer: B groups");
  const int N = b_mn ? B.size(2) : B.size(1), Kb = b_mn ? B.size(1) : B.size(2);
  TORCH_CHECK(Kb == K, "gemm_peer: K mismatch");
  const int M = n_seg * (int)seg_M;
  GemmParams p{};
  p.M = M; p.N = N; p.K = (int)K; p.G = G;
  p.epi = (int)epi; p.a_g_off = (int)a_g_off;
  torch::Tensor out;
  if (!out_ptrs.empty()) {
    TORCH_CHECK((int)out_ptrs.size() == n_seg, "gemm_peer: one output base per segment");
    for (int i = 0; i < n_seg; ++i) p.out_seg[i] = reinterpret_cast<void*>(out_ptrs[i]);
    p.out_seg_on = 1; p.out_g_off = (int)out_g_off; p.ldo = (int)out_ld; p.out_gs = out_gs;
    p.out = p.out_seg[0];
    TORCH_CHECK(out_ld % 8 == 0 && out_gs % 8 == 0, "gemm_peer: output pitches");
  } else {
    out = (out_local.has_value() && out_local->defined()) ? *out_local : torch::empty({G, M, N}, b.options());
    TORCH_CHECK(out.dim() == 3 && out.size(0) == G && out.size(1) == M && out.size(2) == N && out.stride(2) == 1, "gemm_peer: out");
    p.out = out.data_ptr(); p.ldo = (int)out.stride(1); p.out_gs = out.stride(0);
  }
  if (out2_.has_value() && out2_->defined()) {
    TORCH_CHECK(out2_->dim() == 3 && out2_->size(1) == M && out2_->stride(2) == 1, "gemm_peer: out2");
    p.out2 = out2_->data_ptr(); p.ldo2 = (int)out2_->stride(1); p.out2_gs = out2_->stride(0);
  }
  if (aux_.has_value() && aux_->defined()) {
    TORCH_CHECK(aux_->dim() == 3 && aux_->size(1) == M && aux_->stride(2) == 1, "gemm_peer: aux");
    p.aux = aux_->data_ptr(); p.ldaux = (int)aux_->stride(1); p.aux_gs = aux_->stride(0);
  }
  TORCH_CHECK(epi != EPI_RELU2 || p.out2 != nullptr, "gemm_peer: relu2 epilogue needs out2");
  p.status = gemm_status_word(b.get_device());
  std::vector<const void*> list(n_seg);
  for (int i = 0; i < n_seg; ++i) list[i] = reinterpret_cast<const void*>(a_ptrs[i]);
  launch_gemm_seg(list.data(), n_seg, (int)seg_M, (int)a_groups, a_pitch, a_gs, false, B.data_ptr(), B.stride(1),
                  G > 1 ? B.stride(0) : 0, b_mn, p, at::cuda::getCurrentCUDAStream(), gemm_sm_count());
  return out;
}

}  // namespace mb
