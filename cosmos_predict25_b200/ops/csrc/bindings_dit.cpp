// The sampling-time path of the DiT in native code: all transformer blocks of a denoising step (and the cross-attention keys / values
// of all blocks for a prompt) as ONE operator each, which launches the package's kernels back to back. A block is 16 launches
// (13 here: q, k and v are one GEMM over three weights, the norms of q and k one launch);
// issued one by one through Python and the dispatcher they cost about 25 us of host time each, more than most of them take on the GPU
// for an image of 256 x 256 (512 tokens with guidance): 12.9 ms a step, 8.0 ms with this loop when it was written, 4.4 ms with the
// kernels of today (about 3 ms of host time beside them). The kernels are those of models/dit.py:
// Block.forward and so are the sums, except where more tiles in a launch change how a contraction is split.

#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/library.h>

#include <algorithm>
#include <cmath>
#include <initializer_list>
#include <vector>

#include "launchers.h"

int* cb200_error_word(int device);
int cb200_sm_count(int device);

namespace {
using at::Tensor;

// a weight matrix [rows, cols] as the GEMM reads it
const void* weight(const Tensor& w, const Tensor& x, int64_t rows, int64_t cols) {
  TORCH_CHECK(w.is_cuda() && w.scalar_type() == at::kBFloat16 && w.is_contiguous() && w.dim() == 2 && w.size(0) == rows && w.size(1) == cols &&
                  w.device() == x.device(), "dit_blocks: weights must be contiguous CUDA bf16 [", rows, ", ", cols, "] on the device of x");
  return w.data_ptr();
}
// a norm weight of 128 values, bf16 or fp32; one that is laid out otherwise is converted and kept alive in `keep`
struct Norm {
  const void* p;
  int bf16;
};
Norm norm(const Tensor& w, const Tensor& x, std::vector<Tensor>& keep) {
  TORCH_CHECK(w.numel() == 128 && w.device() == x.device(), "dit_blocks: norm weights hold 128 values on the device of x");
  const bool ok = (w.scalar_type() == at::kFloat || w.scalar_type() == at::kBFloat16) && w.is_contiguous() &&
                  reinterpret_cast<uintptr_t>(w.data_ptr()) % 16 == 0;
  if (ok) return {w.data_ptr(), w.scalar_type() == at::kBFloat16 ? 1 : 0};
  keep.push_back(w.to(at::kFloat).clone(at::MemoryFormat::Contiguous));
  return {keep.back().data_ptr(), 0};
}

struct Launcher {
  int* err;
  int sms;
  cudaStream_t st;
  void gemm(const void* a, const void* w, void* c, int64_t M, int64_t N, int64_t K, int act = 0, const void* resid = nullptr,
            const float* gate = nullptr, int64_t ld_gate = 0, int64_t L = 1) const {
    const int rc = cb200_gemm_bf16(a, w, c, (int)M, (int)N, (int)K, 0, 0, nullptr, act, nullptr, resid, gate, ld_gate, (int)L, err, sms, st);
    TORCH_CHECK(rc == 0, "tcgen05 GEMM launch failed with code ", rc);
  }
  void gemms(const void* a, std::initializer_list<const void*> w, std::initializer_list<void*> c, int64_t M, int64_t N, int64_t K) const {
    const int rc = cb200_gemm_bf16_group(a, w.begin(), c.begin(), (int)w.size(), (int)M, (int)N, (int)K, err, sms, st);
    TORCH_CHECK(rc == 0, "tcgen05 GEMM (several weights) launch failed with code ", rc);
  }
  void attention(const void* q, const void* k, const void* v, void* o, float* lse, int64_t B, int64_t Sq, int64_t Skv, int64_t H) const {
    const int rc = cb200_fa_fwd(q, k, v, o, lse, (int)B, (int)Sq, (int)Skv, (int)H, (float)(1.0 / std::sqrt(128.0)), 0, sms, err, st);
    TORCH_CHECK(rc == 0, "fa_fwd launch failed with code ", rc);
  }
};

constexpr int kPerBlock = 11;   // self q, k, v, out, q norm, k norm; cross q, out, q norm; MLP in, out

// x [B, T, L, D]; mods [3 * blocks, B, T, 3 D] fp32 (shift, scale, gate of self-attention, cross-attention, MLP); cos / sin [T * L, 64]
// or absent; weights: kPerBlock per block; kv: keys and values of every block's cross-attention [B, S, H, 128]
Tensor dit_blocks(const Tensor& x, const Tensor& mods, const c10::optional<Tensor>& cosv, const c10::optional<Tensor>& sinv,
                  at::TensorList weights, at::TensorList kv, double ln_eps, double rms_eps) {
  TORCH_CHECK(x.is_cuda() && x.scalar_type() == at::kBFloat16 && x.is_contiguous() && x.dim() == 4, "dit_blocks: x must be contiguous CUDA bf16 [B, T, L, D]");
  const int64_t B = x.size(0), T = x.size(1), L = x.size(2), D = x.size(3), S = T * L, M = B * S, H = D / 128;
  const int64_t n = (int64_t)weights.size() / kPerBlock;
  TORCH_CHECK(x.numel() > 0 && D % 128 == 0 && D <= 8192 && M % 8 == 0 && n > 0 && (int64_t)weights.size() == n * kPerBlock && (int64_t)kv.size() == 2 * n,
              "dit_blocks: heads of 128 channels, tokens a multiple of 8, 11 weights and 2 context tensors per block");
  TORCH_CHECK(mods.is_cuda() && mods.scalar_type() == at::kFloat && mods.is_contiguous() && mods.device() == x.device() &&
                  mods.numel() == 3 * n * B * T * 3 * D && reinterpret_cast<uintptr_t>(mods.data_ptr()) % 16 == 0,
              "dit_blocks: mods must be contiguous fp32 [3 * blocks, B, T, 3 D]");
  TORCH_CHECK(cosv.has_value() == sinv.has_value(), "give both rotation tables or neither");
  const float *cp = nullptr, *sp = nullptr;
  if (cosv.has_value()) {
    for (const Tensor* t : {&*cosv, &*sinv})
      TORCH_CHECK(t->is_cuda() && t->scalar_type() == at::kFloat && t->is_contiguous() && t->dim() == 2 && t->size(0) == S && t->size(1) == 64 &&
                      t->device() == x.device(), "cos / sin must be contiguous fp32 [T * L, 64]");
    cp = cosv->data_ptr<float>();
    sp = sinv->data_ptr<float>();
  }
  int64_t F = 0;
  for (int64_t i = 0; i < n; ++i) F = std::max(F, weights[i * kPerBlock + 9].size(0));
  TORCH_CHECK(F % 64 == 0, "dit_blocks: the MLP width must be a multiple of 64");
  for (const Tensor& t : kv)
    TORCH_CHECK(t.is_cuda() && t.scalar_type() == at::kBFloat16 && t.is_contiguous() && t.dim() == 4 && t.size(0) == B && t.size(2) == H &&
                    t.size(3) == 128 && t.size(1) > 0 && t.device() == x.device(), "dit_blocks: keys / values must be contiguous CUDA bf16 [B, S, H, 128]");
  c10::cuda::CUDAGuard guard(x.device());
  const int dev = x.get_device();
  const Launcher run{cb200_error_word(dev), cb200_sm_count(dev), at::cuda::getCurrentCUDAStream().stream()};
  const auto f32 = x.options().dtype(at::kFloat);
  // two residual streams in turn, the normalised input, and one buffer that is q, k, v, attention output and then the MLP's hidden layer
  Tensor r0 = at::empty({M, D}, x.options()), r1 = at::empty({M, D}, x.options()), h = at::empty({M, D}, x.options());
  Tensor wide = at::empty({std::max(4 * D, F) * M}, x.options());
  Tensor stats = at::empty({2 * M}, f32), rstd = at::empty({2 * M * H}, f32), lse = at::empty({B * H * S}, f32);
  auto part = [&](int64_t i) { return static_cast<void*>(static_cast<char*>(wide.data_ptr()) + i * M * D * 2); };
  void *q = part(0), *k = part(1), *v = part(2), *o = part(3), *hp = h.data_ptr();
  float *mean = stats.data_ptr<float>(), *rs = mean + M, *rn = rstd.data_ptr<float>(), *lp = lse.data_ptr<float>();
  const void* cur = x.data_ptr();
  void *nxt = r0.data_ptr(), *spare = r1.data_ptr();
  auto step = [&]() {               // the sum just written becomes the residual stream
    cur = nxt;
    std::swap(nxt, spare);
  };
  std::vector<Tensor> keep;
  auto rms = [&](const void* raw, const Norm& w, const float* c, const float* s, void* dst) {
    cb200_rmsnorm_rope_fwd(raw, w.p, w.bf16, c, s, dst, rn, M * H, (int)S, (int)H, 128, (float)rms_eps, run.st);
  };
  for (int64_t i = 0; i < n; ++i) {
    const Tensor* w = &weights[i * kPerBlock];
    const int64_t Fi = w[9].size(0), Skv = kv[2 * i].size(1);
    TORCH_CHECK(kv[2 * i + 1].size(1) == Skv && Fi % 64 == 0, "dit_blocks: keys and values of different length");
    const float* m = mods.data_ptr<float>() + 3 * i * B * T * 3 * D;
    auto ln = [&](int64_t j) {
      const float* mj = m + j * B * T * 3 * D;
      cb200_ln_modulate_fwd(cur, mj, mj + D, hp, mean, rs, M, (int)D, (int)L, 3 * D, 3 * D, (float)ln_eps, run.st);
    };
    auto add = [&](int64_t j, const void* a, const void* wt, int64_t K) {
      run.gemm(a, wt, nxt, M, D, K, 0, cur, m + j * B * T * 3 * D + 2 * D, 3 * D, L);
      step();
    };
    ln(0);
    // the attention output's and the next residual stream's places hold the raw projections meanwhile
    run.gemms(hp, {weight(w[0], x, D, D), weight(w[1], x, D, D), weight(w[2], x, D, D)}, {o, nxt, v}, M, D, D);
    {
      // both in one launch: a launch of its own took k 3.9 us at 512 tokens, bound by its start
      const Norm nq = norm(w[4], x, keep), nk = norm(w[5], x, keep);
      const void *raw[2] = {o, nxt}, *nw[2] = {nq.p, nk.p};
      const int nb[2] = {nq.bf16, nk.bf16};
      void* dst[2] = {q, k};
      float* rr[2] = {rn, rn + M * H};
      cb200_rmsnorm_rope_fwd_pair(raw, nw, nb, cp, sp, dst, rr, M * H, (int)S, (int)H, 128, (float)rms_eps, run.st);
    }
    run.attention(q, k, v, o, lp, B, S, S, H);
    add(0, o, weight(w[3], x, D, D), D);
    ln(1);
    run.gemm(hp, weight(w[6], x, D, D), o, M, D, D);
    rms(o, norm(w[8], x, keep), nullptr, nullptr, q);
    run.attention(q, kv[2 * i].data_ptr(), kv[2 * i + 1].data_ptr(), o, lp, B, S, Skv, H);
    add(1, o, weight(w[7], x, D, D), D);
    ln(2);
    run.gemm(hp, weight(w[9], x, Fi, D), wide.data_ptr(), M, Fi, D, 1);
    add(2, wide.data_ptr(), weight(w[10], x, D, Fi), Fi);
  }
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  return (cur == r0.data_ptr() ? r0 : r1).view({B, T, L, D});
}

// blocks whose context keys and values one launch computes: those of equal width, if it has tiles enough; else 0
int64_t context_blocks_per_launch(int64_t rows, int64_t C, at::IntArrayRef widths, int sms) {
  if (widths.empty()) return 0;
  for (int64_t d : widths)
    if (d != widths[0]) return 0;
  const int64_t n = std::min<int64_t>(2 * (int64_t)widths.size(), 1 << 20);
  return cb200_gemm_many_weights((int)n, (int)rows, (int)widths[0], (int)C, sms) / 2;
}
// launches of dit_context_kv for blocks of these widths
int64_t dit_context_launches(int64_t rows, int64_t C, at::IntArrayRef widths) {
  const int64_t n = (int64_t)widths.size(), per = context_blocks_per_launch(rows, C, widths, cb200_sm_count(at::cuda::current_device()));
  return per > 0 ? (n + per - 1) / per : n * (1 + cb200_gemm_group_launches((int)rows, 2));
}

// Cross-attention keys (normalised) and values of every block for one context [B, S, C]; weights: key projection, value projection,
// key norm per block. Returns k_0, v_0, k_1, v_1, ...
std::vector<Tensor> dit_context_kv(const Tensor& context, at::TensorList weights, double rms_eps) {
  TORCH_CHECK(context.is_cuda() && context.scalar_type() == at::kBFloat16 && context.is_contiguous() && context.dim() == 3 && context.numel() > 0,
              "dit_context_kv: the context must be contiguous CUDA bf16 [B, S, C]");
  const int64_t B = context.size(0), S = context.size(1), C = context.size(2), M = B * S, n = (int64_t)weights.size() / 3;
  TORCH_CHECK((int64_t)weights.size() == 3 * n && C % 64 == 0 && M % 8 == 0, "dit_context_kv: three weights per block, C a multiple of 64, B * S of 8");
  c10::cuda::CUDAGuard guard(context.device());
  const int dev = context.get_device();
  const Launcher run{cb200_error_word(dev), cb200_sm_count(dev), at::cuda::getCurrentCUDAStream().stream()};
  std::vector<Tensor> out, keep;
  Tensor rstd, raw;
  std::vector<int64_t> widths;
  for (int64_t i = 0; i < n; ++i) widths.push_back(weights[3 * i].dim() == 2 ? weights[3 * i].size(0) : 0);
  const int64_t D0 = n > 0 ? widths[0] : 0, per = context_blocks_per_launch(M, C, widths, run.sms);
  TORCH_CHECK(per == 0 || D0 % 128 == 0, "dit_context_kv: heads of 128 channels");
  // A block's keys and values as a launch of 64 tiles and a norm took 15.7 us for 2 x 512 tokens and 2048 channels, 440 us for 28 blocks
  for (int64_t i0 = 0; per > 0 && i0 < n; i0 += per) {
    const int m = (int)std::min<int64_t>(per, n - i0);
    std::vector<const void*> w, nw;
    std::vector<uint8_t> nb;
    std::vector<void*> c;
    for (int64_t i = i0; i < i0 + m; ++i) {
      const Norm nk = norm(weights[3 * i + 2], context, keep);
      for (int j = 0; j < 2; ++j) {
        out.push_back(at::empty({B, S, D0 / 128, 128}, context.options()));
        w.push_back(weight(weights[3 * i + j], context, D0, C));
        nw.push_back(j == 0 ? nk.p : nullptr);
        nb.push_back(j == 0 ? (uint8_t)nk.bf16 : 0);
        c.push_back(out.back().data_ptr());
      }
    }
    const int rc = cb200_gemm_bf16_many(context.data_ptr(), w.data(), c.data(), nw.data(), nb.data(), 2 * m, (int)M, (int)D0, (int)C,
                                        (float)rms_eps, run.err, run.sms, run.st);
    TORCH_CHECK(rc == 0, "tcgen05 GEMM (many weights) launch failed with code ", rc);
  }
  for (int64_t i = per > 0 ? n : 0; i < n; ++i) {
    const int64_t D = weights[3 * i].size(0), H = D / 128;
    TORCH_CHECK(D % 128 == 0, "dit_context_kv: heads of 128 channels");
    Tensor k = at::empty({B, S, H, 128}, context.options()), v = at::empty({B, S, H, 128}, context.options());
    if (!rstd.defined() || rstd.numel() < M * H) {
      rstd = at::empty({M * H}, context.options().dtype(at::kFloat));
      raw = at::empty({M * D}, context.options());
    }
    run.gemms(context.data_ptr(), {weight(weights[3 * i], context, D, C), weight(weights[3 * i + 1], context, D, C)}, {raw.data_ptr(), v.data_ptr()}, M, D, C);
    const Norm w = norm(weights[3 * i + 2], context, keep);
    cb200_rmsnorm_rope_fwd(raw.data_ptr(), w.p, w.bf16, nullptr, nullptr, k.data_ptr(), rstd.data_ptr<float>(), M * H, (int)S, (int)H, 128,
                           (float)rms_eps, run.st);
    out.push_back(k);
    out.push_back(v);
  }
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  return out;
}
}  // namespace

void register_dit_ops(torch::Library& m) {
  m.def("dit_blocks(Tensor x, Tensor mods, Tensor? cosv, Tensor? sinv, Tensor[] weights, Tensor[] kv, float ln_eps, float rms_eps) -> Tensor", &dit_blocks);
  m.def("dit_context_kv(Tensor context, Tensor[] weights, float rms_eps) -> Tensor[]", &dit_context_kv);
  m.def("dit_context_launches(int rows, int channels, int[] widths) -> int", &dit_context_launches);
}
