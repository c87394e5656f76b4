// Convolution operators of torch.ops.cosmos_b200 (kernels in conv3d_cl.cu): channels-last implicit-GEMM convolution and the
// RMS-norm + SiLU that precedes it in the VAE's residual blocks.

#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/library.h>

#include <vector>

#include "launchers.h"

int* cb200_error_word(int device);
int cb200_sm_count(int device);

namespace {
using at::Tensor;

// x [T_in, H_in, W_in, Cin] bf16; w [n_rows, ntaps * ceil(Cin / 64) * 64] bf16 (tap-major, channels zero-padded to 64);
// taps: ntaps * 3 ints (dt, dh, dw) added to the (strided) output coordinate, dt counted from the first of `pad` frames in front of
// x: the frames of `cache` are the last of these, frames before them are zeros; out_map: 10 ints (see ConvParams); y is written in place.
void conv_cl(const Tensor& x, const Tensor& w, int64_t n_tile, int64_t Cout, c10::ArrayRef<int64_t> taps, int64_t T_out, int64_t H_out,
             int64_t W_out, c10::ArrayRef<int64_t> out_map, Tensor y, const c10::optional<Tensor>& resid,
             const c10::optional<Tensor>& bias, const c10::optional<Tensor>& cache, int64_t pad, int64_t t_stride, int64_t hw_stride,
             const c10::optional<Tensor>& y_norm, const c10::optional<Tensor>& gamma, bool silu, bool write_raw) {
  TORCH_CHECK(x.is_cuda() && x.scalar_type() == at::kBFloat16 && x.is_contiguous() && x.dim() == 4, "x must be contiguous CUDA bf16 [T, H, W, C]");
  TORCH_CHECK(w.is_cuda() && w.scalar_type() == at::kBFloat16 && w.is_contiguous() && w.dim() == 2 && w.device() == x.device(),
              "w must be contiguous CUDA bf16 [rows, K] on the device of x");
  TORCH_CHECK(y.is_cuda() && y.scalar_type() == at::kBFloat16 && y.is_contiguous() && y.device() == x.device(), "y must be contiguous CUDA bf16");
  const int64_t ntaps = (int64_t)taps.size() / 3, Cin = x.size(3), kblocks = (Cin + 63) / 64;
  TORCH_CHECK(taps.size() % 3 == 0 && ntaps >= 1 && ntaps <= 27, "taps: 1..27 triples");
  TORCH_CHECK(out_map.size() == 10, "out_map: 10 integers");
  TORCH_CHECK(Cin % 16 == 0, "input channels must be a multiple of 16");
  TORCH_CHECK(n_tile % 16 == 0 && n_tile >= 16 && n_tile <= 256 && w.size(0) % n_tile == 0 && Cout >= 1 && Cout <= w.size(0), "bad N tiling");
  TORCH_CHECK(w.size(1) == ntaps * kblocks * 64, "weight K extent must be taps * ceil(Cin / 64) * 64");
  TORCH_CHECK(pad >= 0 && pad <= 64 && t_stride >= 1 && t_stride <= 8 && (hw_stride == 1 || hw_stride == 2), "pad 0..64, time stride 1..8, spatial stride 1 or 2");
  if (cache.has_value())
    TORCH_CHECK(cache->is_cuda() && cache->scalar_type() == at::kBFloat16 && cache->is_contiguous() && cache->device() == x.device() && cache->dim() == 4 &&
                    cache->size(0) >= 1 && cache->size(0) <= pad && cache->sizes().slice(1) == x.sizes().slice(1),
                "cache must be contiguous CUDA bf16 [1..pad, H, W, C] like x");
  TORCH_CHECK(T_out >= 1 && H_out >= 1 && W_out >= 1, "empty output grid");
  // the largest output element the kernel can touch must lie inside y (and inside resid)
  const int64_t ot_mul = out_map[0], ot_add = out_map[1], oh_mul = out_map[2], oh_add = out_map[3], ow_mul = out_map[4], ow_add = out_map[5],
                out_H = out_map[6], out_W = out_map[7], out_C = out_map[8], oc_add = out_map[9];
  TORCH_CHECK(ot_mul >= 1 && oh_mul >= 1 && ow_mul >= 1 && ot_add >= 0 && oh_add >= 0 && ow_add >= 0 && oc_add >= 0, "bad output map");
  TORCH_CHECK((H_out - 1) * oh_mul + oh_add < out_H && (W_out - 1) * ow_mul + ow_add < out_W && oc_add + Cout <= out_C, "output map leaves the frame");
  const int64_t last = ((((T_out - 1) * ot_mul + ot_add) * out_H + out_H - 1) * out_W + out_W - 1) * out_C + out_C;
  TORCH_CHECK(last <= y.numel(), "output map runs past y");
  if (resid.has_value())
    TORCH_CHECK(resid->is_cuda() && resid->scalar_type() == at::kBFloat16 && resid->is_contiguous() && resid->device() == x.device() &&
                    resid->numel() >= last, "resid must be contiguous CUDA bf16 covering the output map");
  if (bias.has_value())
    TORCH_CHECK(bias->is_cuda() && bias->scalar_type() == at::kFloat && bias->is_contiguous() && bias->device() == x.device() &&
                    bias->numel() >= Cout, "bias must be contiguous CUDA fp32 [Cout]");
  TORCH_CHECK(y_norm.has_value() == gamma.has_value() && (write_raw || y_norm.has_value()), "give gamma with y_norm; without it the raw output is written");
  if (y_norm.has_value())
    TORCH_CHECK(y_norm->is_cuda() && y_norm->scalar_type() == at::kBFloat16 && y_norm->is_contiguous() && y_norm->device() == x.device() &&
                    y_norm->numel() >= last && Cout <= n_tile && Cout % 8 == 0 && out_C % 8 == 0 && oc_add % 8 == 0 && gamma->is_cuda() &&
                    gamma->scalar_type() == at::kFloat && gamma->is_contiguous() && gamma->numel() == Cout && gamma->device() == x.device(),
                "y_norm must cover the output map, gamma be fp32 [Cout], and all channels lie in one N tile");
  if (((out_C | oc_add | Cout) & 7) == 0)      // voxels move as 16-byte pieces
    for (const Tensor* t : {(const Tensor*)&y, resid.has_value() ? &*resid : nullptr, y_norm.has_value() ? &*y_norm : nullptr})
      TORCH_CHECK(t == nullptr || reinterpret_cast<uintptr_t>(t->data_ptr()) % 16 == 0, "y, resid and y_norm must start on a 16-byte boundary");
  c10::cuda::CUDAGuard g(x.device());
  std::vector<int> tp(taps.begin(), taps.end()), om(out_map.begin(), out_map.end());
  const int dev = x.get_device();
  const int rc = cb200_conv_cl(x.data_ptr(), (int)x.size(0), (int)x.size(1), (int)x.size(2), (int)Cin,
                               cache.has_value() ? cache->data_ptr() : nullptr, cache.has_value() ? (int)cache->size(0) : 0, (int)pad,
                               (int)t_stride, (int)hw_stride, w.data_ptr(), (int)w.size(0), (int)n_tile, (int)Cout, tp.data(), (int)ntaps, (int)T_out, (int)H_out, (int)W_out, om.data(), y.data_ptr(),
                               resid.has_value() ? resid->data_ptr() : nullptr, bias.has_value() ? bias->data_ptr<float>() : nullptr,
                               y_norm.has_value() ? y_norm->data_ptr() : nullptr, gamma.has_value() ? gamma->data_ptr<float>() : nullptr,
                               silu ? 1 : 0, write_raw ? 1 : 0, cb200_error_word(dev), cb200_sm_count(dev), at::cuda::getCurrentCUDAStream().stream());
  TORCH_CHECK(rc == 0, "conv_cl launch failed with code ", rc);
}

// y = [silu](x / max(||x||_2, 1e-12) * sqrt(C) * gamma) over the last dimension of a channels-last tensor
Tensor rmsnorm_silu_cl(const Tensor& x, const Tensor& gamma, bool silu) {
  TORCH_CHECK(x.is_cuda() && x.scalar_type() == at::kBFloat16 && x.is_contiguous() && x.dim() >= 2, "x must be contiguous CUDA bf16 [..., C]");
  const int64_t C = x.size(-1);
  TORCH_CHECK(gamma.is_cuda() && gamma.scalar_type() == at::kFloat && gamma.is_contiguous() && gamma.numel() == C && gamma.device() == x.device(),
              "gamma must be contiguous CUDA fp32 [C] on the device of x");
  TORCH_CHECK(C % 8 == 0 && C <= 1024, "channels must be a multiple of 8, at most 1024");
  c10::cuda::CUDAGuard g(x.device());
  Tensor y = at::empty_like(x);
  const Tensor gm = reinterpret_cast<uintptr_t>(gamma.data_ptr()) % 16 == 0 ? gamma : gamma.clone();   // read as float4
  const int rc = cb200_rmsnorm_silu_cl(x.data_ptr(), gm.data_ptr<float>(), y.data_ptr(), x.numel() / C, (int)C, silu ? 1 : 0,
                                       at::cuda::getCurrentCUDAStream().stream());
  TORCH_CHECK(rc == 0, "rmsnorm_silu_cl launch failed with code ", rc);
  return y;
}

// softmax(q k^T * scale) v for one head of 384 channels: q [B, Sq, 384], k, v [B, Skv, 384] bf16, rows of any 16-byte aligned stride
Tensor fa_wide(const Tensor& q, const Tensor& k, const Tensor& v, double scale) {
  for (const Tensor* t : {&q, &k, &v}) {
    TORCH_CHECK(t->is_cuda() && t->scalar_type() == at::kBFloat16 && t->dim() == 3 && t->size(2) == 384 && t->stride(2) == 1 &&
                    t->device() == q.device() && t->size(0) == q.size(0), "fa_wide: q, k, v must be CUDA bf16 [B, S, 384] with dense channels");
    TORCH_CHECK(t->stride(1) % 8 == 0 && t->stride(0) % 8 == 0 && t->stride(1) > 0 && t->stride(0) > 0 &&
                    reinterpret_cast<uintptr_t>(t->data_ptr()) % 16 == 0, "fa_wide: rows must start on 16-byte boundaries");
  }
  TORCH_CHECK(scale > 0, "fa_wide: the softmax scale must be positive (the row maximum is taken before it is applied)");
  TORCH_CHECK(k.size(1) == v.size(1) && q.numel() > 0 && k.numel() > 0, "fa_wide: empty input or k / v of different length");
  c10::cuda::CUDAGuard g(q.device());
  Tensor o = at::empty({q.size(0), q.size(1), 384}, q.options());
  const int rc = cb200_fa_wide(q.data_ptr(), q.stride(1), q.stride(0), k.data_ptr(), k.stride(1), k.stride(0), v.data_ptr(), v.stride(1),
                               v.stride(0), o.data_ptr(), (int)q.size(0), (int)q.size(1), (int)k.size(1), (float)scale,
                               cb200_error_word(q.get_device()), at::cuda::getCurrentCUDAStream().stream());
  TORCH_CHECK(rc == 0, "fa_wide launch failed with code ", rc);
  return o;
}
}  // namespace

void register_conv_ops(torch::Library& m) {
  m.def("conv_cl(Tensor x, Tensor w, int n_tile, int Cout, int[] taps, int T_out, int H_out, int W_out, int[] out_map, Tensor(a!) y, "
        "Tensor? resid, Tensor? bias, Tensor? cache=None, int pad=0, int t_stride=1, int hw_stride=1, "
        "Tensor(b!)? y_norm=None, Tensor? gamma=None, bool silu=True, bool write_raw=True) -> ()", &conv_cl);
  m.def("conv_panels(int[] taps, int hw_stride, int Cin, int n_tile) -> int[]", [](c10::ArrayRef<int64_t> taps, int64_t hw_stride, int64_t Cin, int64_t n_tile) {
    TORCH_CHECK(taps.size() % 3 == 0 && taps.size() >= 3 && taps.size() <= 81, "taps: 1..27 triples");
    const std::vector<int> tp(taps.begin(), taps.end());
    int out[3 + 27 * 6];
    const int n = cb200_conv_panels(tp.data(), (int)tp.size() / 3, (int)hw_stride, (int)Cin, (int)n_tile, out);
    return std::vector<int64_t>(out, out + n);
  });
  m.def("fa_wide(Tensor q, Tensor k, Tensor v, float scale) -> Tensor", &fa_wide);
  m.def("rmsnorm_silu_cl(Tensor x, Tensor gamma, bool silu) -> Tensor", &rmsnorm_silu_cl);
}
