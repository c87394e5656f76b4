// Memory-bound fused kernels of the DiT block and of the optimizer (sm_100a).
//
//   ln_modulate      LayerNorm(no affine) * (1 + scale[frame]) + shift[frame]       fwd + bwd
//   gate_residual    x + gate[frame] * y                                             fwd + bwd
//   rmsnorm_rope     per-head RMSNorm (learnable weight) + rotate-half RoPE          fwd + bwd
//   gelu             exact (erf) GELU                                                fwd + bwd
//   cfg_combine      cond + g * (cond - uncond)
//   grad_cast_norm   bf16 grad -> fp32 * scale, NaN/Inf scrub, squared-norm partials
//   adamw_ema_shard  AdamW on fp32 masters + EMA + bf16 write-back, clip coefficient read on device
//
// Every kernel moves each byte once: 16-byte vector accesses, fp32 math in registers, one pass.
// Reductions over tokens (dshift/dscale/dgate/dweight) are two-stage and deterministic: per-CTA
// partials go to a scratch buffer, a second kernel sums them in a fixed order.

#include "common.cuh"
#include "launchers.h"
#include <algorithm>

#include "sm100.cuh"   // packed fp32x2 arithmetic

namespace cb200 {
using sm100::add2;
using sm100::fma2;
using sm100::mul2;

// element pair i of an 8-value register row
#define CB200_P2(arr, i) make_float2((arr)[2 * (i)], (arr)[2 * (i) + 1])

constexpr int kThreads = 256;
constexpr int kMaxVec = 4;  // up to 256*4*8 = 8192 channels per row

__device__ __forceinline__ float2 block_sum2(float a, float b, float* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  a = warp_sum(a);
  b = warp_sum(b);
  __syncthreads();
  if (lane == 0) {
    red[warp] = a;
    red[32 + warp] = b;
  }
  __syncthreads();
  const int nwarps = (blockDim.x + 31) >> 5;
  float ta = (lane < nwarps) ? red[lane] : 0.f;
  float tb = (lane < nwarps) ? red[32 + lane] : 0.f;
  return make_float2(warp_sum(ta), warp_sum(tb));
}

__device__ __forceinline__ void load_f8(const float* p, float (&f)[8]) {
  float4 a = *reinterpret_cast<const float4*>(p);
  float4 b = *reinterpret_cast<const float4*>(p + 4);
  f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w;
  f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}

__device__ __forceinline__ void store_f8(float* p, const float (&f)[8]) {
  *reinterpret_cast<float4*>(p) = make_float4(f[0], f[1], f[2], f[3]);
  *reinterpret_cast<float4*>(p + 4) = make_float4(f[4], f[5], f[6], f[7]);
}

// ------------------------------------------------------------------------------------------------
// LayerNorm + modulate, forward: one CTA per token row
// ------------------------------------------------------------------------------------------------
// For few rows and short frames. Few rows are bound by latency: the row and its modulation vectors
// are loaded together, a thread holds NV pieces of 16 bytes, and each of the two sums is one barrier. With a warp per row, its two
// reductions and then its loads of the modulation in a row, 512 rows of 2048 took 5.6 us in a row of launches, now 3.5 (1024 rows 7.1
// and 3.7; a launch that does nothing about 2). Thousands of rows that a warp holds are bound by the start of CTAs: ROWS rows to a CTA then,
// a warp each (8192 frames of one row of 256 9.2 us with a CTA a row, now 4.2; 2048 frames of three rows of 512 7.7 and 5.3; 64 frames of 64
// rows of 256 in batches 3.7, now 3.4).
template <int NV, int THREADS, int ROWS>
__global__ void __launch_bounds__(THREADS * ROWS) ln_modulate_fwd_row_kernel(
    const bf16* __restrict__ x, const float* __restrict__ shift, const float* __restrict__ scale,
    bf16* __restrict__ y, float* __restrict__ mean_out, float* __restrict__ rstd_out, long rows, int D, int L, long ld_shift, long ld_scale,
    float eps) {
  static_assert(ROWS == 1 || THREADS == 32, "several rows in a CTA: a warp each");
  __shared__ float red[2][THREADS / 32];
  pdl_trigger();                     // launched with programmatic serialisation (see common.cuh)
  pdl_wait();
  const unsigned tid = ROWS == 1 ? threadIdx.x : threadIdx.x & 31;
  const long row = ROWS == 1 ? (long)blockIdx.x : (long)blockIdx.x * ROWS + (threadIdx.x >> 5);
  if (ROWS > 1 && row >= rows) return;
  const long frame = row / L;
  const int nvec = D >> 3, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bf16x8* xr = reinterpret_cast<const bf16x8*>(x + row * D);
  const float* sh = shift + frame * ld_shift;
  const float* sc = scale + frame * ld_scale;
  bf16x8 v[NV];
  float a[NV][8], b[NV][8];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = tid + i * THREADS;
    v[i] = c < nvec ? xr[c] : bf16x8{};
  }
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = tid + i * THREADS;
    if (c < nvec) {
      load_f8(sh + c * 8, a[i]);
      load_f8(sc + c * 8, b[i]);
    }
  }
  auto total = [&](float2 s2, float* slots) -> float {
    const float s = warp_sum(s2.x + s2.y);
    if (THREADS == 32) return s;
    if (lane == 0) slots[warp] = s;
    __syncthreads();
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < THREADS / 32; ++w) t += slots[w];
    return t;
  };
  float2 s2 = make_float2(0.f, 0.f);
#pragma unroll
  for (int i = 0; i < NV; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) s2 = add2(s2, __bfloat1622float2(v[i].v[j]));
  const float mean = total(s2, red[0]) / D;
  const float2 nm = make_float2(-mean, -mean);
  float2 q2 = make_float2(0.f, 0.f);
#pragma unroll
  for (int i = 0; i < NV; ++i)
    if (tid + i * THREADS < nvec) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 d = add2(__bfloat1622float2(v[i].v[j]), nm);
        q2 = fma2(d, d, q2);
      }
    }
  const float rstd = rsqrtf(total(q2, red[1]) / D + eps);
  if (tid == 0) {
    mean_out[row] = mean;
    rstd_out[row] = rstd;
  }
  const float2 one2 = make_float2(1.f, 1.f), rs2 = make_float2(rstd, rstd);
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = tid + i * THREADS;
    if (c < nvec) {
      bf16x8 o;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 t = fma2(mul2(add2(__bfloat1622float2(v[i].v[j]), nm), rs2), add2(CB200_P2(b[i], j), one2), CB200_P2(a[i], j));
        o.v[j] = __floats2bfloat162_rn(t.x, t.y);
      }
      reinterpret_cast<bf16x8*>(y + row * D)[c] = o;
    }
  }
}

// Same operator for many rows: a CTA walks over `rows_per_cta` rows of one frame, four at a time, and a thread keeps the modulation of its
// NV pieces of 16 bytes in registers (read for every row or pair of rows they are four or two times its bytes). The loads of the
// next four rows are in flight while four are reduced; each warp reduces its part of a row to a sum and a sum of squares about
// its own mean, and the parts are put together behind one barrier.
// Bound by memory: 46,800 rows of 2048 (383 MB) 107 us with a pair of rows per warp, now 84 (4.6 TB/s; the bytes take 59 us), 7040 rows
// in L2 13.5 and 13.2, 46,800 rows of 5120 325 (a CTA per row) and 238, 46,800 rows of 1024 51 and 42. Two rows at a time are a tenth
// slower at 2048 channels, from 2056 channels on four spill registers. A spill costs more than a CTA more on the SM gives.
// sums over the warp of R values a lane (two or four): lane l receives the total of value l / (32 / R)
template <int R>
__device__ __forceinline__ float warp_sums(const float (&v)[R], int lane) {
  static_assert(R == 2 || R == 4, "two or four values");
  const bool hi = lane & 16, odd = lane & 8;
  float k;
  if constexpr (R == 4) {
    const float k0 = (hi ? v[2] : v[0]) + __shfl_xor_sync(0xffffffffu, hi ? v[0] : v[2], 16);
    const float k1 = (hi ? v[3] : v[1]) + __shfl_xor_sync(0xffffffffu, hi ? v[1] : v[3], 16);
    k = (odd ? k1 : k0) + __shfl_xor_sync(0xffffffffu, odd ? k0 : k1, 8);
  } else {
    k = (hi ? v[1] : v[0]) + __shfl_xor_sync(0xffffffffu, hi ? v[0] : v[1], 16);
    k += __shfl_xor_sync(0xffffffffu, k, 8);
  }
  k += __shfl_xor_sync(0xffffffffu, k, 4);
  k += __shfl_xor_sync(0xffffffffu, k, 2);
  k += __shfl_xor_sync(0xffffffffu, k, 1);
  return k;
}

template <int NV, int MAXT, int kLnRows, int MINB>
__global__ void __launch_bounds__(MAXT, MINB) ln_modulate_fwd_rows_kernel(
    const bf16* __restrict__ x, const float* __restrict__ shift, const float* __restrict__ scale,
    bf16* __restrict__ y, float* __restrict__ mean_out, float* __restrict__ rstd_out, int D, int L, int rows_per_cta, int groups_per_frame,
    long ld_shift, long ld_scale, float eps) {
  static_assert(MAXT <= 512, "sixteen warps");
  constexpr int G = 32 / kLnRows;            // lanes that put the parts of one row together, 16 / G parts each
  constexpr bool two = G == 8;
  __shared__ float2 red[2][kLnRows][16];     // (sum, squares about the warp's mean) of row r in warp w; two sets in turn
  pdl_trigger();                     // launched with programmatic serialisation (see common.cuh)
  pdl_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, T = blockDim.x, nw = T >> 5, nvec = D >> 3;
  const long frame = blockIdx.x / groups_per_frame;
  const int r0 = (int)(blockIdx.x % groups_per_frame) * rows_per_cta, r1 = min(r0 + rows_per_cta, L);
  const bf16* xf = x + frame * L * D;
  bf16* yf = y + frame * L * D;
  bf16x8 nx[kLnRows][NV];
  auto fetch = [&](int r) {
#pragma unroll
    for (int k = 0; k < kLnRows; ++k)
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const int c = threadIdx.x + i * T;
        nx[k][i] = r + k < r1 && c < nvec ? reinterpret_cast<const bf16x8*>(xf + (long)(r + k) * D)[c] : bf16x8{};
      }
  };
  fetch(r0);
  float a[NV][8], b[NV][8];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = threadIdx.x + i * T;
    if (c < nvec) {
      load_f8(shift + frame * ld_shift + c * 8, a[i]);
      load_f8(scale + frame * ld_scale + c * 8, b[i]);
#pragma unroll
      for (int j = 0; j < 8; ++j) b[i][j] += 1.f;
    }
  }
  // channels of a row that warp w holds
  auto channels = [&](int w) -> float {
    int n = 0;
#pragma unroll
    for (int i = 0; i < NV; ++i) n += 8 * max(0, min(32, nvec - (w * 32 + i * T)));
    return (float)n;
  };
  const float inv_own = 1.f / channels(warp);
  const int w0 = lane % G, w1 = w0 + 8, row_in = lane / G;       // the parts of a row that this lane puts together
  const float n0 = w0 < nw ? channels(w0) : 0.f, n1 = two && w1 < nw ? channels(w1) : 0.f;
  const float i0 = n0 > 0.f ? 1.f / n0 : 0.f, i1 = n1 > 0.f ? 1.f / n1 : 0.f, inv_d = 1.f / D;
  int set = 0;
  for (int r = r0; r < r1; r += kLnRows, set ^= 1) {
    bf16x8 v[kLnRows][NV];
#pragma unroll
    for (int k = 0; k < kLnRows; ++k)
#pragma unroll
      for (int i = 0; i < NV; ++i) v[k][i] = nx[k][i];
    if (r + kLnRows < r1) fetch(r + kLnRows);
    float part[kLnRows];
#pragma unroll
    for (int k = 0; k < kLnRows; ++k) {
      float2 s2 = make_float2(0.f, 0.f);
#pragma unroll
      for (int i = 0; i < NV; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) s2 = add2(s2, __bfloat1622float2(v[k][i].v[j]));
      part[k] = s2.x + s2.y;
    }
    const float sum = warp_sums(part, lane);
    const float own_mean = sum * inv_own;
#pragma unroll
    for (int k = 0; k < kLnRows; ++k) {
      const float m = __shfl_sync(0xffffffffu, own_mean, k * G);
      const float2 nm = make_float2(-m, -m);
      float2 q2 = make_float2(0.f, 0.f);
#pragma unroll
      for (int i = 0; i < NV; ++i)
        if (threadIdx.x + i * T < nvec) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 d = add2(__bfloat1622float2(v[k][i].v[j]), nm);
            q2 = fma2(d, d, q2);
          }
        }
      part[k] = q2.x + q2.y;
    }
    const float squares = warp_sums(part, lane);
    if (w0 == 0) red[set][row_in][warp] = make_float2(sum, squares);
    __syncthreads();
    const float2 p0 = w0 < nw ? red[set][row_in][w0] : make_float2(0.f, 0.f), p1 = two && w1 < nw ? red[set][row_in][w1] : make_float2(0.f, 0.f);
    float mean = p0.x + p1.x;
    if (!two) mean += __shfl_xor_sync(0xffffffffu, mean, 8);
    mean += __shfl_xor_sync(0xffffffffu, mean, 4);
    mean += __shfl_xor_sync(0xffffffffu, mean, 2);
    mean += __shfl_xor_sync(0xffffffffu, mean, 1);
    mean *= inv_d;
    const float d0 = p0.x * i0 - mean, d1 = p1.x * i1 - mean;
    float var = p0.y + p1.y + n0 * d0 * d0 + n1 * d1 * d1;
    if (!two) var += __shfl_xor_sync(0xffffffffu, var, 8);
    var += __shfl_xor_sync(0xffffffffu, var, 4);
    var += __shfl_xor_sync(0xffffffffu, var, 2);
    var += __shfl_xor_sync(0xffffffffu, var, 1);
    const float rstd = rsqrtf(var * inv_d + eps);
    if (warp == 0 && w0 == 0 && r + row_in < r1) {
      mean_out[frame * L + r + row_in] = mean;
      rstd_out[frame * L + r + row_in] = rstd;
    }
#pragma unroll
    for (int k = 0; k < kLnRows; ++k) {
      const float m = __shfl_sync(0xffffffffu, mean, k * G), rs = __shfl_sync(0xffffffffu, rstd, k * G);
      const float2 nm = make_float2(-m, -m), rs2 = make_float2(rs, rs);
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const int c = threadIdx.x + i * T;
        if (r + k < r1 && c < nvec) {
          bf16x8 o;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 t = fma2(mul2(add2(__bfloat1622float2(v[k][i].v[j]), nm), rs2), CB200_P2(b[i], j), CB200_P2(a[i], j));
            o.v[j] = __floats2bfloat162_rn(t.x, t.y);
          }
          reinterpret_cast<bf16x8*>(yf + (long)(r + k) * D)[c] = o;
        }
      }
    }
  }
}

// backward: one CTA per group of `rows_per_cta` rows of one frame; writes dx and the per-group
// partials of dshift (sum dy) and dscale (sum dy * xhat) to `partials` [groups, 2, D].
template <int MV>
__global__ void __launch_bounds__(kThreads) ln_modulate_bwd_kernel(
    const bf16* __restrict__ dy, const bf16* __restrict__ x, const float* __restrict__ mean_in,
    const float* __restrict__ rstd_in, const float* __restrict__ scale, bf16* __restrict__ dx,
    float* __restrict__ partials, int D, int L, int rows_per_cta, int groups_per_frame, long ld_scale) {
  __shared__ float red[64];
  const long frame = blockIdx.x / groups_per_frame;
  const int g = blockIdx.x % groups_per_frame;
  const int r0 = g * rows_per_cta;
  const int r1 = min(r0 + rows_per_cta, L);
  const int nvec = D >> 3;
  float acc_sh[MV][8], acc_sc[MV][8], onep[MV][8];
#pragma unroll
  for (int i = 0; i < MV; ++i) {
    const int c = threadIdx.x + i * kThreads;
#pragma unroll
    for (int j = 0; j < 8; ++j) acc_sh[i][j] = acc_sc[i][j] = 0.f;
    if (c < nvec) {
      load_f8(scale + frame * ld_scale + c * 8, onep[i]);
#pragma unroll
      for (int j = 0; j < 8; ++j) onep[i][j] += 1.f;
    }
  }
  // software pipeline: the loads of row r + 1 are in flight while row r is reduced and written
  bf16x8 nd[MV], nx[MV];
  float nmean = 0.f, nrstd = 0.f;
  auto fetch = [&](int r) {
    const long row = frame * L + r;
    nmean = mean_in[row];
    nrstd = rstd_in[row];
#pragma unroll
    for (int i = 0; i < MV; ++i) {
      const int c = threadIdx.x + i * kThreads;
      if (c < nvec) {
        nd[i] = reinterpret_cast<const bf16x8*>(dy + row * D)[c];
        nx[i] = reinterpret_cast<const bf16x8*>(x + row * D)[c];
      }
    }
  };
  if (r0 < r1) fetch(r0);
  for (int r = r0; r < r1; ++r) {
    const long row = frame * L + r;
    const float mean = nmean, rstd = nrstd;
    bf16x8 cd[MV], cx[MV];
#pragma unroll
    for (int i = 0; i < MV; ++i) {
      cd[i] = nd[i];
      cx[i] = nx[i];
    }
    if (r + 1 < r1) fetch(r + 1);
    float gval[MV][8], xh[MV][8];
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int i = 0; i < MV; ++i) {
      const int c = threadIdx.x + i * kThreads;
      if (c < nvec) {
        float d[8], xv[8];
        unpack8(cd[i], d);
        unpack8(cx[i], xv);
        const float2 nm = make_float2(-mean, -mean), rs2 = make_float2(rstd, rstd);
        float2 t1 = make_float2(0.f, 0.f), t2 = make_float2(0.f, 0.f);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 dj = CB200_P2(d, j);
          const float2 h = mul2(add2(CB200_P2(xv, j), nm), rs2);
          const float2 sh = add2(CB200_P2(acc_sh[i], j), dj);
          const float2 sc = fma2(dj, h, CB200_P2(acc_sc[i], j));
          const float2 gj = mul2(dj, CB200_P2(onep[i], j));
          t1 = add2(t1, gj);
          t2 = fma2(gj, h, t2);
          xh[i][2 * j] = h.x; xh[i][2 * j + 1] = h.y;
          acc_sh[i][2 * j] = sh.x; acc_sh[i][2 * j + 1] = sh.y;
          acc_sc[i][2 * j] = sc.x; acc_sc[i][2 * j + 1] = sc.y;
          gval[i][2 * j] = gj.x; gval[i][2 * j + 1] = gj.y;
        }
        s1 += t1.x + t1.y;
        s2 += t2.x + t2.y;
      }
    }
    const float2 t = block_sum2(s1, s2, red);
    const float m1 = t.x / D, m2 = t.y / D;
    bf16x8* dxr = reinterpret_cast<bf16x8*>(dx + row * D);
#pragma unroll
    for (int i = 0; i < MV; ++i) {
      const int c = threadIdx.x + i * kThreads;
      if (c < nvec) {
        float o[8];
        const float2 nm1 = make_float2(-m1, -m1), nm2 = make_float2(-m2, -m2), rs2 = make_float2(rstd, rstd);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 t = mul2(rs2, fma2(CB200_P2(xh[i], j), nm2, add2(CB200_P2(gval[i], j), nm1)));
          o[2 * j] = t.x;
          o[2 * j + 1] = t.y;
        }
        dxr[c] = pack8(o);
      }
    }
  }
  float* p = partials + (long)blockIdx.x * 2 * D;
#pragma unroll
  for (int i = 0; i < MV; ++i) {
    const int c = threadIdx.x + i * kThreads;
    if (c < nvec) {
      store_f8(p + c * 8, acc_sh[i]);
      store_f8(p + D + c * 8, acc_sc[i]);
    }
  }
}

// out[frame, k, d] = sum over groups of partials[frame*G + g, k, d]; K slabs per group
__global__ void reduce_partials_kernel(const float* __restrict__ partials, float* __restrict__ out0,
                                       float* __restrict__ out1, int D, int groups_per_frame, int K) {
  const int d = blockIdx.x * blockDim.x + threadIdx.x;
  const long frame = blockIdx.y;
  if (d >= D) return;
  for (int k = 0; k < K; ++k) {
    float s = 0.f;
    const float* p = partials + (frame * groups_per_frame) * (long)K * D + (long)k * D + d;
    for (int g = 0; g < groups_per_frame; ++g) s += p[(long)g * K * D];
    float* o = (k == 0) ? out0 : out1;
    o[frame * D + d] = s;
  }
}

// out[d] = sum over rows of partials[row, d] for many rows and few columns (the weight gradient of the per-head RMSNorm:
// thousands of CTA partials of 64 / 128 columns). A CTA owns 32 columns; 32 warps stride over the rows with coalesced 128-byte
// loads, then the 32 per-warp sums of a column are added in a fixed order: deterministic.
__global__ void __launch_bounds__(1024) reduce_rows_kernel(const float* __restrict__ partials, float* __restrict__ out, int D, int rows) {
  __shared__ float sm[32][33];
  const int lane = threadIdx.x & 31, part = threadIdx.x >> 5;
  const int d = blockIdx.x * 32 + lane;
  float s = 0.f;
  if (d < D)
    for (int r = part; r < rows; r += 32) s += partials[(long)r * D + d];
  sm[part][lane] = s;
  __syncthreads();
  if (part == 0 && d < D) {
    float t = 0.f;
#pragma unroll
    for (int k = 0; k < 32; ++k) t += sm[k][lane];
    out[d] = t;
  }
}

// ------------------------------------------------------------------------------------------------
// gated residual
// ------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads) gate_residual_fwd_kernel(
    const bf16* __restrict__ x, const float* __restrict__ gate, const bf16* __restrict__ y, bf16* __restrict__ out,
    long nvec_total, int D, int L, long ld_gate) {
  const int nvec = D >> 3;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < nvec_total; i += (long)gridDim.x * blockDim.x) {
    const long row = i / nvec;
    const int c = (int)(i - row * nvec);
    const long frame = row / L;
    float a[8], b[8], g[8], o[8];
    unpack8(reinterpret_cast<const bf16x8*>(x)[i], a);
    unpack8(reinterpret_cast<const bf16x8*>(y)[i], b);
    load_f8(gate + frame * ld_gate + c * 8, g);
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = a[j] + g[j] * b[j];
    reinterpret_cast<bf16x8*>(out)[i] = pack8(o);
  }
}

template <int MV>
__global__ void __launch_bounds__(kThreads) gate_residual_bwd_kernel(
    const bf16* __restrict__ dout, const float* __restrict__ gate, const bf16* __restrict__ y, bf16* __restrict__ dy,
    float* __restrict__ partials, int D, int L, int rows_per_cta, int groups_per_frame, long ld_gate) {
  const long frame = blockIdx.x / groups_per_frame;
  const int g = blockIdx.x % groups_per_frame;
  const int r0 = g * rows_per_cta, r1 = min(r0 + rows_per_cta, L);
  const int nvec = D >> 3;
  float acc[MV][8], gt[MV][8];
#pragma unroll
  for (int i = 0; i < MV; ++i) {
    const int c = threadIdx.x + i * kThreads;
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
    if (c < nvec) load_f8(gate + frame * ld_gate + c * 8, gt[i]);
  }
  for (int r = r0; r < r1; ++r) {
    const long row = frame * L + r;
    const bf16x8* dor = reinterpret_cast<const bf16x8*>(dout + row * D);
    const bf16x8* yr = reinterpret_cast<const bf16x8*>(y + row * D);
    bf16x8* dyr = reinterpret_cast<bf16x8*>(dy + row * D);
#pragma unroll
    for (int i = 0; i < MV; ++i) {
      const int c = threadIdx.x + i * kThreads;
      if (c < nvec) {
        float d[8], yv[8], o[8];
        unpack8(dor[c], d);
        unpack8(yr[c], yv);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          acc[i][j] += d[j] * yv[j];
          o[j] = d[j] * gt[i][j];
        }
        dyr[c] = pack8(o);
      }
    }
  }
  float* p = partials + (long)blockIdx.x * D;
#pragma unroll
  for (int i = 0; i < MV; ++i) {
    const int c = threadIdx.x + i * kThreads;
    if (c < nvec) store_f8(p + c * 8, acc[i]);
  }
}

// ------------------------------------------------------------------------------------------------
// per-head RMSNorm + RoPE: one warp per (token, head), head_dim in {64, 128}; lane holds HD/32 values
// ------------------------------------------------------------------------------------------------
// Sixteen lanes per (token, head) row, two rows per warp pass. A lane holds P = HD / 32 elements of each half of the row, at the same
// offset, so that the rotation partner of every element is in the lane itself and one cosine / sine vector serves both; reductions
// stay inside the 16-lane half. Token and head of a row are counted along instead of divided out (64-bit divisions per row, a
// shuffle per element and twice the table loads bound the first layout by instruction issue). Bound by memory and by the warps in flight:
// the rows of later passes wait as bf16 (72 registers a thread before, 62 now: four CTAs on an SM for three) and the table's rows are
// loaded with them: one where a lane's rows are heads of one token (a multiple of eight heads), else one for each (loaded pass by pass behind
// the sums, 512 x 2 tokens with one head of 64 took 2.7 us, now 2.1). 46,800 tokens x 16 heads 88 us before, 68 now, without rotation
// 67 and 57 (the bytes take 59 us; part of them are in L2); 7040 tokens 10.4 and 8.0, 46,800 tokens x 40 heads 209 and 156.
constexpr int kRmsPasses = 4;        // forward: passes (of two rows) whose loads a warp keeps in flight together

template <int P>
__device__ __forceinline__ void load_raw(const bf16* p, __nv_bfloat162 (&v)[P / 2]) {
  if constexpr (P == 4) {
    const uint2 raw = *reinterpret_cast<const uint2*>(p);
    v[0] = *reinterpret_cast<const __nv_bfloat162*>(&raw.x);
    v[1] = *reinterpret_cast<const __nv_bfloat162*>(&raw.y);
  } else {
    v[0] = *reinterpret_cast<const __nv_bfloat162*>(p);
  }
}
template <int P>
__device__ __forceinline__ void load_part(const bf16* p, float2 (&v)[P / 2]) {
  if constexpr (P == 4) {
    const uint2 raw = *reinterpret_cast<const uint2*>(p);
    v[0] = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
    v[1] = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
  } else {
    v[0] = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p));
  }
}
template <int P>
__device__ __forceinline__ void store_part(bf16* p, const float2 (&v)[P / 2]) {
  if constexpr (P == 4) {
    uint2 raw;
    *reinterpret_cast<__nv_bfloat162*>(&raw.x) = __floats2bfloat162_rn(v[0].x, v[0].y);
    *reinterpret_cast<__nv_bfloat162*>(&raw.y) = __floats2bfloat162_rn(v[1].x, v[1].y);
    *reinterpret_cast<uint2*>(p) = raw;
  } else {
    *reinterpret_cast<__nv_bfloat162*>(p) = __floats2bfloat162_rn(v[0].x, v[0].y);
  }
}
template <int P>
__device__ __forceinline__ void load_f32_part(const float* p, float2 (&v)[P / 2]) {
  if constexpr (P == 4) {
    const float4 a = *reinterpret_cast<const float4*>(p);
    v[0] = make_float2(a.x, a.y);
    v[1] = make_float2(a.z, a.w);
  } else {
    v[0] = *reinterpret_cast<const float2*>(p);
  }
}
// norm weights starting at element `at`, stored as fp32 or bf16 (parameters are bf16: converting them on the host side cost a
// launch per call)
template <int P>
__device__ __forceinline__ void load_weight_part(const void* w, int w_bf16, int at, float2 (&v)[P / 2]) {
  if (w_bf16) load_part<P>(reinterpret_cast<const bf16*>(w) + at, v);
  else load_f32_part<P>(reinterpret_cast<const float*>(w) + at, v);
}
__device__ __forceinline__ float half_warp_sum(float v) {   // over the 16 lanes of this half
  v += __shfl_xor_sync(0xffffffffu, v, 8);
  v += __shfl_xor_sync(0xffffffffu, v, 4);
  v += __shfl_xor_sync(0xffffffffu, v, 2);
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v;
}
// position in the sequence of consecutive (token, head) rows
struct RowCursor {
  int s, h;
  __device__ RowCursor(long row, int S, int H) {
    const long token = row / H;
    h = (int)(row - token * H);
    s = (int)(token % S);
  }
  __device__ void advance(int rows, int S, int H) {
    h += rows;
    while (h >= H) {
      h -= H;
      if (++s == S) s = 0;
    }
  }
};

// One tensor or two of the same shape (q and k of a self-attention) in a launch: tensor blockIdx.y.
struct RmsTensors {
  const bf16* x[2];
  const void* w[2];
  int w_bf16[2];
  bf16* y[2];
  float* rstd[2];
};

// ROPE: 0 none; 1: all rows of a lane are heads of one token; 2: any tokens
template <int HD, int ROPE>
__global__ void __launch_bounds__(256) rmsnorm_rope_fwd_kernel(
    const __grid_constant__ RmsTensors tensors, const float* __restrict__ cosv, const float* __restrict__ sinv, long n_rows, int S, int H,
    float eps) {
  constexpr int P = HD / 32, Q = P / 2;
  constexpr int U = kRmsPasses;
  pdl_trigger();                     // launched with programmatic serialisation (see common.cuh)
  pdl_wait();
  const bf16* __restrict__ x = tensors.x[blockIdx.y];
  const void* __restrict__ w = tensors.w[blockIdx.y];
  const int w_bf16 = tensors.w_bf16[blockIdx.y];
  bf16* __restrict__ y = tensors.y[blockIdx.y];
  float* __restrict__ rstd_out = tensors.rstd[blockIdx.y];
  const int lane = threadIdx.x & 31, sub = lane & 15, half = lane >> 4;
  const long row0 = ((long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * (2 * U) + half;   // this lane's rows: row0 + 2u
  __nv_bfloat162 raw_lo[U][Q], raw_hi[U][Q];        // as bf16 until their pass: half the registers, one CTA more on an SM
#pragma unroll
  for (int u = 0; u < U; ++u) {
    if (row0 + 2 * u < n_rows) {
      const bf16* xr = x + (row0 + 2 * u) * HD + sub * P;
      load_raw<P>(xr, raw_lo[u]);
      load_raw<P>(xr + HD / 2, raw_hi[u]);
    } else {
#pragma unroll
      for (int j = 0; j < Q; ++j) raw_lo[u][j] = raw_hi[u][j] = __floats2bfloat162_rn(0.f, 0.f);
    }
  }
  float2 wl[Q], wh[Q];
  load_weight_part<P>(w, w_bf16, sub * P, wl);
  load_weight_part<P>(w, w_bf16, HD / 2 + sub * P, wh);
  float2 c[ROPE == 2 ? U : 1][Q], sn[ROPE == 2 ? U : 1][Q];
  if (ROPE != 0) {
    RowCursor token(row0 < n_rows ? row0 : 0, S, H);
#pragma unroll
    for (int u = 0; u < (ROPE == 2 ? U : 1); ++u) {
      if (row0 + 2 * u < n_rows) {
        load_f32_part<P>(cosv + (long)token.s * (HD / 2) + sub * P, c[u]);
        load_f32_part<P>(sinv + (long)token.s * (HD / 2) + sub * P, sn[u]);
      }
      token.advance(2, S, H);
    }
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const long row = row0 + 2 * u;
    const bool valid = row < n_rows;          // both halves run every shuffle; only the accesses are predicated
    float2 lo[Q], hi[Q];
#pragma unroll
    for (int j = 0; j < Q; ++j) {
      lo[j] = __bfloat1622float2(raw_lo[u][j]);
      hi[j] = __bfloat1622float2(raw_hi[u][j]);
    }
    float2 ss2 = make_float2(0.f, 0.f);
#pragma unroll
    for (int j = 0; j < Q; ++j) ss2 = fma2(hi[j], hi[j], fma2(lo[j], lo[j], ss2));
    const float ss = half_warp_sum(ss2.x + ss2.y);
    const float rstd = rsqrtf(ss / HD + eps);
    if (sub == 0 && valid) rstd_out[row] = rstd;
    const float2 rs2 = make_float2(rstd, rstd);
#pragma unroll
    for (int j = 0; j < Q; ++j) {
      lo[j] = mul2(mul2(lo[j], rs2), wl[j]);
      hi[j] = mul2(mul2(hi[j], rs2), wh[j]);
    }
    if (ROPE != 0) {
      constexpr int kTables = ROPE == 2 ? U : 1;
      const float2(&cu)[Q] = c[u < kTables ? u : 0];
      const float2(&su)[Q] = sn[u < kTables ? u : 0];
#pragma unroll
      for (int j = 0; j < Q; ++j) {
        const float2 a = lo[j], b = hi[j], ns = make_float2(-su[j].x, -su[j].y);
        lo[j] = fma2(b, ns, mul2(a, cu[j]));
        hi[j] = fma2(a, su[j], mul2(b, cu[j]));
      }
    }
    if (valid) {
      bf16* yr = y + row * HD + sub * P;
      store_part<P>(yr, lo);
      store_part<P>(yr + HD / 2, hi);
    }
  }
}

// backward: `rows_per_warp` consecutive rows per warp (two per pass) to amortise the weight-gradient partial.
template <int HD>
__global__ void __launch_bounds__(256) rmsnorm_rope_bwd_kernel(
    const bf16* __restrict__ dy, const bf16* __restrict__ x, const void* __restrict__ w, int w_bf16,
    const float* __restrict__ rstd_in, const float* __restrict__ cosv, const float* __restrict__ sinv,
    bf16* __restrict__ dx, float* __restrict__ dw_partials, long n_rows, int S, int H, int rows_per_warp) {
  constexpr int P = HD / 32, Q = P / 2;
  __shared__ float sm[8][HD];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane & 15, half = lane >> 4;
  const long warp_global = (long)blockIdx.x * 8 + warp;
  const long r0 = warp_global * rows_per_warp;
  const long r_end = min(r0 + (long)rows_per_warp, n_rows);
  float2 wl[Q], wh[Q], dwl[Q], dwh[Q];
  load_weight_part<P>(w, w_bf16, sub * P, wl);
  load_weight_part<P>(w, w_bf16, HD / 2 + sub * P, wh);
#pragma unroll
  for (int j = 0; j < Q; ++j) dwl[j] = dwh[j] = make_float2(0.f, 0.f);
  constexpr int U = 4;      // passes (of two rows) whose loads are in flight together
  RowCursor at(min(r0 + half, n_rows - 1), S, H);
  for (long rb = r0; rb < r_end; rb += 2 * U) {
    float2 dl[U][Q], dh[U][Q], xl[U][Q], xh[U][Q];
    float rsU[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long row = rb + 2 * u + half;
      if (row < r_end) {
        load_part<P>(dy + row * HD + sub * P, dl[u]);
        load_part<P>(dy + row * HD + HD / 2 + sub * P, dh[u]);
        load_part<P>(x + row * HD + sub * P, xl[u]);
        load_part<P>(x + row * HD + HD / 2 + sub * P, xh[u]);
        rsU[u] = rstd_in[row];
      } else {
#pragma unroll
        for (int j = 0; j < Q; ++j) dl[u][j] = dh[u][j] = xl[u][j] = xh[u][j] = make_float2(0.f, 0.f);
        rsU[u] = 0.f;
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long row = rb + 2 * u + half;
      const bool valid = row < r_end;
      if (cosv != nullptr && valid) {
        float2 c[Q], sn[Q];
        load_f32_part<P>(cosv + (long)at.s * (HD / 2) + sub * P, c);
        load_f32_part<P>(sinv + (long)at.s * (HD / 2) + sub * P, sn);
#pragma unroll
        for (int j = 0; j < Q; ++j) {
          const float2 a = dl[u][j], b = dh[u][j], ns = make_float2(-sn[j].x, -sn[j].y);
          dl[u][j] = fma2(b, sn[j], mul2(a, c[j]));
          dh[u][j] = fma2(a, ns, mul2(b, c[j]));
        }
      }
      const float rstd = rsU[u];
      const float2 rs2 = make_float2(rstd, rstd);
      float2 dot2 = make_float2(0.f, 0.f);
#pragma unroll
      for (int j = 0; j < Q; ++j) {
        dwl[j] = fma2(mul2(dl[u][j], xl[u][j]), rs2, dwl[j]);
        dwh[j] = fma2(mul2(dh[u][j], xh[u][j]), rs2, dwh[j]);
        dl[u][j] = mul2(dl[u][j], wl[j]);
        dh[u][j] = mul2(dh[u][j], wh[j]);
        dot2 = fma2(dh[u][j], xh[u][j], fma2(dl[u][j], xl[u][j], dot2));
      }
      const float dot = half_warp_sum(dot2.x + dot2.y);
      const float k = dot * rstd * rstd * rstd / HD;
      const float2 nk = make_float2(-k, -k);
#pragma unroll
      for (int j = 0; j < Q; ++j) {
        dl[u][j] = fma2(xl[u][j], nk, mul2(dl[u][j], rs2));
        dh[u][j] = fma2(xh[u][j], nk, mul2(dh[u][j], rs2));
      }
      if (valid) {
        store_part<P>(dx + row * HD + sub * P, dl[u]);
        store_part<P>(dx + row * HD + HD / 2 + sub * P, dh[u]);
      }
      at.advance(2, S, H);
    }
  }
  // the two halves of the warp hold partial sums of the same columns
#pragma unroll
  for (int j = 0; j < Q; ++j) {
    dwl[j].x += __shfl_xor_sync(0xffffffffu, dwl[j].x, 16);
    dwl[j].y += __shfl_xor_sync(0xffffffffu, dwl[j].y, 16);
    dwh[j].x += __shfl_xor_sync(0xffffffffu, dwh[j].x, 16);
    dwh[j].y += __shfl_xor_sync(0xffffffffu, dwh[j].y, 16);
  }
  if (half == 0) {
#pragma unroll
    for (int j = 0; j < Q; ++j) {
      sm[warp][sub * P + 2 * j] = dwl[j].x;
      sm[warp][sub * P + 2 * j + 1] = dwl[j].y;
      sm[warp][HD / 2 + sub * P + 2 * j] = dwh[j].x;
      sm[warp][HD / 2 + sub * P + 2 * j + 1] = dwh[j].y;
    }
  }
  __syncthreads();
  if (threadIdx.x < HD) {
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) s += sm[k][threadIdx.x];
    dw_partials[(long)blockIdx.x * HD + threadIdx.x] = s;
  }
}

// ------------------------------------------------------------------------------------------------
// GELU (erf), elementwise
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ float gelu_f(float x) { return 0.5f * x * (1.f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad_f(float x) {
  const float cdf = 0.5f * (1.f + erff(x * 0.70710678118654752f));
  const float pdf = 0.39894228040143268f * __expf(-0.5f * x * x);
  return cdf + x * pdf;
}

__global__ void __launch_bounds__(kThreads) gelu_fwd_kernel(const bf16* __restrict__ x, bf16* __restrict__ y, long nvec) {
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < nvec; i += (long)gridDim.x * blockDim.x) {
    float a[8];
    unpack8(reinterpret_cast<const bf16x8*>(x)[i], a);
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] = gelu_f(a[j]);
    reinterpret_cast<bf16x8*>(y)[i] = pack8(a);
  }
}

__global__ void __launch_bounds__(kThreads) gelu_bwd_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ x,
                                                             bf16* __restrict__ dx, long nvec) {
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < nvec; i += (long)gridDim.x * blockDim.x) {
    float a[8], d[8];
    unpack8(reinterpret_cast<const bf16x8*>(x)[i], a);
    unpack8(reinterpret_cast<const bf16x8*>(dy)[i], d);
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] = d[j] * gelu_grad_f(a[j]);
    reinterpret_cast<bf16x8*>(dx)[i] = pack8(a);
  }
}

__global__ void __launch_bounds__(kThreads) cfg_combine_kernel(const float* __restrict__ c, const float* __restrict__ u,
                                                                float* __restrict__ o, float g, long n) {
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    o[i] = c[i] + g * (c[i] - u[i]);
}

// ------------------------------------------------------------------------------------------------
// optimizer path
// ------------------------------------------------------------------------------------------------
// g32 = scrub(scale * g16); partial[blockIdx] = sum g32^2
__global__ void __launch_bounds__(kThreads) grad_cast_norm_kernel(const bf16* __restrict__ g16, float* __restrict__ g32,
                                                                   float* __restrict__ partials, float scale, long n) {
  __shared__ float red[32];
  float ss = 0.f;
  const long nvec = n >> 3;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < nvec; i += (long)gridDim.x * blockDim.x) {
    float a[8];
    unpack8(reinterpret_cast<const bf16x8*>(g16)[i], a);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      a[j] = scrub(a[j] * scale);
      ss += a[j] * a[j];
    }
    store_f8(g32 + i * 8, a);
  }
  if (blockIdx.x == 0) {
    for (long i = (nvec << 3) + threadIdx.x; i < n; i += blockDim.x) {
      const float a = scrub(__bfloat162float(g16[i]) * scale);
      g32[i] = a;
      ss += a * a;
    }
  }
  const float t = block_sum(ss, red);
  if (threadIdx.x == 0) partials[blockIdx.x] = t;
}

__global__ void sum_partials_kernel(const float* __restrict__ partials, float* __restrict__ out, int n) {
  __shared__ float red[32];
  float s = 0.f;
  for (int i = threadIdx.x; i < n; i += blockDim.x) s += partials[i];
  s = block_sum(s, red);
  if (threadIdx.x == 0) out[0] = s;
}

__global__ void __launch_bounds__(kThreads) adamw_ema_shard_kernel(
    float* __restrict__ master, const float* __restrict__ grad, float* __restrict__ m, float* __restrict__ v,
    float* __restrict__ ema, bf16* __restrict__ out16, const float* __restrict__ clip_coef, float lr, float beta1,
    float beta2, float eps, float wd, float bc1, float rsqrt_bc2, float ema_beta, long n) {
  const float clip = clip_coef ? clip_coef[0] : 1.f;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const float g = grad[i] * clip;
    float p = master[i] * (1.f - lr * wd);
    const float mi = beta1 * m[i] + (1.f - beta1) * g;
    const float vi = beta2 * v[i] + (1.f - beta2) * g * g;
    const float denom = sqrtf(vi) * rsqrt_bc2 + eps;
    p -= (lr / bc1) * (mi / denom);
    master[i] = p;
    m[i] = mi;
    v[i] = vi;
    if (ema != nullptr && ema_beta >= 0.f) ema[i] = ema_beta * ema[i] + (1.f - ema_beta) * p;
    if (out16 != nullptr) out16[i] = __float2bfloat16(p);
  }
}

__global__ void __launch_bounds__(kThreads) cast_f32_bf16_kernel(const float* __restrict__ src, bf16* __restrict__ dst, long n) {
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    dst[i] = __float2bfloat16(src[i]);
}

static inline int grid_for(long n, int threads, int max_blocks = 148 * 8) {
  long b = (n + threads - 1) / threads;
  if (b < 1) b = 1;
  return (int)(b > max_blocks ? max_blocks : b);
}

}  // namespace cb200

using namespace cb200;

// ------------------------------------------------------------------------------------------------
// host launchers
// ------------------------------------------------------------------------------------------------
extern "C" {

int cb200_ln_groups_per_frame(int L, int rows_per_cta) { return (L + rows_per_cta - 1) / rows_per_cta; }

void cb200_ln_modulate_fwd(const void* x, const float* shift, const float* scale, void* y, float* mean, float* rstd,
                           long rows, int D, int L, long ld_shift, long ld_scale, float eps, cudaStream_t st) {
  auto by_row = [&](auto kern, int threads, int per_cta) {
    launch_pdl(kern, dim3((unsigned)((rows + per_cta - 1) / per_cta)), dim3(threads * per_cta), 0, st, (const bf16*)x, shift, scale, (bf16*)y, mean, rstd, rows,
               D, L, ld_shift, ld_scale, eps);
  };
  // Many rows that a warp holds, where a walk over a frame's rows has little to walk over (frames of up to three rows) or few CTAs would walk
  // (rows of 256: 8192 in frames of 16 4.1 us by warp and 4.8 in batches, 16,384 7.3 and 7.2): a warp for each.
  if (D <= 512 && rows >= 2048 && (L < 4 || (D <= 256 && rows >= 3072 && rows < 12288))) {
    if (D <= 256) by_row(ln_modulate_fwd_row_kernel<1, 32, 8>, 32, 8); else by_row(ln_modulate_fwd_row_kernel<2, 32, 8>, 32, 8);
    return;
  }
  // Few rows (or frames of fewer rows than a CTA takes at a time): a CTA for each. The line: 2048 rows of 2048 6.4 us that way and 6.2 us in
  // batches, 1024 rows 3.7 and 4.4; 1024 rows of 5120 8.6 and 6.9, 512 rows 4.9 and 6.3.
  if (rows < (D <= 2048 ? 2048 : 1024) || L < 4) {
    if (D <= 1024) by_row(ln_modulate_fwd_row_kernel<1, 128, 1>, 128, 1);
    else if (D <= 2048) by_row(ln_modulate_fwd_row_kernel<2, 128, 1>, 128, 1);
    else if (D <= 4096) by_row(ln_modulate_fwd_row_kernel<2, 256, 1>, 256, 1);
    else by_row(ln_modulate_fwd_row_kernel<4, 256, 1>, 256, 1);
    return;
  }
  // rows of a CTA: two waves of CTAs while they are few, at most 20 (longer walks leave the last wave emptier)
  const int resident = 148 * (D <= 512 ? 12 : D <= 1024 ? 6 : D <= 2048 ? 3 : 2);
  const int per = (int)std::min<long>((rows / (2 * resident) + 4) / 4 * 4, 20);
  const int groups = (L + per - 1) / per, nvec = D / 8;
  auto launch = [&](auto kern, int nv) {
    const int threads = ((nvec + nv - 1) / nv + 31) / 32 * 32;
    launch_pdl(kern, dim3((unsigned)(rows / L * groups)), dim3(threads), 0, st, (const bf16*)x, shift, scale, (bf16*)y, mean, rstd, D, L, per, groups,
               ld_shift, ld_scale, eps);
  };
  if (D <= 2048) launch(ln_modulate_fwd_rows_kernel<1, 256, 4, 3>, 1);
  else if (D <= 5120) launch(ln_modulate_fwd_rows_kernel<2, 320, 2, 2>, 2);
  else launch(ln_modulate_fwd_rows_kernel<2, 512, 2, 1>, 2);
}

void cb200_ln_modulate_bwd(const void* dy, const void* x, const float* mean, const float* rstd, const float* scale,
                           void* dx, float* dshift, float* dscale, float* partials, long frames, int D, int L,
                           int rows_per_cta, long ld_scale, cudaStream_t st) {
  const int G = cb200_ln_groups_per_frame(L, rows_per_cta);
#define LAUNCH(MV) ln_modulate_bwd_kernel<MV><<<(unsigned)(frames * G), kThreads, 0, st>>>((const bf16*)dy, (const bf16*)x, mean, rstd, scale, (bf16*)dx, partials, D, L, rows_per_cta, G, ld_scale)
  if (D <= 2048) LAUNCH(1); else if (D <= 4096) LAUNCH(2); else LAUNCH(4);
#undef LAUNCH
  dim3 grid((D + 255) / 256, (unsigned)frames);
  reduce_partials_kernel<<<grid, 256, 0, st>>>(partials, dshift, dscale, D, G, 2);
}

void cb200_gate_residual_fwd(const void* x, const float* gate, const void* y, void* out, long rows, int D, int L,
                             long ld_gate, cudaStream_t st) {
  const long nvec = rows * (D >> 3);
  gate_residual_fwd_kernel<<<grid_for(nvec, kThreads, 148 * 16), kThreads, 0, st>>>((const bf16*)x, gate, (const bf16*)y,
                                                                                    (bf16*)out, nvec, D, L, ld_gate);
}

void cb200_gate_residual_bwd(const void* dout, const float* gate, const void* y, void* dy, float* dgate, float* partials,
                             long frames, int D, int L, int rows_per_cta, long ld_gate, cudaStream_t st) {
  const int G = cb200_ln_groups_per_frame(L, rows_per_cta);
#define LAUNCH(MV) gate_residual_bwd_kernel<MV><<<(unsigned)(frames * G), kThreads, 0, st>>>((const bf16*)dout, gate, (const bf16*)y, (bf16*)dy, partials, D, L, rows_per_cta, G, ld_gate)
  if (D <= 2048) LAUNCH(1); else if (D <= 4096) LAUNCH(2); else LAUNCH(4);
#undef LAUNCH
  dim3 grid((D + 255) / 256, (unsigned)frames);
  reduce_partials_kernel<<<grid, 256, 0, st>>>(partials, dgate, nullptr, D, G, 1);
}

static void launch_rmsnorm_rope_fwd(const RmsTensors& tensors, int n, const float* cosv, const float* sinv, long n_rows, int S, int H, int HD,
                                    float eps, cudaStream_t st) {
  const dim3 blocks((unsigned)((n_rows + 16 * kRmsPasses - 1) / (16 * kRmsPasses)), n);   // 8 warps x 2 rows x passes per CTA
  auto launch = [&](auto kern) { launch_pdl(kern, blocks, dim3(256), 0, st, tensors, cosv, sinv, n_rows, S, H, eps); };
  const bool one_token = H % (2 * kRmsPasses) == 0;
  if (cosv == nullptr) HD == 128 ? launch(rmsnorm_rope_fwd_kernel<128, 0>) : launch(rmsnorm_rope_fwd_kernel<64, 0>);
  else if (one_token) HD == 128 ? launch(rmsnorm_rope_fwd_kernel<128, 1>) : launch(rmsnorm_rope_fwd_kernel<64, 1>);
  else HD == 128 ? launch(rmsnorm_rope_fwd_kernel<128, 2>) : launch(rmsnorm_rope_fwd_kernel<64, 2>);
}

void cb200_rmsnorm_rope_fwd(const void* x, const void* w, int w_bf16, const float* cosv, const float* sinv, void* y, float* rstd,
                            long n_rows, int S, int H, int HD, float eps, cudaStream_t st) {
  launch_rmsnorm_rope_fwd({{(const bf16*)x}, {w}, {w_bf16}, {(bf16*)y}, {rstd}}, 1, cosv, sinv, n_rows, S, H, HD, eps, st);
}

void cb200_rmsnorm_rope_fwd_pair(const void* const* x, const void* const* w, const int* w_bf16, const float* cosv, const float* sinv,
                                 void* const* y, float* const* rstd, long n_rows, int S, int H, int HD, float eps, cudaStream_t st) {
  launch_rmsnorm_rope_fwd({{(const bf16*)x[0], (const bf16*)x[1]}, {w[0], w[1]}, {w_bf16[0], w_bf16[1]}, {(bf16*)y[0], (bf16*)y[1]},
                           {rstd[0], rstd[1]}}, 2, cosv, sinv, n_rows, S, H, HD, eps, st);
}

long cb200_rmsnorm_bwd_blocks(long n_rows, int rows_per_warp) {
  const long warps = (n_rows + rows_per_warp - 1) / rows_per_warp;
  return (warps + 7) / 8;
}

void cb200_rmsnorm_rope_bwd(const void* dy, const void* x, const void* w, int w_bf16, const float* rstd, const float* cosv,
                            const float* sinv, void* dx, float* dw, float* partials, long n_rows, int S, int H, int HD,
                            int rows_per_warp, cudaStream_t st) {
  const long blocks = cb200_rmsnorm_bwd_blocks(n_rows, rows_per_warp);
  if (HD == 128)
    rmsnorm_rope_bwd_kernel<128><<<(unsigned)blocks, 256, 0, st>>>((const bf16*)dy, (const bf16*)x, w, w_bf16, rstd, cosv, sinv,
                                                                   (bf16*)dx, partials, n_rows, S, H, rows_per_warp);
  else
    rmsnorm_rope_bwd_kernel<64><<<(unsigned)blocks, 256, 0, st>>>((const bf16*)dy, (const bf16*)x, w, w_bf16, rstd, cosv, sinv,
                                                                  (bf16*)dx, partials, n_rows, S, H, rows_per_warp);
  reduce_rows_kernel<<<(HD + 31) / 32, 1024, 0, st>>>(partials, dw, HD, (int)blocks);
}

void cb200_gelu_fwd(const void* x, void* y, long n, cudaStream_t st) {
  gelu_fwd_kernel<<<grid_for(n >> 3, kThreads, 148 * 16), kThreads, 0, st>>>((const bf16*)x, (bf16*)y, n >> 3);
}

void cb200_gelu_bwd(const void* dy, const void* x, void* dx, long n, cudaStream_t st) {
  gelu_bwd_kernel<<<grid_for(n >> 3, kThreads, 148 * 16), kThreads, 0, st>>>((const bf16*)dy, (const bf16*)x, (bf16*)dx, n >> 3);
}

void cb200_cfg_combine(const float* c, const float* u, float* o, float g, long n, cudaStream_t st) {
  cfg_combine_kernel<<<grid_for(n, kThreads), kThreads, 0, st>>>(c, u, o, g, n);
}

int cb200_grad_cast_norm_blocks(long n) { return grid_for(n >> 3, kThreads, 148 * 4); }

void cb200_grad_cast_norm(const void* g16, float* g32, float* sumsq, float* partials, float scale, long n, cudaStream_t st) {
  const int blocks = cb200_grad_cast_norm_blocks(n);
  grad_cast_norm_kernel<<<blocks, kThreads, 0, st>>>((const bf16*)g16, g32, partials, scale, n);
  sum_partials_kernel<<<1, 256, 0, st>>>(partials, sumsq, blocks);
}

void cb200_adamw_ema_shard(float* master, const float* grad, float* m, float* v, float* ema, void* out16,
                           const float* clip_coef, float lr, float beta1, float beta2, float eps, float wd, long step,
                           float ema_beta, long n, cudaStream_t st) {
  const float bc1 = 1.f - powf(beta1, (float)step);
  const float bc2 = 1.f - powf(beta2, (float)step);
  adamw_ema_shard_kernel<<<grid_for(n, kThreads, 148 * 8), kThreads, 0, st>>>(
      master, grad, m, v, ema, (bf16*)out16, clip_coef, lr, beta1, beta2, eps, wd, bc1, 1.f / sqrtf(bc2), ema_beta, n);
}

void cb200_cast_f32_bf16(const float* src, void* dst, long n, cudaStream_t st) {
  cast_f32_bf16_kernel<<<grid_for(n, kThreads, 148 * 8), kThreads, 0, st>>>(src, (bf16*)dst, n);
}

}  // extern "C"
