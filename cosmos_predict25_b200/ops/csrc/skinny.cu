// Batched fp32 GEMM for "skinny" problems: a handful of rows (batch x frames of timestep embeddings) against many small weight
// matrices, e.g. the 3 AdaLN-LoRA modulation MLPs of every transformer block and the timestep embedder
// (cosmos_predict2/_src/predict2/networks/minimal_v4_dit.py:776-783, 1131-1162). These run in fp32 (the fp32 island of the
// reference) on a few dozen rows: too few rows for a 128-row tensor-core tile and too many launches as single library GEMMs
// (2 per MLP, 85 MLPs per forward). One launch computes all Z problems
//
//     C[z][r, n] = sum_k fa(A[z][r, k]) * fb(B[z][n, k])  (+ add[r, n] for n < add_cols)
//
// with arbitrary element strides for A and B, so that the same kernel serves the forward (B = weight, k contiguous), the input
// gradient (B = weight read along its rows) and the weight gradient (the reduction runs over the few rows). A is fp32, B is
// bf16 or fp32 and is addressed through a pointer table (weights of different modules) or a base pointer + stride; fa / fb are
// identity or SiLU. Accumulation is fp32 on the CUDA cores in a fixed order: the result is deterministic.

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "common.cuh"
#include "launchers.h"
#include "sm100.cuh"

namespace cb200 {

struct SkinnyParams {
  const float* a;
  long a_z, a_r, a_k;
  const long long* b_ptrs;   // per-problem base addresses of B, or nullptr
  const void* b_base;
  long b_z, b_n, b_k;
  void* c;
  long c_z;
  int ldc;
  const float* add;
  int ld_add, add_cols;
  int R, N, K;
  int silu_a, silu_b;
  int ksplit;   // the reduction is cut into this many ranges; range s of problem z writes C[z * ksplit + s]
};

constexpr int kSkTile = 64;     // rows and columns of C per CTA
constexpr int kSkK = 32;        // reduction elements per shared-memory stage
constexpr int kSkLd = kSkTile + 4;

__device__ __forceinline__ float silu_f(float v) { return v / (1.f + __expf(-v)); }
__device__ __forceinline__ float to_f32(float v) { return v; }
__device__ __forceinline__ float to_f32(__nv_bfloat16 v) { return __bfloat162float(v); }
__device__ __forceinline__ void store_c(float* p, float v) { *p = v; }
__device__ __forceinline__ void store_c(__nv_bfloat16* p, float v) { *p = __float2bfloat16_rn(v); }

template <typename TB, typename TC>
__global__ void __launch_bounds__(256, 2) skinny_bgemm_kernel(SkinnyParams p) {
  __shared__ __align__(16) float As[kSkK][kSkLd];
  __shared__ __align__(16) float Bs[kSkK][kSkLd];
  const int z = blockIdx.z / p.ksplit, ks = blockIdx.z % p.ksplit;
  const int k_per = ((p.K + p.ksplit - 1) / p.ksplit + kSkK - 1) / kSkK * kSkK;
  const int k_lo = ks * k_per, k_hi = min(p.K, k_lo + k_per);
  const int r0 = blockIdx.y * kSkTile, n0 = blockIdx.x * kSkTile;
  const float* A = p.a + (long)z * p.a_z;
  const TB* B = p.b_ptrs ? reinterpret_cast<const TB*>(p.b_ptrs[z]) : reinterpret_cast<const TB*>(p.b_base) + (long)z * p.b_z;
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  // the thread index runs along whichever of (row, k) is contiguous in memory
  const bool a_k_fast = p.a_k == 1, b_k_fast = p.b_k == 1;
  for (int k0 = k_lo; k0 < k_hi; k0 += kSkK) {
#pragma unroll
    for (int it = 0; it < kSkTile * kSkK / 256; ++it) {
      const int idx = it * 256 + tid;
      {
        const int kk = a_k_fast ? idx % kSkK : idx / kSkTile, rr = a_k_fast ? idx / kSkK : idx % kSkTile;
        const int r = r0 + rr, k = k0 + kk;
        float v = 0.f;
        if (r < p.R && k < k_hi) {
          v = A[(long)r * p.a_r + (long)k * p.a_k];
          if (p.silu_a) v = silu_f(v);
        }
        As[kk][rr] = v;
      }
      {
        const int kk = b_k_fast ? idx % kSkK : idx / kSkTile, nn = b_k_fast ? idx / kSkK : idx % kSkTile;
        const int n = n0 + nn, k = k0 + kk;
        float v = 0.f;
        if (n < p.N && k < k_hi) {
          v = to_f32(B[(long)n * p.b_n + (long)k * p.b_k]);
          if (p.silu_b) v = silu_f(v);
        }
        Bs[kk][nn] = v;
      }
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < kSkK; ++kk) {
      const float4 a4 = *reinterpret_cast<const float4*>(&As[kk][ty * 4]);
      const float4 b4 = *reinterpret_cast<const float4*>(&Bs[kk][tx * 4]);
      const float av[4] = {a4.x, a4.y, a4.z, a4.w}, bv[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
    }
    __syncthreads();
  }
  TC* C = reinterpret_cast<TC*>(p.c) + (long)blockIdx.z * p.c_z;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = r0 + ty * 4 + i;
    if (r >= p.R) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + tx * 4 + j;
      if (n >= p.N) continue;
      float v = acc[i][j];
      if (p.add != nullptr && ks == 0 && n < p.add_cols) v += p.add[(long)r * p.ld_add + n];
      store_c(C + (long)r * p.ldc + n, v);
    }
  }
}

// ------------------------------------------------------------------------------------------------------------------------------
// The same contraction for bf16 weights and row-major A (every forward and input-gradient call of the modulation MLPs): the weights
// are read once and bound the kernel while there are few rows (84 weights of 6144 x 256: 264 MB), the fp32 multiply-adds beyond
// about twenty. A CTA owns 256 columns x RT rows: each of its 128 threads keeps 2 columns x RT rows in registers and adds two rows
// per instruction (packed fp32). Weights pass through two 64-deep stages filled by cp.async; activations (SiLU applied) lie
// transposed beside them, so that all lanes read one address. Per MLP pair of the 28-block network's 84 MLPs, 2 / 48 rows: 2.10 / 2.96 ms with the
// 64 x 64 tile above, 0.14 / 0.87 ms here.
// KFAST: the reduction index is contiguous in the weight (forward); otherwise the column index is (input gradient).
constexpr int kFsN = 256, kFsK = 64, kFsThreads = 128;
constexpr int kFsPitchK = kFsK + 8;      // bf16 per column row, KFAST: 144 bytes, no bank conflicts for 16-byte reads
constexpr int kFsPitchN = kFsN + 8;      // bf16 per reduction row otherwise
template <int RT, bool KFAST>
struct FsShape {
  static constexpr int kW = KFAST ? kFsN * kFsPitchK : kFsK * kFsPitchN;   // bf16 elements of a weight stage
  static constexpr int kA = kFsK * RT;                                     // floats of an activation stage
  static constexpr size_t kSmem = 2 * (size_t)(kW * 2 + kA * 4);
};

__device__ __forceinline__ void cp_async16(void* dst, const void* src, int bytes) {   // the rest of the 16 bytes is zeroed
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}

template <int RT, bool KFAST>
__global__ void __launch_bounds__(kFsThreads) skinny_wide_kernel(SkinnyParams p) {
  using Sh = FsShape<RT, KFAST>;
  pdl_trigger();                       // launched with programmatic serialisation (see common.cuh)
  pdl_wait();
  extern __shared__ __align__(16) uint8_t fs_smem[];
  __nv_bfloat16* Ws = reinterpret_cast<__nv_bfloat16*>(fs_smem);
  float* As = reinterpret_cast<float*>(fs_smem + 2 * (size_t)Sh::kW * 2);
  const int z = blockIdx.z / p.ksplit, ks = blockIdx.z % p.ksplit;
  const int k_per = ((p.K + p.ksplit - 1) / p.ksplit + kFsK - 1) / kFsK * kFsK;
  const int k_lo = min(p.K, ks * k_per), k_hi = min(p.K, k_lo + k_per);
  const int r0 = blockIdx.y * RT, n0 = blockIdx.x * kFsN;
  const float* A = p.a + (long)z * p.a_z;
  const __nv_bfloat16* B = p.b_ptrs ? reinterpret_cast<const __nv_bfloat16*>(p.b_ptrs[z])
                                    : reinterpret_cast<const __nv_bfloat16*>(p.b_base) + (long)z * p.b_z;
  const int tid = threadIdx.x;
  // a weight that does not start on a 16-byte boundary (a slice of a larger buffer) is staged element by element
  const bool vec = (reinterpret_cast<uintptr_t>(B) & 15) == 0;

  auto stage_w = [&](int buf, int k0) {
    __nv_bfloat16* w = Ws + buf * Sh::kW;
    constexpr int kPer = KFAST ? kFsK / 8 : kFsN / 8;                 // 16-byte pieces per shared-memory row
    constexpr int kRows = KFAST ? kFsN : kFsK;
#pragma unroll 4
    for (int i = tid; i < kRows * kPer; i += kFsThreads) {
      const int row = i / kPer, piece = i % kPer;
      const int n = n0 + (KFAST ? row : piece * 8), k = k0 + (KFAST ? piece * 8 : row);
      __nv_bfloat16* dst = w + row * (KFAST ? kFsPitchK : kFsPitchN) + piece * 8;
      const bool in = n < p.N && k < k_hi;
      const int left = in ? min(8, KFAST ? k_hi - k : p.N - n) : 0;   // valid elements of the piece
      const __nv_bfloat16* src = B + (in ? (long)n * p.b_n + (long)k * p.b_k : 0);
      if (vec) {
        cp_async16(dst, src, left * 2);
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) dst[j] = j < left ? src[j] : __float2bfloat16(0.f);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // consecutive threads take consecutive rows: conflict-free transposed stores; A is small and stays in L2
  constexpr int kALoads = (RT * (kFsK / 4) + kFsThreads - 1) / kFsThreads;
  float4 av[kALoads];
  auto load_a = [&](int k0) {
#pragma unroll
    for (int i = 0; i < kALoads; ++i) {
      const int idx = tid + i * kFsThreads, r = idx % RT, k = k0 + idx / RT * 4;
      float v[4] = {0.f, 0.f, 0.f, 0.f};
      if (idx < RT * (kFsK / 4) && r0 + r < p.R) {
        const float* src = A + (long)(r0 + r) * p.a_r + k;
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (k + j < k_hi) v[j] = src[j];
      }
      av[i] = make_float4(v[0], v[1], v[2], v[3]);
    }
  };
  auto store_a = [&](int buf) {
    float* a = As + buf * Sh::kA;
#pragma unroll
    for (int i = 0; i < kALoads; ++i) {
      const int idx = tid + i * kFsThreads, r = idx % RT, k = idx / RT * 4;
      if (idx < RT * (kFsK / 4)) {
        float v[4] = {av[i].x, av[i].y, av[i].z, av[i].w};
#pragma unroll
        for (int j = 0; j < 4; ++j) a[(k + j) * RT + r] = p.silu_a ? silu_f(v[j]) : v[j];
      }
    }
  };

  float2 acc[2][RT / 2];
#pragma unroll
  for (int c = 0; c < 2; ++c)
#pragma unroll
    for (int i = 0; i < RT / 2; ++i) acc[c][i] = make_float2(0.f, 0.f);
  // this thread's two columns: neighbours when the column index is contiguous in the weight, else 128 apart
  const int c0 = KFAST ? tid : 2 * tid, c1 = KFAST ? tid + kFsThreads : 2 * tid + 1;

  int buf = 0;
  if (k_lo < k_hi) {
    stage_w(0, k_lo);
    load_a(k_lo);
    store_a(0);
  }
  for (int k0 = k_lo; k0 < k_hi; k0 += kFsK, buf ^= 1) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                       // this stage is in, and everybody is done with the other one
    const bool more = k0 + kFsK < k_hi;
    if (more) {
      stage_w(buf ^ 1, k0 + kFsK);
      load_a(k0 + kFsK);
    }
    const __nv_bfloat16* w = Ws + buf * Sh::kW;
    const float* a = As + buf * Sh::kA;
#pragma unroll 1
    for (int kk = 0; kk < kFsK; kk += 8) {
      float w0[8], w1[8];
      if (KFAST) {
        unpack8(*reinterpret_cast<const bf16x8*>(w + c0 * kFsPitchK + kk), w0);
        unpack8(*reinterpret_cast<const bf16x8*>(w + c1 * kFsPitchK + kk), w1);
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(w + (kk + j) * kFsPitchN + c0));
          w0[j] = f.x;
          w1[j] = f.y;
        }
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float2 x0 = make_float2(w0[j], w0[j]), x1 = make_float2(w1[j], w1[j]);
        const float4* ar = reinterpret_cast<const float4*>(a + (kk + j) * RT);
#pragma unroll
        for (int i = 0; i < RT / 4; ++i) {
          const float4 v = ar[i];
          acc[0][2 * i] = sm100::fma2(make_float2(v.x, v.y), x0, acc[0][2 * i]);
          acc[0][2 * i + 1] = sm100::fma2(make_float2(v.z, v.w), x0, acc[0][2 * i + 1]);
          acc[1][2 * i] = sm100::fma2(make_float2(v.x, v.y), x1, acc[1][2 * i]);
          acc[1][2 * i + 1] = sm100::fma2(make_float2(v.z, v.w), x1, acc[1][2 * i + 1]);
        }
      }
    }
    if (more) store_a(buf ^ 1);            // read by nobody before the next barrier
  }
  float* C = reinterpret_cast<float*>(p.c) + (long)blockIdx.z * p.c_z;
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    const int n = n0 + (c == 0 ? c0 : c1);
    if (n >= p.N) continue;
    const bool plus = p.add != nullptr && ks == 0 && n < p.add_cols;
#pragma unroll
    for (int i = 0; i < RT; ++i) {
      const int r = r0 + i;
      if (r >= p.R) break;
      float v = (i & 1) ? acc[c][i / 2].y : acc[c][i / 2].x;
      if (plus) v += p.add[(long)r * p.ld_add + n];
      C[(long)r * p.ldc + n] = v;
    }
  }
}

template <int RT, bool KFAST>
static int launch_skinny_wide(const SkinnyParams& p, int Z, cudaStream_t st) {
  using Sh = FsShape<RT, KFAST>;
  static bool attr = false;
  if (!attr) {
    cudaError_t e = cudaFuncSetAttribute(skinny_wide_kernel<RT, KFAST>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Sh::kSmem);
    if (e != cudaSuccess) return 100 + (int)e;
    attr = true;
  }
  dim3 grid((p.N + kFsN - 1) / kFsN, (p.R + RT - 1) / RT, Z * p.ksplit);
  return (int)launch_pdl(skinny_wide_kernel<RT, KFAST>, grid, dim3(kFsThreads), Sh::kSmem, st, p);
}

// ------------------------------------------------------------------------------------------------------------------------------
// The same for up to four rows and K <= 2048: the weights, read once, are what counts, then the sums over the lanes. A lane keeps its eight
// elements of the rows in registers for good (which is what ends at 2048: eight warps of 256 elements to a weight row) and takes one 16-byte
// piece of eight weight rows at a time, the next eight in flight; the warps' sums of 32 lanes meet in shared memory. No stages of weights
// in shared memory and no split of the reduction over CTAs (whose sums took a launch more). Times and the rule: cb200_skinny_rows below.
// 88 MB of weights (84 x 256 x 2048) go at 3.9 TB/s with one row, 2.9 with two.
constexpr int kRowsN = 8;                // weight rows of a warp at a time
template <int RT>
__global__ void __launch_bounds__(256) skinny_rows_kernel(SkinnyParams p, int wk, int per_cta) {
  __shared__ float part[2][8][kRowsN * RT];      // two sets in turn: [warp][weight row, row]
  pdl_trigger();                       // launched with programmatic serialisation (see common.cuh)
  pdl_wait();
  constexpr int V = kRowsN * RT;       // sums of a warp: 8, 16 or 32
  const int z = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kpart = warp % wk, npart = warp / wk, wn = 8 / wk, k = kpart * 256 + lane * 8;
  const float* A = p.a + (long)z * p.a_z;
  const __nv_bfloat16* B = p.b_ptrs ? reinterpret_cast<const __nv_bfloat16*>(p.b_ptrs[z])
                                    : reinterpret_cast<const __nv_bfloat16*>(p.b_base) + (long)z * p.b_z;
  // a weight that does not start on a 16-byte boundary (a slice of a larger buffer) is read element by element
  const bool vec = (reinterpret_cast<uintptr_t>(B) & 15) == 0;
  const int n_lo = (int)blockIdx.x * per_cta, n_hi = min(p.N, n_lo + per_cta);
  float a[RT][8];
#pragma unroll
  for (int r = 0; r < RT; ++r)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float v = r < p.R && k + j < p.K ? A[(long)r * p.a_r + k + j] : 0.f;
      a[r][j] = p.silu_a ? silu_f(v) : v;
    }
  bf16x8 next[kRowsN];
  auto fetch = [&](int n0) {
#pragma unroll
    for (int i = 0; i < kRowsN; ++i) {
      const int n = n0 + i;
      next[i] = bf16x8{};
      if (n < n_hi && k < p.K) {                       // K is a multiple of 8
        const __nv_bfloat16* src = B + (long)n * p.b_n + k;
        if (vec) {
          next[i] = *reinterpret_cast<const bf16x8*>(src);
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j) next[i].v[j] = __halves2bfloat162(src[2 * j], src[2 * j + 1]);
        }
      }
    }
  };
  float* C = reinterpret_cast<float*>(p.c) + (long)z * p.c_z;
  const int stride = wn * kRowsN;
  fetch(n_lo + npart * kRowsN);
  int set = 0;
  for (int n0 = n_lo; n0 < n_hi; n0 += stride, set ^= 1) {
    float sum[V];
#pragma unroll
    for (int i = 0; i < kRowsN; ++i) {
      float w[8];
      unpack8(next[i], w);
#pragma unroll
      for (int r = 0; r < RT; ++r) {
        float s = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) s = fmaf(w[j], a[r][j], s);
        sum[i * RT + r] = s;
      }
    }
    fetch(n0 + stride + npart * kRowsN);
    // halves of the values change hands until every lane holds one: value v lies in the lanes whose top bits spell it
#pragma unroll
    for (int half = V / 2, d = 16; half >= 1; half /= 2, d /= 2) {
      const bool up = (lane & d) != 0;
#pragma unroll
      for (int i = 0; i < half; ++i) {
        const float mine = up ? sum[i + half] : sum[i], other = up ? sum[i] : sum[i + half];
        sum[i] = mine + __shfl_xor_sync(0xffffffffu, other, d);
      }
    }
#pragma unroll
    for (int d = 16 / V; d >= 1; d /= 2) sum[0] += __shfl_xor_sync(0xffffffffu, sum[0], d);
    if (lane % (32 / V) == 0) part[set][warp][lane / (32 / V)] = sum[0];
    __syncthreads();
    // one thread per value of the CTA's `stride` weight rows; the parts of a row in the order of its elements
    for (int v = threadIdx.x; v < wn * V; v += 256) {
      const int np = v / V, i = v % V, n = n0 + np * kRowsN + i / RT, r = i % RT;
      if (n < n_hi && r < p.R) {
        float t = 0.f;
        for (int q = 0; q < wk; ++q) t += part[set][np * wk + q][i];
        if (p.add != nullptr && n < p.add_cols) t += p.add[(long)r * p.ld_add + n];
        C[(long)r * p.ldc + n] = t;
      }
    }
  }
}

template <int RT>
static int launch_skinny_rows(const SkinnyParams& p, int Z, cudaStream_t st) {
  int wk = 1;
  while (wk * 256 < p.K) wk *= 2;
  // weight rows of a CTA: about four CTAs on every SM over all problems, whole steps of the CTA
  const int step = 8 / wk * kRowsN;
  const long want = ((long)p.N * Z + 148 * 4 - 1) / (148 * 4);
  const int per_cta = (int)std::min<long>((p.N + step - 1) / step, std::max<long>(1, (want + step - 1) / step)) * step;
  return (int)launch_pdl(skinny_rows_kernel<RT>, dim3((p.N + per_cta - 1) / per_cta, Z), dim3(256), 0, st, p, wk, per_cta);
}

}  // namespace cb200

using namespace cb200;

// Whether a call goes to the kernel for a few rows, which does not split reductions. Its time goes with E, the weight elements with a row
// padded to its warps (256, 512, 1024 or 2048), times the rows; the wide kernel takes about 9 us as soon as it splits, since the sums are a
// launch more (from K = 256 on, up to 296 tiles of 256 columns), and 256 columns' time for few columns. us of the wide kernel and of this
// one, launches back to back with the weights in L2 as far as they fit, and behind a flush of L2 (two layers of 28 blocks' modulation are
// 84 x 256 x 2048 and 84 x 6144 x 256; a network's weights come from HBM). The second of these with two rows stays here although it is slower by
// itself: inside a denoising step of a 256 x 256 image the step takes 4,407 us with it and 4,413 with the wide kernel (spread below 2 us).
//   rows                  1                         2                         4
//   1 x 256 x 2048     9.9  3.6, 17.8 10.2      10.4  4.2, 19.5 10.2      11.2  5.1, 21.5 10.2
//   1 x 4096 x 256     8.9  3.8, 17.4 10.2       9.2  4.6, 17.4 10.2      10.4  6.1, 19.4 12.3
//   84 x 64 x 2048    32.1 10.8, 37.9 14.4      32.2  9.8, 39.8 16.4      32.6 14.1, 40.0 20.5
//   84 x 256 x 2048   32.9 22.5, 46.0 28.7      33.7 30.2, 46.1 37.8      34.7 33.1, 48.1 39.9
//   84 x 6144 x 256   68.6 54.7, 77.8 65.6      70.5 72.0, 79.9 84.0      74.3 90.3, 84.0 97.3     unsplit: one and two rows
//   1 x 6144 x 2048   12.5 10.8, 21.5 14.4      13.0 10.4, 23.6 16.4      13.3 17.8, 25.6 20.5
//   3 x 6144 x 1032   15.8 13.8, 25.7 20.5      16.4 20.2, 27.6 27.5      17.2 23.7, 29.7 30.7     half of the lanes idle
//   84 x 768 x 64      5.3  8.4, 10.3 14.3       5.6 10.9, 12.3 18.4       6.4 14.9, 13.2 20.5     most of the lanes idle: to 4096 columns
extern "C" int cb200_skinny_rows(long a_k, long b_n, long b_k, int b_is_bf16, int c_is_bf16, int silu_b, int Z, int R, int N, int K) {
  if (!(b_is_bf16 && !c_is_bf16 && !silu_b && a_k == 1 && b_k == 1 && b_n % 8 == 0 && K % 8 == 0 && K <= 2048 && R <= 4 && N >= 1)) return 0;
  long padded = 256;
  while (padded < K) padded *= 2;
  const long cols = (long)Z * N, E = cols * padded;
  const bool split = K >= 256 && (long)Z * ((N + 255) / 256) <= 296, full = K * 5 >= padded * 4;
  if (K < 128) return cols <= 4096;
  if (R == 1 && (split || full || (K >= 256 && K * 3 >= padded * 2))) return 1;
  if (K < 256) return cols <= 16384;
  if (N <= 128 || E <= 6L << 20) return 1;
  if (full) return split || R == 2;
  return split && R == 2 && E <= 14L << 20;
}

// whether a call goes to the wide kernel (the split of long reductions counts its tiles): bf16 weights with one contiguous index and
// 8-element rows, row-major A, fp32 result
extern "C" int cb200_skinny_wide(long a_k, long b_n, long b_k, int b_is_bf16, int c_is_bf16, int silu_b, int N, int K) {
  if (!b_is_bf16 || c_is_bf16 || silu_b || a_k != 1) return 0;
  return (b_k == 1 && b_n % 8 == 0 && K % 8 == 0) || (b_n == 1 && b_k % 8 == 0 && N % 8 == 0) ? 1 : 0;
}

extern "C" int cb200_skinny_bgemm(const float* a, long a_z, long a_r, long a_k, const long long* b_ptrs, const void* b_base, long b_z,
                                  long b_n, long b_k, int b_is_bf16, void* c, long c_z, int ldc, int c_is_bf16, const float* add,
                                  int ld_add, int add_cols, int Z, int R, int N, int K, int silu_a, int silu_b, int ksplit, cudaStream_t st) {
  if (Z <= 0 || R <= 0 || N <= 0 || K <= 0) return 0;
  if (ksplit < 1 || (long)Z * ksplit > 65535 || (R + kSkTile - 1) / kSkTile > 65535) return -1;
  SkinnyParams p{a, a_z, a_r, a_k, b_ptrs, b_base, b_z, b_n, b_k, c, c_z, ldc, add, ld_add, add_cols, R, N, K, silu_a, silu_b, ksplit};
  if (ksplit == 1 && Z <= 65535 && cb200_skinny_rows(a_k, b_n, b_k, b_is_bf16, c_is_bf16, silu_b, Z, R, N, K))
    return R == 1 ? launch_skinny_rows<1>(p, Z, st) : R == 2 ? launch_skinny_rows<2>(p, Z, st) : launch_skinny_rows<4>(p, Z, st);
  // (row tiles of 48 reach the grid's limit before those of 64)
  if (cb200_skinny_wide(a_k, b_n, b_k, b_is_bf16, c_is_bf16, silu_b, N, K) && (R + 47) / 48 <= 65535) {
    // rows per CTA: the smallest that holds them all; with several row tiles the weights are read again from L2
    if (b_k == 1)
      return R <= 4 ? launch_skinny_wide<4, true>(p, Z, st) : R <= 16 ? launch_skinny_wide<16, true>(p, Z, st)
           : R <= 32 ? launch_skinny_wide<32, true>(p, Z, st) : launch_skinny_wide<48, true>(p, Z, st);
    return R <= 4 ? launch_skinny_wide<4, false>(p, Z, st) : R <= 16 ? launch_skinny_wide<16, false>(p, Z, st)
         : R <= 32 ? launch_skinny_wide<32, false>(p, Z, st) : launch_skinny_wide<48, false>(p, Z, st);
  }
  dim3 grid((N + kSkTile - 1) / kSkTile, (R + kSkTile - 1) / kSkTile, Z * ksplit);
  if (b_is_bf16) {
    if (c_is_bf16) skinny_bgemm_kernel<__nv_bfloat16, __nv_bfloat16><<<grid, 256, 0, st>>>(p);
    else skinny_bgemm_kernel<__nv_bfloat16, float><<<grid, 256, 0, st>>>(p);
  } else {
    if (c_is_bf16) skinny_bgemm_kernel<float, __nv_bfloat16><<<grid, 256, 0, st>>>(p);
    else skinny_bgemm_kernel<float, float><<<grid, 256, 0, st>>>(p);
  }
  return 0;
}
