// Single-head attention with head dimension 384 on tcgen05 / TMEM (sm_100a), bf16, non-causal: the frame attention of the VAE's
// middle block (cosmos_predict2/_src/predict2/tokenizers/wan2pt1.py:217-256).
//
// The width decides the shape. A CTA owns 128 query rows of one frame; their fp32 output takes 384 of the 512 TMEM columns, which
// leaves two score buffers of 64 keys, so the keys are walked in tiles of 64 and the softmax of tile j runs while the tensor pipe does
// Q.K^T of tile j + 1 and P.V of tile j - 1. Q stays in shared memory (96 KB); K and V pass through a ring of eight 16 KB slots
// (64 keys x 128 channels; three slots each per key tile).
//
//   warps 0-3  softmax: thread i <-> query row i <-> TMEM lane i; probabilities go back over the score buffer as bf16
//   warp  4    TMA producer, warp 5 MMA issuer: S_b = Q K_j^T (SS, 128 x 64), O += P_b V_j (TS, 128 x 128 per channel block)
//
// What bounds it: shared-memory operand reads of the 128 x 64 score MMAs (48 clocks instead of 32 of tensor time), 0.8 of the
// tensor pipe at best. One 88 x 160 frame (14,080 queries and keys): 1.85 ms with the library's mma.sync kernel, 0.30 ms here; its 110
// CTAs leave a quarter of the SMs idle, on the others the tensor pipe is 63 % busy and the operand pipe 85 %.
// Online softmax and bounded waits as in fa_fwd.cu.

#include <math.h>

#include "common.cuh"
#include "launchers.h"
#include "sm100.cuh"
#include "tmap.h"

namespace cb200 {
using namespace sm100;

namespace fw {
constexpr int D = 384, NB = D / 128;           // channels, and 128-channel blocks
constexpr int BQ = 128, BKV = 64;
constexpr int kSubBytes = BKV * 128;           // 64 keys x 64 channels
constexpr int kSlotBytes = 2 * kSubBytes;      // 64 keys x 128 channels
constexpr int kRing = 8;
constexpr int kQSub = BQ * 128;                // 128 rows x 64 channels
constexpr int kQBytes = (D / 64) * kQSub;      // 96 KB
constexpr int kThreads = 192;
constexpr size_t kSmem = (size_t)kQBytes + kRing * kSlotBytes + 1024 + 256;
constexpr uint32_t kSCol = D;                  // TMEM: O [0, 384), S_b [384 + 64 b, +64)
constexpr float kRescaleThreshold = 8.0f;      // log2 units
}  // namespace fw

__device__ __forceinline__ float fw_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__global__ void __launch_bounds__(fw::kThreads, 1)
fa_wide_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
               bf16* __restrict__ O, int Sq, int Skv, float scale_log2, int* __restrict__ err) {
  using namespace fw;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* sQ = smem;
  uint8_t* sR = smem + kQBytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sR + kRing * kSlotBytes);
  uint64_t* q_full = bars;                    // [1]
  uint64_t* r_full = bars + 1;                // [kRing]
  uint64_t* r_empty = r_full + kRing;         // [kRing]
  uint64_t* s_full = r_empty + kRing;         // [2] scores of buffer b ready
  uint64_t* p_ready = s_full + 2;             // [2] probabilities of buffer b written
  uint64_t* o_done = p_ready + 2;             // [2] P.V from buffer b complete
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_done + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int q_base = blockIdx.x * BQ, b = blockIdx.y;
  const int n_kv = (Skv + BKV - 1) / BKV;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int i = 0; i < kRing; ++i) {
      mbar_init(&r_full[i], 1);
      mbar_init(&r_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&s_full[i], 1);
      mbar_init(&p_ready[i], 4);
      mbar_init(&o_done[i], 1);
    }
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 5) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_trigger();                              // launched with programmatic serialisation (see common.cuh)
  pdl_wait();
  if (threadIdx.x == 0) *abort_flag = *reinterpret_cast<volatile int*>(err);   // an earlier error: drain the grid at once
  __syncthreads();
  const bool stopped = *abort_flag != 0;
  __syncthreads();

  if (stopped) {
  } else if (warp == 4) {
    // -------------------------------------------------------------------- TMA producer
    if (lane == 0) {
      prefetch_tmap(&tm_q);
      prefetch_tmap(&tm_k);
      prefetch_tmap(&tm_v);
      mbar_arrive_expect_tx(q_full, kQBytes);
      for (int c = 0; c < D / 64; ++c) tma_load_3d(sQ + c * kQSub, &tm_q, q_full, c * 64, q_base, b);
      bool ok = true;
      int slot = 0;
      uint32_t ph = 0;
      // the order in which the issuer consumes: K_0 K_1 V_0 K_2 V_1 ... V_{n-2} V_{n-1}
      auto tile = [&](const CUtensorMap* tm, int j) {
        for (int n = 0; n < NB && ok; ++n) {
          if (!mbar_wait(&r_empty[slot], ph ^ 1, abort_flag)) { ok = false; break; }
          mbar_arrive_expect_tx(&r_full[slot], kSlotBytes);
          for (int c = 0; c < 2; ++c) tma_load_3d(sR + slot * kSlotBytes + c * kSubBytes, tm, &r_full[slot], n * 128 + c * 64, j * BKV, b);
          if (++slot == kRing) { slot = 0; ph ^= 1; }
        }
      };
      tile(&tm_k, 0);
      for (int j = 0; j < n_kv && ok; ++j) {
        if (j + 1 < n_kv) tile(&tm_k, j + 1);
        tile(&tm_v, j);
      }
      if (!ok) { atomicCAS(err, 0, 91); *abort_flag = 1; }
    }
  } else if (warp == 5) {
    // -------------------------------------------------------------------- MMA issuer (warp-uniform; the elected lane issues)
    const uint32_t leader = elect_one() ? 1u : 0u;
    auto wait_all = [&](uint64_t* bar, uint32_t parity) -> bool { return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag)); };
    constexpr uint32_t idesc_qk = umma_idesc_bf16(BQ, BKV, 0, 0);
    constexpr uint32_t idesc_pv = umma_idesc_bf16(BQ, 128, 0, 1);
    const uint64_t dQ = umma_desc_sw128(smem_u32(sQ), 16, 1024);            // Q blocks as K-major A
    const uint64_t dK = umma_desc_sw128(smem_u32(sR), 16, 1024);            // ring slot as K-major B
    const uint64_t dV = umma_desc_sw128(smem_u32(sR), kSubBytes, 1024);     // ring slot as N-major B
    bool ok = wait_all(q_full, 0);
    int slot = 0;
    uint32_t ph = 0;
    auto advance = [&]() { if (++slot == kRing) { slot = 0; ph ^= 1; } };
    auto qk = [&](int j) {
      for (int n = 0; n < NB && ok; ++n) {
        if (!wait_all(&r_full[slot], ph)) { ok = false; break; }
        tc_fence_after();
        const uint64_t k0 = dK + (uint64_t)(slot * (kSlotBytes >> 4)), q0 = dQ + (uint64_t)(n * (2 * kQSub >> 4));
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)
          umma_ss_w(tmem_base + kSCol + (j & 1) * BKV, q0 + (uint32_t)(((kk >> 2) * kQSub + (kk & 3) * 32) >> 4),
                    k0 + (uint32_t)(((kk >> 2) * kSubBytes + (kk & 3) * 32) >> 4), idesc_qk, (kk > 0 || n > 0) ? 1u : 0u, leader);
        umma_commit_w(&r_empty[slot], leader);
        advance();
      }
      if (ok) umma_commit_w(&s_full[j & 1], leader);
    };
    if (ok) qk(0);
    for (int j = 0; j < n_kv && ok; ++j) {
      if (j + 1 < n_kv) qk(j + 1);      // its buffer's probabilities were consumed by P.V of tile j - 1, issued before
      if (!ok || !wait_all(&p_ready[j & 1], (j >> 1) & 1)) { ok = false; break; }
      tc_fence_after();
      for (int n = 0; n < NB && ok; ++n) {
        if (!wait_all(&r_full[slot], ph)) { ok = false; break; }
        tc_fence_after();
        const uint64_t v0 = dV + (uint64_t)(slot * (kSlotBytes >> 4));
#pragma unroll
        for (int kk = 0; kk < BKV / 16; ++kk)
          umma_ts_w(tmem_base + n * 128, tmem_base + kSCol + (j & 1) * BKV + kk * 8, v0 + (uint32_t)(kk * (2048 >> 4)), idesc_pv,
                    (j > 0 || kk > 0) ? 1u : 0u, leader);
        umma_commit_w(&r_empty[slot], leader);
        advance();
      }
      if (ok) umma_commit_w(&o_done[j & 1], leader);
    }
    if (!ok && lane == 0) { atomicCAS(err, 0, 92); *abort_flag = 1; }
  } else {
    // -------------------------------------------------------------------- softmax
    const int quarter = warp;
    const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
    const uint32_t tO = tmem_base + lane_off;
    float m_ref = -INFINITY, l = 0.f;     // reference maximum of the exponent (log2 domain), sum of probabilities
    bool ok = true;
    for (int j = 0; j < n_kv; ++j) {
      const uint32_t tS = tmem_base + kSCol + (j & 1) * BKV + lane_off;
      if (!mbar_wait_warp(&s_full[j & 1], (j >> 1) & 1, abort_flag)) { ok = false; break; }
      tc_fence_after();
      uint32_t r[2][32];
      tmem_ld32(tS, r[0]);
      tmem_ld32(tS + 32, r[1]);
      tmem_ld_wait();
      const int n_valid = Skv - j * BKV;
      if (n_valid < BKV) {
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (c * 32 + i >= n_valid) r[c][i] = 0xff800000u;  // -inf
      }
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int i = 0; i < 32; ++i) mx4[i & 3] = fmaxf(mx4[i & 3], __uint_as_float(r[c][i]));
      const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * scale_log2;
      const bool need = mx > m_ref + kRescaleThreshold;
      float alpha = 1.f;
      if (need) {
        alpha = (m_ref == -INFINITY) ? 0.f : fw_ex2(m_ref - mx);
        m_ref = mx;
        l *= alpha;
      }
      if (j > 0 && __any_sync(0xffffffffu, need)) {
        // Rescale this warp's output rows; P.V of the previous tile has to be complete. A parity tells two neighbouring phases apart,
        // so the barrier must be neither a phase ahead (P.V of tile j + 1, the next on this barrier, needs this warp's probabilities
        // of tile j first) nor one behind (that of tile j - 3 was complete before the scores of tile j - 1 were begun). One barrier
        // for all tiles would not do: it can be a phase ahead of a warp that is late, which then waits for itself.
        if (!mbar_wait_warp(&o_done[(j - 1) & 1], ((j - 1) >> 1) & 1, abort_flag)) { ok = false; break; }
        tc_fence_after();
#pragma unroll 1
        for (int c = 0; c < D / 32; ++c) {
          uint32_t o[32];
          tmem_ld32(tO + c * 32, o);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
          tmem_st32(tO + c * 32, o);
        }
        tmem_st_wait();
      }
      const float2 sc2 = make_float2(scale_log2, scale_log2), nm2 = make_float2(-m_ref, -m_ref);
      float2 lsum2 = make_float2(0.f, 0.f);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t pk[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float2 x = fma2(make_float2(__uint_as_float(r[c][2 * i]), __uint_as_float(r[c][2 * i + 1])), sc2, nm2);
          const float2 p = make_float2(fw_ex2(x.x), fw_ex2(x.y));
          lsum2 = add2(lsum2, p);
          __nv_bfloat162 pb = __floats2bfloat162_rn(p.x, p.y);
          pk[i] = *reinterpret_cast<uint32_t*>(&pb);
        }
        tmem_st16(tS + c * 16, pk);
      }
      l += lsum2.x + lsum2.y;
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_ready[j & 1]);
    }
    if (ok) ok = mbar_wait_warp(&o_done[(n_kv - 1) & 1], ((n_kv - 1) >> 1) & 1, abort_flag);
    if (ok) {
      tc_fence_after();
      const float inv_l = 1.f / l;
      // rows leave through shared memory (Q is no longer read) so that 16 lanes store 256 contiguous bytes of a row
      uint8_t* stage_warp = sQ + quarter * (32 * 256);
      uint8_t* stage_row = stage_warp + lane * 256;
#pragma unroll 1
      for (int n = 0; n < NB; ++n) {
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
          uint32_t o[32];
          tmem_ld32(tO + n * 128 + c * 32, o);
          tmem_ld_wait();
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            uint4 ov;
            __nv_bfloat162* o2 = reinterpret_cast<__nv_bfloat162*>(&ov);
#pragma unroll
            for (int i = 0; i < 4; ++i)
              o2[i] = __floats2bfloat162_rn(__uint_as_float(o[q * 8 + 2 * i]) * inv_l, __uint_as_float(o[q * 8 + 2 * i + 1]) * inv_l);
            *reinterpret_cast<uint4*>(stage_row + (((c * 4 + q) ^ (lane & 7)) << 4)) = ov;
          }
        }
        __syncwarp();
#pragma unroll 4
        for (int it = 0; it < 16; ++it) {
          const int r_src = it * 2 + (lane >> 4), chunk = lane & 15, row = q_base + quarter * 32 + r_src;
          const uint4 v = *reinterpret_cast<const uint4*>(stage_warp + r_src * 256 + ((chunk ^ (r_src & 7)) << 4));
          if (row < Sq) *reinterpret_cast<uint4*>(O + ((size_t)b * Sq + row) * D + n * 128 + chunk * 8) = v;
        }
        __syncwarp();
      }
    } else if (lane == 0) {
      atomicCAS(err, 0, 93);
      *abort_flag = 1;
    }
  }

  __syncwarp();
  if (*abort_flag && !stopped) {
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 5) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace cb200

using namespace cb200;

// q [B, Sq, 384], k, v [B, Skv, 384] bf16 with rows `*_row` and batches `*_batch` elements apart; o [B, Sq, 384] contiguous.
extern "C" int cb200_fa_wide(const void* q, long q_row, long q_batch, const void* k, long k_row, long k_batch, const void* v, long v_row,
                             long v_batch, void* o, int B, int Sq, int Skv, float scale, int* err, cudaStream_t st) {
  using namespace fw;
  if (B < 1 || B > 65535 || Sq < 1 || Skv < 1) return -61;
  CUtensorMap tq, tk, tv;
  auto make = [&](CUtensorMap* m, const void* p, int S, long row, long batch, uint32_t rows) {
    const uint64_t dims[3] = {(uint64_t)D, (uint64_t)S, (uint64_t)B};
    const uint64_t strides[2] = {(uint64_t)row * 2, (uint64_t)batch * 2};
    const uint32_t box[3] = {64, rows, 1};
    return make_tmap_bf16(m, p, 3, dims, strides, box);
  };
  int rc = make(&tq, q, Sq, q_row, q_batch, BQ);
  if (rc) return rc;
  if ((rc = make(&tk, k, Skv, k_row, k_batch, BKV))) return rc;
  if ((rc = make(&tv, v, Skv, v_row, v_batch, BKV))) return rc;
  static bool attr = false;
  if (!attr) {
    cudaError_t e = cudaFuncSetAttribute(fa_wide_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
    if (e != cudaSuccess) return 100 + (int)e;
    attr = true;
  }
  return (int)launch_pdl(fa_wide_kernel, dim3((Sq + BQ - 1) / BQ, B), dim3(kThreads), kSmem, st, tq, tk, tv, (bf16*)o, Sq, Skv,
                         scale * 1.4426950408889634f, err);
}
