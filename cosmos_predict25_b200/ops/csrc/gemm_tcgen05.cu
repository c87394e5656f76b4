// bf16 GEMM on the 5th-generation tensor cores (sm_100a): C[M,N] = epilogue(A x B), fp32 accumulation.
//
// Persistent, warp-specialised kernel, one CTA per SM, in three forms:
//   CTA pairs (from 256 rows on): clusters of two CTAs work on a 256 x 256 tile with cta_group::2 MMAs, six 32 KB stages; a cluster of two
//            to four pairs shares a tile where there are few of them (see the kernel below);
//   single CTAs (fewer rows, and the gather mode): 128 x 256 tiles, four 48 KB stages.
// Roles: warp 0 is the TMA producer (128x64 A tiles and 256x64 B tiles, 128-byte swizzle, through the ring of stages; completion by
//   mbarrier transaction bytes), warp 1 issues tcgen05.mma from shared-memory descriptors into one of two 128x256 fp32 accumulators
//   in TMEM (2 x 256 = all 512 columns) and releases ring slots with tcgen05.commit, warps 2-9 are the epilogue: two warps per
//   32-lane quarter of TMEM, 128 columns each, apply the fused epilogue in registers and store bf16 through a staging block while
//   warp 1 already accumulates the next tile into the other TMEM buffer.
//
// Operand majors are template parameters so the same kernel serves forward (x @ W^T: both K-major),
// dgrad (dy @ W: B is N-major) and wgrad (dy^T @ x: both MN-major) without transposing in memory.
// Fused epilogues: + bias, exact GELU (optionally also writing the pre-activation for backward),
// and the AdaLN gated residual  out = resid + gate[row / L, col] * acc.
//
// FSDP all-gather fused into the GEMM (template flag GATHER): the B operand is a weight [rows, ld] whose rows are sharded over P
// ranks (rank r holds rows [r * chunk_rows, (r + 1) * chunk_rows) in its own memory). Four extra warps per CTA pull the shards -
// plain 16-byte loads from the owners' memory, local or over NVLink - into a local full-size copy, in groups of 256 rows cut into
// slices, and publish every finished slice with a release increment of the group's counter. The TMA producer acquires the
// counter of the group a B box lies in before it issues the load, so tiles are computed while later groups are still in
// flight and every remote row crosses NVLink exactly once. The same code serves the forward GEMM (groups along N) and dgrad
// (groups along the contraction dimension).
//
// All mbarrier waits are bounded; on timeout the CTA records an error code in `err`, lets in-flight
// copies land, frees its TMEM and returns.

#include <math.h>

#include "launchers.h"
#include <algorithm>
#include <cstdlib>

#include "common.cuh"
#include "sm100.cuh"
#include "tmap.h"

namespace cb200 {
using namespace sm100;

constexpr int BM = 128, BN = 256, BK = 64, UK = 16;
constexpr int kStages = 4;
constexpr int kABytes = BM * BK * 2;  // 16 KB
constexpr int kBBytes = BN * BK * 2;  // 32 KB
constexpr int kStageBytes = kABytes + kBBytes;
constexpr int kGemmThreads = 320;  // TMA warp, MMA warp, 8 epilogue warps (two per TMEM lane quarter, 128 columns each)
constexpr int kPrefetchBlocks = 8;    // k-blocks of the first tile's B operand asked into L2 ahead of the wait
constexpr int kStageOutBytes = 8 * 32 * 128;  // one 32-row x 128-byte staging block per epilogue warp
constexpr size_t kSmemBytes = (size_t)kStages * kStageBytes + 1024 /*alignment slack*/ + 256 /*barriers*/ + kStageOutBytes;

// Ulysses exchange fused into the epilogue: the output [M, N] is a projection to H = N / 128 heads of a local sequence of S
// tokens per batch item; head h of token (b, s) is normalised (optional per-head RMSNorm), rotated (optional rotate-half
// RoPE) and stored straight into the staging buffer of the rank that owns the head, at its place in the gathered sequence.
struct HeadScatter {
  int64_t ptrs[8];    // staging buffers of the P ranks, each [B, P * S, Hl, 128] bf16
  const void* w;      // [128] RMSNorm weight (fp32, or bf16 with w_bf16) or nullptr
  int w_bf16;
  const float* cosv;  // [S, 64] or nullptr
  const float* sinv;
  int S, Hl, P, rank;
  float eps;
  bf16* raw;          // optional [M, N]: the un-normalised projection, kept locally for the RMSNorm backward (training)
  float* rstd_out;    // optional [M, N / 128]: reciprocal RMS of every (token, head), with ``raw``
};

__device__ __forceinline__ float norm_weight(const HeadScatter& hs, int i) {
  return hs.w_bf16 ? __bfloat162float(reinterpret_cast<const bf16*>(hs.w)[i]) : reinterpret_cast<const float*>(hs.w)[i];
}

// Products of one A with up to NW weights of the same shape [N, K] in one launch: N tiles [g tiles, (g + 1) tiles) belong to weight g.
// Three (q, k, v) is what every launch carries; kManyWeights (the context's keys and values of all blocks) is a kernel of its own,
// since the parameters are copied for each launch.
constexpr int kManyWeights = 80;
template <int NW>
struct GemmWeights {
  CUtensorMap map[NW];
  bf16* out[NW];
  // many weights: per-head RMSNorm weight [128] of the product's heads (fp32, or bf16 where `norm_bf16` says so), or null: plain product
  const void* norm[NW > 3 ? NW : 1];
  uint8_t norm_bf16[NW > 3 ? NW : 1];
};

struct GemmEpilogue {
  HeadScatter hs;     // hs.P == 0: disabled
  int groups;         // weights; more than one only without bias, activation, residual and head scatter
  float norm_eps;     // many weights: of their norms
  bf16* pre;          // optional second output: the pre-activation (act == 1) or the product before the gated residual
                      // (full 256-column tiles only)
  const bf16* bias;   // optional [N]
  const bf16* resid;  // optional [M, N] (gated residual)
  const float* gate;  // optional [M / L] rows of N, ld_gate elements apart
  long ld_gate;
  int act;            // 0 none, 1 gelu(erf)
  int L;              // rows per gate vector
};

// Exact GELU of a pair of values: x Phi(x) = (x + |x|) / 2 - |x| Phi(-|x|), and Phi(-a) = exp(-a^2 / 2) R(a), where R = erfcx(a / sqrt 2) / 2
// falls smoothly from 1/2: a degree-11 polynomial in a scaled to [-1, 1] on [0, 5.5], fitted for the relative error (4.2e-6; a thousandth
// of a bf16 rounding; 1 + erff is at 1.3e-7 for positive arguments, at 1.2e-5 for -3 and lost below. Behind the rounding to bf16, the only type
// that leaves here, the 2-norm error is the same to eight digits for arguments of 0.25 to 4 in spread). a R(a) hardly changes beyond 5.5, where the product is below 1e-7: a is held there. The difference 1 + erff
// that stood here loses its digits for x below -3, and took twice the instructions, which an epilogue has to itself when a CTA has one tile:
// 512 x 8192 x 2048 with GELU 20.6 us before, now 18.6 (without GELU 16.1).
// Coefficients are negated: the sum is a fused multiply-add. Infinities and NaN give what the product x Phi(x) gives.
__device__ __forceinline__ float2 gelu2(float2 x) {
  constexpr float kC[12] = {-0.130724221f,  0.108487532f,  -0.0841316134f, 0.0614620969f,  -0.0422496423f, 0.0284217875f,
                            -0.0201631337f, 0.0114772478f, -0.00272275996f, 0.00254054717f, -0.00517878076f, 0.00243854383f};
  const float2 a = make_float2(fabsf(x.x), fabsf(x.y));
  const float2 held = make_float2(fminf(a.x, 5.5f), fminf(a.y, 5.5f));
  const float2 u = fma2(held, make_float2(2.f / 5.5f, 2.f / 5.5f), make_float2(-1.f, -1.f));
  float2 r = make_float2(kC[11], kC[11]);
#pragma unroll
  for (int k = 10; k >= 0; --k) r = fma2(r, u, make_float2(kC[k], kC[k]));
  constexpr float kHalfLog2e = -0.72134752044448171f;
  const float2 t = mul2(mul2(x, x), make_float2(kHalfLog2e, kHalfLog2e));
  const float2 q = mul2(make_float2(exp2f(t.x), exp2f(t.y)), r);
  const float2 half = make_float2(0.5f, 0.5f);
  return fma2(held, q, fma2(x, half, mul2(a, half)));
}
__device__ __forceinline__ void gelu32(float (&v)[32]) {
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    const float2 g = gelu2(make_float2(v[2 * j], v[2 * j + 1]));
    v[2 * j] = g.x;
    v[2 * j + 1] = g.y;
  }
}

// Row-sharded B operand gathered inside the kernel (see the header comment).
constexpr int kGatherWarps = 2;   // with the 10 GEMM warps: three warpgroups, 168 registers per thread (four more warps
                                  // would cap the epilogue at 128 registers and make it spill)
constexpr int kGatherGroupRows = 256;
struct GatherB {
  int64_t ptrs[8];     // rank r: its rows [r * chunk_rows, ...) of the weight, row-major with `ld` elements per row
  bf16* ws;            // local full copy [rows, ld]; the B tensor map is built on it
  int* counters;       // one per 256-row group, zeroed by the host before the launch
  int P, chunk_rows, rows, ld;
  int slices;          // pieces a group is cut into; a group is complete when its counter reaches this value
};

__device__ __forceinline__ int ld_acquire_gpu(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void red_release_gpu_add(int* p, int v) {
  asm volatile("red.release.gpu.global.add.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// CTA2: two CTAs of a cluster share one 256 x 256 output tile (tcgen05 cta_group::2). CTA r of the pair loads rows
// [128 r, 128 r + 128) of the A tile and of the B tile into its own shared memory (half the B bytes per CTA and per MMA), the even
// CTA issues M = 256 MMAs that read both shared memories, each CTA's TMEM receives its 128 rows and its epilogue warps drain them.
// Six 32 KB stages instead of four 48 KB ones.
//
// SPLIT > 1: a cluster of SPLIT pairs works on ONE tile, each pair on its share of the contraction dimension, for outputs of so few
// tiles that most of the GPU would idle while a handful of SMs pull the operands (a 512 x 2048 output is 16 tiles: 32 SMs fetch 1 MB
// each at K = 2048). The fp32 partial tiles are exchanged through distributed shared memory - pair s receives the SPLIT - 1 other
// partials of its share of the columns (in units of 64) in the shared memory that the operand ring no longer needs - added in a fixed order (the
// result is deterministic) and put back into TMEM, from where the ordinary epilogue finishes those columns.
template <int A_MN, int B_MN, bool GATHER, bool CTA2 = false, int SPLIT = 1, int NW = 3>
__global__ void __launch_bounds__(kGemmThreads + (GATHER ? kGatherWarps * 32 : 0), 1)
gemm_bf16_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ GemmWeights<NW> bw, int M, int N, int K, GemmEpilogue ep,
                 GatherB gb, int* __restrict__ err) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  static_assert(!(CTA2 && GATHER), "the gather mode runs on single-CTA tiles");
  static_assert(SPLIT == 1 || (CTA2 && SPLIT >= 2 && SPLIT <= 4), "split tiles: clusters of two to four pairs");
  // SPLIT > 1: pair s finishes the 64-column units [unit_first(s), unit_first(s + 1)) of the tile: two each, two / one / one, one each
  auto unit_first = [](int s) -> int { return SPLIT == 3 ? (s == 0 ? 0 : s + 1) : s * 4 / SPLIT; };
  constexpr int STG = CTA2 ? 6 : kStages;                                   // pipeline stages
  constexpr int STG_BYTES = CTA2 ? (kABytes + kBBytes / 2) : kStageBytes;   // bytes per stage in this CTA
  constexpr int TM = CTA2 ? 2 * BM : BM;                                    // output rows per tile (per pair with CTA2)
  static_assert(STG * STG_BYTES == kStages * kStageBytes, "both layouts fill the same shared-memory window");
  const uint32_t cta_rank = CTA2 ? cluster_ctarank() : 0u, pair_rank = cta_rank & 1u, lead_rank = cta_rank & ~1u;
  const int split = (int)(cta_rank >> 1);                    // this pair's share of the tile's contraction (SPLIT > 1)
  const uint16_t pair_mask = (uint16_t)(3u << lead_rank);
  constexpr int kCtasPerTile = CTA2 ? 2 * SPLIT : 1;
  const int first_tile = (int)blockIdx.x / kCtasPerTile, tile_step = (int)gridDim.x / kCtasPerTile;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + STG * STG_BYTES);
  uint64_t* full = bars;                    // [STG]
  uint64_t* empty = bars + STG;             // [STG]
  uint64_t* acc_full = bars + 2 * STG;      // [2]
  uint64_t* acc_empty = acc_full + 2;       // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  // the shuffle makes the warp index (and every role branch below) provably warp-uniform for the compiler
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int tiles_m = (M + TM - 1) / TM, tiles_g = (N + BN - 1) / BN;
  const int tiles_n = CTA2 ? tiles_g * ep.groups : tiles_g;      // N tiles of all weights
  const int n_tiles = tiles_m * tiles_n;
  // Tile t's row and column. Neighbours run at the same time and share their row of A, whose columns fit L2 - except with many weights,
  // which together do not: there neighbours share a weight's columns, so that every weight is read from HBM once.
  auto tile_row = [&](int t) -> int { return NW > 3 ? t % tiles_m : t / tiles_n; };
  auto tile_col = [&](int t) -> int { return NW > 3 ? t / tiles_m : t % tiles_n; };
  const int k_all = (K + BK - 1) / BK;
  const int kb_first = SPLIT > 1 ? k_all * split / SPLIT : 0, k_blocks = SPLIT > 1 ? k_all * (split + 1) / SPLIT - kb_first : k_all;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STG; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&acc_full[a], 1);
      mbar_init(&acc_empty[a], CTA2 ? 16 : 8);      // the pair leader hears from the epilogue warps of both CTAs
    }
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    if (CTA2) {
      tmem_alloc_pair(tmem_slot, 512);
      tmem_relinquish_pair();
    } else {
      tmem_alloc(tmem_slot, 512);
      tmem_relinquish();
    }
  }
  tc_fence_before();
  __syncthreads();
  if (CTA2) cluster_sync_relaxed();  // the other CTA's barriers exist before anything signals them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  if (CTA2) {                        // launched with programmatic serialisation (see common.cuh)
    pdl_trigger();
    if (warp == 0 && lane == 0) {
      // The first tile's B operand, as a rule a weight that only HBM holds, on its way into L2 while the kernel in front still runs.
      prefetch_tmap(&tma_a);
      const int grp = tile_col(first_tile) / tiles_g;
      const CUtensorMap* tb = &bw.map[grp];
      prefetch_tmap(tb);
      const int n0 = (tile_col(first_tile) - grp * tiles_g) * BN + (int)pair_rank * (BN / 2);
      const int ahead = min(k_blocks, kPrefetchBlocks);
      for (int kb = 0; kb < ahead; ++kb) {
        const int k0 = (kb_first + kb) * BK;
        if (B_MN == 0) {
          tma_prefetch_l2_2d(tb, k0, n0);
        } else {
#pragma unroll
          for (int j = 0; j < BN / 128; ++j) tma_prefetch_l2_2d(tb, n0 + j * 64, k0);
        }
      }
    }
    pdl_wait();
  }

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      if (!CTA2) {
        prefetch_tmap(&tma_a);
        prefetch_tmap(&bw.map[0]);
      }
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      // GATHER: groups of B rows whose gather this thread has already seen complete (a bit per group, 128 groups)
      unsigned long long seen[2] = {0ull, 0ull};
      auto group_ready = [&](int row) -> bool {
        const int g = row / kGatherGroupRows;
        if (g < 128 && ((seen[g >> 6] >> (g & 63)) & 1ull)) return true;
        const unsigned long long t0 = global_timer_ns();
        while (ld_acquire_gpu(gb.counters + g) < gb.slices) {
          __nanosleep(64);
          if (*abort_flag || global_timer_ns() - t0 > kWaitLimitNs) return false;
        }
        fence_proxy_async_all();    // the rows were written by ordinary stores; the TMA load below reads them through the async proxy
        if (g < 128) seen[g >> 6] |= 1ull << (g & 63);
        return true;
      };
      for (int t = first_tile; t < n_tiles && ok; t += tile_step) {
        // with CTA2 this CTA fetches its 128 rows of the pair's A tile and its 128 rows of the B tile
        const int grp = CTA2 ? tile_col(t) / tiles_g : 0;
        const CUtensorMap* tb = &bw.map[grp];
        const int m0 = tile_row(t) * TM + (CTA2 ? (int)pair_rank * BM : 0);
        const int n0 = (tile_col(t) - grp * tiles_g) * BN + (CTA2 ? (int)pair_rank * (BN / 2) : 0);
        for (int kb = 0; kb < k_blocks; ++kb) {
          if (GATHER) {
            // rows of the weight this stage reads: an N tile of 256 rows (forward) or 64 rows of the contraction dimension (dgrad)
            if (B_MN == 0) {
              if (kb == 0 && !group_ready(n0)) { ok = false; break; }
            } else if (!group_ready(kb * BK)) { ok = false; break; }
          }
          if (!mbar_wait(&empty[s], ph ^ 1, abort_flag)) { ok = false; break; }
          uint8_t* sa = smem + s * STG_BYTES;
          uint8_t* sb = sa + kABytes;
          const int k0 = (kb_first + kb) * BK;
          if (CTA2) {
            // all bytes of the pair's stage are counted on the leader's barrier: the leader announces them, both CTAs load
            if (pair_rank == 0) mbar_arrive_expect_tx(&full[s], 2 * STG_BYTES);
            const uint32_t bar = mapa_shared(smem_u32(&full[s]), lead_rank);
            if (A_MN == 0) {
              tma_load_2d_pair(sa, &tma_a, bar, k0, m0);
            } else {
#pragma unroll
              for (int j = 0; j < BM / 64; ++j) tma_load_2d_pair(sa + j * 8192, &tma_a, bar, m0 + j * 64, k0);
            }
            if (B_MN == 0) {
              tma_load_2d_pair(sb, tb, bar, k0, n0);
            } else {
#pragma unroll
              for (int j = 0; j < BN / 128; ++j) tma_load_2d_pair(sb + j * 8192, tb, bar, n0 + j * 64, k0);
            }
          } else {
            mbar_arrive_expect_tx(&full[s], kStageBytes);
            if (A_MN == 0) {
              tma_load_2d(sa, &tma_a, &full[s], k0, m0);
            } else {
#pragma unroll
              for (int j = 0; j < BM / 64; ++j) tma_load_2d(sa + j * 8192, &tma_a, &full[s], m0 + j * 64, k0);
            }
            if (B_MN == 0) {
              tma_load_2d(sb, tb, &full[s], k0, n0);
            } else {
#pragma unroll
              for (int j = 0; j < BN / 64; ++j) tma_load_2d(sb + j * 8192, tb, &full[s], n0 + j * 64, k0);
            }
          }
          if (++s == STG) { s = 0; ph ^= 1; }
        }
      }
      if (!ok) { atomicCAS(err, 0, 1); *abort_flag = 1; }
    }
    if (SPLIT > 1) {                 // the two exchange barriers of the epilogue warps below take every warp of the cluster
      __syncwarp();
      cluster_sync_relaxed();
      cluster_sync_all();
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    // The whole warp runs this loop with identical values and only the elected lane issues: warp-uniform control flow and
    // descriptor arithmetic stay on the uniform datapath, which lowers the issue cost per MMA.
    {
      const uint32_t leader = elect_one() ? 1u : 0u;
      auto wait_all = [&](uint64_t* bar, uint32_t parity) -> bool { return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag)); };
      constexpr uint32_t idesc = umma_idesc_bf16(TM, BN, A_MN, B_MN);
      // stage-0 descriptors; a stage / k-slice is a constant added to the address field (16-byte units)
      const uint64_t da0 = A_MN ? umma_desc_sw128(smem_u32(smem), 8192, 1024) : umma_desc_sw128(smem_u32(smem), 16, 1024);
      const uint64_t db0 = B_MN ? umma_desc_sw128(smem_u32(smem) + kABytes, 8192, 1024) : umma_desc_sw128(smem_u32(smem) + kABytes, 16, 1024);
      int s = 0;
      uint32_t ph = 0;
      int acc = 0;
      uint32_t acc_ph = 0;
      bool ok = true;
      for (int t = first_tile; t < n_tiles && ok && pair_rank == 0; t += tile_step) {     // only the pair leader issues
        if (!wait_all(&acc_empty[acc], acc_ph ^ 1)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * BN;
        for (int kb = 0; kb < k_blocks; ++kb) {
          if (!wait_all(&full[s], ph)) { ok = false; break; }
          tc_fence_after();
          const uint64_t da_s = da0 + (uint64_t)(s * (STG_BYTES >> 4)), db_s = db0 + (uint64_t)(s * (STG_BYTES >> 4));
#pragma unroll
          for (int k = 0; k < BK / UK; ++k) {
            const uint64_t da = da_s + (uint32_t)((A_MN ? k * (UK * 128) : k * (UK * 2)) >> 4);
            const uint64_t db = db_s + (uint32_t)((B_MN ? k * (UK * 128) : k * (UK * 2)) >> 4);
            if (CTA2) umma_ss_pair_w(d_tmem, da, db, idesc, (kb > 0 || k > 0) ? 1u : 0u, leader);
            else umma_ss_w(d_tmem, da, db, idesc, (kb > 0 || k > 0) ? 1u : 0u, leader);
          }
          // slot reusable once these MMAs have read it (with CTA2: in both CTAs)
          if (CTA2) umma_commit_pair_w(&empty[s], leader, pair_mask);
          else umma_commit_w(&empty[s], leader);
          if (++s == STG) { s = 0; ph ^= 1; }
        }
        if (!ok) break;
        if (CTA2) umma_commit_pair_w(&acc_full[acc], leader, pair_mask);
        else umma_commit_w(&acc_full[acc], leader);
        if (++acc == 2) { acc = 0; acc_ph ^= 1; }
      }
      if (!ok && lane == 0) { atomicCAS(err, 0, 2); *abort_flag = 1; }
    }
    if (SPLIT > 1) {
      __syncwarp();
      cluster_sync_relaxed();
      cluster_sync_all();
    }
  } else if (GATHER && warp >= 10) {
    // ------------------------------------------------------------------ gather warps
    // item = (group, slice); CTA b takes items b, b + grid, ...; item i works on group i % n_groups, so the CTAs' first
    // items cover every group at once and the group of a CTA's own first tile is among the first to complete
    const int tid = threadIdx.x - 10 * 32;
    const int n_groups = (gb.rows + kGatherGroupRows - 1) / kGatherGroupRows;
    const int n_items = n_groups * gb.slices;
    const int row_vecs = gb.ld >> 3;                       // 16-byte pieces per row
    for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
      const int g = item % n_groups, sl = item / n_groups;
      const int g_lo = g * kGatherGroupRows, g_hi = min(gb.rows, g_lo + kGatherGroupRows);
      const int per = (g_hi - g_lo + gb.slices - 1) / gb.slices;
      const int r_lo = min(g_hi, g_lo + sl * per), r_hi = min(g_hi, r_lo + per);
      const long n_vec = (long)(r_hi - r_lo) * row_vecs;
      // 16 independent 16-byte loads per thread and round: enough bytes in flight per SM to cover the NVLink round trip
      constexpr int kInFlight = 16;
      // consecutive lanes take consecutive 16-byte pieces: one warp load is 512 contiguous bytes on the link
      constexpr int kGatherThreads = kGatherWarps * 32;
      for (long v0 = tid; v0 < n_vec; v0 += (long)kGatherThreads * kInFlight) {
        uint4 buf[kInFlight];
#pragma unroll
        for (int u = 0; u < kInFlight; ++u) {
          const long v = v0 + (long)u * kGatherThreads;
          if (v < n_vec) {
            const int row = r_lo + (int)(v / row_vecs), piece = (int)(v % row_vecs);
            const int owner = row / gb.chunk_rows;
            const bf16* src = reinterpret_cast<const bf16*>(gb.ptrs[owner]) + (size_t)(row - owner * gb.chunk_rows) * gb.ld;
            buf[u] = *(reinterpret_cast<const uint4*>(src) + piece);
          }
        }
#pragma unroll
        for (int u = 0; u < kInFlight; ++u) {
          const long v = v0 + (long)u * kGatherThreads;
          if (v < n_vec) {
            const int row = r_lo + (int)(v / row_vecs), piece = (int)(v % row_vecs);
            *(reinterpret_cast<uint4*>(gb.ws + (size_t)row * gb.ld) + piece) = buf[u];
          }
        }
      }
      __threadfence();
      asm volatile("bar.sync 1, %0;" ::"n"(kGatherWarps * 32) : "memory");   // every gather thread has stored and fenced
      if (tid == 0) red_release_gpu_add(gb.counters + g, 1);
    }
  } else {
    // ------------------------------------------------------------------ epilogue warps
    const int quarter = warp & 3;      // TMEM lanes [32*quarter, 32*quarter + 32)
    const int part = (warp - 2) >> 2;  // accumulator columns [128*part, 128*part + 128)
    uint8_t* stage_warp = smem + STG * STG_BYTES + 256 + (warp - 2) * (32 * 128);
    uint8_t* stage_row = stage_warp + lane * 128;
    int acc = 0;
    uint32_t acc_ph = 0;
    bool ok = true;
    const bool vec_ok = (N % 8) == 0;
    // SPLIT > 1: the 64-column unit of the tile that this warp finishes; the two warps of a lane quarter share the pair's slice
    constexpr int kSliceMax = SPLIT == 4 ? 64 : 128;
    const int my_unit = SPLIT > 1 && unit_first(split) + part < unit_first(split + 1) ? unit_first(split) + part : -1;
    // Gated residual: the rows of the residual that a pass of 64 columns needs are fetched ahead - the first pass's while the tile's
    // products are still being summed, the next one's while this one is finished - and the gate of 32 columns is one batch of loads.
    // Loaded where they were used, a tile paid their latency once per 16 bytes: 46,800 x 2048 x 2048 400 us, now 270 (the plain product
    // 255), 7040 x 2048 x 2048 74 and 51 us, 512 x 2048 x 2048 22.0 and 15.5 us.
    auto fetch_resid = [&](uint4 (&ahead)[8], int row0, int colbase) {
#pragma unroll
      for (int it = 0; it < 8; ++it) {
        const int r = row0 + it * 4 + (lane >> 3);
        ahead[it] = make_uint4(0, 0, 0, 0);
        if (r < M) ahead[it] = *reinterpret_cast<const uint4*>(ep.resid + (size_t)r * N + colbase + (lane & 7) * 8);
      }
    };
    const uint32_t acc_empty_leader[2] = {CTA2 ? mapa_shared(smem_u32(&acc_empty[0]), lead_rank) : 0u,
                                          CTA2 ? mapa_shared(smem_u32(&acc_empty[1]), lead_rank) : 0u};
    for (int t = first_tile; t < n_tiles && ok; t += tile_step) {
      const int grp = CTA2 ? tile_col(t) / tiles_g : 0;
      bf16* const out = bw.out[grp];
      const int m0 = tile_row(t) * TM + (CTA2 ? (int)pair_rank * BM : 0), n0 = (tile_col(t) - grp * tiles_g) * BN;
      const bool whole = vec_ok && n0 + BN <= N;            // a tile of full width: vector accesses through the staging block
      uint4 ahead[8];
#pragma unroll
      for (int it = 0; it < 8; ++it) ahead[it] = make_uint4(0, 0, 0, 0);
      if (whole && ep.gate != nullptr && ep.hs.P == 0 && (SPLIT == 1 || my_unit >= 0))
        fetch_resid(ahead, m0 + quarter * 32, n0 + (SPLIT > 1 ? my_unit * 64 : part * 128));
      ok = mbar_wait_warp(&acc_full[acc], acc_ph, abort_flag);
      if (SPLIT == 1 && !ok) break;
      tc_fence_after();
      const int row = m0 + quarter * 32 + lane;
      const uint32_t t_row = tmem_base + acc * BN + ((uint32_t)(quarter * 32) << 16);
      if (SPLIT > 1) {
        // One tile per cluster: this code runs once. Block (src, float4 column g of the slice) of the receiving CTA holds 128 rows x
        // 16 bytes, so that the lanes of a warp write and read 512 contiguous bytes.
        const int r_tile = quarter * 32 + lane;
        __syncwarp();
        cluster_sync_relaxed();        // every pair's MMAs are complete: the operand rings are free
        if (ok) {
#pragma unroll 1
          for (int c = part * 4; c < part * 4 + 4; ++c) {
            int dst = SPLIT - 1;       // the pair that finishes this 32-column chunk
            while (unit_first(dst) * 2 > c) --dst;
            if (dst == split) continue;
            uint32_t r[32];
            tmem_ld32(t_row + c * 32, r);
            tmem_ld_wait();
            const uint32_t base = mapa_shared(smem_u32(smem), (uint32_t)(2 * dst) + pair_rank) +
                                  (uint32_t)((split * (kSliceMax / 4) + (c * 32 - unit_first(dst) * 64) / 4) * (BM * 16) + r_tile * 16);
#pragma unroll
            for (int q = 0; q < 8; ++q)
              st_cluster_v4(base + q * (BM * 16), __uint_as_float(r[q * 4]), __uint_as_float(r[q * 4 + 1]), __uint_as_float(r[q * 4 + 2]),
                            __uint_as_float(r[q * 4 + 3]));
          }
        }
        __syncwarp();
        cluster_sync_all();            // every partial has arrived
        if (!ok) break;
        if (my_unit < 0) break;        // no unit left for this warp
#pragma unroll 1
        for (int c = my_unit * 2; c < my_unit * 2 + 2; ++c) {
          uint32_t own[32];
          tmem_ld32(t_row + c * 32, own);
          tmem_ld_wait();
          float sum[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) sum[j] = 0.f;
#pragma unroll
          for (int src = 0; src < SPLIT; ++src) {
            if (src == split) {
#pragma unroll
              for (int j = 0; j < 32; ++j) sum[j] += __uint_as_float(own[j]);
            } else {
              const uint8_t* in = smem + (src * (kSliceMax / 4) + (c * 32 - unit_first(split) * 64) / 4) * (BM * 16) + r_tile * 16;
#pragma unroll
              for (int q = 0; q < 8; ++q) {
                const float4 f = *reinterpret_cast<const float4*>(in + q * (BM * 16));
                sum[q * 4] += f.x; sum[q * 4 + 1] += f.y; sum[q * 4 + 2] += f.z; sum[q * 4 + 3] += f.w;
              }
            }
          }
#pragma unroll
          for (int j = 0; j < 32; ++j) own[j] = __float_as_uint(sum[j]);
          tmem_st32(t_row + c * 32, own);
        }
        tmem_st_wait();
      }
      if (ep.hs.P > 0) {
        // ---- fused head scatter: this thread owns one token row; a 256-wide tile holds two complete heads
        // tcgen05.ld is warp-collective: every lane runs every load, rows past M only skip their stores
        const bool valid = row < M;
        {
          const int row_c = valid ? row : M - 1;
          const int b_idx = row_c / ep.hs.S, s_idx = row_c % ep.hs.S;
          for (int hh = part; hh == part; ++hh) {      // this warp's head of the tile
            const int head = (n0 + hh * 128) >> 7;
            if ((head + 1) * 128 > N) break;
            const uint32_t t_head = t_row + hh * 128;
            float rstd = 1.f;
            if (ep.hs.w != nullptr) {          // pass 1: sum of squares over the head (TMEM re-reads are cheap)
              float ss = 0.f;
#pragma unroll 1
              for (int c = 0; c < 4; ++c) {
                uint32_t r[32];
                tmem_ld32(t_head + c * 32, r);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 32; ++j) ss = fmaf(__uint_as_float(r[j]), __uint_as_float(r[j]), ss);
              }
              rstd = rsqrtf(ss * (1.f / 128.f) + ep.hs.eps);
              if (ep.hs.rstd_out != nullptr && valid) ep.hs.rstd_out[(size_t)row * (N >> 7) + head] = rstd;
            }
            const unsigned long long raw_u =
                ep.hs.raw != nullptr ? reinterpret_cast<unsigned long long>(ep.hs.raw + (size_t)row_c * N + (size_t)head * 128) : 0ull;
            const int dst_rank = head / ep.hs.Hl, hl = head - dst_rank * ep.hs.Hl;
            bf16* dst = reinterpret_cast<bf16*>(ep.hs.ptrs[dst_rank]) +
                        ((((size_t)b_idx * ep.hs.P + ep.hs.rank) * ep.hs.S + s_idx) * ep.hs.Hl + hl) * 128;
            int c_cur = 0;
            // this thread's row (columns [32c, 32c + 32) in ``lo32`` and their rotation partners [64 + 32c, ...) in ``hi32``) goes to
            // the warp's staging block, 16-byte chunks XOR-swizzled by the row (no bank conflicts); then 4 lanes cover a 64-byte
            // run of a head row, so a warp store is eight contiguous 64-byte segments (local memory or a peer's over NVLink)
            // instead of 32 scattered 16-byte pieces
            auto emit = [&](const float (&lo32)[32], const float (&hi32)[32], unsigned long long dst_u) {
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                uint4 o0, o1;
                __nv_bfloat162* p0 = reinterpret_cast<__nv_bfloat162*>(&o0);
                __nv_bfloat162* p1 = reinterpret_cast<__nv_bfloat162*>(&o1);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  p0[j] = __floats2bfloat162_rn(lo32[q * 8 + 2 * j], lo32[q * 8 + 2 * j + 1]);
                  p1[j] = __floats2bfloat162_rn(hi32[q * 8 + 2 * j], hi32[q * 8 + 2 * j + 1]);
                }
                *reinterpret_cast<uint4*>(stage_row + ((q ^ (lane & 7)) << 4)) = o0;
                *reinterpret_cast<uint4*>(stage_row + (((4 + q) ^ (lane & 7)) << 4)) = o1;
              }
              __syncwarp();
#pragma unroll 4
              for (int it = 0; it < 8; ++it) {
                const int r_src = it * 4 + (lane >> 3), chunk = lane & 7;
                const unsigned long long d = __shfl_sync(0xffffffffu, dst_u, r_src);
                const int ok_row = __shfl_sync(0xffffffffu, (int)valid, r_src);
                const uint4 v = *reinterpret_cast<const uint4*>(stage_warp + r_src * 128 + ((chunk ^ (r_src & 7)) << 4));
                const int col = (chunk < 4 ? c_cur * 32 + chunk * 8 : 64 + c_cur * 32 + (chunk - 4) * 8);
                if (ok_row) *reinterpret_cast<uint4*>(d + col * 2) = v;
              }
              __syncwarp();
            };
#pragma unroll 1
            for (int c = 0; c < 2; ++c) {      // pass 2: columns [32c, 32c+32) and their rotation partners [64+32c, 64+32c+32)
              uint32_t lo[32], hi[32];
              tmem_ld32(t_head + c * 32, lo);
              tmem_ld32(t_head + 64 + c * 32, hi);
              tmem_ld_wait();
              float a[32], bb[32];
#pragma unroll
              for (int j = 0; j < 32; ++j) {
                a[j] = __uint_as_float(lo[j]);
                bb[j] = __uint_as_float(hi[j]);
              }
              c_cur = c;
              if (raw_u != 0ull) emit(a, bb, raw_u);        // warp-uniform: every lane of the kernel sees the same ep.hs.raw
              if (ep.hs.w != nullptr) {
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                  a[j] *= rstd * norm_weight(ep.hs, c * 32 + j);
                  bb[j] *= rstd * norm_weight(ep.hs, 64 + c * 32 + j);
                }
                if (ep.hs.cosv != nullptr) {
                  // this row's 32 cosines and sines come in through the staging block with coalesced loads (8 lanes per
                  // 128-byte run, 4 rows per instruction); reading them per thread straight from global memory would be
                  // 32 scattered 16-byte loads per instruction
                  float cs[32], sn[32];
                  auto fetch_rows = [&](const float* table, float (&out)[32]) {
#pragma unroll 4
                    for (int it = 0; it < 8; ++it) {
                      const int r_src = it * 4 + (lane >> 3), chunk = lane & 7;
                      const int s_src = __shfl_sync(0xffffffffu, s_idx, r_src);
                      const uint4 v4 = *reinterpret_cast<const uint4*>(table + (size_t)s_src * 64 + c * 32 + chunk * 4);
                      *reinterpret_cast<uint4*>(stage_warp + r_src * 128 + ((chunk ^ (r_src & 7)) << 4)) = v4;
                    }
                    __syncwarp();
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                      const float4 f = *reinterpret_cast<const float4*>(stage_row + ((q ^ (lane & 7)) << 4));
                      out[q * 4] = f.x; out[q * 4 + 1] = f.y; out[q * 4 + 2] = f.z; out[q * 4 + 3] = f.w;
                    }
                    __syncwarp();
                  };
                  fetch_rows(ep.hs.cosv, cs);
                  fetch_rows(ep.hs.sinv, sn);
#pragma unroll
                  for (int j = 0; j < 32; ++j) {
                    const float x0 = a[j], x1 = bb[j], cc = cs[j], s1 = sn[j];
                    a[j] = x0 * cc - x1 * s1;
                    bb[j] = x1 * cc + x0 * s1;
                  }
                }
              }
              emit(a, bb, reinterpret_cast<unsigned long long>(dst));
            }
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (CTA2) mbar_arrive_cluster_tmem(acc_empty_leader[acc]);
          else mbar_arrive(&acc_empty[acc]);
        }
        if (++acc == 2) { acc = 0; acc_ph ^= 1; }
        continue;
      }
      const float* gate_row = (ep.gate != nullptr && row < M) ? ep.gate + (size_t)(row / ep.L) * ep.ld_gate : nullptr;
      if (whole) {
        // ---- full-width tile: every global access of the epilogue goes through the warp's 4 KB staging block, so that a
        // warp instruction moves four contiguous 128-byte row segments instead of 32 scattered 16-byte pieces (the scattered
        // form made K = 2048 GEMMs epilogue-bound).  This warp owns 128 columns: two passes of 64; TMEM loads stay
        // warp-uniform.
        const int row0 = m0 + quarter * 32;
        auto write_out = [&](bf16* base, int colbase) {       // staged [32 rows x 64 cols] -> base[row, colbase ...]
          __syncwarp();
#pragma unroll 4
          for (int it = 0; it < 8; ++it) {
            const int r_src = it * 4 + (lane >> 3), chunk = lane & 7;
            const uint4 v4 = *reinterpret_cast<const uint4*>(stage_warp + r_src * 128 + ((chunk ^ (r_src & 7)) << 4));
            if (row0 + r_src < M) *reinterpret_cast<uint4*>(base + (size_t)(row0 + r_src) * N + colbase + chunk * 8) = v4;
          }
          __syncwarp();
        };
        auto stage_chunk = [&](int c, const float (&v)[32]) {   // this thread's columns [32c, 32c + 32) of the pass
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            uint4 o;
            __nv_bfloat162* o2 = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
            for (int j = 0; j < 4; ++j) o2[j] = __floats2bfloat162_rn(v[q * 8 + 2 * j], v[q * 8 + 2 * j + 1]);
            *reinterpret_cast<uint4*>(stage_row + (((c * 4 + q) ^ (lane & 7)) << 4)) = o;
          }
        };
        // many weights: this warp's 128 columns are one head, this thread's accumulator row all of it: the norm needs no exchange
        const void* const norm_w = NW > 3 ? bw.norm[NW > 3 ? grp : 0] : nullptr;
        float rstd = 1.f;
        if (NW > 3 && norm_w != nullptr) {
          float2 ss[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll 1
          for (int c = 0; c < 4; ++c) {
            uint32_t r[32];
            tmem_ld32(t_row + part * 128 + c * 32, r);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              const float2 v = make_float2(__uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1]));
              ss[j & 1] = fma2(v, v, ss[j & 1]);
            }
          }
          const float2 t2 = add2(ss[0], ss[1]);
          rstd = rsqrtf((t2.x + t2.y) * (1.f / 128.f) + ep.norm_eps);
        }
#pragma unroll 1
        for (int pass = 0; pass < (SPLIT > 1 ? 1 : 2); ++pass) {
          const int coff = SPLIT > 1 ? my_unit * 64 : part * 128 + pass * 64;   // column offset inside the tile
          const int colbase = n0 + coff;
          if (ep.pre != nullptr && (ep.act == 1 || ep.gate != nullptr)) {
            // second output first (TMEM is read again below): the pre-activation of a GELU, or the plain product of a
            // gated-residual GEMM (training keeps it for the gate gradient)
#pragma unroll 1
            for (int c = 0; c < 2; ++c) {
              uint32_t r[32];
              tmem_ld32(t_row + coff + c * 32, r);
              tmem_ld_wait();
              float v[32];
#pragma unroll
              for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
              if (ep.bias != nullptr) {
#pragma unroll
                for (int j = 0; j < 32; ++j) v[j] += __bfloat162float(ep.bias[colbase + c * 32 + j]);
              }
              stage_chunk(c, v);
            }
            write_out(ep.pre, colbase);
          }
          if (ep.gate != nullptr) {                             // residual rows, fetched coalesced
#pragma unroll
            for (int it = 0; it < 8; ++it) {
              const int r_src = it * 4 + (lane >> 3), chunk = lane & 7;
              *reinterpret_cast<uint4*>(stage_warp + r_src * 128 + ((chunk ^ (r_src & 7)) << 4)) = ahead[it];
            }
            __syncwarp();
            if (SPLIT == 1 && pass == 0) fetch_resid(ahead, row0, colbase + 64);
          }
#pragma unroll 1
          for (int c = 0; c < 2; ++c) {
            const int col0 = colbase + c * 32;
            uint32_t r[32];
            tmem_ld32(t_row + coff + c * 32, r);
            tmem_ld_wait();
            float v[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
            if (NW > 3) {
              if (norm_w != nullptr) {
                const int i0 = pass * 64 + c * 32;          // channel of the head
                const bool wb = bw.norm_bf16[NW > 3 ? grp : 0] != 0;
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                  float w8[8];
                  if (wb) {
                    unpack8(*reinterpret_cast<const bf16x8*>(reinterpret_cast<const bf16*>(norm_w) + i0 + q * 8), w8);
                  } else {
                    const float4* w4 = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(norm_w) + i0 + q * 8);
                    const float4 f0 = w4[0], f1 = w4[1];
                    w8[0] = f0.x; w8[1] = f0.y; w8[2] = f0.z; w8[3] = f0.w; w8[4] = f1.x; w8[5] = f1.y; w8[6] = f1.z; w8[7] = f1.w;
                  }
#pragma unroll
                  for (int j = 0; j < 8; ++j) v[q * 8 + j] = v[q * 8 + j] * rstd * w8[j];
                }
              }
              stage_chunk(c, v);
              continue;
            }
            if (ep.bias != nullptr) {
#pragma unroll
              for (int j = 0; j < 32; ++j) v[j] += __bfloat162float(ep.bias[col0 + j]);
            }
            if (ep.act == 1) gelu32(v);
            if (ep.gate != nullptr) {
              float4 g4[8];                                     // all of the chunk's gate values at once: one latency
#pragma unroll
              for (int q = 0; q < 8; ++q)
                g4[q] = gate_row != nullptr ? *reinterpret_cast<const float4*>(gate_row + col0 + q * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                const uint4 rr = *reinterpret_cast<const uint4*>(stage_row + (((c * 4 + q) ^ (lane & 7)) << 4));
                const __nv_bfloat162* r2 = reinterpret_cast<const __nv_bfloat162*>(&rr);
                const float4 g0 = g4[2 * q], g1 = g4[2 * q + 1];
                const float g[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  const float2 rf = __bfloat1622float2(r2[j]);
                  v[q * 8 + 2 * j] = rf.x + g[2 * j] * v[q * 8 + 2 * j];
                  v[q * 8 + 2 * j + 1] = rf.y + g[2 * j + 1] * v[q * 8 + 2 * j + 1];
                }
              }
            }
            stage_chunk(c, v);                                  // in place: a thread only ever touches its own row here
          }
          write_out(out, colbase);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (CTA2) mbar_arrive_cluster_tmem(acc_empty_leader[acc]);
          else mbar_arrive(&acc_empty[acc]);
        }
        if (++acc == 2) { acc = 0; acc_ph ^= 1; }
        continue;
      }
#pragma unroll 1
      for (int c = part * 4; c < part * 4 + 4; ++c) {
        uint32_t r[32];
        tmem_ld32(t_row + c * 32, r);
        tmem_ld_wait();
        const int col0 = n0 + c * 32;
        if (row < M && col0 < N) {
          float v[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
          const bool full_chunk = vec_ok && (col0 + 32 <= N);
          const size_t off = (size_t)row * N + col0;
          if (ep.bias != nullptr) {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (full_chunk || col0 + j < N) v[j] += __bfloat162float(ep.bias[col0 + j]);
          }
          if (ep.act == 1) {
            if (ep.pre != nullptr) {
              if (full_chunk) {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                  uint4 o;
                  __nv_bfloat162* o2 = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
                  for (int j = 0; j < 4; ++j) o2[j] = __floats2bfloat162_rn(v[q * 8 + 2 * j], v[q * 8 + 2 * j + 1]);
                  *reinterpret_cast<uint4*>(ep.pre + off + q * 8) = o;
                }
              } else {
                for (int j = 0; j < 32 && col0 + j < N; ++j) ep.pre[off + j] = __float2bfloat16(v[j]);
              }
            }
            gelu32(v);
          }
          if (gate_row != nullptr) {
            if (full_chunk) {
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                const uint4 rr = *reinterpret_cast<const uint4*>(ep.resid + off + q * 8);
                const __nv_bfloat162* r2 = reinterpret_cast<const __nv_bfloat162*>(&rr);
                const float4 g0 = *reinterpret_cast<const float4*>(gate_row + col0 + q * 8);
                const float4 g1 = *reinterpret_cast<const float4*>(gate_row + col0 + q * 8 + 4);
                const float g[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  const float2 rf = __bfloat1622float2(r2[j]);
                  v[q * 8 + 2 * j] = rf.x + g[2 * j] * v[q * 8 + 2 * j];
                  v[q * 8 + 2 * j + 1] = rf.y + g[2 * j + 1] * v[q * 8 + 2 * j + 1];
                }
              }
            } else {
              for (int j = 0; j < 32 && col0 + j < N; ++j)
                v[j] = __bfloat162float(ep.resid[off + j]) + gate_row[col0 + j] * v[j];
            }
          }
          if (full_chunk) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              uint4 o;
              __nv_bfloat162* o2 = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
              for (int j = 0; j < 4; ++j) o2[j] = __floats2bfloat162_rn(v[q * 8 + 2 * j], v[q * 8 + 2 * j + 1]);
              *reinterpret_cast<uint4*>(out + off + q * 8) = o;
            }
          } else {
            for (int j = 0; j < 32 && col0 + j < N; ++j) out[off + j] = __float2bfloat16(v[j]);
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
          if (CTA2) mbar_arrive_cluster_tmem(acc_empty_leader[acc]);
          else mbar_arrive(&acc_empty[acc]);
        }
      if (++acc == 2) { acc = 0; acc_ph ^= 1; }
    }
    if (!ok && lane == 0) { atomicCAS(err, 0, 3); *abort_flag = 1; }
  }

  // ---------------------------------------------------------------------- teardown
  __syncwarp();
  if (*abort_flag) {
    // let outstanding bulk copies / MMAs drain before shared memory and TMEM go away
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  if (CTA2) cluster_sync_relaxed();  // neither CTA leaves (or frees TMEM) while the other may still signal it or read its tiles
  if (warp == 1) {
    tc_fence_after();
    if (CTA2) tmem_dealloc_pair(tmem_base, 512);
    else tmem_dealloc(tmem_base, 512);
  }
}

// Few tiles of a very long contraction (the projection of a prompt: 100,352 deep, 4 to 74 tiles). Clusters of pairs per tile leave SMs idle
// where the tiles times a whole number of pairs do not fill the GPU, and take four pairs at most. Here `per_tile` pairs share a tile's k-blocks
// in turn, all tiles in step, so that what neighbouring tiles have in common comes from L2; pairs left over share the last `tail` k-blocks of
// all tiles, tile by tile. Each pair writes its sums as fp32 partial tiles to global memory and gemm_stream_finish_kernel adds them in a fixed
// order: no CTA waits for another pair's work. (With equal shares of all tiles' k-blocks in a row no two pairs were at the same k-block, and
// 1024 x 1024 read 1.6 GB instead of 0.4: 215 us.) Both operands K-major, N a multiple of 256.
// ws: [slot][64 column quadruples][256 rows] float4; slots: pair turn * tiles + tile, then three for each pair of the tail.
// From K = 100,352 to 1024 columns, before and now: 256 rows 125 and 72 us, 512 127 and 83, 768 133 and 115, 1024 174 and 154, 1536 251 and 206,
// 3072 490 and 441; 2048 rows (32 tiles, two pairs each) would go from 282 to 332 and stay with clusters. Where the line lies: cb200_gemm_stream.
struct StreamPlan {
  int tiles, tiles_n, k_all;
  int per_tile, extra, tail;     // pairs a tile, pairs of the tail, k-blocks of a tile that are theirs
};
constexpr int kStreamSlots = 3;  // tiles that a pair of the tail can touch: at most two tiles' worth of tails (see stream_plan)
__host__ __device__ inline int stream_tail_first(const StreamPlan& pl, int e) { return (int)((long)e * pl.tiles * pl.tail / pl.extra); }

__global__ void __launch_bounds__(kGemmThreads, 1)
gemm_stream_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b, float* __restrict__ ws, StreamPlan pl,
                   int* __restrict__ err) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  constexpr int STG = 6, STG_BYTES = kABytes + kBBytes / 2, TM = 2 * BM;
  const uint32_t rank = cluster_ctarank();
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + STG * STG_BYTES);
  uint64_t* full = bars;                    // [STG]
  uint64_t* empty = bars + STG;             // [STG]
  uint64_t* acc_full = bars + 2 * STG;      // [2]
  uint64_t* acc_empty = acc_full + 2;       // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int pair = (int)blockIdx.x >> 1, tail_pair = pair - pl.per_tile * pl.tiles;
  const int g0 = tail_pair >= 0 ? stream_tail_first(pl, tail_pair) : 0, g1 = tail_pair >= 0 ? stream_tail_first(pl, tail_pair + 1) : 0;
  const int t0 = tail_pair >= 0 ? g0 / pl.tail : pair % pl.tiles, n_seg = tail_pair < 0 ? 1 : g1 > g0 ? (g1 - 1) / pl.tail - t0 + 1 : 0;
  const int slot0 = tail_pair < 0 ? pair : pl.per_tile * pl.tiles + tail_pair * kStreamSlots;
  const int head = pl.k_all - pl.tail;             // k-blocks that the pairs of a tile share
  // k-blocks lo, lo + step, ... below hi of segment s, which lies in tile t0 + s
  const int step = tail_pair < 0 ? pl.per_tile : 1;
  auto range = [&](int s, int& lo, int& hi) {
    if (tail_pair < 0) {
      lo = pair / pl.tiles;
      hi = head;
    } else {
      lo = head + max(g0 - (t0 + s) * pl.tail, 0);
      hi = head + min(g1 - (t0 + s) * pl.tail, pl.tail);
    }
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < STG; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&acc_full[a], 1);
      mbar_init(&acc_empty[a], 16);         // the even CTA hears from the epilogue warps of both
    }
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, 512);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_relaxed();            // the other CTA's barriers exist before anything signals them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_trigger();                     // launched with programmatic serialisation (see common.cuh)
  pdl_wait();

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      prefetch_tmap(&tma_a);
      prefetch_tmap(&tma_b);
      int st = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int s = 0; s < n_seg && ok; ++s) {
        int lo, hi;
        range(s, lo, hi);
        const int m0 = (t0 + s) / pl.tiles_n * TM + (int)rank * BM, n0 = (t0 + s) % pl.tiles_n * BN + (int)rank * (BN / 2);
        for (int kb = lo; kb < hi; kb += step) {
          if (!mbar_wait(&empty[st], ph ^ 1, abort_flag)) { ok = false; break; }
          uint8_t* sa = smem + st * STG_BYTES;
          if (rank == 0) mbar_arrive_expect_tx(&full[st], 2 * STG_BYTES);
          const uint32_t bar = mapa_shared(smem_u32(&full[st]), 0);
          tma_load_2d_pair(sa, &tma_a, bar, kb * BK, m0);
          tma_load_2d_pair(sa + kABytes, &tma_b, bar, kb * BK, n0);
          if (++st == STG) { st = 0; ph ^= 1; }
        }
      }
      if (!ok) { atomicCAS(err, 0, 4); *abort_flag = 1; }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (warp-uniform; the elected lane issues)
    const uint32_t leader = elect_one() ? 1u : 0u;
    auto wait_all = [&](uint64_t* bar, uint32_t parity) -> bool { return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag)); };
    constexpr uint32_t idesc = umma_idesc_bf16(TM, BN, 0, 0);
    const uint64_t da0 = umma_desc_sw128(smem_u32(smem), 16, 1024), db0 = umma_desc_sw128(smem_u32(smem) + kABytes, 16, 1024);
    int st = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int s = 0; s < n_seg && ok && rank == 0; ++s) {     // only the even CTA issues
      int lo, hi;
      range(s, lo, hi);
      if (!wait_all(&acc_empty[s & 1], ((s >> 1) & 1) ^ 1)) { ok = false; break; }
      tc_fence_after();
      for (int kb = lo; kb < hi; kb += step) {
        if (!wait_all(&full[st], ph)) { ok = false; break; }
        tc_fence_after();
        const uint64_t da = da0 + (uint64_t)(st * (STG_BYTES >> 4)), db = db0 + (uint64_t)(st * (STG_BYTES >> 4));
#pragma unroll
        for (int k = 0; k < BK / UK; ++k)
          umma_ss_pair_w(tmem_base + (s & 1) * BN, da + (uint32_t)((k * UK * 2) >> 4), db + (uint32_t)((k * UK * 2) >> 4), idesc,
                         (kb > lo || k > 0) ? 1u : 0u, leader);
        umma_commit_pair_w(&empty[st], leader);
        if (++st == STG) { st = 0; ph ^= 1; }
      }
      if (ok) umma_commit_pair_w(&acc_full[s & 1], leader);
    }
    if (!ok && lane == 0) { atomicCAS(err, 0, 5); *abort_flag = 1; }
  } else {
    // ------------------------------------------------------------------ epilogue warps: 32 rows x 128 columns of each partial tile
    const int quarter = warp & 3, part = (warp - 2) >> 2;
    bool ok = true;
    for (int s = 0; s < n_seg && ok; ++s) {
      ok = mbar_wait_warp(&acc_full[s & 1], (s >> 1) & 1, abort_flag);
      if (!ok) break;
      tc_fence_after();
      float4* dst = reinterpret_cast<float4*>(ws) + ((size_t)(slot0 + s) * (BN / 4)) * TM + rank * BM + quarter * 32 + lane;
#pragma unroll 1
      for (int c = part * 4; c < part * 4 + 4; ++c) {
        uint32_t r[32];
        tmem_ld32(tmem_base + (s & 1) * BN + ((uint32_t)(quarter * 32) << 16) + c * 32, r);
        tmem_ld_wait();
#pragma unroll
        for (int q = 0; q < 8; ++q)
          dst[(size_t)(c * 8 + q) * TM] = make_float4(__uint_as_float(r[q * 4]), __uint_as_float(r[q * 4 + 1]), __uint_as_float(r[q * 4 + 2]),
                                                      __uint_as_float(r[q * 4 + 3]));
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster_tmem(mapa_shared(smem_u32(&acc_empty[s & 1]), 0));
    }
    if (!ok && lane == 0) { atomicCAS(err, 0, 6); *abort_flag = 1; }
  }

  __syncwarp();
  if (*abort_flag) {
    // let outstanding bulk copies / MMAs drain before shared memory and TMEM go away
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_relaxed();            // neither CTA leaves (or frees TMEM) while the other may still signal it or read its tiles
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

// C = act(sum of the partial tiles + bias), optionally also the value in front of the activation. A CTA takes 32 rows x 64 columns of a tile, a
// warp 8 of the columns.
__global__ void __launch_bounds__(256) gemm_stream_finish_kernel(const float* __restrict__ ws, bf16* __restrict__ C, bf16* __restrict__ pre,
                                                                 const bf16* __restrict__ bias, int act, int M, int N, StreamPlan pl) {
  pdl_trigger();                     // launched with programmatic serialisation (see common.cuh)
  pdl_wait();
  constexpr int TM = 2 * BM;
  const int tile = (int)blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int r = (int)(blockIdx.x >> 2) * 32 + lane, c8 = (int)(blockIdx.x & 3) * 8 + warp;        // row and 8-column group of the tile
  const int row = tile / pl.tiles_n * TM + r, col = tile % pl.tiles_n * BN + c8 * 8;
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
  auto add = [&](int slot) {
    const float4* src = reinterpret_cast<const float4*>(ws) + ((size_t)slot * (BN / 4) + c8 * 2) * TM + r;
    const float4 u = src[0], v = src[TM];
    a.x += u.x; a.y += u.y; a.z += u.z; a.w += u.w;
    b.x += v.x; b.y += v.y; b.z += v.z; b.w += v.w;
  };
#pragma unroll 4
  for (int i = 0; i < pl.per_tile; ++i) add(i * pl.tiles + tile);
  if (pl.tail > 0) {
    // the pairs of the tail whose range [first, next) meets this tile's [tile * tail, (tile + 1) * tail)
    for (int e = 0; e < pl.extra; ++e) {
      const int g0 = stream_tail_first(pl, e), g1 = stream_tail_first(pl, e + 1);
      if (g0 < (tile + 1) * pl.tail && g1 > tile * pl.tail && g1 > g0)
        add(pl.per_tile * pl.tiles + e * kStreamSlots + tile - g0 / pl.tail);
    }
  }
  if (row >= M) return;
  float o[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
  if (bias != nullptr) {
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] += __bfloat162float(bias[col + j]);
  }
  if (act == 1) {
    if (pre != nullptr) *reinterpret_cast<bf16x8*>(pre + (size_t)row * N + col) = pack8(o);
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
      const float2 g = gelu2(make_float2(o[j], o[j + 1]));
      o[j] = g.x;
      o[j + 1] = g.y;
    }
  }
  *reinterpret_cast<bf16x8*>(C + (size_t)row * N + col) = pack8(o);
}

}  // namespace cb200

using namespace cb200;

template <int A_MN, int B_MN, bool GATHER = false>
static int launch_gemm(const void* A, const void* B, bf16* C, int M, int N, int K, const GemmEpilogue& ep, int* err, int sms,
                       cudaStream_t st, const GatherB& gb = GatherB{}) {
  CUtensorMap ta;
  GemmWeights<3> bw{};
  CUtensorMap& tb = bw.map[0];
  int rc;
  // A: K-major [M,K] -> dims {K, M}, box {64, 128};  MN-major stored [K,M] -> dims {M, K}, box {64, 64}
  if (A_MN == 0) rc = make_tmap_2d_bf16(&ta, A, (uint64_t)K, (uint64_t)M, (uint64_t)K * 2, BK, BM);
  else rc = make_tmap_2d_bf16(&ta, A, (uint64_t)M, (uint64_t)K, (uint64_t)M * 2, 64, BK);
  if (rc) return rc;
  if (B_MN == 0) rc = make_tmap_2d_bf16(&tb, B, (uint64_t)K, (uint64_t)N, (uint64_t)K * 2, BK, BN);
  else rc = make_tmap_2d_bf16(&tb, B, (uint64_t)N, (uint64_t)K, (uint64_t)N * 2, 64, BK);
  if (rc) return rc;
  bw.out[0] = C;
  static bool attr_set = false;      // one flag per template instantiation
  auto kern = gemm_bf16_kernel<A_MN, B_MN, GATHER>;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes);
    if (e != cudaSuccess) return 100 + (int)e;
    attr_set = true;
  }
  const int tiles = ((M + BM - 1) / BM) * ((N + BN - 1) / BN);
  // with a gather every SM takes part (its gather warps work even when it has no tile): the grid is the whole machine
  const int grid = GATHER ? sms : (tiles < sms ? tiles : sms);
  kern<<<grid, kGemmThreads + (GATHER ? kGatherWarps * 32 : 0), kSmemBytes, st>>>(ta, bw, M, N, K, ep, gb, err);
  return (int)cudaGetLastError();
}

// Same contraction on CTA pairs (template flag CTA2): clusters of SPLIT pairs, one 256 x 256 tile per cluster.
struct PairLaunch {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[2];
  PairLaunch(int split, int clusters, cudaStream_t st) {
    cfg.gridDim = dim3(2 * split * clusters);
    cfg.blockDim = dim3(kGemmThreads);
    cfg.dynamicSmemBytes = kSmemBytes;
    cfg.stream = st;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2 * split;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 2;
  }
  PairLaunch(const PairLaunch&) = delete;
};

extern "C" int cb200_gemm_pair_mode(int mode);

// clusters that the GPU holds at once: none where it has no room for one (a share of a GPU)
template <int A_MN, int B_MN, int SPLIT, int NW = 3>
static int resident_clusters(int* clusters) {
  static int resident = -1;
  if (resident < 0) {
    const auto kern = gemm_bf16_kernel<A_MN, B_MN, false, true, SPLIT, NW>;
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes);
    if (e != cudaSuccess) return 100 + (int)e;
    PairLaunch l(SPLIT, 1, nullptr);
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &l.cfg) != cudaSuccess) {
      cudaGetLastError();
      n = 0;
    }
    resident = n;
  }
  *clusters = resident;
  return 0;
}

template <int A_MN, int B_MN, int SPLIT, int NW = 3>
static int launch_gemm_pairs(const void* A, const void* const* B, void* const* C, int M, int N, int K, const GemmEpilogue& ep, int clusters,
                             int* err, cudaStream_t st, const void* const* norm = nullptr, const uint8_t* norm_bf16 = nullptr) {
  CUtensorMap ta;
  GemmWeights<NW> bw{};
  int rc;
  if (A_MN == 0) rc = make_tmap_2d_bf16(&ta, A, (uint64_t)K, (uint64_t)M, (uint64_t)K * 2, BK, BM);
  else rc = make_tmap_2d_bf16(&ta, A, (uint64_t)M, (uint64_t)K, (uint64_t)M * 2, 64, BK);
  if (rc) return rc;
  for (int g = 0; g < ep.groups; ++g) {
    if (B_MN == 0) rc = make_tmap_2d_bf16(&bw.map[g], B[g], (uint64_t)K, (uint64_t)N, (uint64_t)K * 2, BK, BN / 2);   // each CTA loads half the columns
    else rc = make_tmap_2d_bf16(&bw.map[g], B[g], (uint64_t)N, (uint64_t)K, (uint64_t)N * 2, 64, BK);
    if (rc) return rc;
    bw.out[g] = (bf16*)C[g];
    if (NW > 3 && norm != nullptr) {
      bw.norm[NW > 3 ? g : 0] = norm[g];
      bw.norm_bf16[NW > 3 ? g : 0] = norm_bf16[g];
    }
  }
  PairLaunch l(SPLIT, clusters, st);
  const cudaError_t e = cudaLaunchKernelEx(&l.cfg, gemm_bf16_kernel<A_MN, B_MN, false, true, SPLIT, NW>, ta, bw, M, N, K, ep, GatherB{}, err);
  return e == cudaSuccess ? 0 : 500 + (int)e;
}

// One tile per pair, or clusters of 2 to 4 pairs per tile: whichever takes fewer k-blocks in a row, waves counted, with kExchange
// k-blocks' time for the exchange of partial tiles, twice that for three pairs (0.27 us a k-block; two pairs 2.4 to 2.9 us, three 4.3).
// Launches back to back with one, two and three pairs per tile: 512 x 2048 from K = 2048 16.0, 14.1, 14.6 us, from K = 8192 43.8, 29.1,
// 25.2 us; 1024 x 1024 from K = 100,352 (the text projection) 449, 230, 181 us. A B200 holds 33 clusters of two pairs, 22 of three and 15
// or 16 of four: for 16 tiles (512 x 2048) four pairs are one wave on some of them and two on the others (38.9 us at K = 8192).
// `c2`, `c4`, `c3`: clusters of 2, 4 and 3 pairs that the GPU holds at once; where it holds none the split is not taken.
extern "C" int cb200_gemm_pairs_per_tile(long tiles, long kb, int pairs, int c2, int c4, int c3) {
  if (2 * tiles > pairs || kb < 8) return 1;
  constexpr long kExchange = 6;
  long best = kb;
  int split = 1;
  if (c2 > 0 && (tiles + c2 - 1) / c2 * ((kb + 1) / 2 + kExchange) < best) {
    best = (tiles + c2 - 1) / c2 * ((kb + 1) / 2 + kExchange);
    split = 2;
  }
  if (c3 > 0 && (tiles + c3 - 1) / c3 * ((kb + 2) / 3 + 2 * kExchange) < best) {
    best = (tiles + c3 - 1) / c3 * ((kb + 2) / 3 + 2 * kExchange);
    split = 3;
  }
  if (c4 > 0 && (tiles + c4 - 1) / c4 * ((kb + 3) / 4 + kExchange) < best + (split == 2 ? 1 : 0)) split = 4;
  return split;
}

// How gemm_stream_kernel would share out `tiles` tiles of `kb` k-blocks over `pairs` pairs. The tail's pairs take equal parts of its k-blocks, two
// tiles' worth at most (three tiles touched); where they are too few for that there is no tail.
static StreamPlan stream_plan(int tiles, int tiles_n, int kb, int pairs) {
  StreamPlan pl{tiles, tiles_n, kb, pairs / tiles, 0, 0};
  pl.extra = pairs - pl.per_tile * tiles;
  pl.tail = 2 * pl.extra >= tiles ? (int)((long)kb * pl.extra / pairs) : 0;
  if (pl.tail == 0) pl.extra = 0;
  return pl;
}
// Whether that takes less time than the rule above or whole waves of tiles. In units of 10 ns, fitted to launches back to back from K = 8192 to
// 100,352: k-blocks in a row of clusters take 5.5 us + 0.31 us each (within 3 %); shared out, a pair's k-block takes 0.43 us (all pairs draw
// on L2 at once), and the second launch 10 us and what it adds up one after another: 0.55 us for each pair of a tile and 0.33 us for each
// pair of the tail. 256 x 256, where 74 partial tiles are added, takes 46 us from any K up to 32,768 and clusters 22 us from 12,288;
// 256 x 768 from 12,288 28.4 and 22.4, from 32,768 33.5 and 45.5; 4096 x 768 (26 pairs of the tail) from 12,288 74.6 and 65.5, from 32,768
// 163 and 167.
extern "C" int cb200_gemm_stream(long tiles, long kb, int pairs, int c2, int c4, int c3, int* per_tile, int* extra, int* tail) {
  constexpr long kExchange = 6;
  if (tiles < 1 || tiles > pairs || kb < pairs) return 0;
  const int split = cb200_gemm_pairs_per_tile(tiles, kb, pairs, c2, c4, c3);
  const long now = split == 2   ? (tiles + c2 - 1) / c2 * ((kb + 1) / 2 + kExchange)
                   : split == 3 ? (tiles + c3 - 1) / c3 * ((kb + 2) / 3 + 2 * kExchange)
                   : split == 4 ? (tiles + c4 - 1) / c4 * ((kb + 3) / 4 + kExchange)
                                : kb;
  const StreamPlan pl = stream_plan((int)tiles, 1, (int)kb, pairs);
  if (per_tile != nullptr) *per_tile = pl.per_tile;
  if (extra != nullptr) *extra = pl.extra;
  if (tail != nullptr) *tail = pl.tail;
  const long share = (kb - pl.tail + pl.per_tile - 1) / pl.per_tile;
  return 1000 + 43 * share + 55 * pl.per_tile + 33 * pl.extra < 550 + 31 * now ? 1 : 0;
}

// pairs that the GPU holds at once for gemm_stream_kernel
static int stream_pairs(int sms, int* pairs) {
  static int resident = -1;
  if (resident < 0) {
    const cudaError_t e = cudaFuncSetAttribute(gemm_stream_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes);
    if (e != cudaSuccess) return 100 + (int)e;
    PairLaunch l(1, 1, nullptr);
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, gemm_stream_kernel, &l.cfg) != cudaSuccess) {
      cudaGetLastError();
      n = 0;
    }
    resident = n;
  }
  *pairs = std::min(resident, sms / 2);
  return 0;
}

// what the rules above count with on this GPU: pairs of gemm_stream_kernel, clusters of 2, 4 and 3 pairs (K-major operands) held at once
extern "C" int cb200_gemm_clusters(int sms, int* pairs, int* c2, int* c4, int* c3) {
  int rc;
  if ((rc = stream_pairs(sms, pairs)) || (rc = resident_clusters<0, 0, 2>(c2)) || (rc = resident_clusters<0, 0, 4>(c4))) return rc;
  return resident_clusters<0, 0, 3>(c3);
}

// fp32 values of scratch with which cb200_gemm_bf16 can share out the k-blocks of this product, 0: it would not
extern "C" long cb200_gemm_stream_floats(int M, int N, int K, int a_mn, int b_mn, int gated, int sms) {
  if (a_mn || b_mn || gated || M < 2 * BM || N % BN != 0 || K % 8 != 0 || K < 64 * BK || cb200_gemm_pair_mode(-1) != 1) return 0;
  int pairs = 0, c2 = 0, c3 = 0, c4 = 0;
  if (cb200_gemm_clusters(sms, &pairs, &c2, &c4, &c3)) return 0;
  const long tiles = (long)((M + 2 * BM - 1) / (2 * BM)) * (N / BN);
  if (!cb200_gemm_stream(tiles, (K + BK - 1) / BK, pairs, c2, c4, c3, nullptr, nullptr, nullptr)) return 0;
  const StreamPlan pl = stream_plan((int)tiles, N / BN, (K + BK - 1) / BK, pairs);
  return (long)(pl.per_tile * pl.tiles + pl.extra * kStreamSlots) * 2 * BM * BN;
}

static int launch_gemm_stream(const void* A, const void* B, void* C, int M, int N, int K, const GemmEpilogue& ep, float* ws, int* err, int sms,
                              cudaStream_t st) {
  CUtensorMap ta, tb;
  int pairs = 0, rc;
  if ((rc = stream_pairs(sms, &pairs))) return rc;
  if ((rc = make_tmap_2d_bf16(&ta, A, (uint64_t)K, (uint64_t)M, (uint64_t)K * 2, BK, BM))) return rc;
  if ((rc = make_tmap_2d_bf16(&tb, B, (uint64_t)K, (uint64_t)N, (uint64_t)K * 2, BK, BN / 2))) return rc;
  const int tiles = (M + 2 * BM - 1) / (2 * BM) * (N / BN);
  const StreamPlan pl = stream_plan(tiles, N / BN, (K + BK - 1) / BK, pairs);
  PairLaunch l(1, pl.per_tile * tiles + pl.extra, st);
  cudaError_t e = cudaLaunchKernelEx(&l.cfg, gemm_stream_kernel, ta, tb, ws, pl, err);
  if (e != cudaSuccess) return 500 + (int)e;
  e = launch_pdl(gemm_stream_finish_kernel, dim3(2 * BM / 32 * 4, tiles), dim3(256), 0, st, ws, (bf16*)C, ep.pre, ep.bias, ep.act, M, N, pl);
  return e == cudaSuccess ? 0 : 500 + (int)e;
}

template <int A_MN, int B_MN>
static int launch_gemm_any(const void* A, const void* const* B, void* const* C, int M, int N, int K, const GemmEpilogue& ep, int* err, int sms,
                          cudaStream_t st) {
  const long tiles = (long)((M + 2 * BM - 1) / (2 * BM)) * ((N + BN - 1) / BN) * ep.groups, kb = (K + BK - 1) / BK;
  const int pairs = sms / 2;
  int c1 = 0, c2 = 0, c3 = 0, c4 = 0, rc;
  if (N % BN == 0 && ep.hs.P == 0 && 2 * tiles <= pairs) {
    if ((rc = resident_clusters<A_MN, B_MN, 2>(&c2)) || (rc = resident_clusters<A_MN, B_MN, 3>(&c3)) || (rc = resident_clusters<A_MN, B_MN, 4>(&c4)))
      return rc;
    const int split = cb200_gemm_pairs_per_tile(tiles, kb, pairs, c2, c4, c3);
    if (split == 4) return launch_gemm_pairs<A_MN, B_MN, 4>(A, B, C, M, N, K, ep, (int)tiles, err, st);
    if (split == 3) return launch_gemm_pairs<A_MN, B_MN, 3>(A, B, C, M, N, K, ep, (int)tiles, err, st);
    if (split == 2) return launch_gemm_pairs<A_MN, B_MN, 2>(A, B, C, M, N, K, ep, (int)tiles, err, st);
  }
  // A persistent grid must be resident as a whole: the pairs that the GPU can hold at once (a pair lives inside one GPC, so a
  // GPC with an odd number of free SMs leaves one out) bound the grid, otherwise late pairs would run after the others.
  if ((rc = resident_clusters<A_MN, B_MN, 1>(&c1))) return rc;
  if (c1 < 1) return 600;
  return launch_gemm_pairs<A_MN, B_MN, 1>(A, B, C, M, N, K, ep, (int)std::min<long>(tiles, std::min(c1, pairs)), err, st);
}

// 0: single-CTA tiles; 1 (default): CTA pairs where the shape allows (measured 8-45 % faster on the 2B shapes: half the B-operand
// bytes per CTA). COSMOS_B200_GEMM_PAIR=0 selects single-CTA tiles; cb200_gemm_pair_mode switches at run time (the kernel
// benchmark compares the two).
static int g_pair_mode = -1;
extern "C" int cb200_gemm_pair_mode(int mode) {
  if (g_pair_mode < 0) {
    const char* e = getenv("COSMOS_B200_GEMM_PAIR");
    g_pair_mode = (e != nullptr && e[0] == '0') ? 0 : 1;
  }
  const int prev = g_pair_mode;
  if (mode >= 0) g_pair_mode = mode;
  return prev;
}

extern "C" int cb200_gemm_bf16(const void* A, const void* B, void* C, int M, int N, int K, int a_mn, int b_mn,
                               const void* bias, int act, void* pre, const void* resid, const float* gate, long ld_gate, int L,
                               int* err, int sms, cudaStream_t st, float* ws) {
  GemmEpilogue ep{};
  ep.groups = 1;
  ep.pre = (bf16*)pre;
  ep.bias = (const bf16*)bias;
  ep.resid = (const bf16*)resid;
  ep.gate = gate;
  ep.ld_gate = ld_gate;
  ep.act = act;
  ep.L = L > 0 ? L : 1;
  if (ws != nullptr && cb200_gemm_stream_floats(M, N, K, a_mn, b_mn, gate != nullptr, sms) > 0)
    return launch_gemm_stream(A, B, C, M, N, K, ep, ws, err, sms, st);
  if (cb200_gemm_pair_mode(-1) == 1 && M >= 2 * BM && N % 8 == 0) {
    if (a_mn == 0 && b_mn == 0) return launch_gemm_any<0, 0>(A, &B, &C, M, N, K, ep, err, sms, st);
    if (a_mn == 0 && b_mn == 1) return launch_gemm_any<0, 1>(A, &B, &C, M, N, K, ep, err, sms, st);
    if (a_mn == 1 && b_mn == 0) return launch_gemm_any<1, 0>(A, &B, &C, M, N, K, ep, err, sms, st);
    return launch_gemm_any<1, 1>(A, &B, &C, M, N, K, ep, err, sms, st);
  }
  if (a_mn == 0 && b_mn == 0) return launch_gemm<0, 0>(A, B, (bf16*)C, M, N, K, ep, err, sms, st);
  if (a_mn == 0 && b_mn == 1) return launch_gemm<0, 1>(A, B, (bf16*)C, M, N, K, ep, err, sms, st);
  if (a_mn == 1 && b_mn == 0) return launch_gemm<1, 0>(A, B, (bf16*)C, M, N, K, ep, err, sms, st);
  return launch_gemm<1, 1>(A, B, (bf16*)C, M, N, K, ep, err, sms, st);
}

// launches of cb200_gemm_bf16_group: one, or one for each weight where there is no CTA-pair tile
extern "C" int cb200_gemm_group_launches(int M, int groups) { return cb200_gemm_pair_mode(-1) == 1 && M >= 2 * BM ? 1 : groups; }

// C[g] = A @ B[g]^T for `groups` (1 to 3) weights [N, K] in one launch; fewer than 256 rows: one launch each.
extern "C" int cb200_gemm_bf16_group(const void* A, const void* const* B, void* const* C, int groups, int M, int N, int K, int* err, int sms,
                                     cudaStream_t st) {
  if (groups < 1 || groups > 3 || N % 8 != 0) return -41;
  if (cb200_gemm_group_launches(M, 2) > 1) {
    for (int g = 0; g < groups; ++g) {
      const int rc = cb200_gemm_bf16(A, B[g], C[g], M, N, K, 0, 0, nullptr, 0, nullptr, nullptr, nullptr, 0, 1, err, sms, st);
      if (rc) return rc;
    }
    return 0;
  }
  GemmEpilogue ep{};
  ep.groups = groups;
  ep.L = 1;
  return launch_gemm_any<0, 0>(A, B, C, M, N, K, ep, err, sms, st);
}

// Weights that one launch of cb200_gemm_bf16_many takes for this shape: none where fewer than 256 rows, a partial N tile or half a head
// rule out the tiles it is made of, or where all of the weights together are less than a wave of tiles, which the grouped launches
// above split over clusters.
extern "C" int cb200_gemm_many_weights(int n, int M, int N, int K, int sms) {
  const long tiles = (long)((M + 2 * BM - 1) / (2 * BM)) * (N / BN) * n;
  return cb200_gemm_pair_mode(-1) == 1 && M >= 2 * BM && N % BN == 0 && K % 8 == 0 && tiles >= sms / 2 ? kManyWeights : 0;
}

// C[i] = A @ B[i]^T for n <= kManyWeights weights [N, K] in one launch, heads of 128 columns RMS-normalised with norm[i] where that is
// not null (fp32, or bf16 with norm_bf16[i]; 16-byte aligned).
extern "C" int cb200_gemm_bf16_many(const void* A, const void* const* B, void* const* C, const void* const* norm, const uint8_t* norm_bf16,
                                    int n, int M, int N, int K, float eps, int* err, int sms, cudaStream_t st) {
  if (n < 1 || n > kManyWeights || M < 2 * BM || N % BN != 0 || K % 8 != 0) return -43;
  GemmEpilogue ep{};
  ep.groups = n;
  ep.norm_eps = eps;
  ep.L = 1;
  int c1 = 0;
  const int rc = resident_clusters<0, 0, 1, kManyWeights>(&c1);
  if (rc) return rc;
  if (c1 < 1) return 600;
  const long tiles = (long)((M + 2 * BM - 1) / (2 * BM)) * (N / BN) * n;
  return launch_gemm_pairs<0, 0, 1, kManyWeights>(A, B, C, M, N, K, ep, (int)std::min<long>(tiles, std::min(c1, sms / 2)), err, st, norm, norm_bf16);
}

// C is not written: row (b, s) of A[M = B*S, K] @ W[N = H*128, K]^T is split into heads, each head is RMS-normalised with
// `norm_w` (optional), rotated by cos/sin [S, 64] (optional, needs norm_w) and stored into staging buffer ptrs[head / Hl] at
// [b, rank * S + s, head % Hl, :].  The buffers may live on peer GPUs (plain stores over NVLink).
extern "C" int cb200_gemm_bf16_scatter_heads(const void* A, const void* W, int M, int N, int K, const int64_t* ptrs, int P,
                                             int rank, int S, const void* norm_w, int norm_bf16, const float* cosv, const float* sinv,
                                             float eps, void* raw, float* rstd_out, int* err, int sms, cudaStream_t st) {
  if (P < 1 || P > 8 || N % 128 != 0 || (N / 128) % P != 0 || S <= 0 || M % S != 0) return -21;
  if (cosv != nullptr && norm_w == nullptr) return -22;
  if ((raw != nullptr) != (rstd_out != nullptr) || (raw != nullptr && norm_w == nullptr)) return -23;
  GemmEpilogue ep{};
  for (int i = 0; i < P; ++i) ep.hs.ptrs[i] = ptrs[i];
  ep.hs.w = norm_w;
  ep.hs.w_bf16 = norm_bf16;
  ep.hs.cosv = cosv;
  ep.hs.sinv = sinv;
  ep.hs.S = S;
  ep.hs.Hl = (N / 128) / P;
  ep.hs.P = P;
  ep.hs.rank = rank;
  ep.hs.eps = eps;
  ep.hs.raw = (bf16*)raw;
  ep.hs.rstd_out = rstd_out;
  ep.L = 1;
  ep.groups = 1;
  void* none = nullptr;
  if (cb200_gemm_pair_mode(-1) == 1 && M >= 2 * BM) return launch_gemm_any<0, 0>(A, &W, &none, M, N, K, ep, err, sms, st);
  return launch_gemm<0, 0>(A, W, nullptr, M, N, K, ep, err, sms, st);
}

// C = epilogue(A @ op(W)) where W [rows, ld] is sharded by rows over P ranks (rank r: shard_ptrs[r] holds rows [r * chunk_rows, ...)).
// b_mn = 0: forward, C[M, rows] = A[M, ld] @ W^T; b_mn = 1: dgrad, C[M, ld] = A[M, rows] @ W. `ws` [rows, ld] receives the gathered
// weight (and stays valid after the call); `counters`: ceil(rows / 256) ints of scratch.
extern "C" int cb200_gemm_bf16_gather(const void* A, void* ws, void* C, int M, int rows, int ld, int b_mn, const int64_t* shard_ptrs,
                                      int P, int chunk_rows, int* counters, const void* bias, int act, void* pre, int* err, int sms,
                                      cudaStream_t st) {
  if (P < 1 || P > 8 || chunk_rows < 1 || (long)chunk_rows * P < rows || ld % 8 != 0) return -31;
  GemmEpilogue ep{};
  ep.pre = (bf16*)pre;
  ep.bias = (const bf16*)bias;
  ep.act = act;
  ep.L = 1;
  GatherB gb{};
  for (int i = 0; i < P; ++i) gb.ptrs[i] = shard_ptrs[i];
  gb.ws = (bf16*)ws;
  gb.counters = counters;
  gb.P = P;
  gb.chunk_rows = chunk_rows;
  gb.rows = rows;
  gb.ld = ld;
  const int n_groups = (rows + kGatherGroupRows - 1) / kGatherGroupRows;
  gb.slices = sms / n_groups < 1 ? 1 : (sms / n_groups > 16 ? 16 : sms / n_groups);
  cudaError_t e = cudaMemsetAsync(counters, 0, (size_t)n_groups * sizeof(int), st);
  if (e != cudaSuccess) return 400 + (int)e;
  if (b_mn == 0) return launch_gemm<0, 0, true>(A, ws, (bf16*)C, M, rows, ld, ep, err, sms, st, gb);
  return launch_gemm<0, 1, true>(A, ws, (bf16*)C, M, ld, rows, ep, err, sms, st, gb);
}
