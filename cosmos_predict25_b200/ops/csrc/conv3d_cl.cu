// Convolution on channels-last activations as an implicit GEMM on the 5th-generation tensor cores (sm_100a), bf16 in / fp32 accumulate.
//
// Serves every convolution of the Wan-style causal VAE decoder (cosmos_predict2/_src/predict2/tokenizers/wan2pt1.py:40-58 causal
// Conv3d, :84-137 resample, :184-215 residual block): 3 x 3 x 3 causal, 3 x 1 x 1 temporal, 3 x 3 spatial (as the four 2 x 2 phase
// convolutions of "nearest 2x up-sampling followed by 3 x 3"), 1 x 1 x 1.
//
//   activation X [T_in, H_in, W_in, C_in]   (C_in a multiple of 16)
//   weights    W [N_pad, taps, C_pad]        (K-major; C_pad = C_in rounded up to 64, N_pad = C_out rounded up to the N tile)
//   output     Y[t, h, w, n] = bias[n] + sum_{tap, c} X[t + dt(tap), h + dh(tap), w + dw(tap), c] * W[n, tap, c]  (+ residual)
//
// There is no im2col buffer: an output tile is 128 voxels = 16 lines of 8 of one frame, and the A operand of ALL n x n spatial taps of one
// frame offset, channel block kb, is ONE TMA box {64 channels, 7 + n, 15 + n, 1 t} of the activation tensor itself. It lands in shared
// memory as rows of 64 channels with 128-byte swizzle, K-major, which is what the MMA wants: eight voxels of a line are one 8-row group, the
// groups are a line of the box apart, and tap (dy, dx) reads the same box from dy lines and dx rows on. The swizzle goes by the address, so
// neither the start of a tap nor the distance of the groups has to be a whole number of 1,024-byte atoms (checked for every shift and
// distance used here against a plain copy of the rows). Layers of 16 input or output channels take a box for each column of taps, as wide
// as the tile (see tap_panels). Coordinates outside the tensor read zeros: that IS the zero padding of the
// convolution (the channel coordinate stays a multiple of 64, so the 16-byte alignment rule of TMA holds).
// The eight voxels run along the width or along the height, whichever leaves fewer tiles over the frame's edge.
//
// The causal time padding is either the leading frames of the input tensor (pad = 0), or `pad` frames in a tensor of their own
// (the stream cache of the previous chunk) of which the oldest may be missing = zeros: taps whose frame lies in zero padding for
// the whole tile are skipped (two thirds of a 3 x 3 x 3 convolution on a single image). Strided convolutions (the encoder's
// down-sampling) step the frame coordinate, and the pixel coordinates through the tensor map's element strides.
//
// CTA pairs (tcgen05 cta_group::2): two consecutive voxel tiles share the B operand, each CTA fetches its own A box and half of
// the B rows, the even CTA issues M = 256 MMAs. A and B have a ring each: a box serves n columns of B boxes. Where a box serves one column only (single taps
// among them) they are one stage on one barrier: a step of a 3 x 1 x 1 convolution is four MMAs, whose issue a second wait and commit
// made up a third of (384 to 768 channels, 4 frames of 120 x 208: 144 us with one barrier, 187 with two). What bounds the kernel is the
// L2 -> shared-memory path of narrow layers and, on long runs, the card's power, to which that traffic adds: 128 voxels of a
// 3 x 3 x 3 convolution with 96 channels took 498 KB with a box for each column of taps, now 290 (with 192 channels 1,035 and 800).
// Decoding 8 latent frames of 720p 196 and 189 ms, encoding 29 frames of 768 x 432 46 and 44, an image of 640 x 640 2.31 and 2.25.
// Two boxes in flight and the rest for B columns is the best split: three boxes the same, four (two columns of B left) 5 % slower.
//
// Persistent, warp-specialised, one CTA per SM, same skeleton as the GEMM of this package: warp 0 TMA producer (a ring of A boxes and
// one of B boxes), warp 1 MMA issuer (two TMEM accumulators of n_tile columns), warps 2-9 epilogue (bias, optional
// residual, bf16 store through a per-voxel output mapping that also expresses the phase interleave of the up-sampling
// convolutions and the frame interleave of the temporal up-sampler). All waits are bounded and report through `err`.

#include <math.h>

#include <algorithm>

#include "common.cuh"
#include "launchers.h"
#include "sm100.cuh"
#include "tmap.h"

namespace cb200 {
using namespace sm100;

namespace cv {
constexpr int BM = 128, BK = 64, TX = 8, TY = 16;   // a tile: TY lines of TX voxels
constexpr int kThreads = 320;                 // TMA warp, MMA warp, 8 epilogue warps
constexpr int kMaxTaps = 27, kMaxRun = 3;     // taps, and lines / columns of taps that share a box
constexpr int kMaxSlots = 8;                  // of each ring
constexpr int kBarBytes = 512;
constexpr int kStageOut = 32 * 64;            // staging block of an epilogue warp: 32 voxels x 32 channels
constexpr int kBiasMax = 1024;                // channels whose bias is kept in shared memory
constexpr int kSmemMax = 227 * 1024, kSmemFixed = 1024 /*alignment slack*/ + kBarBytes + 8 * kStageOut;
constexpr int kSumSq = 2 * 2 * BM * 4;       // partial sums of squares: buffer, column half, row
}  // namespace cv

struct ConvParams {
  int T_out, X_out, Y_out;      // output grid walked by the tiles; X, Y: width and height, or height and width
  int Cin, Cout;
  int n_tile, tiles_n;          // N per tile (multiple of 16, <= 256) and number of N tiles
  int npanels, kblocks;         // K loop: panels of RUN x RUN taps of one frame offset (by ascending dt) x 64-channel blocks
  int a_slots, b_slots;         // ring depths
  int pad, cache_frames;        // frames of causal padding in front of X; tm_c holds the last `cache_frames` of them, the rest is zero
  int t_stride, xy_stride;      // input coordinate = output coordinate x stride + offset
  int8_t dt[cv::kMaxTaps], dx[cv::kMaxTaps], dy[cv::kMaxTaps];   // per panel: input coordinate = output coordinate + offset
  int8_t tap[cv::kMaxTaps][cv::kMaxRun][cv::kMaxRun];            // weight column block of the panel's tap in column i (width), row j (height)
  // element offset of output voxel (t, x, y), channel n: out_at + t * out_t + x * out_x + y * out_y + n
  long out_at, out_t, out_x, out_y;
  int vec;                      // voxels can be moved as 16-byte pieces
  bf16* Y;
  const bf16* resid;            // optional, same addressing as Y
  const float* bias;            // optional [Cout]
  // optional: the RMS-norm (+ SiLU) that the next convolution's input goes through, of the finished value and in the same epilogue:
  // Yn = [silu](v / max(||v||, 1e-12) * norm_scale * gamma) over the channels, same addressing as Y. Needs all channels in one N tile.
  bf16* Yn;
  const float* gamma;           // [Cout], 16-byte aligned
  float norm_scale;             // sqrt(Cout)
  int silu, write_raw;          // write_raw 0: only Yn is stored
};

// STACK = 2 (narrow layers, N tile <= 128): a CTA owns two voxel tiles side by side, 16 x 16 voxels, with an accumulator each; their A
// box is one of 18 x 18 voxels and every B row in shared memory serves both.
// BY_HEIGHT: X is the frame's height. The order of a sum - columns of taps along the width, their rows, channels - is the same either way, so that
// a band of rows gives the bits of the whole frame.
// COLS: columns of taps that an A box serves: all RUN of a square, or 1, a column of RUN rows and a box as wide as the tile. Then the box and its
// taps' B rows are one stage on one barrier (JOINT; always so with single taps).
template <int RUN, int STACK, bool BY_HEIGHT, int COLS>
__global__ void __launch_bounds__(cv::kThreads, 1)
conv_cl_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_c, const __grid_constant__ CUtensorMap tm_w,
               const __grid_constant__ ConvParams p, int* __restrict__ err) {
  using namespace cv;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int b_half = p.n_tile * (BK * 2 / 2);                  // bytes of one tap's B rows in this CTA (half of the N tile)
  static_assert(COLS == RUN || (COLS == 1 && !BY_HEIGHT), "a box of one column lies along the width");
  constexpr bool JOINT = COLS == 1;
  constexpr int kLine = TX * STACK + COLS - 1;                 // voxels of a line of the A box
  constexpr int kBoxBytes = kLine * (TY + RUN - 1) * BK * 2, kASlot = (kBoxBytes + 1023) / 1024 * 1024;
  const int b_slot = RUN * b_half;                             // the taps of one column
  uint8_t* const ring_b = smem + p.a_slots * kASlot;
  uint64_t* bars = reinterpret_cast<uint64_t*>(ring_b + p.b_slots * b_slot);
  uint64_t* a_full = bars;                    // [a_slots], the even CTA's count the bytes of both
  uint64_t* a_empty = bars + kMaxSlots;       // [a_slots]
  uint64_t* b_full = bars + 2 * kMaxSlots;    // [b_slots]
  uint64_t* b_empty = bars + 3 * kMaxSlots;   // [b_slots]
  uint64_t* acc_full = bars + 4 * kMaxSlots;  // [2]
  uint64_t* acc_empty = acc_full + 2;         // [2]
  uint64_t* sums_in = acc_empty + 2;          // [2][4] sums of squares of a lane quarter's two warps written (buffer, quarter)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sums_in + 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  static_assert((4 * kMaxSlots + 2 + 2 + 8) * 8 + 8 <= kBarBytes, "barriers, tensor-memory address and flag");
  uint8_t* stage_out = reinterpret_cast<uint8_t*>(bars) + kBarBytes;
  float* ssq = reinterpret_cast<float*>(stage_out + 8 * kStageOut);      // with a fused norm: sums of squares, then gamma
  float* gamma_s = ssq + kSumSq / 4;
  float* bias_s = p.Yn != nullptr ? gamma_s + 256 : ssq;   // [Cout] when Cout <= kBiasMax

  // the shuffle makes the warp index (and every role branch below) provably warp-uniform for the compiler
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int tiles_x = (p.X_out + TX * STACK - 1) / (TX * STACK), tiles_y = (p.Y_out + TY - 1) / TY;
  const int vox_tiles = p.T_out * tiles_y * tiles_x;
  const int first_tile = (int)(blockIdx.x >> 1), tile_step = (int)(gridDim.x >> 1);

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.a_slots; ++s) {
      mbar_init(&a_full[s], 1);
      mbar_init(&a_empty[s], 1);
    }
    for (int s = 0; s < p.b_slots; ++s) {
      mbar_init(&b_full[s], 1);
      mbar_init(&b_empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&acc_full[a], 1);
      mbar_init(&acc_empty[a], 16);           // the even CTA hears from the epilogue warps of both
      for (int q = 0; q < 4; ++q) mbar_init(&sums_in[a * 4 + q], 2);
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
  cluster_sync_relaxed();                     // the other CTA's barriers exist before anything signals them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_trigger();                              // launched with programmatic serialisation (see common.cuh)
  pdl_wait();
  if (p.bias != nullptr && p.Cout <= kBiasMax)
    for (int i = threadIdx.x; i < p.Cout; i += kThreads) bias_s[i] = p.bias[i];
  if (p.Yn != nullptr)
    for (int i = threadIdx.x; i < p.Cout; i += kThreads) gamma_s[i] = p.gamma[i] * p.norm_scale;
  if (threadIdx.x == 0) *abort_flag = *reinterpret_cast<volatile int*>(err);   // an earlier error: drain the grid at once
  __syncthreads();
  // tiles of the pair: two voxel tiles x one N tile; after an earlier error none
  const int n_tiles = *abort_flag != 0 ? 0 : (vox_tiles + 1) / 2 * p.tiles_n;
  __syncthreads();

  // pair tile -> N tile and this CTA's voxel tile (a trailing odd tile is computed by both CTAs and stored by the even one);
  // N tiles of one voxel pair are neighbours so that they run at the same time and share the activation boxes through L2
  auto decode = [&](int t, int& nt, int& x0, int& y0, int& tf, bool& mine) {
    nt = t % p.tiles_n;
    int v = t / p.tiles_n * 2 + (int)rank;
    mine = v < vox_tiles;
    v = min(v, vox_tiles - 1);
    x0 = (v % tiles_x) * (TX * STACK);
    v /= tiles_x;
    y0 = (v % tiles_y) * TY;
    tf = v / tiles_y;
  };
  // panels whose frame is zero padding for both tiles of the pair are left out: the later tile's frame decides, and the panels
  // are in the order of their frames
  auto first_panel = [&](int t) {
    const int tf_last = min(t / p.tiles_n * 2 + 1, vox_tiles - 1) / (tiles_y * tiles_x);
    int g = 0;
    while (g < p.npanels - 1 && tf_last * p.t_stride + p.dt[g] < p.pad - p.cache_frames) ++g;
    return g;
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      prefetch_tmap(&tm_x);
      prefetch_tmap(&tm_c);
      prefetch_tmap(&tm_w);
      int as = 0, bs = 0;
      uint32_t aph = 0, bph = 0;
      bool ok = true;
      for (int t = first_tile; t < n_tiles && ok; t += tile_step) {
        int nt, x0, y0, tf;
        bool mine;
        decode(t, nt, x0, y0, tf, mine);
        const int n0 = nt * p.n_tile + (int)rank * (p.n_tile / 2);
        for (int g = first_panel(t); g < p.npanels && ok; ++g) {
          const int tx = tf * p.t_stride + p.dt[g] - p.pad;          // frame of X; negative: a cached frame or padding
          const bool cached = tx < 0 && p.cache_frames > 0;
          const CUtensorMap* tm = cached ? &tm_c : &tm_x;
          const int tc = cached ? tx + p.cache_frames : tx;
          const int xx = x0 * p.xy_stride + p.dx[g], xy = y0 * p.xy_stride + p.dy[g];
          for (int kb = 0; kb < p.kblocks && ok; ++kb) {
            if (!JOINT) {
              if (!mbar_wait(&a_empty[as], aph ^ 1, abort_flag)) { ok = false; break; }
              if (rank == 0) mbar_arrive_expect_tx(&a_full[as], 2 * kBoxBytes);
              tma_load_4d_pair(smem + as * kASlot, tm, mapa_shared(smem_u32(&a_full[as]), 0), kb * BK, xx, xy, tc);
              if (++as == p.a_slots) { as = 0; aph ^= 1; }
            }
#pragma unroll
            for (int i = 0; i < COLS; ++i) {
              if (!mbar_wait(&b_empty[bs], bph ^ 1, abort_flag)) { ok = false; break; }
              if (rank == 0) mbar_arrive_expect_tx(&b_full[bs], 2 * (b_slot + (JOINT ? kBoxBytes : 0)));
              const uint32_t bar = mapa_shared(smem_u32(&b_full[bs]), 0);
              if (JOINT) tma_load_4d_pair(smem + bs * kASlot, tm, bar, kb * BK, xx, xy, tc);
#pragma unroll
              for (int j = 0; j < RUN; ++j)
                tma_load_2d_pair(ring_b + bs * b_slot + j * b_half, &tm_w, bar, (p.tap[g][i][j] * p.kblocks + kb) * BK, n0);
              if (++bs == p.b_slots) { bs = 0; bph ^= 1; }
            }
          }
        }
      }
      if (!ok) { atomicCAS(err, 0, 61); *abort_flag = 1; }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (warp-uniform; the elected lane issues)
    const uint32_t leader = elect_one() ? 1u : 0u;
    auto wait_all = [&](uint64_t* bar, uint32_t parity) -> bool { return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag)); };
    const uint32_t idesc = umma_idesc_bf16(2 * BM, p.n_tile, 0, 0);
    const uint64_t da0 = umma_desc_sw128(smem_u32(smem), 16, kLine * BK * 2);
    const uint64_t db0 = umma_desc_sw128(smem_u32(ring_b), 16, 1024);
    int as = 0, bs = 0;
    uint32_t aph = 0, bph = 0;
    int acc = 0;
    uint32_t acc_ph = 0;
    bool ok = true;
    for (int t = first_tile; t < n_tiles && ok && rank == 0; t += tile_step) {      // only the even CTA issues
      if (!wait_all(&acc_empty[acc], acc_ph ^ 1)) { ok = false; break; }
      tc_fence_after();
      const uint32_t d_tmem = tmem_base + acc * 256;
      uint32_t first = 0;
      for (int g = first_panel(t); g < p.npanels && ok; ++g) {
        for (int kb = 0; kb < p.kblocks && ok; ++kb) {
          if (!JOINT && !wait_all(&a_full[as], aph)) { ok = false; break; }
          const uint64_t da_s = da0 + (uint64_t)((JOINT ? bs : as) * (kASlot >> 4));
          const int ksteps = (p.Cin - kb * BK) / 16;   // below 4 in the last block of, e.g., C_in = 96: 32 real channels
#pragma unroll
          for (int i = 0; i < COLS; ++i) {
            if (!wait_all(&b_full[bs], bph)) { ok = false; break; }
            tc_fence_after();
            const uint64_t db_s = db0 + (uint64_t)(bs * (b_slot >> 4));
            // straight-line issue: one warp issues every MMA of the pair, and a narrow MMA (N = 96: 48 clocks) is over before a
            // loop with descriptor arithmetic gets to the next one (64 -> 16 channels, 27 taps: 6.8 us a tile as loops, 4.4 us)
            auto issue = [&](int j, int k) {
              const uint64_t db = db_s + (uint32_t)(j * (b_half >> 4) + k * 2);
#pragma unroll
              for (int u = 0; u < STACK; ++u)
                umma_ss_pair_w(d_tmem + u * 128, da_s + (uint32_t)((((BY_HEIGHT ? i * kLine + j : j * kLine + i) + u * TX) * BK * 2 + k * 32) >> 4), db, idesc,
                               (i | j | k) ? 1u : first, leader);
            };
            if (ksteps >= 4) {
#pragma unroll
              for (int j = 0; j < RUN; ++j)
#pragma unroll
                for (int k = 0; k < 4; ++k) issue(j, k);
            } else if (ksteps == 2) {
#pragma unroll
              for (int j = 0; j < RUN; ++j)
#pragma unroll
                for (int k = 0; k < 2; ++k) issue(j, k);
            } else {
              for (int j = 0; j < RUN; ++j)
                for (int k = 0; k < ksteps; ++k) issue(j, k);
            }
            umma_commit_pair_w(&b_empty[bs], leader);  // slot reusable in both CTAs once these MMAs have read it
            if (++bs == p.b_slots) { bs = 0; bph ^= 1; }
          }
          first = 1u;
          if (!JOINT) {
            umma_commit_pair_w(&a_empty[as], leader);
            if (++as == p.a_slots) { as = 0; aph ^= 1; }
          }
        }
      }
      if (!ok) break;
      umma_commit_pair_w(&acc_full[acc], leader);
      if (++acc == 2) { acc = 0; acc_ph ^= 1; }
    }
    if (!ok && lane == 0) { atomicCAS(err, 0, 62); *abort_flag = 1; }
  } else {
    // ------------------------------------------------------------------ epilogue warps
    // A thread owns one output voxel of the accumulator and stages 32 channels of it; then 4 lanes cover the 64 contiguous bytes
    // of a voxel. Storing (and reading the residual) per thread made 32 partly filled requests per instruction and bound every
    // convolution with a short K loop (1 x 1, 64 -> 192 channels with residual: 13.5 us a tile, now 5.1 us).
    const int quarter = warp & 3;      // TMEM lanes [32 quarter, +32)
    const int part = (warp - 2) >> 2;  // which half of the tile's 32-column chunks
    const int nch = (p.n_tile + 31) >> 5, c_lo = part == 0 ? 0 : (nch + 1) / 2, c_hi = part == 0 ? (nch + 1) / 2 : nch;
    uint8_t* stage_warp = stage_out + (warp - 2) * kStageOut;
    int acc = 0;
    uint32_t acc_ph = 0;
    bool ok = true;
    int sums = 0;                        // exchanges of sums of squares so far: buffer sums & 1, phase sums >> 1
    const bool vec_ok = p.vec != 0;
    const float* bias = p.bias != nullptr && p.Cout <= kBiasMax ? bias_s : p.bias;
    const uint32_t acc_empty_leader[2] = {mapa_shared(smem_u32(&acc_empty[0]), 0), mapa_shared(smem_u32(&acc_empty[1]), 0)};
    for (int t = first_tile; t < n_tiles && ok; t += tile_step) {
      int nt, x0, y0, tf;
      bool mine;
      decode(t, nt, x0, y0, tf, mine);
      bool arrived = false;              // whether the accumulators of this tile have been waited for
#pragma unroll 1
      for (int u = 0; u < STACK; ++u, x0 += TX) {
        // element offset of a voxel of the tile (row r = 8 y + x), or -1 outside the frame
        auto offset = [&](int r) -> long {
          const int x = x0 + (r & 7), y = y0 + (r >> 3);
          if (!mine || x >= p.X_out || y >= p.Y_out) return -1;
          return p.out_at + tf * p.out_t + x * p.out_x + y * p.out_y;
        };
        const uint32_t t_row = tmem_base + acc * 256 + u * 128 + ((uint32_t)(quarter * 32) << 16);
        if (vec_ok) {
          const int piece = lane & 3;                       // 16-byte piece of the 64-byte run that this lane moves
          long off[4];                                      // voxels quarter * 32 + 8 it + lane / 4
#pragma unroll
          for (int it = 0; it < 4; ++it) off[it] = offset(quarter * 32 + it * 8 + (lane >> 2));
          auto slot = [&](int row, int pc) { return stage_warp + row * 64 + ((pc ^ ((row >> 1) & 3)) << 4); };   // no bank conflicts
          // residual of the first chunk: on its way while the accumulator is still being computed
          uint4 res[4];
          auto fetch = [&](int c) {
            const int n = nt * p.n_tile + c * 32 + piece * 8;
#pragma unroll
            for (int it = 0; it < 4; ++it)
              if (off[it] >= 0 && n < p.Cout) res[it] = *reinterpret_cast<const uint4*>(p.resid + off[it] + n);
          };
          if (p.resid != nullptr && c_lo < c_hi) fetch(c_lo);
          if (!arrived && !mbar_wait_warp(&acc_full[acc], acc_ph, abort_flag)) { ok = false; break; }
          arrived = true;
          tc_fence_after();
          // this thread's 32 channels of chunk c, staged and stored as 64-byte runs
          auto emit = [&](bf16* dst, int c, const uint32_t (&a)[32]) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              uint4 o;
              __nv_bfloat162* o2 = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
              for (int j = 0; j < 4; ++j)
                o2[j] = __floats2bfloat162_rn(__uint_as_float(a[q * 8 + 2 * j]), __uint_as_float(a[q * 8 + 2 * j + 1]));
              *reinterpret_cast<uint4*>(slot(lane, q)) = o;
            }
            __syncwarp();
            const int n = nt * p.n_tile + c * 32 + piece * 8;
#pragma unroll
            for (int it = 0; it < 4; ++it)
              if (off[it] >= 0 && n < p.Cout && c * 32 + piece * 8 < p.n_tile)
                *reinterpret_cast<uint4*>(dst + off[it] + n) = *reinterpret_cast<const uint4*>(slot(it * 8 + (lane >> 2), piece));
            __syncwarp();
          };
          float ss = 0.f;
#pragma unroll 1
          for (int c = c_lo; c < c_hi; ++c) {
            const int n0 = nt * p.n_tile + c * 32;
            uint32_t a[32];
            tmem_ld32(t_row + c * 32, a);                   // warp-collective; columns past the tile are loaded and not stored
            tmem_ld_wait();
            if (bias != nullptr) {
              if (n0 + 32 <= p.Cout && bias == bias_s) {
#pragma unroll
                for (int j = 0; j < 32; j += 4) {
                  const float4 f = *reinterpret_cast<const float4*>(bias_s + n0 + j);
                  a[j] = __float_as_uint(__uint_as_float(a[j]) + f.x);
                  a[j + 1] = __float_as_uint(__uint_as_float(a[j + 1]) + f.y);
                  a[j + 2] = __float_as_uint(__uint_as_float(a[j + 2]) + f.z);
                  a[j + 3] = __float_as_uint(__uint_as_float(a[j + 3]) + f.w);
                }
              } else {
#pragma unroll
                for (int j = 0; j < 32; ++j)
                  if (n0 + j < p.Cout) a[j] = __float_as_uint(__uint_as_float(a[j]) + bias[n0 + j]);
              }
            }
            if (p.resid != nullptr) {
              // the sum is rounded once: the residual comes through the staging block to the thread that owns the voxel
#pragma unroll
              for (int it = 0; it < 4; ++it) *reinterpret_cast<uint4*>(slot(it * 8 + (lane >> 2), piece)) = res[it];
              if (c + 1 < c_hi) fetch(c + 1);
              __syncwarp();
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                const uint4 rr = *reinterpret_cast<const uint4*>(slot(lane, q));
                const __nv_bfloat162* r2 = reinterpret_cast<const __nv_bfloat162*>(&rr);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  const float2 rf = __bfloat1622float2(r2[j]);
                  a[q * 8 + 2 * j] = __float_as_uint(__uint_as_float(a[q * 8 + 2 * j]) + rf.x);
                  a[q * 8 + 2 * j + 1] = __float_as_uint(__uint_as_float(a[q * 8 + 2 * j + 1]) + rf.y);
                }
              }
            }
            if (p.Yn != nullptr) {
              // the finished values go back to TMEM for the second pass
              if (n0 + 32 <= p.Cout) {
                float2 s2[4] = {make_float2(ss, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                  const float2 v = make_float2(__uint_as_float(a[2 * j]), __uint_as_float(a[2 * j + 1]));
                  s2[j & 3] = fma2(v, v, s2[j & 3]);
                }
                const float2 t = add2(add2(s2[0], s2[1]), add2(s2[2], s2[3]));
                ss = t.x + t.y;
              } else {
#pragma unroll
                for (int j = 0; j < 32; ++j)
                  if (n0 + j < p.Cout) ss = fmaf(__uint_as_float(a[j]), __uint_as_float(a[j]), ss);
              }
              tmem_st32(t_row + c * 32, a);
            }
            if (p.write_raw) emit(p.Y, c, a);
          }
          if (p.Yn != nullptr) {
            // the two warps of a lane quarter hold half of a voxel's channels each. Two buffers: a warp is at most one tile ahead of its
            // partner. The partner may have given up, so this wait is bounded like every other (a named barrier is not)
            const int ss_buf = sums & 1;
            float* mine_s = ssq + (ss_buf * 2 + part) * BM + quarter * 32 + lane;
            const float* other_s = ssq + (ss_buf * 2 + (part ^ 1)) * BM + quarter * 32 + lane;
            uint64_t* bar = &sums_in[ss_buf * 4 + quarter];
            *mine_s = ss;
            tmem_st_wait();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar);
            if (!mbar_wait_warp(bar, (sums >> 1) & 1, abort_flag)) { ok = false; break; }
            ++sums;
            const float total = part == 0 ? ss + *other_s : *other_s + ss;
            const float inv = 1.f / fmaxf(sqrtf(total), 1e-12f);
#pragma unroll 1
            for (int c = c_lo; c < c_hi; ++c) {
              uint32_t a[32];
              tmem_ld32(t_row + c * 32, a);
              tmem_ld_wait();
              const float2 inv2 = make_float2(inv, inv);
#pragma unroll
              for (int j = 0; j < 32; j += 4) {
                // gamma past the last channel is whatever follows it in shared memory: those columns are not stored
                const float4 g = *reinterpret_cast<const float4*>(gamma_s + c * 32 + j);
                const float2 z0 = mul2(mul2(make_float2(__uint_as_float(a[j]), __uint_as_float(a[j + 1])), inv2), make_float2(g.x, g.y));
                const float2 z1 = mul2(mul2(make_float2(__uint_as_float(a[j + 2]), __uint_as_float(a[j + 3])), inv2), make_float2(g.z, g.w));
                a[j] = __float_as_uint(z0.x);
                a[j + 1] = __float_as_uint(z0.y);
                a[j + 2] = __float_as_uint(z1.x);
                a[j + 3] = __float_as_uint(z1.y);
              }
              if (p.silu) {
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                  const float z = __uint_as_float(a[j]);
                  a[j] = __float_as_uint(z / (1.f + __expf(-z)));
                }
              }
              emit(p.Yn, c, a);
            }
          }
        } else {
          const long base = offset(quarter * 32 + lane);
          if (!arrived && !mbar_wait_warp(&acc_full[acc], acc_ph, abort_flag)) { ok = false; break; }
          arrived = true;
          tc_fence_after();
#pragma unroll 1
          for (int c = c_lo; c < c_hi; ++c) {
            uint32_t a[32];
            tmem_ld32(t_row + c * 32, a);
            tmem_ld_wait();
            const int n0 = nt * p.n_tile + c * 32;
            if (base >= 0) {
#pragma unroll
              for (int j = 0; j < 32; ++j)
                if (n0 + j < p.Cout && c * 32 + j < p.n_tile) {
                  float o = __uint_as_float(a[j]);
                  if (bias != nullptr) o += bias[n0 + j];
                  if (p.resid != nullptr) o += __bfloat162float(p.resid[base + n0 + j]);
                  p.Y[base + n0 + j] = __float2bfloat16(o);
                }
            }
          }
        }
      }
      if (!ok) break;
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster_tmem(acc_empty_leader[acc]);
      if (++acc == 2) { acc = 0; acc_ph ^= 1; }
    }
    if (!ok && lane == 0) { atomicCAS(err, 0, 63); *abort_flag = 1; }
  }

  __syncwarp();
  if (*abort_flag && n_tiles > 0) {
    // let outstanding bulk copies / MMAs drain before shared memory and TMEM go away
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_relaxed();              // neither CTA leaves (or frees TMEM) while the other may still signal it or read its tiles
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

// y[v, :] = silu(x[v, :] / max(||x[v, :]||_2, 1e-12) * sqrt(C) * gamma): the RMS-norm + SiLU in front of every convolution of a
// residual block, on channels-last rows. Bound by memory (one read, one write). G lanes share a voxel and each holds NV 16-byte
// pieces of it, so that every lane of a warp loads whatever C is (pieces past C are skipped, G * NV * 8 >= C). The lanes go on from voxel to voxel
// with their part of gamma in registers - read for every voxel it is twice the voxel's bytes - and the next voxel's pieces in flight.
// 25,600 voxels of 384 channels 10.4 us before (a voxel per lane group), now 9.3; 56,320 19.7 and 16.9, 102,400 of 192 18.6 and 15.5, 4 frames
// of 704 x 1280 x 96 316 and 281 (4.9 TB/s). Three CTAs an SM are what its registers hold: held to the registers of four
// the kernel spills (25,600 voxels 13 us).
constexpr int kRmsCtas = 148 * 3;
template <int G, int NV>
__global__ void __launch_bounds__(256) rmsnorm_silu_cl_kernel(const bf16* __restrict__ x, const float* __restrict__ gamma,
                                                                bf16* __restrict__ y, long n_vox, int C, float scale, int silu) {
  pdl_trigger();                                       // launched with programmatic serialisation (see common.cuh)
  pdl_wait();
  const int sub = threadIdx.x % G;
  const int nvec = C >> 3;
  const long step = (long)gridDim.x * (256 / G);
  bf16x8 next[NV];
  auto fetch = [&](long v) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int idx = sub + i * G;
      next[i] = v < n_vox && idx < nvec ? *reinterpret_cast<const bf16x8*>(x + v * C + idx * 8) : bf16x8{};
    }
  };
  long v = (long)blockIdx.x * (256 / G) + threadIdx.x / G;
  fetch(v);
  float g[NV][8];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int idx = sub + i * G;
#pragma unroll
    for (int j = 0; j < 8; j += 4) {
      const float4 f = idx < nvec ? *reinterpret_cast<const float4*>(gamma + idx * 8 + j) : make_float4(0.f, 0.f, 0.f, 0.f);
      g[i][j] = f.x; g[i][j + 1] = f.y; g[i][j + 2] = f.z; g[i][j + 3] = f.w;
    }
  }
  // the reduction below is warp-wide: the lanes of a warp leave the loop together
  for (; __any_sync(0xffffffffu, v < n_vox); v += step) {
    bf16x8 cur[NV];
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) cur[i] = next[i];
    fetch(v + step);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      float f[8];
      unpack8(cur[i], f);
#pragma unroll
      for (int j = 0; j < 8; ++j) ss = fmaf(f[j], f[j], ss);
    }
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if (v >= n_vox) continue;
    const float inv = scale / fmaxf(sqrtf(ss), 1e-12f);
    bf16* out = y + v * C;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int idx = sub + i * G;
      if (idx < nvec) {
        float o[8], f[8];
        unpack8(cur[i], f);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float z = f[j] * inv * g[i][j];
          o[j] = silu ? z / (1.f + __expf(-z)) : z;
        }
        *reinterpret_cast<bf16x8*>(out + idx * 8) = pack8(o);
      }
    }
  }
}

}  // namespace cb200

using namespace cb200;

// As in the GEMM: the persistent grid is bounded by the pairs that the GPU can hold at once. One CTA per SM whatever the ring depths
// (the rings are over half of the shared memory), so the figure for the largest shared-memory size holds for all.
template <int RUN, int STACK, bool BY_HEIGHT, int COLS>
static int launch_conv(cudaLaunchConfig_t& cfg, long tiles, int sms, const CUtensorMap& tx, const CUtensorMap& tc,
                       const CUtensorMap& tw, const ConvParams& p, int* err) {
  const auto kern = conv_cl_kernel<RUN, STACK, BY_HEIGHT, COLS>;
  static int max_pairs = 0;
  if (max_pairs == 0) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, cv::kSmemMax);
    if (e != cudaSuccess) return 100 + (int)e;
    int n = 0;
    cudaLaunchConfig_t c = cfg;
    c.dynamicSmemBytes = cv::kSmemMax;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &c) != cudaSuccess || n < 1) return 600;
    max_pairs = n;
  }
  cfg.gridDim = dim3(2 * (unsigned)std::min<long>(tiles, std::min(max_pairs, sms / 2)));
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, tx, tc, tw, p, err);
  return e == cudaSuccess ? 0 : 500 + (int)e;
}

// The K loop of a list of taps: panels of one frame offset, run rows x cols columns each, by ascending frame.
struct TapPanels {
  int run, cols, n;
  int dt[cv::kMaxTaps], dh[cv::kMaxTaps], dw[cv::kMaxTaps];      // of a panel's first row and column
  int tap[cv::kMaxTaps][cv::kMaxRun][cv::kMaxRun];               // [panel][column][row] -> index in the list
};

// The whole list has to fall into squares of 3 x 3 or 2 x 2 taps or columns of three or two rows, tried in that order, else each tap is its own
// (with a spatial stride neighbouring taps do not share rows of a strided box).
static TapPanels tap_panels(const int* taps, int ntaps, int hw_stride, int Cin, int n_tile) {
  using namespace cv;
  constexpr int kShapes[5][2] = {{3, 3}, {3, 1}, {2, 2}, {2, 1}, {1, 1}};
  TapPanels tp{};
  int order[kMaxTaps];
  for (int i = 0; i < ntaps; ++i) order[i] = i;
  std::stable_sort(order, order + ntaps, [&](int a, int b) { return taps[3 * a] < taps[3 * b]; });
  for (int shape = hw_stride == 1 ? 0 : 4; shape < 5; ++shape) {
    const int run = kShapes[shape][0], cols = kShapes[shape][1];
    bool used[kMaxTaps] = {};
    bool fits = ntaps % (run * cols) == 0;
    tp.n = 0;
    for (int q = 0; q < ntaps && fits; ++q) {
      const int i = order[q];
      if (used[i]) continue;
      // the corner of the panel: the first row among the frame offset's unused taps (of the tap's column, for columns), and the first
      // column of that row
      int dh0 = taps[3 * i + 1], dw0 = taps[3 * i + 2];
      if (run > 1)
        for (int k = 0; k < ntaps; ++k)
          if (!used[k] && taps[3 * k] == taps[3 * i] && (cols > 1 || taps[3 * k + 2] == taps[3 * i + 2]) &&
              (taps[3 * k + 1] < dh0 || (taps[3 * k + 1] == dh0 && taps[3 * k + 2] < dw0))) {
            dh0 = taps[3 * k + 1];
            dw0 = taps[3 * k + 2];
          }
      for (int j = 0; j < run * cols && fits; ++j) {
        int found = run > 1 ? -1 : i;
        for (int k = 0; k < ntaps && found < 0; ++k)
          if (!used[k] && taps[3 * k] == taps[3 * i] && taps[3 * k + 1] == dh0 + j / cols && taps[3 * k + 2] == dw0 + j % cols) found = k;
        fits = found >= 0;
        if (fits) {
          used[found] = true;
          tp.tap[tp.n][j % cols][j / cols] = found;
        }
      }
      tp.dt[tp.n] = taps[3 * i];
      tp.dh[tp.n] = dh0;
      tp.dw[tp.n] = dw0;
      ++tp.n;
    }
    tp.run = run;
    tp.cols = cols;
    if (fits) break;
  }
  // Squares go column by column where a shared box costs more than it saves. 16 output channels: an MMA is over as soon as its A rows are
  // read, and rows that do not start on 1,024 bytes are read slower (96 to 3 channels, 704 x 1280: 9 taps 114 us with one box, 88 by
  // columns, 27 taps 231 and 217). 16 input channels: a column is three MMAs, in whose time the wait for another barrier does not hide (16 to
  // 384, 27 taps, 88 x 160 16.9 and 15.2 us, 352 x 640 143 and 132). With 32 channels on either side the shared box is as fast or faster.
  // (The frame's size has no say: a band of rows has to give the bits of the whole frame.)
  if (tp.cols == 3 && (Cin == 16 || (n_tile == 16 && Cin > 32))) {
    const TapPanels square = tp;
    tp.cols = 1;
    tp.n = square.n * 3;
    for (int c = 0; c < tp.n; ++c) {
      const int g = c / 3, i = c % 3;
      tp.dt[c] = square.dt[g];
      tp.dh[c] = square.dh[g];
      tp.dw[c] = square.dw[g] + i;
      for (int j = 0; j < 3; ++j) tp.tap[c][0][j] = square.tap[g][i][j];
    }
  }
  return tp;
}

// rows and columns of the panels, their number, then of each panel: dt, dh, dw and its taps by column and row; returns the number of values
extern "C" int cb200_conv_panels(const int* taps, int ntaps, int hw_stride, int Cin, int n_tile, int* out) {
  if (ntaps < 1 || ntaps > cv::kMaxTaps) return 0;
  const TapPanels tp = tap_panels(taps, ntaps, hw_stride, Cin, n_tile);
  int n = 0;
  for (int v : {tp.run, tp.cols, tp.n}) out[n++] = v;
  for (int g = 0; g < tp.n; ++g) {
    for (int v : {tp.dt[g], tp.dh[g], tp.dw[g]}) out[n++] = v;
    for (int i = 0; i < tp.cols; ++i)
      for (int j = 0; j < tp.run; ++j) out[n++] = tp.tap[g][i][j];
  }
  return n;
}

// x [T_in, H_in, W_in, Cin] bf16; cache [cache_frames <= pad, H_in, W_in, Cin] or null; w [n_rows, ntaps * kblocks * 64] bf16 with
// n_rows = tiles_n * n_tile; taps: ntaps x (dt, dh, dw), dt counted from the first of the `pad` frames in front of x.
// out_map: {ot_mul, ot_add, oh_mul, oh_add, ow_mul, ow_add, out_H, out_W, out_C, oc_add}.
extern "C" int cb200_conv_cl(const void* x, int T_in, int H_in, int W_in, int Cin, const void* cache, int cache_frames, int pad, int t_stride,
                             int hw_stride, const void* w, int n_rows, int n_tile, int Cout, const int* taps, int ntaps, int T_out, int H_out, int W_out, const int* out_map,
                             void* y, const void* resid, const float* bias, void* y_norm, const float* gamma, int silu, int write_raw,
                             int* err, int sms, cudaStream_t st) {
  using namespace cv;
  if (Cin % 16 != 0 || Cin < 16 || ntaps < 1 || ntaps > kMaxTaps || n_tile % 16 != 0 || n_tile < 16 || n_tile > 256 ||
      n_rows % n_tile != 0 || Cout > n_rows || Cout < 1 || pad < 0 || pad > 64 || cache_frames < 0 || cache_frames > pad || t_stride < 1 || t_stride > 8 || hw_stride < 1 || hw_stride > 2)
    return -51;
  ConvParams p{};
  p.T_out = T_out;
  p.Cin = Cin;
  p.Cout = Cout;
  p.n_tile = n_tile;
  p.tiles_n = (Cout + n_tile - 1) / n_tile;
  p.kblocks = (Cin + BK - 1) / BK;
  p.pad = pad;
  p.cache_frames = cache != nullptr ? cache_frames : 0;
  p.t_stride = t_stride;
  p.xy_stride = hw_stride;
  int max_dt = -128;
  for (int i = 0; i < ntaps; ++i) {
    const int dt = taps[3 * i], dh = taps[3 * i + 1], dw = taps[3 * i + 2];
    if (dt < -64 || dt > 64 || dh < -64 || dh > 64 || dw < -64 || dw > 64) return -52;
    max_dt = std::max(max_dt, dt);
  }
  if (pad > 0 && max_dt < pad) return -52;      // the newest tap has to read X itself: otherwise a frame could be all padding
  const TapPanels tp = tap_panels(taps, ntaps, hw_stride, Cin, n_tile);
  const int run = tp.run, cols = tp.cols;
  p.npanels = tp.n;
  // Voxels of a line along the width, or along the height where that leaves fewer tiles; two tiles side by side for narrow layers, unless
  // 16 x 16 voxels leave more than a fifth over.
  auto up = [](int a, int b) -> long { return (a + b - 1) / b; };
  const long along_w = up(W_out, TX) * up(H_out, TY), along_h = up(H_out, TX) * up(W_out, TY), pairs = 2 * up(W_out, 2 * TX) * up(H_out, TY);
  const int stack = run == 3 && n_tile <= 128 && pairs * 10 <= std::min(along_w, along_h) * 12 ? 2 : 1;
  const bool by_height = stack == 1 && along_h < along_w && (cols > 1 || run == 1);
  p.X_out = by_height ? H_out : W_out;
  p.Y_out = by_height ? W_out : H_out;
  for (int g = 0; g < p.npanels; ++g) {
    p.dt[g] = (int8_t)tp.dt[g];
    p.dx[g] = (int8_t)(by_height ? tp.dh[g] : tp.dw[g]);
    p.dy[g] = (int8_t)(by_height ? tp.dw[g] : tp.dh[g]);
    for (int i = 0; i < cols; ++i)
      for (int j = 0; j < run; ++j) p.tap[g][i][j] = (int8_t)tp.tap[g][i][j];
  }
  const int box_x = TX * stack + cols - 1, box_y = TY + run - 1;
  const int a_slot = (box_x * box_y * BK * 2 + 1023) / 1024 * 1024, b_slot = run * n_tile * BK;
  const int fixed = kSmemFixed + (Cout <= kBiasMax ? (Cout * 4 + 15) / 16 * 16 : 0) + (y_norm != nullptr ? kSumSq + 256 * 4 : 0);
  // ring depths: as many columns of taps ahead as both rings hold
  int ahead = 0;
  for (int a = 1; a <= kMaxSlots; ++a) {
    const int b = cols == 1 ? (a * (a_slot + b_slot) <= kSmemMax - fixed ? a : 0) : std::min(kMaxSlots, (kSmemMax - fixed - a * a_slot) / b_slot);
    const int reach = std::min(a * cols, b);
    if (b >= 1 && (reach > ahead || (reach == ahead && a == 2))) {       // a second box even where it does not reach further
      ahead = reach;
      p.a_slots = a;
      p.b_slots = b;
    }
  }
  if (ahead == 0) return -57;
  {
    const long ot_mul = out_map[0], ot_add = out_map[1], oh_mul = out_map[2], oh_add = out_map[3], ow_mul = out_map[4], ow_add = out_map[5],
               out_H = out_map[6], out_W = out_map[7], out_C = out_map[8], oc_add = out_map[9];
    p.out_t = ot_mul * out_H * out_W * out_C;
    const long per_h = oh_mul * out_W * out_C, per_w = ow_mul * out_C;
    p.out_x = by_height ? per_h : per_w;
    p.out_y = by_height ? per_w : per_h;
    p.out_at = ((ot_add * out_H + oh_add) * out_W + ow_add) * out_C + oc_add;
    p.vec = ((out_C | oc_add | Cout) & 7) == 0;
  }
  p.Y = (bf16*)y;
  p.resid = (const bf16*)resid;
  p.bias = bias;
  if (y_norm != nullptr && (p.tiles_n != 1 || gamma == nullptr || !p.vec)) return -55;
  if (y_norm == nullptr && !write_raw) return -55;
  p.Yn = (bf16*)y_norm;
  p.gamma = gamma;
  p.norm_scale = sqrtf((float)Cout);
  p.silu = silu;
  p.write_raw = write_raw;
  CUtensorMap tx, tc, tw;
  const uint64_t per_w = (uint64_t)Cin * 2, per_h = (uint64_t)W_in * Cin * 2;
  const uint64_t strides[3] = {by_height ? per_h : per_w, by_height ? per_w : per_h, (uint64_t)H_in * W_in * Cin * 2};
  const uint64_t in_x = (uint64_t)(by_height ? H_in : W_in), in_y = (uint64_t)(by_height ? W_in : H_in);
  const uint32_t hw = (uint32_t)hw_stride, box[4] = {BK, (uint32_t)box_x * hw, (uint32_t)box_y * hw, 1}, step[4] = {1, hw, hw, 1};
  {
    const uint64_t dims[4] = {(uint64_t)Cin, in_x, in_y, (uint64_t)T_in};
    const int rc = make_tmap_bf16(&tx, x, 4, dims, strides, box, 1, step);
    if (rc) return rc;
  }
  tc = tx;
  if (p.cache_frames > 0) {
    const uint64_t dims[4] = {(uint64_t)Cin, in_x, in_y, (uint64_t)p.cache_frames};
    const int rc = make_tmap_bf16(&tc, cache, 4, dims, strides, box, 1, step);
    if (rc) return rc;
  }
  {
    const uint64_t kdim = (uint64_t)ntaps * p.kblocks * BK;
    const int rc = make_tmap_2d_bf16(&tw, w, kdim, (uint64_t)n_rows, kdim * 2, BK, (uint32_t)(n_tile / 2));
    if (rc) return rc;
  }
  const long vox = (long)T_out * up(p.X_out, TX * stack) * up(p.Y_out, TY);
  const long tiles = (vox + 1) / 2 * p.tiles_n;
  if (tiles <= 0 || 2 * tiles > 0x7fffffffL) return -53;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * (sms / 2));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = (size_t)p.a_slots * a_slot + (size_t)p.b_slots * b_slot + fixed;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 2;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.numAttrs = 2;
  // (with one tap per panel both orders of the axes run the same code)
  auto go = [&](auto launch) { return launch(cfg, tiles, sms, tx, tc, tw, p, err); };
  if (run == 1) return go(launch_conv<1, 1, false, 1>);
  if (run == 2 && cols == 1) return go(launch_conv<2, 1, false, 1>);
  if (run == 2) return by_height ? go(launch_conv<2, 1, true, 2>) : go(launch_conv<2, 1, false, 2>);
  if (cols == 1) return stack == 2 ? go(launch_conv<3, 2, false, 1>) : go(launch_conv<3, 1, false, 1>);
  if (stack == 2) return go(launch_conv<3, 2, false, 3>);
  return by_height ? go(launch_conv<3, 1, true, 3>) : go(launch_conv<3, 1, false, 3>);
}

extern "C" int cb200_rmsnorm_silu_cl(const void* x, const float* gamma, void* y, long n_vox, int C, int silu, cudaStream_t st) {
  if (C % 8 != 0 || C > 1024 || n_vox <= 0) return -54;
  const float scale = sqrtf((float)C);
  auto run = [&](auto kern, int lanes) {
    const int per_block = 256 / lanes;
    launch_pdl(kern, dim3((unsigned)std::min<long>((n_vox + per_block - 1) / per_block, kRmsCtas)), dim3(256), 0, st, (const bf16*)x, gamma, (bf16*)y, n_vox, C, scale, silu);
  };
  // three pieces per lane while that fills the lanes (C = 96, 192, 384, 768: no idle lane), never more than the row has: a lane keeps gamma for
  // all of its pieces, and with four pieces for 512 channels the kernel was slower than without (25,600 voxels 13.1 and 17.3 us)
  if (C <= 16) run(rmsnorm_silu_cl_kernel<2, 1>, 2);
  else if (C <= 48) run(rmsnorm_silu_cl_kernel<2, 3>, 2);
  else if (C <= 96) run(rmsnorm_silu_cl_kernel<4, 3>, 4);
  else if (C <= 192) run(rmsnorm_silu_cl_kernel<8, 3>, 8);
  else if (C <= 384) run(rmsnorm_silu_cl_kernel<16, 3>, 16);
  else if (C <= 512) run(rmsnorm_silu_cl_kernel<32, 2>, 32);
  else if (C <= 768) run(rmsnorm_silu_cl_kernel<32, 3>, 32);
  else run(rmsnorm_silu_cl_kernel<32, 4>, 32);
  return (int)cudaGetLastError();
}
