// Shared device helpers for the sm_100a kernels of this package.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace cb200 {

using bf16 = __nv_bfloat16;

// 16-byte vector of 8 bf16 values
struct alignas(16) bf16x8 {
  __nv_bfloat162 v[4];
};

__device__ __forceinline__ void unpack8(const bf16x8& p, float (&f)[8]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 t = __bfloat1622float2(p.v[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}

__device__ __forceinline__ bf16x8 pack8(const float (&f)[8]) {
  bf16x8 p;
#pragma unroll
  for (int i = 0; i < 4; ++i) p.v[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return p;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Block-wide sum for up to 1024 threads; every thread receives the total. `red` is 32 floats of smem.
__device__ __forceinline__ float block_sum(float v, float* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  v = warp_sum(v);
  __syncthreads();  // protect `red` from a previous use
  if (lane == 0) red[warp] = v;
  __syncthreads();
  const int nwarps = (blockDim.x + 31) >> 5;
  float t = (lane < nwarps) ? red[lane] : 0.f;
  t = warp_sum(t);
  return t;
}

__device__ __forceinline__ float scrub(float x) {
  // NaN and +-Inf become 0 (the reference's nan_to_num(0,0,0) before clipping)
  return (fabsf(x) <= 3.402823466e+38f) ? x : 0.f;
}

// Programmatic dependent launch: a kernel launched with `launch_pdl` may start before the kernel in front of it on the stream has
// ended - its set-up (barriers, TMEM, descriptors) and its launch then overlap that kernel's tail. Every thread block of such a kernel
// calls pdl_wait() before its first access to global memory (the device's error word apart, which the kernel reads again behind it); the
// call returns when the kernel in front is complete and its writes are visible. Hints that ask a tile into L2 may come ahead of it: they read
// nothing into the kernel, and L2 is where the writes of the kernel in front meet the loads behind the wait. pdl_trigger() lets the next kernel start; it comes after the block's own TMEM allocation, so that a waiting kernel
// never holds what a block of this one still needs (the next kernel starts only when every block has triggered or ended).
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... P, typename... A>
static inline cudaError_t launch_pdl(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
}

}  // namespace cb200
