// Small device helpers shared by the bandwidth-bound kernels (norms, RoPE, activations, optimizer,
// losses): 128-bit vector access, warp/block reductions, bf16 pack/unpack.
#pragma once
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>

namespace sx {

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
__device__ __forceinline__ bf16x8 ld8(const __nv_bfloat16* p) { return *reinterpret_cast<const bf16x8*>(p); }
__device__ __forceinline__ void st8(__nv_bfloat16* p, const bf16x8& v) { *reinterpret_cast<bf16x8*>(p) = v; }

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
// Block-wide sum; `red` is shared scratch of >= 33 floats. All threads receive the result.
__device__ __forceinline__ float block_sum(float v, float* red) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  if (w == 0) {
    float t = lane < nw ? red[lane] : 0.f;
    t = warp_sum(t);
    if (lane == 0) red[32] = t;
  }
  __syncthreads();
  return red[32];
}
__device__ __forceinline__ float block_max(float v, float* red) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_max(v);
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  if (w == 0) {
    float t = lane < nw ? red[lane] : -INFINITY;
    t = warp_max(t);
    if (lane == 0) red[32] = t;
  }
  __syncthreads();
  return red[32];
}

// Launch of a kernel whose blocks may be set up while the kernel before it on the stream still runs (programmatic dependent launch), so that what lies
// between the two is the wait, not a launch. In a decode step of an 8B-width model half of the kernels take 2 to 3 us, most of it that.
// The kernel executes griddepcontrol.wait before it touches anything that an earlier kernel writes or reads. Its pointers are not __restrict__: that
// would promise the compiler that nobody else writes the memory while the kernel runs, and let it load around the cache's coherence or ahead of the
// wait, but until the wait returns the kernel before does write it. Whether it lets its own successor start early is up to it: after_predecessor()
// does, the paged decode kernel does not.
// A chain of kernels that signal before they wait holds nothing back. Loads in front of a wait (the static weights of a decode product) may pass all of
// them, up to the last kernel that was not launched this way or did not signal: no kernel behind that one may write what is loaded so.
// When to let the successor start: at once where this kernel leaves the SMs nearly empty, so that the successor's set-up and first loads of weights lie
// under the wait (eight norms and products of one row of 768: 78 us, 83 behind the wait; a step of an 8B decoder for one sequence 7.9 and 8.2 ms); behind the
// wait from three warps an SM on, because kernels that wait hold places, and what follows is dealt out unevenly around them (eight norms of 300 rows of
// 16384 106 and 69 us, 73 launched ordinarily). `most` CTAs: above that not at all, for the same reason where a CTA's share is long (600 rows: 159 us, 111).
__device__ __forceinline__ void after_predecessor(unsigned most = 0xffffffffu) {
  const unsigned ctas = gridDim.x * gridDim.y * gridDim.z;
  const bool small = (unsigned long long)ctas * (blockDim.x * blockDim.y) <= 148 * 96;
  if (small) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");                // all that kernels before this one wrote is there
  if (!small && ctas <= most) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <typename... K, typename... A>
inline cudaError_t launch_dependent(void (*kern)(K...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, static_cast<K>(args)...);
}

// Launch shape of a kernel whose thread takes one of `items` pieces of a token: block (pieces, tokens), grid (tokens, pieces). Tokens of fewer
// than 128 pieces share a CTA, so that it has 8 warps (one token each left 32 threads to a CTA: rotating 131072 tokens of one head of 16 took
// 72 us, 6 so). Larger ones go over several CTAs, of 128 threads where tokens are few, because a thread that takes pieces one after another
// waits for each (500 tokens of 48 heads of 256: 10.3 us with 512 threads a token, 8.3 so).
inline void token_grid(long long tokens, int items, dim3* grid, dim3* block) {
  if (items < 128) {
    *block = dim3(items, 256 / items);
    *grid = dim3((unsigned)((tokens + block->y - 1) / block->y));
  } else {
    const int most = tokens < 148 ? 128 : 512, parts = (items + most - 1) / most;
    *block = dim3(((items + parts - 1) / parts + 31) / 32 * 32);
    *grid = dim3((unsigned)tokens, parts);
  }
}

}  // namespace sx
