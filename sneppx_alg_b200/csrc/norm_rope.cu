// N1: RMSNorm forward/backward with the residual add fused in, and LayerNorm forward.
// R1: rotary position embedding (rotate-half and adjacent-pair conventions) of the fused QKV activation,
//     into a new buffer or in place, forward and backward.
// SwiGLU / GeGLU gating forward and backward.
// All bf16 in/out with fp32 math; rows are read with 128-bit loads. These replace the
// reference's layernorm / rmsnorm / rope kernels (kernel/cuda/tensor_cuda.cu:393-441,
// kernel/cuda/autodiff_cuda.cu:444-487, kernel/cuda/attention_cuda.cu:895-943) and the CPU gated
// activations (kernel/activations/gated_activations.c:33-118).
#include "common.cuh"
#include "sx_api.h"

namespace sx {

// Sum over the block with one barrier: every thread adds the warps' partial sums. `red`: 32 floats, not reused before the next barrier.
__device__ __forceinline__ float row_sum(float v, float* red) {
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  v = warp_sum(v);
  if (lane == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  return warp_sum(lane < nw ? red[lane] : 0.f);
}

// Rows that are read once: they leave the weights' place in L1 alone. (What these kernels read may be written until their wait returns, so the
// non-coherent loads that would do that are not open to them.)
__device__ __forceinline__ bf16x8 ld8_once(const __nv_bfloat16* p) {
  bf16x8 v;
  uint32_t* u = reinterpret_cast<uint32_t*>(&v);
  asm volatile("ld.global.L1::no_allocate.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]) : "l"(p) : "memory");
  return v;
}

// y = rmsnorm(x + res_in) * w ; res_out = x + res_in ; rstd saved for backward.
// Bound: memory. A row stays in the registers of one CTA between the sum and the output (V vectors of 8 a thread), so it is read once and
// all of its loads are in flight together; rows are spread over CTAs and overlap. Two vectors a thread keep CTAs small enough that
// several share an SM; the weights come from L1 or L2 when the sum is there, because registers for them cost CTAs, too. Warm, with / without a
// residual: [8192, 6144] 64 / 46 us (85 / 47 with the weights fetched first, through the read-only path), [8192, 2560] 30 / 21 (37 / 23),
// [4096, 4096] 22 / 14 (26 / 16). RES: with a residual; without one the registers for it cost CTAs an SM.
template <int V, bool RES>
__global__ void __launch_bounds__(512) rmsnorm_fwd_kernel(const __nv_bfloat16* x, const __nv_bfloat16* res_in, const __nv_bfloat16* w,
                                                          __nv_bfloat16* y, __nv_bfloat16* res_out, float* rstd, int d, float eps) {
  after_predecessor(2 * 148);
  __shared__ float red[32];
  const long long row = blockIdx.x;
  const int nvec = d >> 3, t = threadIdx.x;
  bf16x8 a[V], b[RES ? V : 1];
#pragma unroll
  for (int k = 0; k < V; ++k) {
    const int i = t + k * blockDim.x;
    if (i < nvec) {
      a[k] = ld8_once(x + row * d + i * 8);
      if (RES) b[k] = ld8_once(res_in + row * d + i * 8);
    }
  }
  float f[V][8], ss = 0.f;
#pragma unroll
  for (int k = 0; k < V; ++k) {
    const int i = t + k * blockDim.x;
#pragma unroll
    for (int j = 0; j < 8; ++j) f[k][j] = 0.f;
    if (i >= nvec) continue;
    unpack8(a[k], f[k]);
    float h[8];
    if (RES) {
      unpack8(b[RES ? k : 0], h);
#pragma unroll
      for (int j = 0; j < 8; ++j) f[k][j] += h[j];
      // round through bf16 so that the statistics match what backward will re-read
      const bf16x8 hp = pack8(f[k]);
      unpack8(hp, h);
      if (res_out) {
        st8(res_out + row * d + i * 8, hp);
        unpack8(hp, f[k]);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) h[j] = f[k][j];
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) ss += h[j] * h[j];
  }
  ss = row_sum(ss, red);
  bf16x8 wv[V];
#pragma unroll
  for (int k = 0; k < V; ++k)
    if (t + k * blockDim.x < nvec) wv[k] = ld8(w + (t + k * blockDim.x) * 8);
  const float r = rsqrtf(ss / d + eps);
  if (t == 0 && rstd) rstd[row] = r;
#pragma unroll
  for (int k = 0; k < V; ++k) {
    const int i = t + k * blockDim.x;
    if (i >= nvec) continue;
    float g[8];
    unpack8(wv[k], g);
#pragma unroll
    for (int j = 0; j < 8; ++j) g[j] = f[k][j] * r * g[j];
    st8(y + row * d + i * 8, pack8(g));
  }
}
// Rows longer than 8192: two passes.
__global__ void __launch_bounds__(256) rmsnorm_fwd_long_kernel(const __nv_bfloat16* x, const __nv_bfloat16* res_in, const __nv_bfloat16* w,
                                                               __nv_bfloat16* y, __nv_bfloat16* res_out, float* rstd, int d, float eps) {
  after_predecessor(2 * 148);
  __shared__ float red[33];
  const long long row = blockIdx.x;
  const __nv_bfloat16* xr = x + row * d;
  const int nvec = d >> 3;
  float ss = 0.f;
  for (int i = threadIdx.x; i < nvec; i += blockDim.x) {
    float f[8];
    unpack8(ld8(xr + i * 8), f);
    if (res_in) {
      float g[8];
      unpack8(ld8(res_in + row * d + i * 8), g);
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] += g[j];
      bf16x8 hp = pack8(f);
      unpack8(hp, f);
      if (res_out) st8(res_out + row * d + i * 8, hp);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) ss += f[j] * f[j];
  }
  ss = block_sum(ss, red);
  const float r = rsqrtf(ss / d + eps);
  if (threadIdx.x == 0 && rstd) rstd[row] = r;
  const __nv_bfloat16* hr = (res_in && res_out) ? res_out + row * d : xr;
  for (int i = threadIdx.x; i < nvec; i += blockDim.x) {
    float f[8], g[8];
    unpack8(ld8(hr + i * 8), f);
    if (res_in && !res_out) {
      unpack8(ld8(res_in + row * d + i * 8), g);
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] += g[j];
    }
    unpack8(ld8(w + i * 8), g);
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = f[j] * r * g[j];
    st8(y + row * d + i * 8, pack8(f));
  }
}

// dx = rstd * (w*dy) - h * rstd^3 * mean(w*dy*h) (+ dres) ; dw partial sums per CTA.
// Each CTA walks rows blockIdx.x, blockIdx.x + gridDim.x, ... and keeps its dw partials in registers (thread t owns column vectors
// t, t + blockDim, ...; at most V of them). Bound: memory. With V <= 2 the loads of the next row are issued before the sum of this one, otherwise
// a CTA has one row in flight and the barrier's latency between rows. [4096, 4096] with dres: 46 us (20 us at copy bandwidth) with the
// reduction of the partials, 75 us before; [8192, 5120]: 122 and 263 us. Four vectors a thread (rows of more than 8192) leave no registers
// for the next row: with it 264 bytes a thread are spilled. [8192, 12288] 180 us, 550 with the next row, 362 with eight vectors a thread.
template <int V>
__global__ void __launch_bounds__(512) rmsnorm_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ h,
                                                          const __nv_bfloat16* __restrict__ w, const float* __restrict__ rstd,
                                                          const __nv_bfloat16* __restrict__ dres, __nv_bfloat16* __restrict__ dx,
                                                          float* __restrict__ dw_partial, int T, int d) {
  constexpr bool AHEAD = V <= 2;
  __shared__ float red[2][32];
  const int nvec = d >> 3, t = threadIdx.x;
  float acc[V][8];
  bf16x8 wv[V], gv[V], hv[V], ev[V], gn[V], hn[V], en[V];
  float rn = 0.f;
#pragma unroll
  for (int k = 0; k < V; ++k) {
    const int i = t + k * blockDim.x;
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[k][j] = 0.f;
    if (i < nvec) wv[k] = ld8(w + i * 8);
  }
  auto fetch = [&](long long row) {
    rn = rstd[row];
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const int i = t + k * blockDim.x;
      if (i < nvec) {
        gn[k] = ld8(dy + row * d + i * 8);
        hn[k] = ld8(h + row * d + i * 8);
        if (dres) en[k] = ld8(dres + row * d + i * 8);
      }
    }
  };
  if (AHEAD && (int)blockIdx.x < T) fetch(blockIdx.x);
  int buf = 0;
  for (long long row = blockIdx.x; row < T; row += gridDim.x, buf ^= 1) {
    if (!AHEAD) fetch(row);
    const float r = rn;
#pragma unroll
    for (int k = 0; k < V; ++k) {
      gv[k] = gn[k];
      hv[k] = hn[k];
      ev[k] = en[k];
    }
    if (AHEAD && row + gridDim.x < T) fetch(row + gridDim.x);
    float dot = 0.f;
#pragma unroll
    for (int k = 0; k < V; ++k) {
      if (t + k * blockDim.x >= nvec) continue;
      float g[8], hh[8], ww[8];
      unpack8(gv[k], g);
      unpack8(hv[k], hh);
      unpack8(wv[k], ww);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        acc[k][j] += g[j] * hh[j] * r;
        dot += g[j] * ww[j] * hh[j];
      }
    }
    dot = row_sum(dot, red[buf]);      // two buffers: the next row's partial sums do not meet slow readers of this one's
    const float c = dot * r * r * r / d;
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const int i = t + k * blockDim.x;
      if (i >= nvec) continue;
      float g[8], hh[8], ww[8];
      unpack8(gv[k], g);
      unpack8(hv[k], hh);
      unpack8(wv[k], ww);
#pragma unroll
      for (int j = 0; j < 8; ++j) g[j] = g[j] * ww[j] * r - hh[j] * c;
      if (dres) {
        unpack8(ev[k], hh);
#pragma unroll
        for (int j = 0; j < 8; ++j) g[j] += hh[j];
      }
      st8(dx + row * d + i * 8, pack8(g));
    }
  }
#pragma unroll
  for (int k = 0; k < V; ++k) {
    const int i = t + k * blockDim.x;
    if (i < nvec) {
      float4* o = reinterpret_cast<float4*>(dw_partial + (long long)blockIdx.x * d + i * 8);
      o[0] = make_float4(acc[k][0], acc[k][1], acc[k][2], acc[k][3]);
      o[1] = make_float4(acc[k][4], acc[k][5], acc[k][6], acc[k][7]);
    }
  }
}

// Column sums of the partial rows: 32 columns x 32 row groups a CTA (one thread a column walked all rows one after another: 16 us at 296
// rows of 4096; with it [512, 512] backward took 21.5 us, now 13).
__global__ void __launch_bounds__(1024) colsum_partials_kernel(const float* __restrict__ part, int nparts, int d,
                                                               __nv_bfloat16* __restrict__ out_bf16, float* __restrict__ out_f32,
                                                               int accumulate) {
  __shared__ float red[32][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5, c = blockIdx.x * 32 + tx;
  float s = 0.f;
  if (c < d) {
#pragma unroll 4
    for (int p = ty; p < nparts; p += 32) s += part[(long long)p * d + c];
  }
  red[ty][tx] = s;
  __syncthreads();
  s = warp_sum(red[tx][ty]);             // warp ty adds column ty of the block
  const int co = blockIdx.x * 32 + ty;
  if (tx != 0 || co >= d) return;
  if (out_f32) out_f32[co] = accumulate ? out_f32[co] + s : s;
  if (out_bf16) out_bf16[co] = __float2bfloat16(accumulate ? __bfloat162float(out_bf16[co]) + s : s);
}

__global__ void __launch_bounds__(256) layernorm_fwd_kernel(const __nv_bfloat16* __restrict__ x,
                                                            const __nv_bfloat16* __restrict__ w,
                                                            const __nv_bfloat16* __restrict__ b,
                                                            __nv_bfloat16* __restrict__ y, float* __restrict__ mean,
                                                            float* __restrict__ rstd, int d, float eps) {
  __shared__ float red[33];
  const long long row = blockIdx.x;
  float s = 0.f;
  for (int i = threadIdx.x; i < d; i += blockDim.x) s += __bfloat162float(x[row * d + i]);
  const float mu = block_sum(s, red) / d;
  float v = 0.f;
  for (int i = threadIdx.x; i < d; i += blockDim.x) {
    const float t = __bfloat162float(x[row * d + i]) - mu;
    v += t * t;
  }
  const float r = rsqrtf(block_sum(v, red) / d + eps);
  if (threadIdx.x == 0) {
    if (mean) mean[row] = mu;
    if (rstd) rstd[row] = r;
  }
  for (int i = threadIdx.x; i < d; i += blockDim.x) {
    float t = (__bfloat162float(x[row * d + i]) - mu) * r * __bfloat162float(w[i]);
    if (b) t += __bfloat162float(b[i]);
    y[row * d + i] = __float2bfloat16(t);
  }
}

// RoPE in place. x: [tokens, row_stride] with `heads` heads of size D starting at column 0.
// table: [max_pos, D/2] cos and sin (fp32). pos: optional per-token position, else token % seq.
__global__ void rope_kernel(__nv_bfloat16* __restrict__ x, const float* __restrict__ cos_t,
                            const float* __restrict__ sin_t, const int* __restrict__ pos, long long tokens,
                            int seq, int heads, int D, long long row_stride, int interleaved, float sign) {
  const int half = D >> 1;
  const long long total = tokens * heads * half;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const int i = idx % half;
    const int hd = (idx / half) % heads;
    const long long t = idx / ((long long)half * heads);
    const int p = pos ? pos[t] : (int)(t % seq);
    const float c = cos_t[(long long)p * half + i];
    const float s = sin_t[(long long)p * half + i] * sign;
    __nv_bfloat16* base = x + t * row_stride + (long long)hd * D;
    const int i1 = interleaved ? 2 * i : i;
    const int i2 = interleaved ? 2 * i + 1 : i + half;
    const float a = __bfloat162float(base[i1]);
    const float b = __bfloat162float(base[i2]);
    base[i1] = __float2bfloat16(a * c - b * s);
    base[i2] = __float2bfloat16(b * c + a * s);
  }
}

// Rotate-half layout from src to dst (which may be the same): 8 rotation pairs per thread, i.e. two 16-byte loads of x (the halves) and 2 x 32
// bytes of cos / sin, which the heads of a token share in L1. Heads from `rot` on are copied. Launch shape: token_grid. Bound: memory; rotating
// into a new buffer replaces a copy followed by a rotation in place ([4096, 48 x 128]: 27 + 23 us before, 27 us).
__global__ void __launch_bounds__(512) rope_vec8_kernel(const __nv_bfloat16* src, __nv_bfloat16* dst, const float* __restrict__ cos_t,
                                                        const float* __restrict__ sin_t, const int* __restrict__ pos, unsigned tokens,
                                                        int seq, int heads, int rot, int D, long long src_stride, long long dst_stride,
                                                        float sign) {
  const int half = D >> 1, hv = half >> 3;
  const unsigned t = blockIdx.x * blockDim.y + threadIdx.y;
  if (t >= tokens) return;
  const long long p = pos ? pos[t] : (int)(t % (unsigned)seq);
  src += t * src_stride;
  dst += t * dst_stride;
  for (int k = blockIdx.y * blockDim.x + threadIdx.x; k < heads * hv; k += gridDim.y * blockDim.x) {
    const int hd = k / hv, i = (k - hd * hv) * 8, o = hd * D + i;
    const bf16x8 pa = ld8(src + o), pb = ld8(src + o + half);
    if (hd >= rot) {
      st8(dst + o, pa);
      st8(dst + o + half, pb);
      continue;
    }
    const float4* cp = reinterpret_cast<const float4*>(cos_t + p * half + i);
    const float4* sp = reinterpret_cast<const float4*>(sin_t + p * half + i);
    const float4 c0 = cp[0], c1 = cp[1], s0 = sp[0], s1 = sp[1];
    const float c[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
    const float sn[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
    float a[8], b[8], ra[8], rb[8];
    unpack8(pa, a);
    unpack8(pb, b);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float s = sn[j] * sign;
      ra[j] = a[j] * c[j] - b[j] * s;
      rb[j] = b[j] * c[j] + a[j] * s;
    }
    st8(dst + o, pack8(ra));
    st8(dst + o + half, pack8(rb));
  }
}
static int rope_vec8(const void* src, void* dst, const float* cos_t, const float* sin_t, const int* pos, long long tokens, int seq, int heads,
                     int rot, int D, long long src_stride, long long dst_stride, int backward, cudaStream_t st) {
  if (heads <= 0) return -11;
  dim3 grid, block;
  token_grid(tokens, heads * (D / 16), &grid, &block);
  rope_vec8_kernel<<<grid, block, 0, st>>>((const __nv_bfloat16*)src, (__nv_bfloat16*)dst, cos_t, sin_t, pos, (unsigned)tokens, seq, heads, rot, D,
                                           src_stride, dst_stride, backward ? -1.f : 1.f);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}
static bool rope_vec8_ok(const void* src, const void* dst, const float* cos_t, const float* sin_t, long long tokens, int D, long long src_stride,
                         long long dst_stride) {
  auto aligned = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  return D % 16 == 0 && src_stride % 8 == 0 && dst_stride % 8 == 0 && tokens <= 0x7fffffffll && aligned(src) && aligned(dst) && aligned(cos_t) &&
         aligned(sin_t);
}

// h = act(gate) * up ; gu = [T, 2F] (gate | up). act: 0 silu (SwiGLU), 1 gelu (GeGLU), 2 relu (ReGLU)
__device__ __forceinline__ float gate_act(float g, int act) {
  if (act == 0) return g / (1.f + __expf(-g));
  if (act == 1) {
    const float k0 = 0.7978845608028654f, k1 = 0.044715f;
    return 0.5f * g * (1.f + tanhf(k0 * (g + k1 * g * g * g)));
  }
  return fmaxf(g, 0.f);
}
__device__ __forceinline__ float gate_act_grad(float g, int act) {
  if (act == 0) {
    const float s = 1.f / (1.f + __expf(-g));
    return s * (1.f + g * (1.f - s));
  }
  if (act == 1) {
    const float k0 = 0.7978845608028654f, k1 = 0.044715f;
    const float u = k0 * (g + k1 * g * g * g);
    const float th = tanhf(u);
    return 0.5f * (1.f + th) + 0.5f * g * (1.f - th * th) * k0 * (1.f + 3.f * k1 * g * g);
  }
  return g > 0.f ? 1.f : 0.f;
}

__global__ void glu_fwd_kernel(const __nv_bfloat16* gu, __nv_bfloat16* h, long long T, int F, int act) {
  after_predecessor();
  const int fv = F >> 3;
  const long long total = T * fv;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const long long t = idx / fv;
    const int c = (idx % fv) * 8;
    float g[8], u[8];
    unpack8(ld8(gu + t * 2 * F + c), g);
    unpack8(ld8(gu + t * 2 * F + F + c), u);
#pragma unroll
    for (int j = 0; j < 8; ++j) g[j] = gate_act(g[j], act) * u[j];
    st8(h + t * F + c, pack8(g));
  }
}

__global__ void glu_bwd_kernel(const __nv_bfloat16* __restrict__ dh, const __nv_bfloat16* __restrict__ gu,
                               __nv_bfloat16* __restrict__ dgu, long long T, int F, int act) {
  const int fv = F >> 3;
  const long long total = T * fv;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const long long t = idx / fv;
    const int c = (idx % fv) * 8;
    float g[8], u[8], d[8], dg[8], du[8];
    unpack8(ld8(gu + t * 2 * F + c), g);
    unpack8(ld8(gu + t * 2 * F + F + c), u);
    unpack8(ld8(dh + t * F + c), d);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      dg[j] = d[j] * u[j] * gate_act_grad(g[j], act);
      du[j] = d[j] * gate_act(g[j], act);
    }
    st8(dgu + t * 2 * F + c, pack8(dg));
    st8(dgu + t * 2 * F + F + c, pack8(du));
  }
}

}  // namespace sx

using namespace sx;

extern "C" int sx_rmsnorm_fwd(const void* x, const void* res_in, const void* w, void* y, void* res_out, float* rstd,
                              long long T, int d, float eps, cudaStream_t st) {
  if (d % 8) return -1;
  if (T == 0) return 0;
  const int nvec = d / 8;
  auto run = [&](auto kern, int threads) {
    launch_dependent(kern, (unsigned)T, threads, 0, st, (const __nv_bfloat16*)x, (const __nv_bfloat16*)res_in, (const __nv_bfloat16*)w,
                     (__nv_bfloat16*)y, (__nv_bfloat16*)res_out, rstd, d, eps);
  };
  auto per = [&](int v) { return ((nvec + v - 1) / v + 31) / 32 * 32; };
  // 256 threads up to 4096 as long as they have a vector each (a thread's share then does not depend on how the row divides), more threads
  // with two vectors up to 8192; a CTA of 1024 threads has an SM to itself, and two passes over L2 are faster then ([1000, 16384]: 37
  // against 43 us)
  if (nvec <= 256) res_in ? run(rmsnorm_fwd_kernel<1, true>, per(1)) : run(rmsnorm_fwd_kernel<1, false>, per(1));
  else if (nvec <= 1024) {
    const int threads = nvec <= 512 ? 256 : per(2);
    res_in ? run(rmsnorm_fwd_kernel<2, true>, threads) : run(rmsnorm_fwd_kernel<2, false>, threads);
  } else run(rmsnorm_fwd_long_kernel, 256);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

// CTAs, and rows of partial weight gradients, of the backward pass: short rows keep as much in flight with four small CTAs an SM as longer ones
// with two large.
extern "C" int sx_rmsnorm_bwd_parts(int d) { return d <= 2048 ? 592 : 296; }

// dw_partial: scratch of sx_rmsnorm_bwd_parts(d) * d floats.
extern "C" int sx_rmsnorm_bwd(const void* dy, const void* h, const void* w, const float* rstd, const void* dres,
                              void* dx, float* dw_partial, void* dw_bf16, float* dw_f32, int accumulate, long long T,
                              int d, cudaStream_t st) {
  if (d % 8) return -1;
  if (T == 0) return 0;
  const int nvec = d / 8;
  const int most = sx_rmsnorm_bwd_parts(d);
  const int parts = T < most ? (int)T : most;
  auto run = [&](auto kern, int v) {
    kern<<<parts, nvec > 256 && nvec <= 512 ? 256 : ((nvec + v - 1) / v + 31) / 32 * 32, 0, st>>>((const __nv_bfloat16*)dy, (const __nv_bfloat16*)h, (const __nv_bfloat16*)w,
                                                               rstd, (const __nv_bfloat16*)dres, (__nv_bfloat16*)dx, dw_partial, (int)T, d);
  };
  if (nvec <= 256) run(rmsnorm_bwd_kernel<1>, 1);
  else if (nvec <= 1024) run(rmsnorm_bwd_kernel<2>, 2);
  else if (nvec <= 2048) run(rmsnorm_bwd_kernel<4>, 4);
  else return -2;
  colsum_partials_kernel<<<(d + 31) / 32, 1024, 0, st>>>(dw_partial, parts, d, (__nv_bfloat16*)dw_bf16, dw_f32, accumulate);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

extern "C" int sx_layernorm_fwd(const void* x, const void* w, const void* b, void* y, float* mean, float* rstd,
                                long long T, int d, float eps, cudaStream_t st) {
  if (T == 0) return 0;
  layernorm_fwd_kernel<<<(unsigned)T, 256, 0, st>>>((const __nv_bfloat16*)x, (const __nv_bfloat16*)w,
                                                    (const __nv_bfloat16*)b, (__nv_bfloat16*)y, mean, rstd, d, eps);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

extern "C" int sx_rope(void* x, const float* cos_t, const float* sin_t, const int* pos, long long tokens, int seq,
                       int heads, int D, long long row_stride, int interleaved, int backward, cudaStream_t st) {
  if (tokens == 0) return 0;
  if (!interleaved && rope_vec8_ok(x, x, cos_t, sin_t, tokens, D, row_stride, row_stride))
    return rope_vec8(x, x, cos_t, sin_t, pos, tokens, seq, heads, heads, D, row_stride, row_stride, backward, st);
  const long long total = tokens * heads * (D / 2);
  const int blocks = (int)((total + 255) / 256 < 148 * 16 ? (total + 255) / 256 : 148 * 16);
  rope_kernel<<<blocks, 256, 0, st>>>((__nv_bfloat16*)x, cos_t, sin_t, pos, tokens, seq, heads, D, row_stride,
                                      interleaved, backward ? -1.f : 1.f);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

// Rotates the first `rot` of `heads` heads from src to dst and copies the others (rotate-half; 16-byte rows and tables: -1 otherwise).
extern "C" int sx_rope_to(const void* src, void* dst, const float* cos_t, const float* sin_t, const int* pos, long long tokens, int seq,
                          int heads, int rot, int D, long long src_stride, long long dst_stride, int backward, cudaStream_t st) {
  if (tokens == 0) return 0;
  if (!rope_vec8_ok(src, dst, cos_t, sin_t, tokens, D, src_stride, dst_stride)) return -1;
  return rope_vec8(src, dst, cos_t, sin_t, pos, tokens, seq, heads, rot, D, src_stride, dst_stride, backward, st);
}

extern "C" int sx_glu_fwd(const void* gu, void* h, long long T, int F, int act, cudaStream_t st) {
  if (F % 8) return -1;
  if (T == 0) return 0;
  const long long total = T * (F / 8);
  const int blocks = (int)((total + 255) / 256 < 148 * 16 ? (total + 255) / 256 : 148 * 16);
  launch_dependent(glu_fwd_kernel, blocks, 256, 0, st, (const __nv_bfloat16*)gu, (__nv_bfloat16*)h, T, F, act);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

extern "C" int sx_glu_bwd(const void* dh, const void* gu, void* dgu, long long T, int F, int act, cudaStream_t st) {
  if (F % 8) return -1;
  if (T == 0) return 0;
  const long long total = T * (F / 8);
  const int blocks = (int)((total + 255) / 256 < 148 * 16 ? (total + 255) / 256 : 148 * 16);
  glu_bwd_kernel<<<blocks, 256, 0, st>>>((const __nv_bfloat16*)dh, (const __nv_bfloat16*)gu, (__nv_bfloat16*)dgu, T,
                                         F, act);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}
