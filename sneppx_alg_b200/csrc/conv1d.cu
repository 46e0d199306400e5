// C1: causal depthwise conv1d (kernel width <= 4) with optional SiLU, channels-last [B, L, C] bf16,
// forward and backward, halo aware: an optional [B, K-1, C] "previous tokens" tensor supplies the left
// context (chunked prefill, decode and context-parallel ranks pass the tail of the previous chunk) and
// the final K-1 tokens can be written out as the next state.
// The reference's conv kernels limit L to one thread block (algorithms/hss/cuda/hss_cuda_extended.cu:208-226)
// and its Mamba-2 block copies instead of convolving (kernel/arch/mamba2.c:82-84).
#include "common.cuh"
#include "tc_common.cuh"
#include "sx_api.h"

namespace sx {

constexpr int CONV_MAXK = 4;

__device__ __forceinline__ float silu_f(float x) { return x / (1.f + __expf(-x)); }
__device__ __forceinline__ float silu_grad(float x) {
  const float s = 1.f / (1.f + __expf(-x));
  return s * (1.f + x * (1.f - s));
}

// V channels of a row: 8 (16 bytes), 4 or 2.
template <int V> struct ConvVec;
template <> struct ConvVec<8> { typedef uint4 T; };
template <> struct ConvVec<4> { typedef uint2 T; };
template <> struct ConvVec<2> { typedef uint32_t T; };
__device__ __forceinline__ float2 bf2(uint32_t v) { return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v)); }
__device__ __forceinline__ uint32_t pk2(float a, float b) {
  const __nv_bfloat162 t = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&t);
}
__device__ __forceinline__ void conv_unpack(uint2 r, float (&f)[4]) {
  const float2 a = bf2(r.x), b = bf2(r.y);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y;
}
__device__ __forceinline__ void conv_unpack(uint4 r, float (&f)[8]) {
  const float2 a = bf2(r.x), b = bf2(r.y), c = bf2(r.z), d = bf2(r.w);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
}
__device__ __forceinline__ void conv_unpack(uint32_t r, float (&f)[2]) {
  const float2 a = bf2(r);
  f[0] = a.x; f[1] = a.y;
}
__device__ __forceinline__ uint4 conv_pack(const float (&f)[8]) { return make_uint4(pk2(f[0], f[1]), pk2(f[2], f[3]), pk2(f[4], f[5]), pk2(f[6], f[7])); }
__device__ __forceinline__ uint2 conv_pack(const float (&f)[4]) { return make_uint2(pk2(f[0], f[1]), pk2(f[2], f[3])); }
__device__ __forceinline__ uint32_t conv_pack(const float (&f)[2]) { return pk2(f[0], f[1]); }
template <int V> __device__ __forceinline__ typename ConvVec<V>::T conv_ld(const __nv_bfloat16* p) {
  return *reinterpret_cast<const typename ConvVec<V>::T*>(p);
}
template <int V> __device__ __forceinline__ void conv_ld(const __nv_bfloat16* p, float (&f)[V]) { conv_unpack(conv_ld<V>(p), f); }
template <int V> __device__ __forceinline__ void conv_st(__nv_bfloat16* p, const float (&f)[V]) {
  *reinterpret_cast<typename ConvVec<V>::T*>(p) = conv_pack(f);
}
__device__ __forceinline__ uint64_t bf16x2_f32x2(uint32_t v) { return pack_f32x2(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u)); }
template <int K, int V>
__device__ __forceinline__ void conv_taps(const __nv_bfloat16* w, int c, float (&wv)[K][V]) {
  if (K == 4 && (reinterpret_cast<uintptr_t>(w) & 7) == 0) {   // a channel's four taps are 8 contiguous bytes
#pragma unroll
    for (int j = 0; j < V; ++j) {
      float t[4];
      conv_ld<4>(w + (c + j) * 4, t);
#pragma unroll
      for (int k = 0; k < K; ++k) wv[k][j] = t[k];
    }
  } else {
#pragma unroll
    for (int k = 0; k < K; ++k)
#pragma unroll
      for (int j = 0; j < V; ++j) wv[k][j] = __bfloat162float(w[(c + j) * K + k]);
  }
}

// One thread: V channels (4, or 8 with one tap, see sx_conv1d_fwd) x `run` consecutive positions. The K taps and the bias live in registers and the K-1 previous inputs slide through
// registers, so each input vector is loaded once and each output costs one load and one store of V channels; consecutive threads own consecutive
// channel vectors (coalesced rows).
// Bound: the instructions of a row (half of them the sigmoid), so pairs of channels go through one packed multiply-add, rounded like two scalar
// ones, and the rows that no state is made of are a loop without conditions. Cold, scalar with conditions -> now, four taps: [8192, 7168]
// 79.9 -> 67.6 us (36 at copy bandwidth), [8192, 5376] 63.5 -> 55.3, [16, 4096, 4352] 348 -> 263, [4, 2048, 1792] 30.7 -> 26.6; [8192, 7168] with
// three taps 70 -> 63.5, two 59 -> 51, one 53 either way. Three CTAs an SM: four (64 registers) spill 64 bytes and take 71.7 us with three or four
// taps, but 51 instead of 57 with two. A 32-bit division for the index spills as well (77.8 us).
template <int K, int V>
__global__ void __launch_bounds__(256, V == 8 || K >= 3 ? 3 : 4) conv1d_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ prev,
                                                            const __nv_bfloat16* __restrict__ w, const __nv_bfloat16* __restrict__ bias,
                                                            __nv_bfloat16* __restrict__ y, __nv_bfloat16* __restrict__ state_out, int B,
                                                            int L, int C, int act, long long xld, int Ly, int run) {
  typedef typename ConvVec<V>::T T;
  constexpr int P = V / 2;
  const unsigned cv = C / V, lchunks = (L + run - 1) / run;
  const long long total = (long long)B * lchunks * cv;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total; idx += (long long)gridDim.x * blockDim.x) {
    const int c = (int)(idx % cv) * V;
    const unsigned bl = (unsigned)(idx / cv);
    const int l0 = (int)(bl % lchunks) * run, b = (int)(bl / lchunks);
    const int l1 = min(L, l0 + run);
    const __nv_bfloat16* xp = x + ((long long)b * L + l0) * xld + c;
    __nv_bfloat16* yp = y + ((long long)b * Ly + l0) * C + c;
    uint64_t wv[K][P], bv[P], xh[K][P];   // pairs of channels; xh[i]: input of the position K - 1 - i before the current one
    {
      float t[K][V], f[V];
      conv_taps<K, V>(w, c, t);
      if (bias) conv_ld<V>(bias + c, f);
#pragma unroll
      for (int j = 0; j < P; ++j) {
#pragma unroll
        for (int k = 0; k < K; ++k) { wv[k][j] = pack_f32x2(t[k][2 * j], t[k][2 * j + 1]); xh[k][j] = 0; }
        bv[j] = bias ? pack_f32x2(f[2 * j], f[2 * j + 1]) : 0;
      }
    }
    auto take = [&](T r, uint64_t (&h)[P]) {
#pragma unroll
      for (int j = 0; j < P; ++j) h[j] = bf16x2_f32x2(reinterpret_cast<const uint32_t*>(&r)[j]);
    };
#pragma unroll
    for (int i = 1; i < K; ++i) {
      const int ls = l0 - K + i;
      if (ls >= 0) take(conv_ld<V>(xp + (long long)(i - K) * xld), xh[i]);
      else if (prev) take(conv_ld<V>(prev + ((long long)b * (K - 1) + (K - 1 + ls)) * C + c), xh[i]);
    }
    auto row = [&](T r) {
#pragma unroll
      for (int i = 0; i + 1 < K; ++i)
#pragma unroll
        for (int j = 0; j < P; ++j) xh[i][j] = xh[i + 1][j];
      take(r, xh[K - 1]);
      float f[V];
#pragma unroll
      for (int j = 0; j < P; ++j) {
        uint64_t a = bv[j];
#pragma unroll
        for (int k = 0; k < K; ++k) a = fma_f32x2(xh[k][j], wv[k][j], a);
        unpack_f32x2(a, f[2 * j], f[2 * j + 1]);
      }
      if (act) {
#pragma unroll
        for (int j = 0; j < V; ++j) f[j] = silu_f(f[j]);
      }
      conv_st<V>(yp, f);
      yp += C;
    };
    const int plain = state_out ? min(l1, L - (K - 1)) : l1;   // from here on rows are of the state too
    int l = l0;
    for (; l + 4 <= plain; l += 4) {
      T r[4];   // four independent loads in flight per thread
#pragma unroll
      for (int u = 0; u < 4; ++u, xp += xld) r[u] = conv_ld<V>(xp);
#pragma unroll
      for (int u = 0; u < 4; ++u) row(r[u]);
    }
    for (; l < l1; l += 4) {
      T r[4];
#pragma unroll
      for (int u = 0; u < 4; ++u, xp += xld)
        if (l + u < l1) r[u] = conv_ld<V>(xp);
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (l + u < l1) {
          row(r[u]);
          if (state_out && l + u >= L - (K - 1)) *reinterpret_cast<T*>(state_out + ((long long)b * (K - 1) + (l + u - (L - (K - 1)))) * C + c) = r[u];
        }
    }
  }
}

// The same for sequences of few positions (one token of each in a decoding step): a thread walks all of them, scalar, and has no division by runs.
// The packed form's taps and main loop stand in front of its first rows. Four taps: [16, 4, 1792] 2.83 us, 3.46 packed (3.17 when this walk served
// every length); [16, 1, 1792] 2.40 (2.70). From 8 positions on the packed form is as fast as that walk was (4.0 us) and then faster (4.8 and 5.6 at 15).
constexpr int CONV_SHORT = 8;
template <int K>
__global__ void __launch_bounds__(256, 3) conv1d_short_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ prev,
                                                              const __nv_bfloat16* __restrict__ w, const __nv_bfloat16* __restrict__ bias,
                                                              __nv_bfloat16* __restrict__ y, __nv_bfloat16* __restrict__ state_out, int B,
                                                              int L, int C, int act, long long xld, int Ly) {
  const int cv = C / 4;
  const long long total = (long long)B * cv;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total; idx += (long long)gridDim.x * blockDim.x) {
    const int c = (int)(idx % cv) * 4;
    const long long b = idx / cv;
    const __nv_bfloat16* xp = x + b * L * xld + c;
    __nv_bfloat16* yp = y + b * Ly * C + c;
    float wv[K][4], bv[4], hist[K][4];   // hist[i]: input of the position K - 1 - i before the current one
    conv_taps<K, 4>(w, c, wv);
    if (bias) conv_ld<4>(bias + c, bv);
    else {
#pragma unroll
      for (int j = 0; j < 4; ++j) bv[j] = 0.f;
    }
#pragma unroll
    for (int i = 0; i < K; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) hist[i][j] = 0.f;
    if (prev) {
#pragma unroll
      for (int i = 0; i < K - 1; ++i) conv_ld<4>(prev + (b * (K - 1) + i) * C + c, hist[i]);
    }
    for (int lb = 0; lb < L; lb += 4) {
      uint2 raw[4];   // four independent loads in flight per thread
#pragma unroll
      for (int u = 0; u < 4; ++u, xp += xld)
        if (lb + u < L) raw[u] = conv_ld<4>(xp);
#pragma unroll
      for (int u = 0; u < 4; ++u, yp += C) {
        const int l = lb + u;
        if (l >= L) break;
        conv_unpack(raw[u], hist[K - 1]);
        float acc[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[j] = bv[j];
#pragma unroll
        for (int k = 0; k < K; ++k)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[j] = fmaf(hist[k][j], wv[k][j], acc[j]);
        if (act) {
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[j] = silu_f(acc[j]);
        }
        conv_st<4>(yp, acc);
        if (state_out && l >= L - (K - 1)) *reinterpret_cast<uint2*>(state_out + (b * (K - 1) + (l - (L - (K - 1)))) * C + c) = raw[u];
#pragma unroll
        for (int i = 0; i + 1 < K; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) hist[i][j] = hist[i + 1][j];
      }
    }
  }
}

// dx and per-CTA partials of dw / dbias. A CTA is 32 pairs of channels (one per lane: 128 contiguous bytes per row) by 8 runs of `run` consecutive
// positions (one per warp). A thread walks its run once: the last K inputs and the last K pre-activation gradients slide through registers, so
// every x and dy value is loaded once (plus the K-1 row overlap between runs) and dx is stored once.
// Bound: the instructions of a row, so both channels go through one packed multiply-add (fma.f32x2), addresses advance by a row, and the rows that
// only warm up, only finish or do both are loops of their own. [8192, 7168], four taps: 159 us, 247 with two scalar channels and conditions in
// every row, 265 with four channels and fewer warps (54 us at copy bandwidth).
// The 8 warps add their dw / db into shared memory and the CTA writes one partial row; conv1d_reduce_partials sums the rows.
// One tap: rows one by one and four CTAs an SM ([8192, 7168] 82 and 89 us with SiLU; 92 and 98 four at a time, 88 and 98 scalar). FEW: sequences of
// fewer than CONV_FEW positions, without the loop of four (512 of one position and 7168 channels, four taps: 27.7 us, 32 with it, 28.4 scalar).
constexpr int CONV_FEW = 5;
template <int K, bool FEW>
__global__ void __launch_bounds__(256, K == 4 || K == 1 ? 4 : 3) conv1d_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                                                            const __nv_bfloat16* __restrict__ prev, const __nv_bfloat16* __restrict__ w,
                                                            const __nv_bfloat16* __restrict__ bias, __nv_bfloat16* __restrict__ dx,
                                                            float* __restrict__ partial, int B, int L, int C, int act, long long xld, int Ly,
                                                            long long dxld, int run) {
  __shared__ float s_acc[32][(CONV_MAXK + 1) * 2 + 1];
  const int lane = threadIdx.x & 31, sub = threadIdx.x >> 5;
  const int v = blockIdx.x * 32 + lane;
  const bool live = v < C / 2;
  const int c = v * 2;
  for (int i = threadIdx.x; i < 32 * ((CONV_MAXK + 1) * 2 + 1); i += 256) (&s_acc[0][0])[i] = 0.f;
  __syncthreads();
  if (live) {
    uint64_t wv[K], dw[K], db = 0, bv = 0;
    {
      float t[K][2];
      conv_taps<K, 2>(w, c, t);
#pragma unroll
      for (int k = 0; k < K; ++k) { wv[k] = pack_f32x2(t[k][0], t[k][1]); dw[k] = 0; }
      if (bias) bv = bf16x2_f32x2(conv_ld<2>(bias + c));
    }
    const int lchunks = (L + run - 1) / run;
    const int nchunks = B * lchunks;
    for (int ch = blockIdx.y * 8 + sub; ch < nchunks; ch += gridDim.y * 8) {
      const int b = ch / lchunks, l0 = (ch % lchunks) * run;
      const int lend = min(l0 + run, L);
      // xh[i], dp[i]: input and pre-activation gradient of the position K - 1 - i before the current one
      uint64_t xh[K], dp[K];
#pragma unroll
      for (int i = 0; i < K; ++i) xh[i] = dp[i] = 0;
#pragma unroll
      for (int i = 1; i < K; ++i) {
        const int ls = l0 - K + i;
        if (ls >= 0) xh[i] = bf16x2_f32x2(conv_ld<2>(x + ((long long)b * L + ls) * xld + c));
        else if (prev) xh[i] = bf16x2_f32x2(conv_ld<2>(prev + ((long long)b * (K - 1) + (K - 1 + ls)) * C + c));
      }
      const __nv_bfloat16* xp = x + ((long long)b * L + l0) * xld + c;
      const __nv_bfloat16* gp = dy + ((long long)b * Ly + l0) * C + c;
      __nv_bfloat16* op = dx + ((long long)b * L + l0) * dxld + c;
      // one position: its pre-activation gradient into dp[K - 1]
      auto enter = [&](uint32_t xr, uint32_t gr) {
#pragma unroll
        for (int i = 0; i + 1 < K; ++i) { xh[i] = xh[i + 1]; dp[i] = dp[i + 1]; }
        xh[K - 1] = bf16x2_f32x2(xr);
        uint64_t g = bf16x2_f32x2(gr);
        if (act) {
          uint64_t pre = bv;
#pragma unroll
          for (int k = 0; k < K; ++k) pre = fma_f32x2(xh[k], wv[k], pre);
          float p0, p1;
          unpack_f32x2(pre, p0, p1);
          g = mul_f32x2(g, pack_f32x2(silu_grad(p0), silu_grad(p1)));
        }
        dp[K - 1] = g;
      };
      auto sums = [&] {   // of the run's own positions: dw[k] += dpre[l] x[l-(K-1)+k], db += dpre[l]
        db = add_f32x2(db, dp[K - 1]);
#pragma unroll
        for (int k = 0; k < K; ++k) dw[k] = fma_f32x2(dp[K - 1], xh[k], dw[k]);
      };
      auto leave = [&] {  // dx of the position K - 1 before: sum_k w[k] dpre[l - k]
        uint64_t a = 0;
#pragma unroll
        for (int k = 0; k < K; ++k) a = fma_f32x2(wv[k], dp[K - 1 - k], a);
        float a0, a1;
        unpack_f32x2(a, a0, a1);
        *reinterpret_cast<uint32_t*>(op) = pk2(a0, a1);
        op += dxld;
      };
      int l = l0;
#pragma unroll
      for (int i = 0; i < K - 1; ++i)
        if (l < lend) {
          enter(conv_ld<2>(xp), conv_ld<2>(gp));
          sums();
          xp += xld; gp += C; ++l;
        }
      if constexpr (!FEW) {
        for (; l + 4 <= lend; l += 4) {
          uint32_t xr[4], gr[4];
#pragma unroll
          for (int u = 0; u < 4; ++u, xp += xld, gp += C) { xr[u] = conv_ld<2>(xp); gr[u] = conv_ld<2>(gp); }
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            enter(xr[u], gr[u]);
            sums();
            leave();
          }
        }
      }
      for (; l < lend; ++l, xp += xld, gp += C) {
        enter(conv_ld<2>(xp), conv_ld<2>(gp));
        sums();
        leave();
      }
      // the positions behind the run, which its last ones feed: zero gradient behind the sequence
      const int short_by = max(0, K - 1 - (lend - l0));      // a run of fewer than K - 1 positions has not left its first ones yet
#pragma unroll
      for (int i = 0; i < K - 1; ++i, ++l, xp += xld, gp += C) {
        if (l < L) enter(conv_ld<2>(xp), conv_ld<2>(gp));
        else {
#pragma unroll
          for (int k = 0; k + 1 < K; ++k) dp[k] = dp[k + 1];
          dp[K - 1] = 0;
        }
        if (i >= short_by) leave();
      }
    }
#pragma unroll
    for (int k = 0; k <= K; ++k) {
      float a0, a1;
      unpack_f32x2(k < K ? dw[k < K ? k : 0] : db, a0, a1);
      atomicAdd(&s_acc[lane][k * 2], a0);
      atomicAdd(&s_acc[lane][k * 2 + 1], a1);
    }
  }
  __syncthreads();
  // partial layout: [part][(K+1) * C]: dw as [c][k] flattened (C*K) then db (C)
  float* pp = partial + (long long)blockIdx.y * (K + 1) * C;
  for (int i = threadIdx.x; i < 32 * (K + 1) * 2; i += 256) {
    const int ln = i / ((K + 1) * 2), r = i % ((K + 1) * 2);
    const int k = r / 2, j = r % 2;
    const int cc = (blockIdx.x * 32 + ln) * 2 + j;
    if (cc >= C) continue;
    if (k < K) pp[(long long)cc * K + k] = s_acc[ln][r];
    else pp[(long long)C * K + cc] = s_acc[ln][r];
  }
}

// out must be zero: blockIdx.y owns every gridDim.y-th partial row and adds its sum with one atomic per element.
__global__ void conv1d_reduce_partials(const float* __restrict__ part, int nparts, int n, float* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float s = 0.f;
#pragma unroll 4
  for (int p = blockIdx.y; p < nparts; p += gridDim.y) s += part[(long long)p * n + i];
  atomicAdd(out + i, s);
}

}  // namespace sx
using namespace sx;

// Sequences are L rows of pitch xld in x and Ly rows of pitch C in y (and in dy below; rows from L on are not touched).
extern "C" int sx_conv1d_fwd(const void* x, const void* prev, const void* w, const void* bias, void* y, void* state_out,
                             int B, int L, int C, int K, int act, long long xld, int Ly, cudaStream_t st) {
  if (C % 8 || K > CONV_MAXK || K < 1 || xld % 8 || xld < C || Ly < L) return -1;
  if ((long long)B * L * C == 0) return 0;
  const bool few = L < CONV_SHORT;
  // With one tap a row is hardly more than its load and its store: from here on, where x and y outgrow L2, 16-byte ones are better ([8192, 7168] 40.2
  // and 43.4 us, with SiLU 43.8 and 46.4; [8192, 1792] 8.4 and 7.6).
  const bool wide = K == 1 && !few && (long long)B * L * C >= 1ll << 25 &&
                    ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(bias)) & 15) == 0;
  const int V = wide ? 8 : 4;
  // Runs of 32 read fewer rows twice, but only where they still fill the SMs twice over ([8192, 7168] 71.7 us with 16, 67.6 with 32; [4, 500, 1792]
  // 14 and 18). With one tap no row is read twice.
  const int run = K > 1 && (long long)B * ((L + 31) / 32) * (C / 4) >= 2ll * 148 * 768 ? 32 : 16;
  auto go = [&](auto kern, auto... more) {
    const long long blocks = ((long long)B * (sizeof...(more) ? (L + run - 1) / run : 1) * (C / V) + 255) / 256;
    kern<<<(int)(blocks < 148 * 1024 ? blocks : 148 * 1024), 256, 0, st>>>(
        (const __nv_bfloat16*)x, (const __nv_bfloat16*)prev, (const __nv_bfloat16*)w, (const __nv_bfloat16*)bias, (__nv_bfloat16*)y,
        (__nv_bfloat16*)state_out, B, L, C, act, xld, Ly, more...);
  };
  switch (K) {
    case 1: few ? go(conv1d_short_kernel<1>) : wide ? go(conv1d_fwd_kernel<1, 8>, run) : go(conv1d_fwd_kernel<1, 4>, run); break;
    case 2: few ? go(conv1d_short_kernel<2>) : go(conv1d_fwd_kernel<2, 4>, run); break;
    case 3: few ? go(conv1d_short_kernel<3>) : go(conv1d_fwd_kernel<3, 4>, run); break;
    default: few ? go(conv1d_short_kernel<4>) : go(conv1d_fwd_kernel<4, 4>, run); break;
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

// Positions of a run: the K - 1 positions behind it are computed twice, so long ones where the runs still fill the SMs twice over ([8192, 7168]
// 159 us, 167 with 32, 4 taps; 126 and 136, 2 taps).
static int conv_bwd_run(int B, int L, int C) { return (long long)B * ((L + 63) / 64) * ((C / 2 + 31) / 32) >= 148ll * 32 * 2 ? 64 : 16; }

// Number of partial rows the backward kernel writes for B sequences of L tokens of C channels.
extern "C" int sx_conv1d_bwd_parts(int B, int L, int C) {
  // 64 positions per warp, four runs of 16 or one of 64: the per-CTA prologue (taps, bias) and epilogue (partial row) cost about as much as 16.
  // Sequences of few positions are counted by those, longer ones by the runs of 16 that they would have (512 sequences of one position and 7168
  // channels: 27.7 us, 47 counted as runs of 64). Inputs that would leave SMs idle that way take as many CTAs as make one wave, down to one
  // run per warp ([4, 500, 1792]: 73 -> 32 us)
  const int run = conv_bwd_run(B, L, C);
  const long long chunks = (long long)B * ((L + run - 1) / run);
  const int cols = (C / 2 + 31) / 32;             // four CTAs an SM
  const long long wave = 148 * 4 / (cols > 0 ? cols : 1), most = (chunks + 7) / 8;
  long long p = ((L < CONV_FEW ? ((long long)B * L + 15) / 16 : (long long)B * ((L + 15) / 16)) + 31) / 32;
  if (p < wave) p = most < wave ? most : wave;
  if (p > most) p = most;
  return (int)(p < 1 ? 1 : (p > 512 ? 512 : p));
}

// partial: scratch of sx_conv1d_bwd_parts(B, L, C) * (K+1) * C floats; dwdb: fp32 [(K+1)*C] = dw [C][K] then db [C].
// dx: rows of pitch dxld.
extern "C" int sx_conv1d_bwd(const void* dy, const void* x, const void* prev, const void* w, const void* bias, void* dx,
                             float* partial, float* dwdb, int B, int L, int C, int K, int act, long long xld, int Ly,
                             long long dxld, cudaStream_t st) {
  if (C % 8 || K > CONV_MAXK || K < 1 || xld % 8 || xld < C || Ly < L || dxld % 4 || dxld < C) return -1;
  if ((long long)B * L == 0) return 0;
  const int parts = sx_conv1d_bwd_parts(B, L, C);
  const bool few = L < CONV_FEW;
  auto run = [&](auto kern) {
    kern<<<dim3((C / 2 + 31) / 32, parts), 256, 0, st>>>((const __nv_bfloat16*)dy, (const __nv_bfloat16*)x, (const __nv_bfloat16*)prev,
                                                         (const __nv_bfloat16*)w, (const __nv_bfloat16*)bias, (__nv_bfloat16*)dx, partial, B, L, C,
                                                         act, xld, Ly, dxld, conv_bwd_run(B, L, C));
  };
  switch (K) {
    case 1: run(conv1d_bwd_kernel<1, true>); break;
    case 2: few ? run(conv1d_bwd_kernel<2, true>) : run(conv1d_bwd_kernel<2, false>); break;
    case 3: few ? run(conv1d_bwd_kernel<3, true>) : run(conv1d_bwd_kernel<3, false>); break;
    default: few ? run(conv1d_bwd_kernel<4, true>) : run(conv1d_bwd_kernel<4, false>); break;
  }
  const int n = (K + 1) * C;
  cudaMemsetAsync(dwdb, 0, sizeof(float) * n, st);
  conv1d_reduce_partials<<<dim3((n + 255) / 256, parts < 8 ? parts : 8), 256, 0, st>>>(partial, parts, n, dwdb);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}
