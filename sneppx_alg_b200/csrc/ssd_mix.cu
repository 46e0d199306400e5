// Small stages of the Mamba-2 mixer's training pass around the chunked scan (ssd.cu, ssd_fwd.cu): step sizes and decays of a chunk, their
// gradients, layouts of B and C, the sum of the score gradients over the heads of a group.
// Each replaces a chain of elementwise, scan and copy launches over [tokens, heads] (22 forward and backward); they are bound by launch
// latency and by reading each array once. Rows r = (bc, q): chunk bc = b * nc + c of Q tokens, tokens from L on are padding (dt = 0).
#include "common.cuh"
#include "ragged.cuh"
#include "sx_api.h"

namespace sx {

constexpr int MX_H = 8;      // heads of a CTA, one warp each: a token's 8 values are one 32-byte sector

__device__ __forceinline__ float warp_scan(float v, int lane) {      // inclusive
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += t;
  }
  return v;
}

// dt = softplus(raw + bias), cs = running sum of -exp(A_log) dt along the chunk. Heads-first dth, csh [BC, H, Q]; token-major
// E = exp(cs), decay = exp(cs_last - cs) dt [BC, Q, H]; tot = exp(cs_last) [BC, H].
__global__ void __launch_bounds__(256) mix_prep_kernel(const __nv_bfloat16* __restrict__ raw, long long ld, const float* __restrict__ bias,
                                                       const float* __restrict__ a_log, float* __restrict__ dth, float* __restrict__ csh,
                                                       float* __restrict__ E, float* __restrict__ decay, float* __restrict__ tot, int nc,
                                                       int L, int H, int Q) {
  __shared__ float s_dt[256][MX_H + 1], s_cs[256][MX_H + 1];
  const int bc = blockIdx.x, h0 = blockIdx.y * MX_H, b = bc / nc, l0 = (bc % nc) * Q, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = threadIdx.x; i < Q * MX_H; i += 256) {
    const int q = i / MX_H, h = h0 + i % MX_H;
    s_dt[q][i % MX_H] = h < H && l0 + q < L ? softplus_f(__bfloat162float(raw[((long long)b * L + l0 + q) * ld + h]) + bias[h]) : 0.f;
  }
  __syncthreads();
  const int h = h0 + warp;
  if (h < H) {
    const float A = -expf(a_log[h]);
    const long long o = ((long long)bc * H + h) * Q;
    float carry = 0.f;
    for (int q0 = 0; q0 < Q; q0 += 32) {
      const int q = q0 + lane;
      const float dt = q < Q ? s_dt[q][warp] : 0.f;
      const float cs = carry + warp_scan(A * dt, lane);
      carry = __shfl_sync(0xffffffffu, cs, 31);
      if (q < Q) {
        s_cs[q][warp] = cs;
        dth[o + q] = dt;
        csh[o + q] = cs;
      }
    }
    if (lane == 0) tot[(long long)bc * H + h] = expf(carry);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < Q * MX_H; i += 256) {
    const int q = i / MX_H, j = i % MX_H;
    if (h0 + j >= H) continue;
    const long long o = ((long long)bc * Q + q) * H + h0 + j;
    const float cs = s_cs[q][j];
    E[o] = expf(cs);
    decay[o] = expf(s_cs[Q - 1][j] - cs) * s_dt[q][j];
  }
}

// Gradients of the above. From ddecay, dcs (through exp(cs) of the read-out) and ddrow = <dy, x>, token-major [BC, Q, H]; rowW, colU
// (through the score matrix, colU without the factor dt), heads-first; dtot [BC, H]:
//   d cs_q = dcs - ddecay decay + rowW - colU dt,  d cs_last += dtot tot + sum_q ddecay decay,  da_q = sum of d cs from q on,
//   d dt = ddecay exp(cs_last - cs) + colU + A da,  d raw = d dt sigmoid(raw + bias)
// part [3, BC, H]: dA_log (da dt summed, times A), dD (ddrow summed), dbias (d raw summed) of the chunk.
__global__ void __launch_bounds__(256) mix_finish_kernel(const __nv_bfloat16* __restrict__ raw, long long ld, const float* __restrict__ bias,
                                                         const float* __restrict__ a_log, const float* __restrict__ dth,
                                                         const float* __restrict__ csh, const float* __restrict__ ddecay,
                                                         const float* __restrict__ dcs, const float* __restrict__ ddrow,
                                                         const float* __restrict__ rowW, const float* __restrict__ colU,
                                                         const float* __restrict__ dtot, const float* __restrict__ tot,
                                                         __nv_bfloat16* __restrict__ draw, long long dld, float* __restrict__ part, int BC,
                                                         int nc, int L, int H, int Q) {
  __shared__ float s_dd[256][MX_H + 1], s_dc[256][MX_H + 1], s_out[256][MX_H + 1];
  const int bc = blockIdx.x, h0 = blockIdx.y * MX_H, b = bc / nc, l0 = (bc % nc) * Q, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = threadIdx.x; i < Q * MX_H; i += 256) {
    const int q = i / MX_H, j = i % MX_H, h = h0 + j;
    if (h >= H) continue;
    const long long o = ((long long)bc * Q + q) * H + h;
    s_dd[q][j] = ddecay[o];
    s_dc[q][j] = dcs[o];
    s_out[q][j] = ddrow[o];
  }
  __syncthreads();
  const int h = h0 + warp;
  if (h < H) {
    const float A = -expf(a_log[h]), bi = bias[h];
    const long long o = ((long long)bc * H + h) * Q, bh = (long long)bc * H + h;
    const float last = csh[o + Q - 1];
    float gsum = 0.f, dd = 0.f;
    for (int q = lane; q < Q; q += 32) {
      gsum += s_dd[q][warp] * expf(last - csh[o + q]) * dth[o + q];
      dd += s_out[q][warp];
    }
    gsum = warp_sum(gsum);
    dd = warp_sum(dd);
    __syncwarp();
    const float dlast = dtot[bh] * tot[bh] + gsum;
    float carry = 0.f, dA = 0.f, db = 0.f;          // carry: d cs of the tokens behind this group of 32
    for (int q0 = (Q - 1) / 32 * 32; q0 >= 0; q0 -= 32) {
      const int q = q0 + 31 - lane;                 // lanes walk backwards, so the inclusive scan sums from q on
      const bool in = q < Q;
      float dt = 0.f, eL = 0.f, cu = 0.f, v = 0.f, de = 0.f;
      if (in) {
        dt = dth[o + q];
        eL = expf(last - csh[o + q]);
        cu = colU[o + q];
        de = s_dd[q][warp];
        v = s_dc[q][warp] - de * eL * dt + rowW[o + q] - cu * dt + (q == Q - 1 ? dlast : 0.f);
      }
      const float da = carry + warp_scan(v, lane);
      carry = __shfl_sync(0xffffffffu, da, 31);
      if (in) {
        dA = fmaf(da, dt, dA);
        float g = 0.f;
        if (l0 + q < L) {
          const float x = __bfloat162float(raw[((long long)b * L + l0 + q) * ld + h]) + bi;
          g = (de * eL + cu + A * da) * sigmoid_f(x);
          db += g;
        }
        s_out[q][warp] = g;                         // this warp alone reads and writes column `warp`
      }
    }
    dA = warp_sum(dA);
    db = warp_sum(db);
    if (lane == 0) {
      part[bh] = dA * A;
      part[(long long)BC * H + bh] = dd;
      part[2ll * BC * H + bh] = db;
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < Q * MX_H; i += 256) {
    const int q = i / MX_H, j = i % MX_H;
    if (h0 + j < H && l0 + q < L) draw[((long long)b * L + l0 + q) * dld + h0 + j] = __float2bfloat16_rn(s_out[q][j]);
  }
}

// Rows of B and C ([tokens, G N] each, pitch ld, C behind B) -> [2][BC, G, Q, N].
__global__ void __launch_bounds__(256) mix_pack_kernel(const __nv_bfloat16* __restrict__ in, long long ld, __nv_bfloat16* __restrict__ out,
                                                       long long rows, int G, int Q, int N) {
  const int nv = N >> 3, per = 2 * G * nv;
  const long long total = rows * per;
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < total; i += gridDim.x * 256ll) {
    const long long r = i / per;
    const int j = (int)(i - r * per), which = j / (G * nv), g = j / nv % G, e = j % nv;
    const long long o = (((which * (rows / Q) + r / Q) * G + g) * Q + r % Q) * nv + e;
    st8(out + o * 8, ld8(in + r * ld + j * 8));
  }
}
// The reverse for fp32 gradients: dB, dC [BC, G, Q, N] -> bf16 rows.
__global__ void __launch_bounds__(256) mix_unpack_kernel(const float* __restrict__ dB, const float* __restrict__ dC,
                                                         __nv_bfloat16* __restrict__ out, long long ld, long long rows, int G, int Q, int N) {
  const int nv = N >> 3, per = 2 * G * nv;
  const long long total = rows * per;
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < total; i += gridDim.x * 256ll) {
    const long long r = i / per;
    const int j = (int)(i - r * per), which = j / (G * nv), g = j / nv % G, e = j % nv;
    const float4* p = reinterpret_cast<const float4*>((which ? dC : dB) + ((((r / Q) * G + g) * Q + r % Q) * nv + e) * 8);
    const float4 a = p[0], b = p[1];
    const float f[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    st8(out + r * ld + j * 8, pack8(f));
  }
}
// out [n, M] = sum over rep of in [n, rep, M]
__global__ void __launch_bounds__(256) mix_sum_kernel(const __nv_bfloat16* __restrict__ in, __nv_bfloat16* __restrict__ out, long long n, int rep,
                                                      int mv) {
  const long long total = n * mv;
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < total; i += gridDim.x * 256ll) {
    const __nv_bfloat16* p = in + ((i / mv) * rep * mv + i % mv) * 8;
    float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (int k = 0; k < rep; ++k) {
      float f[8];
      unpack8(ld8(p + (long long)k * mv * 8), f);
#pragma unroll
      for (int j = 0; j < 8; ++j) s[j] += f[j];
    }
    st8(out + i * 8, pack8(s));
  }
}

}  // namespace sx
using namespace sx;

static unsigned mix_grid(long long total) {
  const long long nb = (total + 255) / 256;
  return (unsigned)(nb < 148 * 16 ? nb : 148 * 16);
}

extern "C" int sx_mix_prep(const void* raw, long long ld, const float* bias, const float* a_log, float* dth, float* csh, float* E,
                           float* decay, float* tot, int B, int nc, int L, int H, int Q, cudaStream_t st) {
  if (Q < 1 || Q > 256) return -1;
  if ((long long)B * nc * H == 0) return 0;
  mix_prep_kernel<<<dim3(B * nc, (H + MX_H - 1) / MX_H), 256, 0, st>>>((const __nv_bfloat16*)raw, ld, bias, a_log, dth, csh, E, decay, tot, nc, L,
                                                                       H, Q);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

extern "C" int sx_mix_finish(const void* raw, long long ld, const float* bias, const float* a_log, const float* dth, const float* csh,
                             const float* ddecay, const float* dcs, const float* ddrow, const float* rowW, const float* colU,
                             const float* dtot, const float* tot, void* draw, long long dld, float* part, int B, int nc, int L, int H, int Q,
                             cudaStream_t st) {
  if (Q < 1 || Q > 256) return -1;
  if ((long long)B * nc * H == 0) return 0;
  mix_finish_kernel<<<dim3(B * nc, (H + MX_H - 1) / MX_H), 256, 0, st>>>((const __nv_bfloat16*)raw, ld, bias, a_log, dth, csh, ddecay, dcs, ddrow,
                                                                         rowW, colU, dtot, tot, (__nv_bfloat16*)draw, dld, part, B * nc, nc, L,
                                                                         H, Q);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

extern "C" int sx_mix_pack(const void* in, long long ld, void* out, long long rows, int G, int Q, int N, cudaStream_t st) {
  if (N % 8 || ld % 8 || rows % Q) return -1;
  if (rows == 0) return 0;
  mix_pack_kernel<<<mix_grid(rows * 2 * G * (N / 8)), 256, 0, st>>>((const __nv_bfloat16*)in, ld, (__nv_bfloat16*)out, rows, G, Q, N);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

extern "C" int sx_mix_unpack(const float* dB, const float* dC, void* out, long long ld, long long rows, int G, int Q, int N, cudaStream_t st) {
  if (N % 8 || ld % 8 || rows % Q) return -1;
  if (rows == 0) return 0;
  mix_unpack_kernel<<<mix_grid(rows * 2 * G * (N / 8)), 256, 0, st>>>(dB, dC, (__nv_bfloat16*)out, ld, rows, G, Q, N);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

extern "C" int sx_mix_sum(const void* in, void* out, long long n, int rep, int M, cudaStream_t st) {
  if (M % 8) return -1;
  if (n == 0) return 0;
  mix_sum_kernel<<<mix_grid(n * (M / 8)), 256, 0, st>>>((const __nv_bfloat16*)in, (__nv_bfloat16*)out, n, rep, M / 8);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}
