// One decode step of a Mamba-2 layer: RMSNorm (+ residual) -> input projection -> convolution, recurrence and output gate of one
// token per sequence -> gated RMSNorm -> output projection.
//   S <- exp(-exp(A_log) dt) S + dt x B^T,   g = (S C + D x) silu(z),   head h reads B and C of group h / (H / G)
//
// Bound: the fp32 state, H P N values per sequence read and written once (84 MB at 16 sequences of 80 x 64 x 128: 13 us), and the two
// projections' weights (gemm_skinny.cu). One CTA per (head, sequence) keeps its P x N state in registers between the read and the
// write: a warp owns whole rows, a lane four neighbouring values of N, so rows move as 512-byte pieces and y needs one warp sum a row.
// The state is fetched before griddepcontrol.wait: no kernel between the last step's and this one writes it, so the fetch runs under the
// input projection, and so does all of the convolution but the newest token. This kernel does not signal its successor, so whatever starts early
// behind it, the next step's fetch too, starts when the states have been written. Four CTAs an SM (64 registers): with two, 1280 CTAs were
// more than four rounds of one chain of loads each (40 us a launch under a profiler, 29 now). Convolution inputs are read from one buffer and the shifted ones written to another, because the heads of a group
// share B and C and run in no order.
// Measured (B200, 8 layers of width 2560, 16 sequences, one step with embedding, head and argmax): 0.76 ms against 9.3 ms when every step
// gathered the states of its sequences, ran the chunked prompt form on one token and copied the states back (76 launches a layer).
#include "common.cuh"
#include "ragged.cuh"
#include "sx_api.h"

namespace sx {

constexpr int MS_WARPS = 8;

// NC: 128-wide pieces of a state row. The rows of a warp are walked 8 / NC at a time, their loads in flight together.
template <int NC>
__global__ void __launch_bounds__(32 * MS_WARPS, 4) mamba_step_kernel(const SxMambaStepArgs p) {
  constexpr int RB = 8 / NC;
  extern __shared__ __align__(16) float sm[];
  float* sB = sm;                 // [N] dt B
  float* sC = sB + p.N;           // [N]
  float* sx = sC + p.N;           // [P]
  float* sy = sx + p.P;           // [P]
  float* sv = sy + p.P;           // [P + 2 N] bias and older taps of the convolutions, each thread's own entries
  float* sw = sv + p.P + 2 * p.N; // [P + 2 N] newest tap
  const int h = blockIdx.x, b = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rep = p.H / p.G, g = h / rep, inner = p.H * p.P, C = inner + 2 * p.G * p.N;
  const long long* t = p.table + b * 3;
  float* st = reinterpret_cast<float*>(t[0]) + ((long long)p.layer * p.H + h) * p.P * p.N;
  float4 S[RB][NC];
  auto load = [&](int r0) {
#pragma unroll
    for (int k = 0; k < RB; ++k)
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const int r = r0 + k * MS_WARPS + warp, n = c * 128 + lane * 4;
        S[k][c] = r < p.P && n < p.N ? __ldcs(reinterpret_cast<const float4*>(st + (r * p.N + n))) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
  };
  load(0);
  const long long cs = (long long)p.layer * (p.taps - 1) * C;
  const __nv_bfloat16* old = reinterpret_cast<const __nv_bfloat16*>(t[1]) + cs;
  __nv_bfloat16* now = reinterpret_cast<__nv_bfloat16*>(t[2]) + cs;
  const __nv_bfloat16* w = reinterpret_cast<const __nv_bfloat16*>(p.conv_w);
  const __nv_bfloat16* cb = reinterpret_cast<const __nv_bfloat16*>(p.conv_b);
  const int n_ch = p.P + 2 * p.N;
  auto channel = [&](int i) {        // convolution channel of entry i: x of this head, then B and C of its group
    const int which = i < p.P ? 0 : 1 + (i - p.P) / p.N;
    return which ? inner + ((which - 1) * p.G + g) * p.N + (i - p.P) % p.N : h * p.P + i;
  };
  // the heads of a group share B and C: its first one keeps them
  auto keeps = [&](int i) { return i < p.P || h % rep == 0; };
  for (int i = tid; i < n_ch; i += 32 * MS_WARPS) {
    const int ch = channel(i);
    __nv_bfloat16 x[3], wv[4];
#pragma unroll
    for (int k = 0; k < 3; ++k)
      if (k < p.taps - 1) x[k] = old[(long long)k * C + ch];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (k < p.taps) wv[k] = w[ch * p.taps + k];
    float v = __bfloat162float(cb[ch]);
#pragma unroll
    for (int k = 0; k < 3; ++k)
      if (k < p.taps - 1) {
        v = fmaf(__bfloat162float(wv[k]), __bfloat162float(x[k]), v);
        if (k > 0 && keeps(i)) now[(long long)(k - 1) * C + ch] = x[k];   // the last step read this buffer, and it is over
      }
    sv[i] = v;
    sw[i] = __bfloat162float(p.taps == 4 ? wv[3] : p.taps == 3 ? wv[2] : wv[1]);
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const __nv_bfloat16* u = reinterpret_cast<const __nv_bfloat16*>(p.zx) + (long long)b * p.zx_ld;
  const float dt = softplus_f(__bfloat162float(u[inner + C + h]) + p.dt_bias[h]);
  const float decay = expf(-expf(p.a_log[h]) * dt);
  for (int i = tid; i < n_ch; i += 32 * MS_WARPS) {
    const int ch = channel(i);
    const __nv_bfloat16 cur = u[inner + ch];
    if (keeps(i)) now[(long long)(p.taps - 2) * C + ch] = cur;
    float v = fmaf(sw[i], __bfloat162float(cur), sv[i]);
    v *= sigmoid_f(v);
    if (i < p.P) sx[i] = v;
    else if (i < p.P + p.N) sB[i - p.P] = v * dt;
    else sC[i - p.P - p.N] = v;
  }
  __syncthreads();
  float4 Bv[NC], Cv[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const int n = c * 128 + lane * 4;
    const bool in = n < p.N;
    Bv[c] = in ? *reinterpret_cast<const float4*>(sB + n) : make_float4(0.f, 0.f, 0.f, 0.f);
    Cv[c] = in ? *reinterpret_cast<const float4*>(sC + n) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  for (int r0 = 0; r0 < p.P; r0 += RB * MS_WARPS) {
    if (r0) load(r0);
#pragma unroll
    for (int k = 0; k < RB; ++k) {
      const int r = r0 + k * MS_WARPS + warp;
      const float x = r < p.P ? sx[r] : 0.f;
      float y = 0.f;
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const int n = c * 128 + lane * 4;
        float4 v = S[k][c];
        v.x = fmaf(decay, v.x, x * Bv[c].x);
        v.y = fmaf(decay, v.y, x * Bv[c].y);
        v.z = fmaf(decay, v.z, x * Bv[c].z);
        v.w = fmaf(decay, v.w, x * Bv[c].w);
        y = fmaf(v.x, Cv[c].x, fmaf(v.y, Cv[c].y, fmaf(v.z, Cv[c].z, fmaf(v.w, Cv[c].w, y))));
        if (r < p.P && n < p.N) __stcs(reinterpret_cast<float4*>(st + (r * p.N + n)), v);
      }
      y = warp_sum(y);
      if (lane == 0 && r < p.P) sy[r] = fmaf(p.D[h], x, y);
    }
  }
  __syncthreads();
  __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(p.g) + (long long)b * inner + h * p.P;
  for (int i = tid; i < p.P; i += 32 * MS_WARPS) {
    const float z = __bfloat162float(u[h * p.P + i]);
    out[i] = __float2bfloat16_rn(sy[i] * z * sigmoid_f(z));
  }
}

}  // namespace sx
using namespace sx;

static int mamba_gemm(const void* x, const void* w, void* y, int M, int N, int K, int* status, cudaStream_t st) {
  SxGemmArgs a = {};
  a.A = x; a.B = w; a.D = y;
  a.M = M; a.N = N; a.K = K; a.batch = 1;
  a.lda = K; a.ldb = K; a.ldd = N;
  a.alpha = 1.f;
  a.status = status;
  a.flags = 1;      // see sx_mamba2_step
  return sx_gemm_bf16(&a, st);
}

// Five launches. The sizes are those that the front-end has checked (serving/mamba_states.py). The weights of both projections are declared static, and
// the norm in front lets their first loads pass it: no kernel in front of the call may write them, unless one that is launched ordinarily lies between
// (the lookup of the tokens in a decode step).
extern "C" int sx_mamba2_step(const SxMambaStepArgs* a, cudaStream_t st) {
  if (a->B <= 0) return 0;
  if (a->B > 65535 || a->H <= 0 || a->G <= 0 || a->H % a->G || a->P <= 0 || a->N <= 0 || a->N % 4 || a->N > 256 || a->taps < 2 || a->taps > 4 || a->d % 8)
    return -1;
  const int inner = a->H * a->P;
  const int smem = (6 * a->N + 4 * a->P) * 4;   // the operands, y, and the convolutions' two arrays of P + 2 N
  if (smem > 48 * 1024 || a->zx_ld != 2 * inner + 2 * a->G * a->N + a->H || inner % 8) return -2;
  int rc = sx_rmsnorm_fwd(a->x, a->res_in, a->norm_w, a->hn, a->res_out, nullptr, a->B, a->d, a->eps, st);
  if (rc) return rc;
  rc = mamba_gemm(a->hn, a->in_w, a->zx, a->B, (int)a->zx_ld, a->d, a->status, st);
  if (rc) return rc;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(a->H, a->B, 1);
  cfg.blockDim = dim3(32 * MS_WARPS, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if ((a->N <= 128 ? cudaLaunchKernelEx(&cfg, mamba_step_kernel<1>, *a) : cudaLaunchKernelEx(&cfg, mamba_step_kernel<2>, *a)) != cudaSuccess)
    return -11;
  rc = sx_rmsnorm_fwd(a->g, nullptr, a->gate_norm_w, a->gn, nullptr, nullptr, a->B, inner, a->gate_eps, st);
  if (rc) return rc;
  return mamba_gemm(a->gn, a->out_w, a->out, a->B, a->d, inner, a->status, st);
}
