// Q2: dequant-GEMM on tcgen05. Y[M, N] = X[M, K] (bf16) x dequant(W)[N, K]^T with W stored as
//   fp8 e4m3 + fp32 scales per 128 x 128 block, or INT4 (two per byte, offset 8) + fp32 scales per (row, 128 columns).
//
// Bound: reading the packed weights once (decode: a few rows of X against the whole matrix). The operands are swapped so that
// 128 weight rows are the MMA's M (TMEM lanes) and BT = 16 / 32 / 64 / 128 rows of X its N, and the reduction is split over the
// CTAs of a cluster, which add their fp32 tiles through distributed shared memory in a fixed order (as gemm_skinny.cu does):
//   TMA        brings 128 rows x 128 bytes of packed weights and the matching columns of X into a ring of stages
//   converters NG groups of four warps, one 128-wide k-block each in turn: a thread reads its row's bytes (swizzled tile, no
//              bank conflicts), turns them into bf16 VALUES WITHOUT SCALE - exact for both formats - and stores them in TMEM, which
//              is where the MMA reads its A operand: the expanded weights never touch shared memory. A group is one chain of
//              dependent instructions (about 1 us a k-block), so several are in flight
//   MMA        eight K = 16 steps per k-block into one of two accumulators, each with an issuing warp of its own: k-blocks do not
//              accumulate into one another, and one thread's waits, issue and commits were the limit
//   promotion  acc[row][m] += scale[row, k-block] * partial in fp32 registers; the scale belongs to the thread's own row (TMEM lane),
//              so it is one multiply-add per value. Products are therefore exact and nothing is rounded to bf16 before the output.
// Two CTAs share an SM up to 32 rows of X, so that one converts while the other waits.
// Measured (B200, graph replay, cold weights), int4 [28672, 4096] at 1 / 16 / 32 / 64 / 128 rows: 24 / 24 / 27 / 33 / 51 us, [4096, 14336]
// 15 / 15 / 16 / 16 / 23 us; 28 / 28 / 30 / 39 / 62 and 16 / 17 / 17 / 19 / 28 us when MMAs were issued behind `lane == 0`
// (tc_common.cuh), 203 / 199 / 199 / 199 / 201 and 361 / 354 / 353 / 353 / 356 us when 128 x 128 output tiles left most SMs idle and four
// converter warps wrote scaled bf16 tiles to shared memory. The floor (packed weights at copy bandwidth) is 9 and 4.5 us. K of 128 or 256 with
// more than one wave of tiles: gemm_dq_short.cu.
// The reference has quantise / dequantise kernels only (kernel/quantization/quantize_cuda.cu), no GEMM on them.
#include "dq_convert.cuh"
#include "tc_common.cuh"
#include "tmap.h"
#include "sx_api.h"

namespace sx {

constexpr int DQ_BM = 128;         // weight rows per tile
constexpr int DQ_BK = 128;         // elements of K per k-block: one scale group
constexpr int DQ_W_BYTES = DQ_BM * 128;   // packed weights of a stage: one k-block (fp8) or two (int4)
constexpr int DQ_MAX_STAGES = 6;

struct DqParams {
  CUtensorMap tmW, tmX;
  const float* scales;    // fp8: [ceil(N/128), K/128]; int4: [N, K/128]
  const float* bias;
  __nv_bfloat16* D;
  long long ldd;
  int M, N, K, stages, early_weights;
  int* status;
};

// BT rows of X per tile. Warps: PW promotion / epilogue, 4 NG converters, 2 MMA, 1 TMA.
// Times below: cold, with the launch. PW: a promotion thread holds BT sums with four warps, and from 64 on they do not fit its registers beside the rest (120 bytes spilled at 64 rows,
// int4 [28672, 4096] 57 us; 48 with eight); at 32 rows eight warps leave 48 registers for two CTAs an SM (43 us, 39 with four).
// NG: four converter groups where one CTA an SM leaves room for them, 48 us at 64 rows, 53 with two; at 128 rows they leave 72 registers for
// promotion threads of 64 sums (184 bytes spilled, 79 us; 72 with two).
template <int BT>
struct DqCfg {
  static constexpr int PW = BT >= 64 ? 8 : 4;           // from 64 columns on two warps per lane quadrant, half of the columns each
  static constexpr int COLS = BT / (PW / 4);            // columns of a promotion thread
  static constexpr int NG = BT == 64 ? 4 : 2;           // converter groups
  // A buffers, k-block i in buffer i % NA: an even number, so that a buffer and its barriers belong to one group and one MMA warp (a phase's parity
  // says nothing to a warp that missed the phase before). Two for each group at 128 rows, whose converters otherwise wait for the MMA of their
  // last k-block: 58 -> 51 us. Up to 32 rows TMEM has room for three in two CTAs; with barriers for each group that gained nothing (24 us).
  static constexpr int NA = BT >= 64 ? 4 : 2;
  static_assert(NA % NG == 0, "a buffer belongs to one group");
  static constexpr int MMA_WARP = PW + 4 * NG;          // two MMA warps, then the TMA warp
  static constexpr int THREADS = 32 * (MMA_WARP + 3);
  static constexpr int CTAS = BT <= 32 ? 2 : 1;         // resident per SM
  static constexpr int X_BYTES = BT * DQ_BK * 2;        // X of one k-block: two 64-column slabs
  static constexpr int TM_D = NA * 64;                  // TMEM: A buffers of 64 columns, then two accumulators
  static constexpr int TMEM_COLS = TM_D + 2 * BT <= 256 ? 256 : 512;
  static_assert(CTAS * TMEM_COLS <= 512 && TM_D + 2 * BT <= TMEM_COLS, "TMEM");
  static constexpr int BUDGET = CTAS == 2 ? 98304 : 196608;
};

__device__ __forceinline__ void dq_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 dq_ld_peer(uint32_t local_addr, uint32_t rank) {
  uint32_t ra;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(local_addr), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(ra)
               : "memory");
  return v;
}

template <int BT, bool INT4>
__global__ void __launch_bounds__(DqCfg<BT>::THREADS, DqCfg<BT>::CTAS) gemm_dq_kernel(const __grid_constant__ DqParams p) {
  using Cfg = DqCfg<BT>;
  constexpr int KPS = INT4 ? 2 : 1;                                   // k-blocks per stage
  constexpr int STAGE_BYTES = DQ_W_BYTES + KPS * Cfg::X_BYTES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  float* sP = reinterpret_cast<float*>(smem);                         // [BT][128] fp32 partial tile, over the drained stages
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + p.stages * STAGE_BYTES);
  uint64_t* full = bars;
  uint64_t* empty = bars + DQ_MAX_STAGES;                             // four converter warps and one MMA warp a k-block
  uint64_t* a_full = bars + 2 * DQ_MAX_STAGES;                        // [NA] four converter warps
  uint64_t* a_empty = a_full + Cfg::NA;                               // [NA] MMA
  uint64_t* d_full = a_empty + Cfg::NA;                               // [2] MMA
  uint64_t* d_empty = d_full + 2;                                     // [2] promotion warps
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(d_empty + 2);
  volatile int* s_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = warp_index(), lane = threadIdx.x & 31;
  uint32_t S, r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(S));
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  const int n0 = (blockIdx.x / S) * DQ_BM, m0 = blockIdx.y * BT;
  const int kblks = p.K / DQ_BK, st_total = (kblks + KPS - 1) / KPS;
  const int per = (st_total + (int)S - 1) / (int)S;
  const int st0 = (int)r * per, st1 = min(st_total, st0 + per);
  const int nst = max(st1 - st0, 0);                                  // stages of this CTA
  const int kb0 = st0 * KPS, nk = nst > 0 ? min(kblks, st1 * KPS) - kb0 : 0;   // k-blocks of this CTA

  if (threadIdx.x == 0) {
    for (int i = 0; i < p.stages; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 5 * KPS);
    }
    for (int i = 0; i < Cfg::NA; ++i) {
      mbar_init(&a_full[i], 4);
      mbar_init(&a_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&d_full[i], 1);
      mbar_init(&d_empty[i], Cfg::PW);
    }
    *s_abort = 0;
    mbar_fence_init();
    tma_prefetch_desc(&p.tmW);
    tma_prefetch_desc(&p.tmX);
  }
  if (warp == Cfg::MMA_WARP) tmem_alloc(tmem_slot, Cfg::TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == Cfg::MMA_WARP + 2) {
    // ------------------------------------------------------------ TMA
    if (elect_one()) {
      auto load_w = [&](int i, int s) {
        mbar_expect_tx(&full[s], STAGE_BYTES);
        tma_load_2d(smem + s * STAGE_BYTES, &p.tmW, &full[s], (st0 + i) * 128, n0);
      };
      auto load_x = [&](int i, int s) {
        // an odd last int4 k-block: the second half of the stage lies past K and arrives as zeros
#pragma unroll
        for (int c = 0; c < 2 * KPS; ++c)
          tma_load_2d(smem + s * STAGE_BYTES + DQ_W_BYTES + c * (Cfg::X_BYTES / 2), &p.tmX, &full[s],
                      (st0 + i) * KPS * DQ_BK + c * 64, m0);
      };
      const int pre = p.early_weights ? min(nst, p.stages) : 0;
      for (int i = 0; i < pre; ++i) load_w(i, i);
      asm volatile("griddepcontrol.wait;" ::: "memory");
      for (int i = 0; i < pre; ++i) load_x(i, i);
      for (int i = pre; i < nst; ++i) {
        const int s = i % p.stages;
        if (!mbar_wait(&empty[s], ((i / p.stages) & 1) ^ 1, s_abort, p.status, ST_TIMEOUT_PRODUCER)) break;
        load_w(i, s);
        load_x(i, s);
      }
    }
  } else if (warp >= Cfg::MMA_WARP) {
    // ------------------------------------------------------------ MMA: this warp's k-blocks i = buf, buf + 2, ...
    if (elect_one()) {
      constexpr uint32_t idesc = umma_idesc_f16(DQ_BM, BT, 1, 0, 0);
      const int buf = warp - Cfg::MMA_WARP;
      const uint32_t tD = tmem_base + Cfg::TM_D + buf * BT;
      const uint32_t sm0 = smem_u32(smem);
      int s = INT4 ? 0 : buf;                                          // stage and its phase, followed without a division
      uint32_t sph = 0, dph = 1, aph = 0;
      int g = buf;                                                     // A buffer and its phase
      for (int i = buf; i < nk; i += 2) {
        if (g >= Cfg::NA) { g -= Cfg::NA; aph ^= 1; }
        if (s >= p.stages) { s -= p.stages; sph ^= 1; }
        // a_full follows full of the stage (the converters read it), but the X tile arrived through the async proxy: wait for it here too
        if (!mbar_wait(&full[s], sph, s_abort, p.status, ST_TIMEOUT_MMA)) break;
        if (!mbar_wait(&d_empty[buf], dph, s_abort, p.status, ST_TIMEOUT_MMA)) break;
        const uint64_t x0 = umma_desc_sw128(sm0 + s * STAGE_BYTES + DQ_W_BYTES + (INT4 ? buf : 0) * Cfg::X_BYTES, 16, 1024);
        if (!mbar_wait(&a_full[g], aph, s_abort, p.status, ST_TIMEOUT_MMA)) break;
        tc_fence_after();
#pragma unroll
        for (int k = 0; k < 8; ++k)
          umma_f16_ts(tD, tmem_base + g * 64 + k * 8, x0 + ((k >> 2) * (Cfg::X_BYTES / 2) + (k & 3) * 32) / 16, idesc, k ? 1u : 0u);
        umma_commit(&d_full[buf]);
        umma_commit(&a_empty[g]);
        umma_commit(&empty[s]);
        s += INT4 ? 1 : 2;
        g += 2;
        dph ^= 1;
      }
    }
  } else if (warp >= Cfg::PW) {
    // ------------------------------------------------------------ converters: group g takes the k-blocks i with i % NG == g
    const int g = (warp - Cfg::PW) >> 2, q = warp & 3;                // q: TMEM lane quadrant of this warp (PW is a multiple of 4)
    const int row = q * 32 + lane;
    int s = g / KPS, ab = g;
    uint32_t sph = 0, aph = 1;
    for (int i = g; i < nk; i += Cfg::NG, s += Cfg::NG / KPS, ab += Cfg::NG) {
      if (ab >= Cfg::NA) { ab -= Cfg::NA; aph ^= 1; }
      const uint32_t tA = tmem_base + ab * 64 + (static_cast<uint32_t>(q * 32) << 16);
      while (s >= p.stages) { s -= p.stages; sph ^= 1; }
      if (!mbar_wait_warp(&full[s], sph, s_abort, p.status, ST_TIMEOUT_CONVERT)) break;
      const uint8_t* src = smem + s * STAGE_BYTES + row * 128;
      bool ok = true;
#pragma unroll
      for (int h = 0; h < (INT4 ? 1 : 2); ++h) {                      // 64 bytes of the row at a time
        uint4 w[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const int ch = (INT4 ? (i & 1) : h) * 4 + c;
          w[c] = *reinterpret_cast<const uint4*>(src + ((ch ^ (row & 7)) << 4));
        }
        if (h == (INT4 ? 0 : 1)) {                                    // the row is in registers: the stage may be refilled
          __syncwarp();
          if (lane == 0) mbar_arrive(&empty[s]);
        }
        if (h == 0) {
          ok = mbar_wait_warp(&a_empty[ab], aph, s_abort, p.status, ST_TIMEOUT_CONVERT);
          if (!ok) break;
          tc_fence_after();
        }
        uint32_t o[16];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          if constexpr (INT4) {
            int4x8_to_bf16(w[c].x, o);
            int4x8_to_bf16(w[c].y, o + 4);
            int4x8_to_bf16(w[c].z, o + 8);
            int4x8_to_bf16(w[c].w, o + 12);
            tmem_st16(tA + c * 16, o);
          } else {
            e4m3x4_to_bf16(w[c].x, o + (c & 1) * 8);
            e4m3x4_to_bf16(w[c].y, o + (c & 1) * 8 + 2);
            e4m3x4_to_bf16(w[c].z, o + (c & 1) * 8 + 4);
            e4m3x4_to_bf16(w[c].w, o + (c & 1) * 8 + 6);
            if (c & 1) tmem_st16(tA + h * 32 + (c >> 1) * 16, o);
          }
        }
      }
      if (!ok) break;
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&a_full[ab]);
    }
  } else {
    // ------------------------------------------------------------ promotion: thread = weight row (TMEM lane)
    const int q = warp & 3, row = q * 32 + lane, c0 = (warp >> 2) * Cfg::COLS;
    const uint32_t tD = tmem_base + Cfg::TM_D + (static_cast<uint32_t>(q * 32) << 16) + c0;
    const float* sc = p.scales + (INT4 ? (long long)min(n0 + row, p.N - 1) * kblks : (long long)(n0 / 128) * kblks) + kb0;
    float acc[Cfg::COLS];
#pragma unroll
    for (int j = 0; j < Cfg::COLS; ++j) acc[j] = 0.f;
    if (!p.early_weights) asm volatile("griddepcontrol.wait;" ::: "memory");   // the scales may come from the kernel before this one
    float next = nk > 0 ? sc[0] : 0.f;
    for (int i = 0; i < nk; ++i) {
      const int buf = i & 1;
      const float scale = next;
      if (i + 1 < nk) next = sc[i + 1];
      if (!mbar_wait_warp(&d_full[buf], (i >> 1) & 1, s_abort, p.status, ST_TIMEOUT_EPILOGUE)) break;
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < Cfg::COLS; c += 16) {
        uint32_t v[16];
        tmem_ld16(tD + buf * BT + c, v);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j) acc[c + j] = fmaf(scale, __uint_as_float(v[j]), acc[c + j]);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&d_empty[buf]);
    }
    // every stage has been consumed by an MMA whose result was read above: the ring is free
#pragma unroll
    for (int j = 0; j < Cfg::COLS; ++j) sP[(c0 + j) * DQ_BM + row] = acc[j];
    if (S == 1) asm volatile("bar.sync 1, %0;" ::"n"(32 * Cfg::PW) : "memory");
  }

  // every thread of every CTA takes part in both cluster barriers, whatever happened above
  if (S > 1) dq_cluster_sync();
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (warp < Cfg::PW) {
    asm volatile("griddepcontrol.wait;" ::: "memory");   // stores come after the kernel before this one
    const int c4 = lane * 4, n = n0 + c4;
    const bool vec = n + 3 < p.N && (p.ldd & 3) == 0 && (reinterpret_cast<uintptr_t>(p.D) & 7) == 0;
    float bias[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) bias[j] = p.bias && n + j < p.N ? p.bias[n + j] : 0.f;
    // CTA r writes the rows r, r + S, ... of the tile, one warp per row
    for (int m = (int)r + warp * (int)S; m < min(BT, p.M - m0); m += Cfg::PW * (int)S) {
      const uint32_t a = smem_u32(&sP[m * DQ_BM + c4]);
      float4 t[8];
#pragma unroll
      for (int s = 0; s < 8; ++s)
        if (s < (int)S) t[s] = S > 1 ? dq_ld_peer(a, (uint32_t)s) : *reinterpret_cast<const float4*>(&sP[m * DQ_BM + c4]);
      float4 v = t[0];
#pragma unroll
      for (int s = 1; s < 8; ++s)
        if (s < (int)S) { v.x += t[s].x; v.y += t[s].y; v.z += t[s].z; v.w += t[s].w; }
      v.x += bias[0]; v.y += bias[1]; v.z += bias[2]; v.w += bias[3];
      __nv_bfloat16* d = p.D + (long long)(m0 + m) * p.ldd + n;
      if (vec) {
        *reinterpret_cast<uint2*>(d) = make_uint2(pack_bf16x2(v.x, v.y), pack_bf16x2(v.z, v.w));
      } else {
        const float o[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (n + j < p.N) d[j] = __float2bfloat16(o[j]);
      }
    }
  }
  if (S > 1) dq_cluster_sync();

  tc_fence_before();
  __syncthreads();
  if (*s_abort) bounded_delay_ns(2000000);
  if (warp == Cfg::MMA_WARP) {
    tc_fence_after();
    tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
  }
}

// K of 128 or 256 and more tiles than one wave (gemm_dq_short.cu)
bool gemm_dq_short_ok(int M, int N, int K, int sms);
int gemm_dq_short(const void* X, long long ldx, const void* W, const float* scales, const float* bias, void* D, long long ldd, int M, int N, int K,
                  int mode, int sms, int* status, cudaStream_t st);

// CTAs of a cluster = slices of K: the fewest that fill the resident slots in as few waves as possible. A CTA costs its stages plus
// a fixed part (set-up and reduction) worth about six of them, as in the bf16 decode kernel.
static int dq_splits(int tiles, int stages, int slots) {
  int best = 1;
  long long best_cost = -1;
  for (int s = 1; s <= 8; s *= 2) {
    const int per = (stages + s - 1) / s;
    if (s > 1 && per < 2) break;
    const long long cost = (long long)(((long long)tiles * s + slots - 1) / slots) * (per + 6);
    if (best_cost < 0 || cost < best_cost) { best_cost = cost; best = s; }
  }
  return best;
}

template <int BT, bool INT4>
static int dq_launch(DqParams& p, int sms, cudaStream_t st) {
  using Cfg = DqCfg<BT>;
  constexpr int STAGE_BYTES = DQ_W_BYTES + (INT4 ? 2 : 1) * Cfg::X_BYTES;
  p.stages = Cfg::BUDGET / STAGE_BYTES < DQ_MAX_STAGES ? Cfg::BUDGET / STAGE_BYTES : DQ_MAX_STAGES;
  static_assert(Cfg::BUDGET / STAGE_BYTES >= 2, "at least two stages");
  static_assert(2 * STAGE_BYTES >= BT * DQ_BM * 4, "the partial tile lies over the stages");
  const int smem = p.stages * STAGE_BYTES + 1024 + 256;
  static int set = 0;
  if (set < smem) {
    if (cudaFuncSetAttribute(gemm_dq_kernel<BT, INT4>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return -10;
    set = smem;
  }
  const int tiles = (p.N + DQ_BM - 1) / DQ_BM, mt = (p.M + BT - 1) / BT;
  const int kblks = p.K / DQ_BK;
  const int S = dq_splits(tiles * mt, INT4 ? (kblks + 1) / 2 : kblks, Cfg::CTAS * sms);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(tiles * S, mt, 1);
  cfg.blockDim = dim3(Cfg::THREADS, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = S;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, gemm_dq_kernel<BT, INT4>, p) == cudaSuccess ? 0 : -11;
}

}  // namespace sx
using namespace sx;

// X: bf16 [M, K] (ldx); W packed (mode 0: fp8 e4m3 [N, K], mode 1: int4 [N, K/2]); D: bf16 [M, N] (ldd).
// static_weights: no kernel before this one on the stream writes W, so its first tiles may be fetched before that kernel ends.
extern "C" int sx_gemm_dequant(const void* X, long long ldx, const void* W, const float* scales, const float* bias,
                               void* D, long long ldd, int M, int N, int K, int mode, int static_weights, int* status,
                               cudaStream_t st) {
  if (K % 128 || ldx % 8 || (reinterpret_cast<uintptr_t>(X) & 15) || (reinterpret_cast<uintptr_t>(W) & 15)) return -1;
  if (M <= 0 || N <= 0) return 0;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (gemm_dq_short_ok(M, N, K, sms)) return gemm_dq_short(X, ldx, W, scales, bias, D, ldd, M, N, K, mode, sms, status, st);
  constexpr int MOST = 65535 * 128;      // rows of a launch: tiles of them are the grid's y
  for (; M > MOST; M -= MOST) {
    const int rc = sx_gemm_dequant(X, ldx, W, scales, bias, D, ldd, MOST, N, K, mode, static_weights, status, st);
    if (rc) return rc;
    X = (const __nv_bfloat16*)X + (long long)MOST * ldx;
    D = (__nv_bfloat16*)D + (long long)MOST * ldd;
  }
  DqParams p;
  const int bt = M <= 16 ? 16 : (M <= 32 ? 32 : (M <= 64 ? 64 : 128));
  {
    const uint64_t row = mode == 0 ? K : K / 2;
    uint64_t dims[2] = {row, (uint64_t)N};
    uint64_t strides[1] = {row};
    uint32_t box[2] = {128, DQ_BM};
    int rc = make_tmap(&p.tmW, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, W, dims, strides, box);
    if (rc) return rc;
  }
  {
    uint64_t dims[2] = {(uint64_t)K, (uint64_t)M};
    uint64_t strides[1] = {(uint64_t)ldx * 2};
    uint32_t box[2] = {64, (uint32_t)bt};
    int rc = make_tmap(&p.tmX, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, X, dims, strides, box);
    if (rc) return rc;
  }
  p.scales = scales; p.bias = bias; p.D = (__nv_bfloat16*)D; p.ldd = ldd;
  p.M = M; p.N = N; p.K = K; p.status = status; p.early_weights = static_weights;
  if (mode == 0) {
    if (bt == 16) return dq_launch<16, false>(p, sms, st);
    if (bt == 32) return dq_launch<32, false>(p, sms, st);
    if (bt == 64) return dq_launch<64, false>(p, sms, st);
    return dq_launch<128, false>(p, sms, st);
  }
  if (bt == 16) return dq_launch<16, true>(p, sms, st);
  if (bt == 32) return dq_launch<32, true>(p, sms, st);
  if (bt == 64) return dq_launch<64, true>(p, sms, st);
  return dq_launch<128, true>(p, sms, st);
}
