// Dequant GEMM (gemm_dq.cu) for K of 128 or 256 and many output tiles. A tile is then a few MMAs, and what counts is that the next one's loads and
// conversions run under this one's epilogue: persistent CTAs, 128 rows of X by 128 weight rows a tile, X by TMA, weights converted to bf16
// values without scale (exact) into the swizzled tile that the MMA reads. Every 128-wide k-block has an accumulator of its own and the epilogue
// adds scale times partial sum in 32 bits, the values and the order of gemm_dq.cu.
// Measured (B200, warm) at 16384 rows, int4 [N, K] = [4096, 128] 100 us, 214 with one CTA a tile (gemm_dq.cu); [4096, 256] 130 and 235; fp8
// [1024, 128] 28 and 52.
// Structure (320 threads): warp 0 TMA (X), warp 1 MMA issue, warps 2-5 converters, warps 6-9 epilogue.
#include "dq_convert.cuh"
#include "tmap.h"
#include "sx_api.h"

namespace sx {

constexpr int DS_BM = 128, DS_BN = 128, DS_BK = 64, DS_STAGES = 6, DS_THREADS = 320, DS_MAX_KB = 2;
constexpr int DS_X_BYTES = DS_BM * DS_BK * 2, DS_STAGE_BYTES = DS_X_BYTES + DS_BN * DS_BK * 2;
constexpr int DS_SMEM = DS_STAGES * DS_STAGE_BYTES + 1024 + 512;
constexpr int DS_ACC_COLS = DS_MAX_KB * DS_BN;      // accumulators of a tile; two tiles in flight

struct DsParams {
  CUtensorMap tmX;
  const uint8_t* W;       // fp8: [N, K] bytes; int4: [N, K/2] bytes
  const float* scales;    // fp8: [ceil(N/128), K/128]; int4: [N, K/128]
  const float* bias;
  __nv_bfloat16* D;
  long long ldd;
  int M, N, K, m_blks;
  long long tiles;
  int* status;
};

template <bool INT4>
__global__ void __launch_bounds__(DS_THREADS, 1) gemm_dq_short_kernel(const __grid_constant__ DsParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + DS_STAGES * DS_STAGE_BYTES);
  uint64_t* x_full = bars;                    // [STAGES] TMA
  uint64_t* w_full = bars + DS_STAGES;        // [STAGES] 4 converter warps
  uint64_t* empty = bars + 2 * DS_STAGES;     // [STAGES] MMA commit
  uint64_t* tfull = bars + 3 * DS_STAGES;     // [2]
  uint64_t* tempty = tfull + 2;               // [2] 4 epilogue warps
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
  volatile int* s_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = warp_index(), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < DS_STAGES; ++s) {
      mbar_init(&x_full[s], 1);
      mbar_init(&w_full[s], 4);
      mbar_init(&empty[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tfull[i], 1);
      mbar_init(&tempty[i], 4);
    }
    *s_abort = 0;
    mbar_fence_init();
    tma_prefetch_desc(&p.tmX);
  }
  if (warp == 1) tmem_alloc(tmem_slot, 2 * DS_ACC_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const int kblks = p.K / 128, steps = p.K / DS_BK;      // steps of 64: two a k-block

  if (warp == 0) {
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (long long t = blockIdx.x; t < p.tiles && ok; t += gridDim.x) {
        const int m_blk = (int)(t % p.m_blks);
        for (int k = 0; k < steps; ++k) {
          if (!mbar_wait(&empty[stage], phase ^ 1, s_abort, p.status, ST_TIMEOUT_PRODUCER)) { ok = false; break; }
          mbar_expect_tx(&x_full[stage], DS_X_BYTES);
          tma_load_2d(smem + stage * DS_STAGE_BYTES, &p.tmX, &x_full[stage], k * DS_BK, m_blk * DS_BM);
          if (++stage == DS_STAGES) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc = umma_idesc_f16(DS_BM, DS_BN, 1, 0, 0);
      int stage = 0, it = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (long long t = blockIdx.x; t < p.tiles && ok; t += gridDim.x, ++it) {
        if (!mbar_wait(&tempty[it & 1], ((it >> 1) & 1) ^ 1, s_abort, p.status, ST_TIMEOUT_MMA)) break;
        tc_fence_after();
        for (int k = 0; k < steps; ++k) {
          if (!mbar_wait(&x_full[stage], phase, s_abort, p.status, ST_TIMEOUT_MMA) ||
              !mbar_wait(&w_full[stage], phase, s_abort, p.status, ST_TIMEOUT_MMA)) { ok = false; break; }
          tc_fence_after();
          const uint32_t sx = smem_u32(smem + stage * DS_STAGE_BYTES), sw = sx + DS_X_BYTES;
          const uint32_t acc = tmem_base + (it & 1) * DS_ACC_COLS + (k >> 1) * DS_BN;
#pragma unroll
          for (int j = 0; j < DS_BK / 16; ++j)
            umma_f16_ss(acc, umma_desc_sw128(sx + j * 32, 16, 1024), umma_desc_sw128(sw + j * 32, 16, 1024), idesc, ((k & 1) | j) ? 1u : 0u);
          umma_commit(&empty[stage]);
          if (++stage == DS_STAGES) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        umma_commit(&tfull[it & 1]);
      }
    }
  } else if (warp < 6) {
    // ------------------------------------------------------------ converters: 128 threads, one weight row each
    const int r = (warp - 2) * 32 + lane;
    constexpr int V = INT4 ? 2 : 4;           // 16-byte pieces of a row's step
    const long long pitch = INT4 ? p.K / 2 : p.K;
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    uint4 raw[V];
    auto fetch = [&](long long t, int k) {    // rows behind N are zeros; their products are not written
      const long long n = t / p.m_blks * DS_BN + r;
#pragma unroll
      for (int i = 0; i < V; ++i)
        raw[i] = n < p.N ? *reinterpret_cast<const uint4*>(p.W + n * pitch + k * (V * 16) + i * 16) : make_uint4(0u, 0u, 0u, 0u);
    };
    if ((long long)blockIdx.x < p.tiles) fetch(blockIdx.x, 0);
    for (long long t = blockIdx.x; t < p.tiles && ok; t += gridDim.x) {
      for (int k = 0; k < steps; ++k) {
        uint4 cur[V];
#pragma unroll
        for (int i = 0; i < V; ++i) cur[i] = raw[i];
        if (k + 1 < steps) fetch(t, k + 1);
        else if (t + gridDim.x < p.tiles) fetch(t + gridDim.x, 0);
        if (!mbar_wait_warp(&empty[stage], phase ^ 1, s_abort, p.status, ST_TIMEOUT_CONVERT)) { ok = false; break; }
        uint8_t* sw = smem + stage * DS_STAGE_BYTES + DS_X_BYTES + r * 128;
        const uint32_t* w = reinterpret_cast<const uint32_t*>(cur);
#pragma unroll
        for (int c = 0; c < 8; ++c) {         // 8 pieces of 8 bf16
          uint32_t o[4];
          if constexpr (INT4) {
            int4x8_to_bf16(w[c], o);
          } else {
            e4m3x4_to_bf16(w[2 * c], o);
            e4m3x4_to_bf16(w[2 * c + 1], o + 2);
          }
          *reinterpret_cast<uint4*>(sw + ((c ^ (r & 7)) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&w_full[stage]);
        if (++stage == DS_STAGES) { stage = 0; phase ^= 1; }
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue: thread = row of X (TMEM lane)
    const int q = warp & 3;
    int it = 0;
    for (long long t = blockIdx.x; t < p.tiles; t += gridDim.x, ++it) {
      const int row = (int)(t % p.m_blks) * DS_BM + q * 32 + lane, n0 = (int)(t / p.m_blks) * DS_BN;
      if (!mbar_wait_warp(&tfull[it & 1], (it >> 1) & 1, s_abort, p.status, ST_TIMEOUT_EPILOGUE)) break;
      tc_fence_after();
#pragma unroll 1
      for (int c = 0; c < DS_BN / 32; ++c) {
        const int col0 = n0 + c * 32;
        if (col0 >= p.N) break;
        float f[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) f[j] = 0.f;
        // lane j holds the scale of column j
        for (int kb = 0; kb < kblks; ++kb) {
          uint32_t v[32];
          tmem_ld32(tmem_base + (it & 1) * DS_ACC_COLS + kb * DS_BN + c * 32 + (static_cast<uint32_t>(q * 32) << 16), v);
          const long long sr = INT4 ? min(col0 + lane, p.N - 1) : n0 / 128;
          const float s = p.scales[sr * kblks + kb];
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j) f[j] = fmaf(__shfl_sync(0xffffffffu, s, j), __uint_as_float(v[j]), f[j]);
        }
        if (p.bias) {
          const float b = p.bias[min(col0 + lane, p.N - 1)];
#pragma unroll
          for (int j = 0; j < 32; ++j) f[j] += __shfl_sync(0xffffffffu, b, j);
        }
        __nv_bfloat16* dp = p.D + (long long)row * p.ldd + col0;
        if (row < p.M && col0 + 32 <= p.N && (reinterpret_cast<uintptr_t>(dp) & 15) == 0) {
#pragma unroll
          for (int j = 0; j < 32; j += 8)
            *reinterpret_cast<uint4*>(dp + j) = make_uint4(pack_bf16x2(f[j], f[j + 1]), pack_bf16x2(f[j + 2], f[j + 3]),
                                                           pack_bf16x2(f[j + 4], f[j + 5]), pack_bf16x2(f[j + 6], f[j + 7]));
        } else if (row < p.M) {
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (col0 + j < p.N) dp[j] = __float2bfloat16(f[j]);
        }
        __syncwarp();
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty[it & 1]);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (*s_abort) bounded_delay_ns(2000000);
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 2 * DS_ACC_COLS);
  }
}

// Up to one wave of tiles the general kernel has less to set up a tile and splits K over CTAs: 128 tiles of K = 128 7.8 us there and 8.3 here, of 256
// 8.4 and 10.4. From the second wave on its CTAs wait for one another's places: 152 tiles 13.7 and 10.4, of K = 256 14.6 and 14.5; 512 tiles 29.5 and
// 17.7, 31.7 and 23.2 (fp8; int4 the same way).
bool gemm_dq_short_ok(int M, int N, int K, int sms) {
  return K / 128 <= DS_MAX_KB && ((long long)M + DS_BM - 1) / DS_BM * ((N + DS_BN - 1) / DS_BN) > sms;
}

int gemm_dq_short(const void* X, long long ldx, const void* W, const float* scales, const float* bias, void* D, long long ldd, int M, int N, int K,
                  int mode, int sms, int* status, cudaStream_t st) {
  DsParams p;
  uint64_t dims[2] = {(uint64_t)K, (uint64_t)M};
  uint64_t strides[1] = {(uint64_t)ldx * 2};
  uint32_t box[2] = {DS_BK, DS_BM};
  int rc = make_tmap(&p.tmX, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, X, dims, strides, box);
  if (rc) return rc;
  p.W = (const uint8_t*)W; p.scales = scales; p.bias = bias; p.D = (__nv_bfloat16*)D; p.ldd = ldd;
  p.M = M; p.N = N; p.K = K; p.status = status;
  p.m_blks = (int)(((long long)M + DS_BM - 1) / DS_BM);
  p.tiles = (long long)p.m_blks * ((N + DS_BN - 1) / DS_BN);
  auto run = [&](auto kern) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, DS_SMEM) != cudaSuccess) return -10;
    kern<<<(unsigned)(p.tiles < sms ? p.tiles : sms), DS_THREADS, DS_SMEM, st>>>(p);
    return cudaGetLastError() == cudaSuccess ? 0 : -11;
  };
  return mode == 0 ? run(gemm_dq_short_kernel<false>) : run(gemm_dq_short_kernel<true>);
}

}  // namespace sx
