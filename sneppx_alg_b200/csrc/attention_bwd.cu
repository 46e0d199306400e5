// A2: flash attention backward on tcgen05 (sm_100a), head_dim 128.
//
// One CTA owns 128 key/value rows of one (batch, kv head) and walks every query head of the GQA
// group and every 64-row query tile that can see those keys. Everything is computed transposed
// (key index on the TMEM lane axis), so that with the saved LSE no row reduction is needed:
//   S^T  = K Q^T            dP^T = V dO^T                         (128 x 64, fp32 in TMEM)
//   P^T  = exp2(S^T*c - LSE)    dS^T = P^T o (dP^T - delta)        (registers -> bf16: P^T to TMEM, dS^T to shared memory)
//   dV  += P^T dO  (A operand read from TMEM)   dK += dS^T Q       (128 x 128 accumulators in TMEM; dK scaled at the end)
//   dQ^T = K^T dS^T         (128 x 64; staged through shared memory and added into dq_accum with bulk fp32
//                            reductions, cp.reduce.async.bulk, by four drain warps; scaled when converted to bf16)
// Pipeline: two tiles are in flight in TMEM, each with S^T and dP^T of its own. P^T takes the columns of S^T that it was computed from, dQ^T
// those of dP^T once dS^T is out, so that both tiles fit beside the dV and dK accumulators (2 x 128 + 2 x 128 columns). One thread issues
//   dV(i)  dQ(i)  dK(i)  S(i+2)  [dQ(i) drained]  dP(i+2)
// while two groups of eight softmax-gradient warps turn S^T / dP^T into P^T / dS^T, the even and the odd tiles. A tile still takes 3400
// cycles (3700 with one S^T / dP^T buffer and all sixteen warps on one tile; causal, 4096 tokens, 32 heads on 8: the kernel 523 -> 509 us,
// 16384 tokens 7.0 - 7.2 ms either way), of which the tensor pipe is busy 2360 and multiplies 1280: the N = 64 products fetch A from shared
// memory at half rate. Leaving out the dQ reductions or their staging changes nothing, leaving out the dQ products takes 15 % off. A loader
// warp keeps up to four Q and three dO tiles and the LSE / delta rows in flight (dO is wanted later than Q;
// the row statistics are fetched two tiles ahead so that their global-load latency is hidden); the drain warps empty dQ^T while the
// next tile's GEMMs run. CTAs are ordered heaviest key tile first. All MN-major operand forms (dO, Q, K^T, dS^T) are
// read from the very tiles TMA brought or the softmax warps wrote; no transposed copy exists. dK/dV need no atomics
// because the whole GQA group is reduced inside the CTA.
// The reference only had a dQ kernel and a cuBLAS-composed backward that materialises P
// (kernel/cuda/attention_cuda.cu:388-492, kernel/cuda/autodiff_cuda.cu:746-862).
#include <limits.h>
#include "tc_common.cuh"
#include "common.cuh"
#include "tmap.h"
#include "sx_api.h"

namespace sx {

constexpr int BWD_KV = 128;
constexpr int BWD_Q = 64;
constexpr int BWD_D = 128;
// Warp roles: 0 loader (TMA + per-row statistics), 1 MMA issue, 2..17 softmax-gradient warps (2 groups that take the tiles in turn, each 2
// halves of 32 query columns x 4 TMEM lane quarters), 18..21 dQ drain warps (one per lane quarter).
constexpr int BWD_SM_WARPS = 16;
constexpr int BWD_DRAIN_WARPS = 4;
constexpr int BWD_THREADS = 32 * (2 + BWD_SM_WARPS + BWD_DRAIN_WARPS);  // 704

struct AttnBwdParams {
  CUtensorMap tmQ, tmK, tmV, tmdO;
  const float* lse;    // [B, Hq, Sq]
  const float* delta;  // [B, Hq, Sq]
  float* dq_accum;     // tiled fp32, see the drain warps
  __nv_bfloat16* dK;
  __nv_bfloat16* dV;
  long long dk_row_stride, dv_row_stride, dk_batch_stride, dv_batch_stride;
  int* status;
  int B, Sq, Skv, Hq, Hk;
  int causal, window;
  float scale, scale_log2;
};

struct BwdCfg {
  static constexpr int Q_STAGES = 4, STAGES = 3;         // Q tiles; dO tiles and row statistics
  static constexpr int KV_BYTES = BWD_KV * BWD_D * 2;  // 32 KB
  static constexpr int Q_BYTES = BWD_Q * BWD_D * 2;    // 16 KB
  static constexpr int PT_BYTES = BWD_KV * BWD_Q * 2;  // 16 KB
  static constexpr int OFF_K = 0;
  static constexpr int OFF_V = KV_BYTES;
  static constexpr int OFF_Q = 2 * KV_BYTES;
  static constexpr int OFF_DO = OFF_Q + Q_STAGES * Q_BYTES;
  static constexpr int OFF_DST = OFF_DO + STAGES * Q_BYTES;     // dS^T, double buffered
  static constexpr int OFF_DQS = OFF_DST + 2 * PT_BYTES;        // dQ staging: 4 drain warps x [32 query rows][32 head-dim] fp32
  static constexpr int DQS_BYTES = 4 * 4096;
  static constexpr int OFF_STAT = OFF_DQS + DQS_BYTES;          // STAGES x {lse * log2e, delta} x 64 floats
  static constexpr int OFF_BAR = OFF_STAT + STAGES * 512;
  static constexpr int SMEM_BYTES = OFF_BAR + 256 + 1024;
  // TMEM columns: two tiles of S^T and dP^T (64 each), dV, dK (128 each). P^T as packed bf16 pairs: the 16 query columns of a column group
  // (one K step of dV) become the first 8 of the group's 16 columns of S^T, which only the warps of that group have read.
  static constexpr uint32_t TM_S = 0, TM_DP = 64, TM_TILE = 128, TM_DV = 256, TM_DK = 384;
};

__global__ void __launch_bounds__(BWD_THREADS, 1) attn_bwd_kernel(const __grid_constant__ AttnBwdParams p) {
  using Cfg = BwdCfg;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sK = smem + Cfg::OFF_K;
  uint8_t* sV = smem + Cfg::OFF_V;
  uint8_t* sQ = smem + Cfg::OFF_Q;
  uint8_t* sdO = smem + Cfg::OFF_DO;
  uint8_t* sDST = smem + Cfg::OFF_DST;
  float* sStat = reinterpret_cast<float*>(smem + Cfg::OFF_STAT);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::OFF_BAR);
  uint64_t* kv_full = bars;          // 1
  uint64_t* q_full = bars + 1;       // [4]
  uint64_t* q_empty = bars + 5;      // [4]
  uint64_t* do_full = bars + 9;      // [3]
  uint64_t* do_empty = bars + 12;    // [3]
  uint64_t* stat_full = bars + 15;   // [3], 1 arrival each
  uint64_t* s_full = bars + 18;      // [2] by tile parity, as are the next two
  uint64_t* dp_full = bars + 20;     // [2]
  uint64_t* pds_ready = bars + 22;   // [2], 8 arrivals
  uint64_t* dq_full = bars + 24;     // 1
  uint64_t* dq_drained = bars + 25;  // 4 arrivals: the dQ^T accumulator has been read out of TMEM
  uint64_t* all_done = bars + 26;    // 1: every MMA of the CTA has executed
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 27);
  volatile int* s_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = warp_index(), lane = threadIdx.x & 31;
  // Heaviest key tiles first (under a causal mask tile 0 sees every query tile): kv head is the fastest block index.
  const int kv_tile = blockIdx.x / p.Hk, kv_head = blockIdx.x % p.Hk, b = blockIdx.z;
  const int G = p.Hq / p.Hk;
  const int kv0 = kv_tile * BWD_KV;
  const int offset = p.Skv - p.Sq;
  const int n_qt_total = (p.Sq + BWD_Q - 1) / BWD_Q;
  int qt_lo = 0, qt_hi = n_qt_total;  // [lo, hi)
  if (p.causal) {
    const int first_q = kv0 - offset;  // smallest query index that sees key kv0
    if (first_q > 0) qt_lo = first_q / BWD_Q;
  }
  if (p.window > 0) {
    const long long last_q = (long long)kv0 + BWD_KV - 1 + p.window - 1 - offset;
    if (last_q < 0) qt_hi = 0;
    else if (last_q / BWD_Q + 1 < qt_hi) qt_hi = (int)(last_q / BWD_Q + 1);
  }
  const int n_qt = max(qt_hi - qt_lo, 0);
  const int n_it = n_qt * G;

  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    for (int i = 0; i < Cfg::Q_STAGES; ++i) {
      mbar_init(&q_full[i], 1);
      mbar_init(&q_empty[i], 1);
    }
    for (int i = 0; i < Cfg::STAGES; ++i) {
      mbar_init(&do_full[i], 1);
      mbar_init(&do_empty[i], 1);
      mbar_init(&stat_full[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&s_full[i], 1);
      mbar_init(&dp_full[i], 1);
      mbar_init(&pds_ready[i], BWD_SM_WARPS / 2);
    }
    mbar_init(all_done, 1);
    mbar_init(dq_full, 1);
    mbar_init(dq_drained, BWD_DRAIN_WARPS);
    *s_abort = 0;
    mbar_fence_init();
    tma_prefetch_desc(&p.tmQ);
    tma_prefetch_desc(&p.tmK);
    tma_prefetch_desc(&p.tmV);
    tma_prefetch_desc(&p.tmdO);
  }
  if (warp == 1) tmem_alloc(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  auto tma5 = [](void* dst, const CUtensorMap* m, uint64_t* bar, int c1, int c3, int c4) {
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
        ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(0), "r"(c1), "r"(0),
        "r"(c3), "r"(c4)
        : "memory");
  };

  if (warp == 0) {
    // ------------------------------------------------------------ loader: TMA tiles + LSE / delta rows
    if (n_it > 0) {
      if (lane == 0) {
        mbar_expect_tx(kv_full, 2 * Cfg::KV_BYTES);
        tma5(sK, &p.tmK, kv_full, kv0, kv_head, b);
        tma5(sV, &p.tmV, kv_full, kv0, kv_head, b);
      }
      // LSE (scaled to log2) and delta of the 64 query rows of a tile: lane i holds rows i and i + 32. The loads run two
      // tiles ahead of their use so that their ~1 us latency never sits on the per-tile critical path.
      auto load_stats = [&](int it, float& l0, float& l1, float& d0, float& d1) {
        const int head = kv_head * G + it / n_qt;
        const int qrow0 = (qt_lo + it % n_qt) * BWD_Q;
        const long long so = ((long long)b * p.Hq + head) * p.Sq + qrow0;
        l0 = INFINITY; l1 = INFINITY; d0 = 0.f; d1 = 0.f;
        if (qrow0 + lane < p.Sq) { l0 = p.lse[so + lane] * 1.4426950408889634f; d0 = p.delta[so + lane]; }
        if (qrow0 + lane + 32 < p.Sq) { l1 = p.lse[so + lane + 32] * 1.4426950408889634f; d1 = p.delta[so + lane + 32]; }
      };
      float cl0, cl1, cd0, cd1, nl0 = INFINITY, nl1 = INFINITY, nd0 = 0.f, nd1 = 0.f;
      load_stats(0, cl0, cl1, cd0, cd1);
      if (n_it > 1) load_stats(1, nl0, nl1, nd0, nd1);
      auto load_q = [&](int it) {
        const int s = it % Cfg::Q_STAGES;
        if (!mbar_wait_warp(&q_empty[s], ((it / Cfg::Q_STAGES) & 1) ^ 1, s_abort, p.status, ST_TIMEOUT_PRODUCER)) return false;
        if (lane == 0) {
          mbar_expect_tx(&q_full[s], Cfg::Q_BYTES);
          tma5(sQ + s * Cfg::Q_BYTES, &p.tmQ, &q_full[s], (qt_lo + it % n_qt) * BWD_Q, kv_head * G + it / n_qt, b);
        }
        return true;
      };
      bool ok = load_q(0);
      for (int it = 0; it < n_it && ok; ++it) {
        const int s = it % Cfg::STAGES;
        if (!mbar_wait_warp(&do_empty[s], ((it / Cfg::STAGES) & 1) ^ 1, s_abort, p.status, ST_TIMEOUT_PRODUCER)) break;
        if (lane == 0) {
          mbar_expect_tx(&do_full[s], Cfg::Q_BYTES);
          tma5(sdO + s * Cfg::Q_BYTES, &p.tmdO, &do_full[s], (qt_lo + it % n_qt) * BWD_Q, kv_head * G + it / n_qt, b);
        }
        if (it + 1 < n_it) ok = load_q(it + 1);
        float* st = sStat + s * 128;
        st[lane] = cl0; st[lane + 32] = cl1; st[64 + lane] = cd0; st[64 + lane + 32] = cd1;
        __syncwarp();
        if (lane == 0) mbar_arrive(&stat_full[s]);
        cl0 = nl0; cl1 = nl1; cd0 = nd0; cd1 = nd1;
        if (it + 2 < n_it) load_stats(it + 2, nl0, nl1, nd0, nd1);
      }
    }
  } else if (warp == 1) {
    if (n_it > 0 && elect_one()) {
      constexpr uint32_t idesc_s = umma_idesc_f16(128, BWD_Q, 1, 0, 0);      // K Q^T, V dO^T
      constexpr uint32_t idesc_acc = umma_idesc_f16(128, BWD_D, 1, 0, 1);    // P^T dO, dS^T Q
      constexpr uint32_t idesc_dq = umma_idesc_f16(128, BWD_Q, 1, 1, 1);     // K^T dS^T
      const uint32_t aK = smem_u32(sK), aV = smem_u32(sV), aDST0 = smem_u32(sDST);
      auto q_ready = [&](int it) {
        return mbar_wait(&q_full[it % Cfg::Q_STAGES], (it / Cfg::Q_STAGES) & 1, s_abort, p.status, ST_TIMEOUT_MMA);
      };
      auto do_ready = [&](int it) {
        return mbar_wait(&do_full[it % Cfg::STAGES], (it / Cfg::STAGES) & 1, s_abort, p.status, ST_TIMEOUT_MMA);
      };
      auto issue_s = [&](int it) {
        const uint32_t q = smem_u32(sQ + (it % Cfg::Q_STAGES) * Cfg::Q_BYTES), t = tmem_base + Cfg::TM_S + (it & 1) * Cfg::TM_TILE;
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
          for (int k = 0; k < 4; ++k)
            umma_f16_ss(t, umma_desc_sw128(aK + c * 16384 + k * 32, 16, 1024), umma_desc_sw128(q + c * 8192 + k * 32, 16, 1024), idesc_s,
                        (c | k) ? 1u : 0u);
        umma_commit(&s_full[it & 1]);
      };
      auto issue_dp = [&](int it) {
        const uint32_t dO = smem_u32(sdO + (it % Cfg::STAGES) * Cfg::Q_BYTES), t = tmem_base + Cfg::TM_DP + (it & 1) * Cfg::TM_TILE;
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
          for (int k = 0; k < 4; ++k)
            umma_f16_ss(t, umma_desc_sw128(aV + c * 16384 + k * 32, 16, 1024), umma_desc_sw128(dO + c * 8192 + k * 32, 16, 1024), idesc_s,
                        (c | k) ? 1u : 0u);
        umma_commit(&dp_full[it & 1]);
      };
      bool ok = mbar_wait(kv_full, 0, s_abort, p.status, ST_TIMEOUT_MMA);
      for (int it = 0; it < 2 && it < n_it && ok; ++it) {
        ok = q_ready(it) && do_ready(it);
        if (!ok) break;
        tc_fence_after();
        issue_s(it);
        issue_dp(it);
      }
      for (int it = 0; it < n_it && ok; ++it) {
        if (!mbar_wait(&pds_ready[it & 1], (it >> 1) & 1, s_abort, p.status, ST_TIMEOUT_MMA)) { ok = false; break; }
        tc_fence_after();
        const uint32_t q = smem_u32(sQ + (it % Cfg::Q_STAGES) * Cfg::Q_BYTES), dO = smem_u32(sdO + (it % Cfg::STAGES) * Cfg::Q_BYTES);
        const uint32_t aDST = aDST0 + (it & 1) * Cfg::PT_BYTES, tT = tmem_base + (it & 1) * Cfg::TM_TILE;
        // dV += P^T dO (P^T read from TMEM)   (K = 64 query rows: 4 k-steps)
#pragma unroll
        for (int k = 0; k < 4; ++k)
          umma_f16_ts(tmem_base + Cfg::TM_DV, tT + Cfg::TM_S + k * 16, umma_desc_sw128(dO + k * 2048, 8192, 1024), idesc_acc,
                      (it | k) ? 1u : 0u);
        umma_commit(&do_empty[it % Cfg::STAGES]);
        // dQ^T = K^T dS^T  (K = 128 key rows: 8 k-steps), over dP^T, which every softmax warp has read
#pragma unroll
        for (int k = 0; k < 8; ++k)
          umma_f16_ss(tT + Cfg::TM_DP, umma_desc_sw128(aK + k * 2048, 16384, 1024), umma_desc_sw128(aDST + k * 2048, 16384, 1024), idesc_dq,
                      k ? 1u : 0u);
        umma_commit(dq_full);
        // dK += dS^T Q
#pragma unroll
        for (int k = 0; k < 4; ++k)
          umma_f16_ss(tmem_base + Cfg::TM_DK, umma_desc_sw128(aDST + k * 32, 16, 1024), umma_desc_sw128(q + k * 2048, 8192, 1024), idesc_acc,
                      (it | k) ? 1u : 0u);
        umma_commit(&q_empty[it % Cfg::Q_STAGES]);
        // S^T of tile it + 2 over P^T, which dV (issued before) has read
        if (it + 2 < n_it) {
          if (!q_ready(it + 2)) { ok = false; break; }
          tc_fence_after();
          issue_s(it + 2);
        }
        // every drain is waited for: its barrier advances one phase a tile
        if (it + 1 < n_it && !mbar_wait(dq_drained, it & 1, s_abort, p.status, ST_TIMEOUT_MMA)) { ok = false; break; }
        if (it + 2 < n_it) {
          if (!do_ready(it + 2)) { ok = false; break; }
          tc_fence_after();
          issue_dp(it + 2);
        }
      }
      if (ok) umma_commit(all_done);
    }
  } else if (warp < 2 + BWD_SM_WARPS) {
    // ------------------------------------------------------------ softmax-gradient warps
    const int cg = (warp - 2) >> 2;     // output columns in the end: halves of dV and dK
    const int grp = cg >> 1;            // tiles of this group of eight warps: it % 2 == grp
    const int qd = warp & 3;            // TMEM lane quarter this warp may touch
    const int r = qd * 32 + lane;       // key row inside the tile == TMEM lane
    const int kv_idx = kv0 + r;
    const uint32_t lane_addr = static_cast<uint32_t>(qd * 32) << 16;
    bool ok = n_it > 0;
    for (int it = grp; it < n_it && ok; it += 2) {
      const int qrow0 = (qt_lo + it % n_qt) * BWD_Q;
      const bool need_mask = (p.causal && kv0 + BWD_KV - 1 > qrow0 + offset) || (kv0 + BWD_KV > p.Skv) ||
                             (p.window > 0 && kv0 < qrow0 + BWD_Q - 1 + offset - p.window + 1);
      const int stg = it % Cfg::STAGES;
      const uint32_t tile = tmem_base + grp * Cfg::TM_TILE + lane_addr;
      uint8_t* dstb = sDST + grp * Cfg::PT_BYTES;
      if (!mbar_wait_warp(&stat_full[stg], (it / Cfg::STAGES) & 1, s_abort, p.status, ST_TIMEOUT_EPILOGUE)) { ok = false; break; }
      if (!mbar_wait_warp(&s_full[grp], (it >> 1) & 1, s_abort, p.status, ST_TIMEOUT_EPILOGUE)) { ok = false; break; }
      tc_fence_after();
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int cc0 = (cg & 1) * 2 + h, c0 = cc0 * 16;      // 16 query columns: one K step of dV
        const float* st = sStat + stg * 128 + c0;
        float pf[16];
        uint32_t pt[8], ds[8];
        {
          uint32_t v[16];
          tmem_ld16(tile + Cfg::TM_S + c0, v);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; i += 4) {
            const float4 a4 = *reinterpret_cast<const float4*>(st + i);
            pf[i] = exp2f(fmaf(__uint_as_float(v[i]), p.scale_log2, -a4.x));
            pf[i + 1] = exp2f(fmaf(__uint_as_float(v[i + 1]), p.scale_log2, -a4.y));
            pf[i + 2] = exp2f(fmaf(__uint_as_float(v[i + 2]), p.scale_log2, -a4.z));
            pf[i + 3] = exp2f(fmaf(__uint_as_float(v[i + 3]), p.scale_log2, -a4.w));
          }
          if (need_mask) {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const int qi = qrow0 + c0 + i + offset;
              bool dead = kv_idx >= p.Skv;
              if (p.causal && kv_idx > qi) dead = true;
              if (p.window > 0 && kv_idx < qi - p.window + 1) dead = true;
              if (dead) pf[i] = 0.f;
            }
          }
#pragma unroll
          for (int i = 0; i < 16; i += 2) pt[i / 2] = pack_bf16x2(pf[i], pf[i + 1]);
        }
        if (h == 0) {
          ok = mbar_wait_warp(&dp_full[grp], (it >> 1) & 1, s_abort, p.status, ST_TIMEOUT_EPILOGUE);
          if (!ok) break;
          tc_fence_after();
        }
        {
          uint32_t v[16];
          tmem_ld16(tile + Cfg::TM_DP + c0, v);
          // Buffer grp of P^T and dS^T was last read by the GEMMs of tile it - 2. Those were issued before S^T of this tile and the GEMMs
          // of one thread execute in order, so s_full already covers them.
          asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(tile + Cfg::TM_S + c0),
                       "r"(pt[0]), "r"(pt[1]), "r"(pt[2]), "r"(pt[3]), "r"(pt[4]), "r"(pt[5]), "r"(pt[6]), "r"(pt[7])
                       : "memory");
          tmem_ld_wait();
          // dS without the softmax scale: dK and dQ are scaled once when they are written out
#pragma unroll
          for (int i = 0; i < 16; i += 4) {
            const float4 d4 = *reinterpret_cast<const float4*>(st + 64 + i);
            ds[i / 2] = pack_bf16x2(pf[i] * (__uint_as_float(v[i]) - d4.x), pf[i + 1] * (__uint_as_float(v[i + 1]) - d4.y));
            ds[i / 2 + 1] = pack_bf16x2(pf[i + 2] * (__uint_as_float(v[i + 2]) - d4.z), pf[i + 3] * (__uint_as_float(v[i + 3]) - d4.w));
          }
        }
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const int off = r * 128 + (((cc0 * 2 + k) ^ (r & 7)) << 4);
          *reinterpret_cast<uint4*>(dstb + off) = make_uint4(ds[k * 4], ds[k * 4 + 1], ds[k * 4 + 2], ds[k * 4 + 3]);
        }
      }
      if (!ok) break;
      tmem_st_wait();
      fence_proxy_async_smem();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&pds_ready[grp]);
    }
    if (ok && n_it > 0) {
      if (mbar_wait_warp(all_done, 0, s_abort, p.status, ST_TIMEOUT_EPILOGUE)) {
        tc_fence_after();
        // dK / dV accumulators -> bf16 rows: column groups 0,1 store the halves of dV, 2,3 the halves of dK (scaled)
        const bool row_ok = kv_idx < p.Skv;
        const bool is_dk = cg >= 2;
        const float mul = is_dk ? p.scale : 1.f;
        __nv_bfloat16* dst = (is_dk ? p.dK + (long long)b * p.dk_batch_stride + (long long)kv_idx * p.dk_row_stride
                                    : p.dV + (long long)b * p.dv_batch_stride + (long long)kv_idx * p.dv_row_stride) +
                             (long long)kv_head * BWD_D + (cg & 1) * 64;
        const uint32_t src = tmem_base + (is_dk ? Cfg::TM_DK : Cfg::TM_DV) + lane_addr + (cg & 1) * 64;
#pragma unroll 1
        for (int c = 0; c < 2; ++c) {
          uint32_t v[32];
          tmem_ld32(src + c * 32, v);
          tmem_ld_wait();
          if (row_ok) {
#pragma unroll
            for (int i = 0; i < 32; i += 8) {
              uint4 o;
              o.x = pack_bf16x2(__uint_as_float(v[i]) * mul, __uint_as_float(v[i + 1]) * mul);
              o.y = pack_bf16x2(__uint_as_float(v[i + 2]) * mul, __uint_as_float(v[i + 3]) * mul);
              o.z = pack_bf16x2(__uint_as_float(v[i + 4]) * mul, __uint_as_float(v[i + 5]) * mul);
              o.w = pack_bf16x2(__uint_as_float(v[i + 6]) * mul, __uint_as_float(v[i + 7]) * mul);
              *reinterpret_cast<uint4*>(dst + c * 32 + i) = o;
            }
          }
        }
      }
    } else if (n_it == 0 && cg == 0) {
      if (kv_idx < p.Skv) {
        __nv_bfloat16* dkr = p.dK + (long long)b * p.dk_batch_stride + (long long)kv_idx * p.dk_row_stride +
                             (long long)kv_head * BWD_D;
        __nv_bfloat16* dvr = p.dV + (long long)b * p.dv_batch_stride + (long long)kv_idx * p.dv_row_stride +
                             (long long)kv_head * BWD_D;
        for (int i = 0; i < BWD_D; i += 8) {
          *reinterpret_cast<uint4*>(dkr + i) = make_uint4(0, 0, 0, 0);
          *reinterpret_cast<uint4*>(dvr + i) = make_uint4(0, 0, 0, 0);
        }
      }
    }
  } else {
    // ------------------------------------------------------------ dQ drain warps
    // dQ^T tile in TMEM: lane = head-dim index, column = query row. Each warp owns one lane quarter and moves it in two
    // halves of 32 query rows: [32 query rows][32 head-dim] fp32 (4 KB, contiguous) staged in shared memory and added
    // into dq_accum with one bulk reduction each. dq_accum is tiled to match:
    // [b][head][q tile][lane quarter][64 query rows][32 head-dim].
    const int qd = warp & 3;
    const uint32_t lane_addr = static_cast<uint32_t>(qd * 32) << 16;
    float* stage = reinterpret_cast<float*>(smem + Cfg::OFF_DQS) + qd * 1024;
    bool ok = true;
    for (int it = 0; it < n_it && ok; ++it) {
      const int head = kv_head * G + it / n_qt;
      const int qt = qt_lo + it % n_qt;
      float* dst = p.dq_accum + ((((long long)b * p.Hq + head) * n_qt_total + qt) * 4 + qd) * 2048;
      if (!mbar_wait_warp(dq_full, it & 1, s_abort, p.status, ST_TIMEOUT_EPILOGUE)) { ok = false; break; }
      tc_fence_after();
      uint32_t v0[32], v1[32];
      const uint32_t src = tmem_base + Cfg::TM_DP + (it & 1) * Cfg::TM_TILE + lane_addr;
      tmem_ld32(src, v0);
      tmem_ld32(src + 32, v1);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(dq_drained);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // the stage has been read
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 32; ++i) stage[i * 32 + lane] = __uint_as_float(h ? v1[i] : v0[i]);
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f32 [%0], [%1], %2;" ::"l"(dst + h * 1024),
                       "r"(smem_u32(stage)), "r"(4096)
                       : "memory");
          asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
      }
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }

  tc_fence_before();
  __syncthreads();
  if (*s_abort) bounded_delay_ns(2000000);
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// delta[b,h,s] = sum_d dO * O, and dq_accum zeroed. Bound: memory (dO and O read, dq_accum written once). 16 lanes a (token, head) row with a
// 16-byte load each, four rows of a lane in flight: [1, 4096, 32, 128] 21 us, 45 us as a memset and a kernel with four bytes a lane. dq_accum holds
// whole tiles of 64 queries, so few queries leave more to zero than their rows have CTAs for: CTAs behind the last row only zero
// ([1, 1, 32, 128], whole backward: 20 us, 36 with one CTA that zeroed 1 MB).
// WIDE: rows of O on 16 bytes; on 4 otherwise, which is all that a caller of sx_attn_bwd has to keep for O.
template <bool WIDE>
__global__ void __launch_bounds__(256) attn_delta_kernel(const __nv_bfloat16* __restrict__ dO, const __nv_bfloat16* __restrict__ O,
                                                         float* __restrict__ delta, float4* __restrict__ acc, long long acc4, unsigned rows,
                                                         unsigned S, unsigned H, long long do_row_stride, long long o_row_stride) {
  constexpr int R = 4;
  const unsigned part = threadIdx.x & 15, r0 = (blockIdx.x * 16u + (threadIdx.x >> 4)) * R;
  const long long threads = (long long)gridDim.x * 256;
  bf16x8 a[R], c[R];
#pragma unroll
  for (int k = 0; k < R; ++k) {
    const unsigned r = min(r0 + k, rows - 1), h = r % H, tok = r / H;
    a[k] = ld8(dO + tok * do_row_stride + h * BWD_D + part * 8);
    const __nv_bfloat16* o = O + tok * o_row_stride + h * BWD_D + part * 8;
    if constexpr (WIDE) c[k] = ld8(o);
    else {
#pragma unroll
      for (int j = 0; j < 4; ++j) reinterpret_cast<uint32_t*>(&c[k])[j] = reinterpret_cast<const uint32_t*>(o)[j];
    }
  }
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < acc4; i += threads) acc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int k = 0; k < R; ++k) {
    float x[8], y[8], s = 0.f;
    unpack8(a[k], x);
    unpack8(c[k], y);
#pragma unroll
    for (int j = 0; j < 8; ++j) s += x[j] * y[j];
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    const unsigned r = r0 + k;
    if (part == 0 && r < rows) {
      const unsigned h = r % H, tok = r / H;
      delta[((long long)(tok / S) * H + h) * S + tok % S] = s;
    }
  }
}

// dq_accum (tiled as the backward kernel writes it) * scale -> bf16 dQ rows. One thread converts 4 values.
__global__ void attn_dq_convert_kernel(const float* __restrict__ acc, __nv_bfloat16* __restrict__ dQ, int B, int Sq,
                                       int Hq, long long dq_row_stride, float scale) {
  const int n_qt = (Sq + BWD_Q - 1) / BWD_Q;
  const long long n = (long long)B * Hq * n_qt * (BWD_Q * BWD_D / 4);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    // i enumerates float4 groups in storage order [tile][lane quarter (4)][query row (64)][head-dim (32)]
    const int di4 = i & 7;
    const int qi = (i >> 3) & 63;
    const int qd = (i >> 9) & 3;
    const long long t = i >> 11;           // (b * Hq + head) * n_qt + tile
    const int tile = t % n_qt;
    const long long bh = t / n_qt;
    const int head = bh % Hq;
    const long long bb = bh / Hq;
    const int srow = tile * BWD_Q + qi;
    if (srow >= Sq) continue;
    const float4 v = *reinterpret_cast<const float4*>(acc + i * 4);
    __nv_bfloat162 lo = __floats2bfloat162_rn(v.x * scale, v.y * scale), hi = __floats2bfloat162_rn(v.z * scale, v.w * scale);
    uint2 o;
    o.x = *reinterpret_cast<uint32_t*>(&lo);
    o.y = *reinterpret_cast<uint32_t*>(&hi);
    *reinterpret_cast<uint2*>(dQ + (bb * Sq + srow) * dq_row_stride + (long long)head * BWD_D + qd * 32 + di4 * 4) = o;
  }
}

static int make_attn_map_bwd(CUtensorMap* tm, const void* base, int B, int S, int H, int D, long long row_stride,
                             long long batch_stride, int box_rows) {
  uint64_t dims[5] = {64, (uint64_t)S, (uint64_t)(D / 64), (uint64_t)H, (uint64_t)B};
  uint64_t strides[4] = {(uint64_t)row_stride * 2, 128, (uint64_t)D * 2, (uint64_t)batch_stride * 2};
  uint32_t box[5] = {64, (uint32_t)box_rows, (uint32_t)(D / 64), 1, 1};
  return make_tmap(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, base, dims, strides, box);
}

}  // namespace sx
using namespace sx;

// Requirements: D == 128, v_head_div == 1, dQ batch stride == Sq * dq_row_stride; dq_accum holds
// B * Hq * ceil(Sq / 64) * 64 * 128 floats.
extern "C" int sx_attn_bwd(const SxAttnArgs* a, cudaStream_t st) {
  if (a->D != BWD_D) return -1;
  if (a->Hq % a->Hk) return -2;
  if (a->v_head_div > 1) return -4;
  if ((a->q_row_stride % 8) || (a->k_row_stride % 8) || (a->v_row_stride % 8) || (a->do_row_stride % 8) ||
      (a->dq_row_stride % 4) || (a->dk_row_stride % 8) || (a->dv_row_stride % 8))
    return -3;
  AttnBwdParams p;
  int rc = make_attn_map_bwd(&p.tmQ, a->Q, a->B, a->Sq, a->Hq, a->D, a->q_row_stride, a->q_batch_stride, BWD_Q);
  if (rc) return rc;
  rc = make_attn_map_bwd(&p.tmdO, a->dO, a->B, a->Sq, a->Hq, a->D, a->do_row_stride, (long long)a->Sq * a->do_row_stride,
                         BWD_Q);
  if (rc) return rc;
  rc = make_attn_map_bwd(&p.tmK, a->K, a->B, a->Skv, a->Hk, a->D, a->k_row_stride, a->k_batch_stride, BWD_KV);
  if (rc) return rc;
  rc = make_attn_map_bwd(&p.tmV, a->V, a->B, a->Skv, a->Hk, a->D, a->v_row_stride, a->v_batch_stride, BWD_KV);
  if (rc) return rc;
  const long long tokens = (long long)a->B * a->Sq;
  const int n_qt = (a->Sq + BWD_Q - 1) / BWD_Q;
  // dq_accum holds whole 64-row query tiles: B * Hq * n_qt * 64 * 128 floats
  const long long acc_floats = (long long)a->B * a->Hq * n_qt * BWD_Q * BWD_D;
  const long long rows = tokens * a->Hq;
  if (rows <= 0 || rows > 0x7fffffffll || (a->o_row_stride % 2) || (reinterpret_cast<uintptr_t>(a->O) & 3)) return -5;
  // CTAs for the rows, and for zeroing enough that a thread has at most 8 pieces, up to four an SM
  const long long acc4 = acc_floats / 4, by_rows = (rows + 63) / 64, by_acc = (acc4 + 2047) / 2048 < 592 ? (acc4 + 2047) / 2048 : 592;
  const bool wide = a->o_row_stride % 8 == 0 && (reinterpret_cast<uintptr_t>(a->O) & 15) == 0;
  auto delta = [&](auto kern) {
    kern<<<(unsigned)(by_rows > by_acc ? by_rows : by_acc), 256, 0, st>>>((const __nv_bfloat16*)a->dO, (const __nv_bfloat16*)a->O, a->delta,
                                                                         (float4*)a->dq_accum, acc4, (unsigned)rows, (unsigned)a->Sq,
                                                                         (unsigned)a->Hq, a->do_row_stride, a->o_row_stride);
  };
  wide ? delta(attn_delta_kernel<true>) : delta(attn_delta_kernel<false>);
  p.lse = a->lse; p.delta = a->delta; p.dq_accum = a->dq_accum;
  p.dK = (__nv_bfloat16*)a->dK; p.dV = (__nv_bfloat16*)a->dV;
  p.dk_row_stride = a->dk_row_stride; p.dv_row_stride = a->dv_row_stride;
  p.dk_batch_stride = a->dk_batch_stride; p.dv_batch_stride = a->dv_batch_stride;
  p.status = a->status;
  p.B = a->B; p.Sq = a->Sq; p.Skv = a->Skv; p.Hq = a->Hq; p.Hk = a->Hk;
  p.causal = a->causal; p.window = a->window;
  p.scale = a->scale; p.scale_log2 = a->scale * 1.4426950408889634f;
  static bool set = false;
  if (!set) {
    if (cudaFuncSetAttribute(attn_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, BwdCfg::SMEM_BYTES) !=
        cudaSuccess)
      return -10;
    set = true;
  }
  dim3 grid(((a->Skv + BWD_KV - 1) / BWD_KV) * a->Hk, 1, a->B);
  attn_bwd_kernel<<<grid, BWD_THREADS, BwdCfg::SMEM_BYTES, st>>>(p);
  {
    const long long n = acc_floats / 4;
    const int blocks = (int)((n + 255) / 256 < 148 * 16 ? (n + 255) / 256 : 148 * 16);
    attn_dq_convert_kernel<<<blocks, 256, 0, st>>>(a->dq_accum, (__nv_bfloat16*)a->dQ, a->B, a->Sq, a->Hq,
                                                   a->dq_row_stride, a->scale);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}
