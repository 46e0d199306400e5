// A2: flash attention backward on tcgen05 (sm_100a), head_dim 128.
//
// One CTA owns 128 key/value rows of one (batch, kv head) and walks every query head of the GQA
// group and every 128-row query tile that can see those keys. Everything but dQ is computed transposed
// (key index on the TMEM lane axis), so that with the saved LSE no row reduction is needed:
//   S^T  = K Q^T            dP^T = V dO^T                         (128 x 128, fp32 in TMEM)
//   P^T  = exp2(S^T*c - LSE)    dS^T = P^T o (dP^T - delta)        (registers -> bf16: P^T to TMEM, dS^T to shared memory)
//   dV  += P^T dO  (A operand read from TMEM)   dK += dS^T Q       (128 x 128 accumulators in TMEM; dK scaled at the end)
//   dQ   = dS K             (128 x 128; staged through shared memory and added into dq_accum with bulk fp32 reductions,
//                            cp.reduce.async.bulk, by eight drain warps; scaled when converted to bf16)
// Pipeline: TMEM is full (S^T, dP^T, dV, dK of 128 columns each): P^T takes the columns of S^T that it was computed from, dQ those of dP^T
// once dS^T is out. One thread issues
//   dV(i)  S(i+1)  dQ(i)  dK(i)  [dQ(i) drained]  dP(i+1)
// while sixteen softmax-gradient warps turn S^T(i+1) into P^T under dQ(i), dK(i) and dP(i+1), and dP^T(i+1) into dS^T under dV(i+1) and S(i+2).
// A loader warp refills each half of dO when dV has read it and a Q tile when dK has. CTAs are ordered heaviest key tile first. All MN-major
// operand forms (dO, Q, K, dS) are read from the very tiles TMA brought or the softmax warps wrote; no transposed copy exists. dK/dV need no
// atomics because the whole GQA group is reduced inside the CTA.
// Bound: shared memory. The 40 products of a tile are 2560 cycles of the tensor pipe, their operands, the tiles, dS and the staged dQ 512 KB,
// 4096 cycles at 128 bytes; a tile takes about 4000. With query tiles of 64 (two in flight) it was 6800 for as many queries: a product of N = 64
// takes its A as often as one of N = 128. B200, warm, whole backward as called (delta, this kernel, conversion),
// before -> now: [1, 4096, 32 / 8 heads] causal 550 -> 367 us, [1, 16384, 32 / 8] 7.4 -> 5.1 ms, [1, 8192, 8 / 2] full 1084 -> 800 us,
// [8, 512, 28 / 4] 185 -> 152 us.
// dQ by 16-byte reductions from registers instead of staging and bulk reductions: 25 cycles per 512 bytes, 64 KB a tile, and shared memory
// accesses queue behind them (488 us at 4096, 425 staged by four warps). The accumulator's columns have to be read before dP^T of the next tile:
// eight drain warps take them into registers at once.
// The reference only had a dQ kernel and a cuBLAS-composed backward that materialises P
// (kernel/cuda/attention_cuda.cu:388-492, kernel/cuda/autodiff_cuda.cu:746-862).
#include <limits.h>
#include "tc_common.cuh"
#include "common.cuh"
#include "tmap.h"
#include "sx_api.h"

namespace sx {

constexpr int BWD_KV = 128;
constexpr int BWD_Q = 128;
constexpr int BWD_D = 128;
// Warp roles: 0 loader (TMA + per-row statistics), 1 MMA issue, 2..17 softmax-gradient warps (4 groups of 32 query columns x 4 TMEM lane
// quarters), 18..25 dQ drain warps (two per lane quarter, half of the columns each).
constexpr int BWD_SM_WARPS = 16;
constexpr int BWD_DRAIN_WARPS = 8;
constexpr int BWD_THREADS = 32 * (2 + BWD_SM_WARPS + BWD_DRAIN_WARPS);  // 832
// dq_accum: [b][head][piece of 32 queries][32 groups of 4 head-dim][32 queries][4] fp32, which a warp's 16-byte stores of one group write
// without bank conflicts; pieces come in pairs (64 queries).
__host__ __device__ constexpr int bwd_pieces(int Sq) { return (Sq + 63) / 64 * 2; }

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
  static constexpr int TILE_BYTES = 128 * BWD_D * 2;   // 32 KB: K, V, Q, dO or dS^T of 128 rows, as two slabs of 64 columns
  static constexpr int SLAB = TILE_BYTES / 2;
  static constexpr int OFF_K = 0;
  static constexpr int OFF_V = TILE_BYTES;
  static constexpr int OFF_Q = 2 * TILE_BYTES;         // two
  static constexpr int OFF_DO = 4 * TILE_BYTES;        // one: each half of its rows is refilled when dV has read it
  static constexpr int OFF_DST = 5 * TILE_BYTES;       // dS^T
  static constexpr int OFF_DQS = 6 * TILE_BYTES;       // dQ staging: 8 drain warps x [8 groups of 4 head-dim][32 queries][4] fp32
  static constexpr int OFF_STAT = OFF_DQS + 8 * 4096;  // 2 x {-lse * log2e, -delta} x 128 floats
  static constexpr int OFF_BAR = OFF_STAT + 2 * 1024;
  static constexpr int SMEM_BYTES = OFF_BAR + 256;     // no room to align the base: it is checked
  static_assert(SMEM_BYTES <= 232448, "227 KB");
  // TMEM columns. P^T as packed bf16 pairs: the 16 query columns of a column group (one K step of dV) become the first 8 of the group's 16
  // columns of S^T, which only the warps of that group have read.
  static constexpr uint32_t TM_S = 0, TM_DP = 128, TM_DV = 256, TM_DK = 384;
};

__global__ void __launch_bounds__(BWD_THREADS, 1) attn_bwd_kernel(const __grid_constant__ AttnBwdParams p) {
  using Cfg = BwdCfg;
  extern __shared__ __align__(1024) uint8_t smem[];
  if (smem_u32(smem) & 1023) {   // swizzled tiles need it; the kernel has no other shared memory, so that the base is 1024
    if (threadIdx.x == 0 && p.status) atomicCAS(p.status, 0, ST_BAD_ARGUMENT);
    return;
  }
  uint8_t* sK = smem + Cfg::OFF_K;
  uint8_t* sV = smem + Cfg::OFF_V;
  uint8_t* sQ = smem + Cfg::OFF_Q;
  uint8_t* sdO = smem + Cfg::OFF_DO;
  uint8_t* sDST = smem + Cfg::OFF_DST;
  float* sStat = reinterpret_cast<float*>(smem + Cfg::OFF_STAT);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::OFF_BAR);
  uint64_t* kv_full = bars;          // 1
  uint64_t* q_full = bars + 1;       // [2]
  uint64_t* q_empty = bars + 3;      // [2]
  uint64_t* do_full = bars + 5;      // 1
  uint64_t* do_empty = bars + 6;     // [2] halves of the rows
  uint64_t* stat_full = bars + 8;    // [2], 1 arrival each
  uint64_t* s_full = bars + 10;      // 1
  uint64_t* dp_full = bars + 11;     // 1
  uint64_t* p_ready = bars + 12;     // 16 arrivals
  uint64_t* ds_ready = bars + 13;    // 16 arrivals
  uint64_t* dq_full = bars + 14;     // 1
  uint64_t* dq_drained = bars + 15;  // 8 arrivals: the dQ accumulator has been read out of TMEM
  uint64_t* all_done = bars + 16;    // 1: every MMA of the CTA has executed
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 17);
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
  // A last tile of at most 64 queries (-1: it has more): dV and dK reduce over those only, and the softmax warps of the columns behind them rest. Few
  // queries and several heads a group are a chain of such tiles: whole backward [1, 1, 28 / 4 heads] 22.2 us, 26.7 with whole tiles, 24.2 when a
  // tile had 64 queries and two were in flight; [1, 64 on 4096 keys, 28 / 4] 30.0, 34.2 and 31.5.
  const int qt_half = (p.Sq - 1) % BWD_Q < 64 ? n_qt_total - 1 : -1;

  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&q_full[i], 1);
      mbar_init(&q_empty[i], 1);
      mbar_init(&do_empty[i], 1);
      mbar_init(&stat_full[i], 1);
    }
    mbar_init(do_full, 1);
    mbar_init(s_full, 1);
    mbar_init(dp_full, 1);
    mbar_init(p_ready, BWD_SM_WARPS);
    mbar_init(ds_ready, BWD_SM_WARPS);
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

  auto tma5 = [](void* dst, const CUtensorMap* m, uint64_t* bar, int c1, int c2, int c3, int c4) {
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
        ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(0), "r"(c1), "r"(c2),
        "r"(c3), "r"(c4)
        : "memory");
  };

  if (warp == 0) {
    // ------------------------------------------------------------ loader: TMA tiles + LSE / delta rows
    if (n_it > 0) {
      if (lane == 0) {
        mbar_expect_tx(kv_full, 2 * Cfg::TILE_BYTES);
        tma5(sK, &p.tmK, kv_full, kv0, 0, kv_head, b);
        tma5(sV, &p.tmV, kv_full, kv0, 0, kv_head, b);
      }
      // LSE (scaled to log2) and delta of the 128 query rows of a tile, negated: lane i holds rows i, i + 32, i + 64 and i + 96. The loads run
      // two tiles ahead of their use so that their ~1 us latency never sits on the per-tile critical path.
      int ls_qt = qt_lo, ls_head = kv_head * G;              // next tile of load_stats, in turn
      auto load_stats = [&](float (&l)[4], float (&d)[4]) {
        const int qrow0 = ls_qt * BWD_Q;
        const long long so = ((long long)b * p.Hq + ls_head) * p.Sq + qrow0;
        if (++ls_qt == qt_hi) { ls_qt = qt_lo; ++ls_head; }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int row = lane + 32 * k;
          l[k] = -INFINITY; d[k] = 0.f;
          if (qrow0 + row < p.Sq) { l[k] = p.lse[so + row] * -1.4426950408889634f; d[k] = -p.delta[so + row]; }
        }
      };
      float cl[4], cd[4], nl[4] = {}, nd[4] = {};
      load_stats(cl, cd);
      if (n_it > 1) load_stats(nl, nd);
      int q_qt = qt_lo, q_head = kv_head * G;                // and of load_q
      auto load_q = [&](int it) {
        const int s = it & 1;
        if (!mbar_wait_warp(&q_empty[s], ((it >> 1) & 1) ^ 1, s_abort, p.status, ST_TIMEOUT_PRODUCER)) return false;
        if (lane == 0) {
          mbar_expect_tx(&q_full[s], Cfg::TILE_BYTES);
          tma5(sQ + s * Cfg::TILE_BYTES, &p.tmQ, &q_full[s], q_qt * BWD_Q, 0, q_head, b);
        }
        if (++q_qt == qt_hi) { q_qt = qt_lo; ++q_head; }
        return true;
      };
      bool ok = load_q(0);
      for (int it = 0, qt = qt_lo, head = kv_head * G; it < n_it && ok; ++it) {
        const int qrow0 = qt * BWD_Q;
        for (int h = 0; h < 2 && ok; ++h) {
          ok = mbar_wait_warp(&do_empty[h], (it & 1) ^ 1, s_abort, p.status, ST_TIMEOUT_PRODUCER);
          if (ok && lane == 0) {
            if (h == 0) mbar_expect_tx(do_full, Cfg::TILE_BYTES);
#pragma unroll
            for (int c = 0; c < 2; ++c) tma5(sdO + c * Cfg::SLAB + h * (Cfg::SLAB / 2), &p.tmdO, do_full, qrow0 + h * 64, c, head, b);
          }
        }
        if (!ok) break;
        if (++qt == qt_hi) { qt = qt_lo; ++head; }
        // the statistics of tile it - 2 were last read before dS^T(it - 2) was handed over, so before dV(it - 1), which freed dO
        float* st = sStat + (it & 1) * 256;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          st[lane + 32 * k] = cl[k];
          st[128 + lane + 32 * k] = cd[k];
          cl[k] = nl[k];
          cd[k] = nd[k];
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&stat_full[it & 1]);
        if (it + 1 < n_it) ok = load_q(it + 1);
        if (it + 2 < n_it) load_stats(nl, nd);
      }
    }
  } else if (warp == 1) {
    if (n_it > 0 && elect_one()) {
      constexpr uint32_t idesc_s = umma_idesc_f16(128, BWD_Q, 1, 0, 0);      // K Q^T, V dO^T
      constexpr uint32_t idesc_acc = umma_idesc_f16(128, BWD_D, 1, 0, 1);    // P^T dO, dS^T Q
      constexpr uint32_t idesc_dq = umma_idesc_f16(128, BWD_D, 1, 1, 1);     // dS K
      const uint32_t aK = smem_u32(sK), aV = smem_u32(sV), aDO = smem_u32(sdO), aDST = smem_u32(sDST);
      auto issue_nt = [&](uint32_t d, uint32_t a, uint32_t bt) {             // both operands row by row over the head-dim
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const uint32_t o = (k >> 2) * Cfg::SLAB + (k & 3) * 32;
          umma_f16_ss(d, umma_desc_sw128(a + o, 16, 1024), umma_desc_sw128(bt + o, 16, 1024), idesc_s, k ? 1u : 0u);
        }
      };
      auto q_ready = [&](int it) { return mbar_wait(&q_full[it & 1], (it >> 1) & 1, s_abort, p.status, ST_TIMEOUT_MMA); };
      bool ok = mbar_wait(kv_full, 0, s_abort, p.status, ST_TIMEOUT_MMA) && q_ready(0);
      if (ok) {
        tc_fence_after();
        issue_nt(tmem_base + Cfg::TM_S, aK, smem_u32(sQ));
        umma_commit(s_full);
        ok = mbar_wait(do_full, 0, s_abort, p.status, ST_TIMEOUT_MMA);
      }
      if (ok) {
        tc_fence_after();
        issue_nt(tmem_base + Cfg::TM_DP, aV, aDO);
        umma_commit(dp_full);
      }
      for (int it = 0, qt = qt_lo; it < n_it && ok; ++it) {
        const bool more = it + 1 < n_it;
        const int ks = qt == qt_half ? 4 : 8;              // K steps over the queries
        if (++qt == qt_hi) qt = qt_lo;
        const uint32_t q = smem_u32(sQ + (it & 1) * Cfg::TILE_BYTES);
        if (!mbar_wait(p_ready, it & 1, s_abort, p.status, ST_TIMEOUT_MMA)) { ok = false; break; }
        tc_fence_after();
        // dV += P^T dO (P^T read from TMEM)
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          if (k >= ks) break;
          umma_f16_ts(tmem_base + Cfg::TM_DV, tmem_base + Cfg::TM_S + k * 16, umma_desc_sw128(aDO + k * 2048, Cfg::SLAB, 1024), idesc_acc,
                      (it | k) ? 1u : 0u);
          if (k == 3) umma_commit(&do_empty[0]);
        }
        umma_commit(&do_empty[1]);
        // S^T of the next tile over P^T, which dV (issued before) has read
        if (more) {
          if (!q_ready(it + 1)) { ok = false; break; }
          tc_fence_after();
          issue_nt(tmem_base + Cfg::TM_S, aK, smem_u32(sQ + ((it + 1) & 1) * Cfg::TILE_BYTES));
          umma_commit(s_full);
        }
        if (!mbar_wait(ds_ready, it & 1, s_abort, p.status, ST_TIMEOUT_MMA)) { ok = false; break; }
        tc_fence_after();
        // dQ = dS K over dP^T, which every softmax warp has read
#pragma unroll
        for (int k = 0; k < 8; ++k)
          umma_f16_ss(tmem_base + Cfg::TM_DP, umma_desc_sw128(aDST + k * 2048, Cfg::SLAB, 1024), umma_desc_sw128(aK + k * 2048, Cfg::SLAB, 1024),
                      idesc_dq, k ? 1u : 0u);
        umma_commit(dq_full);
        // dK += dS^T Q
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          if (k >= ks) break;
          umma_f16_ss(tmem_base + Cfg::TM_DK, umma_desc_sw128(aDST + (k >> 2) * Cfg::SLAB + (k & 3) * 32, 16, 1024),
                      umma_desc_sw128(q + k * 2048, Cfg::SLAB, 1024), idesc_acc, (it | k) ? 1u : 0u);
        }
        umma_commit(&q_empty[it & 1]);
        if (more) {
          if (!mbar_wait(dq_drained, it & 1, s_abort, p.status, ST_TIMEOUT_MMA) ||
              !mbar_wait(do_full, (it + 1) & 1, s_abort, p.status, ST_TIMEOUT_MMA)) { ok = false; break; }
          tc_fence_after();
          issue_nt(tmem_base + Cfg::TM_DP, aV, aDO);
          umma_commit(dp_full);
        }
      }
      if (ok) umma_commit(all_done);
    }
  } else if (warp < 2 + BWD_SM_WARPS) {
    // ------------------------------------------------------------ softmax-gradient warps
    const int cg = (warp - 2) >> 2;     // group of 32 query columns; in the end: halves of dV and dK
    const int qd = warp & 3;            // TMEM lane quarter this warp may touch
    const int r = qd * 32 + lane;       // key row inside the tile == TMEM lane
    const int kv_idx = kv0 + r;
    const uint32_t lane_addr = static_cast<uint32_t>(qd * 32) << 16;
    const uint32_t tile = tmem_base + lane_addr + cg * 32;
    const uint64_t scale2 = pack_f32x2(p.scale_log2, p.scale_log2);
    // dS^T row of this key: 16-byte pieces of the column group, swizzled
    uint8_t* dst_row = sDST + (cg >> 1) * Cfg::SLAB + r * 128;
    const int piece0 = (cg & 1) * 4;
    bool ok = n_it > 0;
    for (int it = 0, qt = qt_lo; it < n_it && ok; ++it) {
      const int qrow0 = qt * BWD_Q;
      const bool idle = cg >= 2 && qt == qt_half;          // this warp's columns are behind the last query, and no product reads them
      if (++qt == qt_hi) qt = qt_lo;
      const bool need_mask = (p.causal && kv0 + BWD_KV - 1 > qrow0 + offset) || (kv0 + BWD_KV > p.Skv) ||
                             (p.window > 0 && kv0 < qrow0 + BWD_Q - 1 + offset - p.window + 1);
      const float* st = sStat + (it & 1) * 256 + cg * 32;
      if (!mbar_wait_warp(&stat_full[it & 1], (it >> 1) & 1, s_abort, p.status, ST_TIMEOUT_EPILOGUE)) { ok = false; break; }
      if (!mbar_wait_warp(s_full, it & 1, s_abort, p.status, ST_TIMEOUT_EPILOGUE)) { ok = false; break; }
      tc_fence_after();
      if (idle) {                                          // the barriers of the tile, in step with the others
        if (lane == 0) mbar_arrive(p_ready);
        if (!mbar_wait_warp(dp_full, it & 1, s_abort, p.status, ST_TIMEOUT_EPILOGUE)) { ok = false; break; }
        if (lane == 0) mbar_arrive(ds_ready);
        continue;
      }
      float pf[32];
      {
        uint32_t v[32];
        tmem_ld32(tile + Cfg::TM_S, v);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
          const ulonglong2 l2 = *reinterpret_cast<const ulonglong2*>(st + i);
          unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(v[i]), __uint_as_float(v[i + 1])), scale2, l2.x), pf[i], pf[i + 1]);
          unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(v[i + 2]), __uint_as_float(v[i + 3])), scale2, l2.y), pf[i + 2], pf[i + 3]);
#pragma unroll
          for (int k = 0; k < 4; ++k) pf[i + k] = exp2f(pf[i + k]);
        }
      }
      if (need_mask) {
        // query columns of this group that see the key: [lo, hi]
        const long long rel = (long long)kv_idx - offset - qrow0 - cg * 32;
        const int lo = kv_idx >= p.Skv ? 32 : (p.causal ? (int)min(max(rel, -1ll), 32ll) : -1);
        const int hi = p.window > 0 ? (int)min(max(rel + p.window - 1, -1ll), 31ll) : 31;
#pragma unroll
        for (int i = 0; i < 32; ++i)
          if (i < lo || i > hi) pf[i] = 0.f;
      }
      // The MMAs of tile it - 1 that read P^T were issued before S^T of this tile and one thread's MMAs execute in order: s_full covers them.
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float* f = pf + h * 16;
        asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(tile + Cfg::TM_S + h * 16),
                     "r"(pack_bf16x2(f[0], f[1])), "r"(pack_bf16x2(f[2], f[3])), "r"(pack_bf16x2(f[4], f[5])), "r"(pack_bf16x2(f[6], f[7])),
                     "r"(pack_bf16x2(f[8], f[9])), "r"(pack_bf16x2(f[10], f[11])), "r"(pack_bf16x2(f[12], f[13])), "r"(pack_bf16x2(f[14], f[15]))
                     : "memory");
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_ready);
      if (!mbar_wait_warp(dp_full, it & 1, s_abort, p.status, ST_TIMEOUT_EPILOGUE)) { ok = false; break; }
      tc_fence_after();
      // dS without the softmax scale: dK and dQ are scaled once when they are written out
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t v[16], ds[8];
        tmem_ld16(tile + Cfg::TM_DP + h * 16, v);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; i += 4) {
          const ulonglong2 d2 = *reinterpret_cast<const ulonglong2*>(st + 128 + h * 16 + i);
          const float* f = pf + h * 16 + i;
          float a0, a1;
          unpack_f32x2(mul_f32x2(pack_f32x2(f[0], f[1]), add_f32x2(pack_f32x2(__uint_as_float(v[i]), __uint_as_float(v[i + 1])), d2.x)), a0, a1);
          ds[i / 2] = pack_bf16x2(a0, a1);
          unpack_f32x2(mul_f32x2(pack_f32x2(f[2], f[3]), add_f32x2(pack_f32x2(__uint_as_float(v[i + 2]), __uint_as_float(v[i + 3])), d2.y)), a0, a1);
          ds[i / 2 + 1] = pack_bf16x2(a0, a1);
        }
        // dQ and dK of tile it - 1, which read this buffer, were issued before dP^T of this tile: dp_full covers them
#pragma unroll
        for (int k = 0; k < 2; ++k)
          *reinterpret_cast<uint4*>(dst_row + (((piece0 + h * 2 + k) ^ (r & 7)) << 4)) =
              make_uint4(ds[k * 4], ds[k * 4 + 1], ds[k * 4 + 2], ds[k * 4 + 3]);
      }
      fence_proxy_async_smem();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(ds_ready);
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
    // dQ tile in TMEM: lane = query row, column = head-dim index. Each warp owns 32 query rows and half of the columns, which it takes into
    // registers at once: dP^T of the next tile waits for that. Then 4 KB (32 columns) at a time are staged in shared memory and added into the
    // warp's piece of dq_accum with a bulk reduction.
    const int qd = warp & 3, half = (warp - 2 - BWD_SM_WARPS) >> 2;
    const uint32_t src = tmem_base + Cfg::TM_DP + (static_cast<uint32_t>(qd * 32) << 16) + half * 64;
    const uint32_t stage = smem_u32(smem + Cfg::OFF_DQS + (warp - 2 - BWD_SM_WARPS) * 4096);
    int head = b * p.Hq + kv_head * G;
    bool ok = true;
    for (int it = 0, qt = qt_lo; it < n_it && ok; ++it) {
      if (!mbar_wait_warp(dq_full, it & 1, s_abort, p.status, ST_TIMEOUT_EPILOGUE)) { ok = false; break; }
      tc_fence_after();
      uint32_t v[2][32];
      tmem_ld32(src, v[0]);
      tmem_ld32(src + 32, v[1]);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(dq_drained);
      const int piece = qt * 4 + qd, pieces = bwd_pieces(p.Sq);
      if (piece < pieces) {   // the last tile may reach behind the accumulator: those queries do not exist
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // the stage has been read
          __syncwarp();
#pragma unroll
          for (int c = 0; c < 8; ++c)
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(stage + c * 512 + lane * 16), "r"(v[k][c * 4]), "r"(v[k][c * 4 + 1]),
                         "r"(v[k][c * 4 + 2]), "r"(v[k][c * 4 + 3])
                         : "memory");
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            float* dst = p.dq_accum + ((long long)head * pieces + piece) * 4096 + half * 2048 + k * 1024;
            asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f32 [%0], [%1], %2;" ::"l"(dst), "r"(stage), "r"(4096)
                         : "memory");
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          }
        }
      }
      if (++qt == qt_hi) { qt = qt_lo; ++head; }
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
// pairs of pieces, 64 queries, so few queries leave more to zero than their rows have CTAs for: CTAs behind the last row only zero
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

// dq_accum (tiled as the backward kernel writes it) * scale -> bf16 dQ rows. One CTA a piece of 32 queries. What bounds it is how many parts of lines
// a warp touches: its lanes take 4 queries by 8 groups of 4 columns, so that a load reads 64 contiguous bytes of each group and a store writes 64 of
// each row. [1, 4096, 32 heads] 14.7 us = 6.8 TB/s, a part of it from L2 (30.4 with 32 queries a warp, which wrote 8 bytes of each of 32 rows; 8 queries by 4 groups 15.9,
// 2 by 16 16.5), 16384 tokens 61.5 us (142; 66; 70). A CTA that walks several pieces is slower by 1 us and 9 us.
__global__ void __launch_bounds__(256) attn_dq_convert_kernel(const float* __restrict__ acc, __nv_bfloat16* __restrict__ dQ, int Sq, int Hq,
                                                              long long dq_row_stride, float scale) {
  const unsigned pieces = bwd_pieces(Sq), piece = blockIdx.x % pieces, bh = blockIdx.x / pieces;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int rows = Sq - (int)piece * 32;   // queries of the piece (0 or less in the padding of Sq to 64)
  const float4* a = reinterpret_cast<const float4*>(acc) + (long long)blockIdx.x * 1024;
  __nv_bfloat16* o = dQ + ((long long)(bh / Hq) * Sq + piece * 32) * dq_row_stride + (long long)(bh % Hq) * BWD_D;
  float4 v[4];
  int q[4], g[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int part = warp * 4 + k;         // 8 parts of 4 queries, 4 parts of 8 groups
    q[k] = part % 8 * 4 + lane % 4;
    g[k] = part / 8 * 8 + lane / 4;
    if (q[k] < rows) v[k] = a[g[k] * 32 + q[k]];
  }
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (q[k] < rows)
      *reinterpret_cast<uint2*>(o + q[k] * dq_row_stride + g[k] * 4) =
          make_uint2(pack_bf16x2(v[k].x * scale, v[k].y * scale), pack_bf16x2(v[k].z * scale, v[k].w * scale));
}

static int make_attn_map_bwd(CUtensorMap* tm, const void* base, int B, int S, int H, int D, long long row_stride,
                             long long batch_stride, int box_rows, int box_slabs) {
  uint64_t dims[5] = {64, (uint64_t)S, (uint64_t)(D / 64), (uint64_t)H, (uint64_t)B};
  uint64_t strides[4] = {(uint64_t)row_stride * 2, 128, (uint64_t)D * 2, (uint64_t)batch_stride * 2};
  uint32_t box[5] = {64, (uint32_t)box_rows, (uint32_t)box_slabs, 1, 1};
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
  int rc = make_attn_map_bwd(&p.tmQ, a->Q, a->B, a->Sq, a->Hq, a->D, a->q_row_stride, a->q_batch_stride, BWD_Q, 2);
  if (rc) return rc;
  rc = make_attn_map_bwd(&p.tmdO, a->dO, a->B, a->Sq, a->Hq, a->D, a->do_row_stride, (long long)a->Sq * a->do_row_stride,
                         64, 1);
  if (rc) return rc;
  rc = make_attn_map_bwd(&p.tmK, a->K, a->B, a->Skv, a->Hk, a->D, a->k_row_stride, a->k_batch_stride, BWD_KV, 2);
  if (rc) return rc;
  rc = make_attn_map_bwd(&p.tmV, a->V, a->B, a->Skv, a->Hk, a->D, a->v_row_stride, a->v_batch_stride, BWD_KV, 2);
  if (rc) return rc;
  const long long tokens = (long long)a->B * a->Sq;
  const long long acc_floats = (long long)a->B * a->Hq * bwd_pieces(a->Sq) * 32 * BWD_D;
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
  attn_dq_convert_kernel<<<(unsigned)(acc_floats / (32 * BWD_D)), 256, 0, st>>>(a->dq_accum, (__nv_bfloat16*)a->dQ, a->Sq, a->Hq,
                                                                             a->dq_row_stride, a->scale);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}
