// A1: flash attention forward on tcgen05 (sm_100a).
//
// One CTA owns 256 query rows of one (batch, head) as two 128-row tiles X in {A, B}, each served
// by its own softmax warpgroup, and walks the visible 128-row KV tiles:
//   S   = Q_X K^T       tcgen05.mma SS, fp32 in TMEM
//   P_X = exp2(S - m)   one query row per thread (TMEM lane == row, no shuffles), packed bf16 in TMEM
//   O_X += P_X V        tcgen05.mma TS: P straight from TMEM, V consumed MN-major from its [kv, d] tile
// Both tiles take turns with one S: a warpgroup has its scores in registers (setmaxnreg: 216 a thread) before it works on them, so that the next
// product may follow at once, and P has columns of its own. A tile's scores are then ready when its warpgroup is, and the row's chain of maximum,
// 128 exponentials and sum is all that a step of it waits for. With P over S, S had to wait for O += P V of the step before, which was a third of
// a step, whatever the exponentials cost (half of them as polynomials: slower; 16 softmax warps, half a row each: slower). The MMA warp issues the
// score products two items (tile, step) ahead of P V, in a fixed order: taking whichever is ready first was slower, the tiles fall into step.
// The running max is only refreshed when it grew by more than 2^8, so rescaling O in TMEM is rare.
// Causal / sliding-window masks, GQA head
// mapping and the differential-attention V mapping (two score heads share one V head) are index
// arithmetic; nothing is materialised. An optional block mask (one byte per 128 x 128 score tile, per head or
// shared) removes whole tiles from the walk: a step whose tile is masked for both query tiles is neither loaded nor
// multiplied (block-sparse / flex-attention patterns at tile granularity).
// Bound: exponentials (16 a cycle and SM: 2048 cycles for a step of both tiles, as many as its products take). B200, warm, captured calls, with one S a
// tile -> now: [1, 4096, 32 / 8 heads, 128] causal 191 -> 135 us, [1, 8192, 8 / 2] full 281 -> 240, [8, 512, 28 / 4] causal 55 -> 43, [1, 16384, 32 / 8]
// causal 2.28 -> 2.00 ms (1100 TFLOP/s, at the power cap). A block of one step is a chain from launch to store: [64, 128, 32 / 8] full 92 us either
// way, 101 when the first loads came behind the block's set-up and each quarter of a row asked for a mask.
// Takes the place of the reference's SIMT flash-attention forward, GQA and block-sparse kernels
// (kernel/cuda/attention_cuda.cu:37-328, 498-573, 1154-1230) and its empty "v3" kernel (:1262-1286).
#include <limits.h>
#include "tc_common.cuh"
#include "tmap.h"
#include "sx_api.h"

namespace sx {

constexpr int ATT_BM = 128;   // rows per q tile (two per CTA)
constexpr int ATT_BN = 128;
// 2 x 4 softmax warps, TMA warp, MMA warp, two idle ones: the last four give registers to the softmax warps, which hold a row of 128 scores
// (2 x 128 x 216 + 128 x 72 = 384 x 168, what the block is launched with; more than that would never be granted, so the launch checks it)
constexpr int ATT_THREADS = 384, ATT_TMA_WARP = 8, ATT_MMA_WARP = 9;
constexpr int ATT_REGS = 168;

struct AttnFwdParams {
  CUtensorMap tmQ, tmK, tmV;
  __nv_bfloat16* O;   // [B, Sq, Hq, D]
  float* lse;         // [B, Hq, Sq]  (natural log)
  int* status;
  long long o_row_stride;  // elements between consecutive tokens of O
  int B, Sq, Skv, Hq, Hk;
  int v_head_div;  // V head = (K head) / v_head_div
  int causal, window;  // window <= 0: unlimited
  int pairs, order;    // pairs of query tiles; what the grid's axes are, see sx_attn_fwd
  float scale_log2;    // softmax scale * log2(e)
  const uint8_t* block_mask;   // optional [B or 1][Hq or 1][q tiles][kv tiles], non-zero = tile takes part
  long long bm_batch_stride, bm_head_stride;
  int bm_kv_tiles;
};

template <int D>
struct AttnCfg {
  static constexpr int Q_BYTES = ATT_BM * D * 2;   // one q tile
  static constexpr int KV_BYTES = ATT_BN * D * 2;
  static constexpr int OFF_K = 2 * Q_BYTES;
  static constexpr int OFF_V = OFF_K + 2 * KV_BYTES;
  static constexpr int OFF_BAR = OFF_V + 2 * KV_BYTES;
  static constexpr int SMEM_BYTES = OFF_BAR + 256 + 1024;
  // TMEM columns: S of whichever tile's turn it is, P of tiles A and B (bf16 pairs), O of both
  static constexpr uint32_t TMEM_COLS = 512, TM_S = 0, TM_P = 128, TM_O = 256;
};

// Visible KV tile range [lo, hi) of a 128-row q tile starting at q0.
__device__ __forceinline__ void kv_range(const AttnFwdParams& p, int q0, int& lo, int& hi) {
  const int offset = p.Skv - p.Sq;
  lo = 0;
  hi = (p.Skv + ATT_BN - 1) / ATT_BN;
  if (q0 >= p.Sq) { hi = 0; return; }
  if (p.causal) {
    const int last = q0 + ATT_BM - 1 + offset;
    hi = last < 0 ? 0 : min(hi, last / ATT_BN + 1);
  }
  if (p.window > 0) {
    const int first = q0 + offset - p.window + 1;
    if (first > 0) lo = first / ATT_BN;
  }
  if (hi < lo) hi = lo;
}

template <int D, bool MASK>
__global__ void __launch_bounds__(ATT_THREADS, 1) attn_fwd_kernel(const __grid_constant__ AttnFwdParams p) {
  using Cfg = AttnCfg<D>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;
  uint8_t* sK = smem + Cfg::OFF_K;
  uint8_t* sV = smem + Cfg::OFF_V;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::OFF_BAR);
  uint64_t* q_full = bars;            // 1
  uint64_t* k_full = bars + 1;        // [2]
  uint64_t* k_empty = bars + 3;       // [2]
  uint64_t* v_full = bars + 5;        // [2]
  uint64_t* v_empty = bars + 7;       // [2]
  uint64_t* s_full = bars + 9;        // [2 tiles]
  uint64_t* p_full = bars + 11;       // [2 tiles]
  uint64_t* pv_done = bars + 13;      // [2 tiles]
  uint64_t* s_free = bars + 15;       // 1
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 16);
  volatile int* s_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = warp_index(), lane = threadIdx.x & 31;
  const unsigned ax = blockIdx.x, ay = blockIdx.y, az = blockIdx.z;
  const int head = p.order < 2 ? ax : ay;
  const int b = p.order == 0 ? ay : p.order == 2 ? ax : az;
  const int pair = p.pairs - 1 - (int)(p.order == 1 ? ay : p.order == 3 ? ax : az);
  const int kv_head = head / (p.Hq / p.Hk);
  const int v_head = kv_head / p.v_head_div;
  const int q0 = pair * 2 * ATT_BM;

  int lo[2], hi[2];
  kv_range(p, q0, lo[0], hi[0]);
  kv_range(p, q0 + ATT_BM, lo[1], hi[1]);
  // union range walked by the loaders; tile X takes part in step j when lo[X] <= j < hi[X]
  int jlo = INT_MAX, jhi = 0;
#pragma unroll
  for (int x = 0; x < 2; ++x)
    if (hi[x] > lo[x]) { jlo = min(jlo, lo[x]); jhi = max(jhi, hi[x]); }
  // tile X takes part in the step of kv tile jt?
  const uint8_t* bm = MASK ? p.block_mask + b * p.bm_batch_stride + head * p.bm_head_stride : nullptr;
  auto on = [&](int x, int jt) -> bool {
    if (jt < lo[x] || jt >= hi[x]) return false;
    if constexpr (!MASK) return true;
    else return bm[(long long)(pair * 2 + x) * p.bm_kv_tiles + jt] != 0;
  };
  // next kv tile after jt that any of the two tiles takes part in (-1: none)
  auto next_step = [&](int jt) -> int {
    if constexpr (!MASK) {
      return jt + 1 < jhi ? jt + 1 : -1;   // without a mask every tile of the union range is taken
    } else {
      for (++jt; jt < jhi; ++jt)
        if (on(0, jt) || on(1, jt)) return jt;
      return -1;
    }
  };
  const int first_step = jhi > jlo ? next_step(jlo - 1) : -1;
  const int n_steps = first_step >= 0 ? 1 : 0;   // only "are there any" is used below

  auto tma5 = [](void* dst, const CUtensorMap* m, uint64_t* bar, int c1, int c3, int c4) {
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
        ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(0), "r"(c1), "r"(0),
        "r"(c3), "r"(c4)
        : "memory");
  };

  // The loader sets up the barriers and sends for the first tiles while the other warps get TMEM and meet: a block of one step takes 12 thousand cycles,
  // 1.5 of them up to there.
  if (warp == ATT_TMA_WARP && elect_one()) {
    mbar_init(q_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&k_full[i], 1);
      mbar_init(&k_empty[i], 1);
      mbar_init(&v_full[i], 1);
      mbar_init(&v_empty[i], 1);
      mbar_init(&s_full[i], 1);
      mbar_init(&p_full[i], 4);
      mbar_init(&pv_done[i], 1);
    }
    mbar_init(s_free, 4);
    *s_abort = 0;
    mbar_fence_init();
    fence_proxy_async_smem();
    if (n_steps > 0) {
      mbar_expect_tx(q_full, 2 * Cfg::Q_BYTES);
      tma5(sQ, &p.tmQ, q_full, q0, head, b);
      tma5(sQ + Cfg::Q_BYTES, &p.tmQ, q_full, q0 + ATT_BM, head, b);
      mbar_expect_tx(&k_full[0], Cfg::KV_BYTES);
      tma5(sK, &p.tmK, &k_full[0], first_step * ATT_BN, kv_head, b);
      mbar_expect_tx(&v_full[0], Cfg::KV_BYTES);
      tma5(sV, &p.tmV, &v_full[0], first_step * ATT_BN, v_head, b);
    }
  }
  __syncwarp();
  if (warp == ATT_MMA_WARP) tmem_alloc(tmem_slot, Cfg::TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp >= 8) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
    if (warp == ATT_TMA_WARP) {
      // ------------------------------------------------------------ TMA producer
      if (n_steps > 0 && elect_one()) {
        int j = 1;   // steps taken so far: the first one is on its way
        for (int jt = next_step(first_step); jt >= 0; jt = next_step(jt), ++j) {
          const int s = j & 1;
          const uint32_t ph = (j >> 1) & 1;
          const int kv0 = jt * ATT_BN;
          if (!mbar_wait(&k_empty[s], ph ^ 1, s_abort, p.status, ST_TIMEOUT_PRODUCER)) break;
          mbar_expect_tx(&k_full[s], Cfg::KV_BYTES);
          tma5(sK + s * Cfg::KV_BYTES, &p.tmK, &k_full[s], kv0, kv_head, b);
          if (!mbar_wait(&v_empty[s], ph ^ 1, s_abort, p.status, ST_TIMEOUT_PRODUCER)) break;
          mbar_expect_tx(&v_full[s], Cfg::KV_BYTES);
          tma5(sV + s * Cfg::KV_BYTES, &p.tmV, &v_full[s], kv0, v_head, b);
        }
      }
    } else if (warp == ATT_MMA_WARP) {
      // ------------------------------------------------------------ MMA issuer
      if (n_steps > 0 && elect_one()) {
        constexpr uint32_t idesc_qk = umma_idesc_f16(ATT_BM, ATT_BN, 1, 0, 0);
        constexpr uint32_t idesc_pv = umma_idesc_f16(ATT_BM, D, 1, 0, 1);
        bool ok = mbar_wait(q_full, 0, s_abort, p.status, ST_TIMEOUT_MMA);
        int cnt_a = 0, cnt_b = 0;                // products P V so far
        // O_x += P_x V of the step in ring slot j & 1; `last`: nobody else multiplies this V
        auto do_pv = [&](int x, int j, bool last) -> bool {
          const int done = x ? cnt_b : cnt_a;
          if (!mbar_wait(&v_full[j & 1], (j >> 1) & 1, s_abort, p.status, ST_TIMEOUT_MMA) ||
              !mbar_wait(&p_full[x], done & 1, s_abort, p.status, ST_TIMEOUT_MMA)) return false;
          tc_fence_after();
          const uint32_t b0 = smem_u32(sV + (j & 1) * Cfg::KV_BYTES);
          const uint32_t dO = tmem_base + Cfg::TM_O + x * 128, aP = tmem_base + Cfg::TM_P + x * 64;
#pragma unroll
          for (int k = 0; k < 8; ++k)
            umma_f16_ts(dO, aP + k * 8, umma_desc_sw128(b0 + k * 2048, ATT_BN * 128, 1024), idesc_pv, (done | k) ? 1u : 0u);
          umma_commit(&pv_done[x]);
          if (last) umma_commit(&v_empty[j & 1]);
          cnt_a += x ^ 1;
          cnt_b += x;
          return true;
        };
        // Products S = Q K^T in the order A, B, A, B ... of the tiles that take part in a step, two ahead of the products P V
        int i = 0, x1 = 0, j1 = 0, x2 = 0, j2 = 0;
        int j = 0;
        for (int jt = first_step; jt >= 0 && ok; jt = next_step(jt), ++j) {
          if (!mbar_wait(&k_full[j & 1], (j >> 1) & 1, s_abort, p.status, ST_TIMEOUT_MMA)) { ok = false; break; }
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            if (!ok || !on(x, jt)) continue;
            if (i > 0 && !mbar_wait(s_free, (i - 1) & 1, s_abort, p.status, ST_TIMEOUT_MMA)) { ok = false; continue; }
            tc_fence_after();
            const uint32_t a0 = smem_u32(sQ + x * Cfg::Q_BYTES), b0 = smem_u32(sK + (j & 1) * Cfg::KV_BYTES);
#pragma unroll
            for (int c = 0; c < D / 64; ++c)
#pragma unroll
              for (int k = 0; k < 4; ++k)
                umma_f16_ss(tmem_base + Cfg::TM_S, umma_desc_sw128(a0 + c * (ATT_BM * 128) + k * 32, 16, 1024),
                            umma_desc_sw128(b0 + c * (ATT_BN * 128) + k * 32, 16, 1024), idesc_qk, (c | k) ? 1u : 0u);
            umma_commit(&s_full[x]);
            if (i >= 2) ok = do_pv(x2, j2, j1 != j2);
            x2 = x1; j2 = j1; x1 = x; j1 = j;
            ++i;
          }
          if (ok) umma_commit(&k_empty[j & 1]);
        }
        if (ok && i >= 2) ok = do_pv(x2, j2, j1 != j2);
        if (ok && i >= 1) do_pv(x1, j1, true);
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
    // ------------------------------------------------------------ softmax warpgroups
    const int x = warp >> 2;                // which q tile
    const int qd = warp & 3;                // TMEM lane quadrant of this warp
    const int row = qd * 32 + lane;         // row inside the tile == TMEM lane
    const int q_idx = q0 + x * ATT_BM + row;
    const int offset = p.Skv - p.Sq;
    const uint32_t lane_addr = static_cast<uint32_t>(qd * 32) << 16;
    const uint32_t tS = tmem_base + Cfg::TM_S + lane_addr, tP = tmem_base + Cfg::TM_P + x * 64 + lane_addr;
    const uint32_t tO = tmem_base + Cfg::TM_O + x * 128 + lane_addr;
    const int my_lo = x ? lo[1] : lo[0], my_hi = x ? hi[1] : hi[0];
    auto mine = [&](int jt) -> bool {
      if constexpr (!MASK) return true;
      else return bm[(long long)(pair * 2 + x) * p.bm_kv_tiles + jt] != 0;
    };
    int n_mine = 0;   // steps this tile takes part in
    for (int jt = my_lo; jt < my_hi; ++jt) n_mine += mine(jt) ? 1 : 0;
    float m_used = -INFINITY;  // running (possibly stale) max, log2 domain
    float l = 0.f;
    bool ok = true;
    // visible keys of this row: [lo_k, hi_k]
    const int hi_k = p.causal ? min(p.Skv - 1, q_idx + offset) : p.Skv - 1;
    const int lo_k = p.window > 0 ? (int)max((long long)q_idx + offset - p.window + 1, -1ll) : -1;
    const int qt0 = q0 + x * ATT_BM;
    // tiles from this one on have keys that some row does not see; before lo_full, too, where there is a window
    const int hi_full = (min(p.Skv, p.causal ? qt0 + offset + 1 : p.Skv)) / ATT_BN;
    const int lo_full = p.window > 0 ? (int)max((long long)qt0 + ATT_BM - 1 + offset - p.window + 1, 0ll) : 0;
    const uint64_t scale2 = pack_f32x2(p.scale_log2, p.scale_log2);
    for (int jt = my_lo, j = 0; jt < my_hi && ok; ++jt) {
      if (!mine(jt)) continue;
      if (!mbar_wait_warp(&s_full[x], j & 1, s_abort, p.status, ST_TIMEOUT_EPILOGUE)) { ok = false; break; }
      tc_fence_after();
      const bool need_mask = jt >= hi_full || jt * ATT_BN < lo_full;
      uint32_t r[ATT_BN];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld32(tS + c * 32, *reinterpret_cast<uint32_t(*)[32]>(&r[c * 32]));
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(s_free);      // the other tile's scores may follow
      // four chains of three-operand maxima: one chain of 128 dependent ones takes as long as the exponentials of half a tile
      float mc[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
      if (need_mask) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const int h = hi_k - jt * ATT_BN - c * 32, w = lo_k - jt * ATT_BN - c * 32;
          const uint32_t seen = (h >= 31 ? 0xffffffffu : h < 0 ? 0u : (2u << h) - 1u) & (w <= 0 ? 0xffffffffu : w > 31 ? 0u : 0xffffffffu << w);
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (!(seen & (1u << i))) r[c * 32 + i] = 0xff800000u;  // -inf
        }
      }
#pragma unroll
      for (int i = 0; i < ATT_BN; i += 8)
#pragma unroll
        for (int k = 0; k < 4; ++k) mc[k] = fmax3(mc[k], __uint_as_float(r[i + 2 * k]), __uint_as_float(r[i + 2 * k + 1]));
      const float mx = fmaxf(fmax3(mc[0], mc[1], mc[2]), mc[3]) * p.scale_log2;
      float alpha = 1.f;
      bool rescale = false;
      if ((mx > m_used + 8.f || m_used == -INFINITY) && mx != -INFINITY) {
        alpha = (m_used == -INFINITY) ? 0.f : exp2f(m_used - mx);
        rescale = (m_used != -INFINITY);
        m_used = mx;
      }
      l *= alpha;
      if (j > 0 && __any_sync(0xffffffffu, rescale)) {
        if (!mbar_wait_warp(&pv_done[x], (j - 1) & 1, s_abort, p.status, ST_TIMEOUT_EPILOGUE)) { ok = false; break; }
        tc_fence_after();
#pragma unroll 1
        for (int c = 0; c < D / 16; ++c) {
          uint32_t o[16];
          tmem_ld16(tO + c * 16, o);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
          tmem_st16(tO + c * 16, o);
        }
      }
      const float m_sub = (m_used == -INFINITY) ? 0.f : m_used;
      const uint64_t m2 = pack_f32x2(-m_sub, -m_sub);
      float lsum = 0.f;
      auto exps = [&](int i0, int i1) {
#pragma unroll
        for (int i = i0; i < i1; i += 2) {
          const uint64_t e = fma_f32x2(pack_f32x2(__uint_as_float(r[i]), __uint_as_float(r[i + 1])), scale2, m2);
          float v0, v1;
          unpack_f32x2(e, v0, v1);
          const uint32_t pb = pack_bf16x2(exp2f(v0), exp2f(v1));
          r[i / 2] = pb;
          // row sum from the rounded values so that l matches what P V sees, in the order of the keys
          lsum += add_bf16x2(pb);
        }
      };
      exps(0, 64);
      // P V of the step before has read P
      if (j > 0) {
        if (!mbar_wait_warp(&pv_done[x], (j - 1) & 1, s_abort, p.status, ST_TIMEOUT_EPILOGUE)) { ok = false; break; }
        tc_fence_after();
      }
      tmem_st32(tP, *reinterpret_cast<uint32_t(*)[32]>(&r[0]));
      exps(64, 128);
      tmem_st32(tP + 32, *reinterpret_cast<uint32_t(*)[32]>(&r[32]));
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[x]);
      l += lsum;
      ++j;
    }
    if (ok && n_mine > 0) {
      if (mbar_wait_warp(&pv_done[x], (n_mine - 1) & 1, s_abort, p.status, ST_TIMEOUT_EPILOGUE)) {
        tc_fence_after();
        const float inv_l = l > 0.f ? 1.f / l : 0.f;
        const bool row_ok = q_idx < p.Sq;
        __nv_bfloat16* orow = p.O + ((long long)b * p.Sq + q_idx) * p.o_row_stride + (long long)head * D;
#pragma unroll 1
        for (int c = 0; c < D / 32; ++c) {
          uint32_t o[32];
          tmem_ld32(tO + c * 32, o);
          tmem_ld_wait();
          if (row_ok) {
#pragma unroll
            for (int i = 0; i < 32; i += 8) {
              uint4 w;
              w.x = pack_bf16x2(__uint_as_float(o[i]) * inv_l, __uint_as_float(o[i + 1]) * inv_l);
              w.y = pack_bf16x2(__uint_as_float(o[i + 2]) * inv_l, __uint_as_float(o[i + 3]) * inv_l);
              w.z = pack_bf16x2(__uint_as_float(o[i + 4]) * inv_l, __uint_as_float(o[i + 5]) * inv_l);
              w.w = pack_bf16x2(__uint_as_float(o[i + 6]) * inv_l, __uint_as_float(o[i + 7]) * inv_l);
              *reinterpret_cast<uint4*>(orow + c * 32 + i) = w;
            }
          }
        }
        if (row_ok && p.lse)
          p.lse[((long long)b * p.Hq + head) * p.Sq + q_idx] =
              (l > 0.f) ? (m_used + log2f(l)) * 0.6931471805599453f : -INFINITY;
      }
    } else if (n_mine <= 0) {
      // no visible keys for this tile: zero output
      if (q_idx < p.Sq) {
        __nv_bfloat16* orow = p.O + ((long long)b * p.Sq + q_idx) * p.o_row_stride + (long long)head * D;
        for (int i = 0; i < D; i += 8) *reinterpret_cast<uint4*>(orow + i) = make_uint4(0, 0, 0, 0);
        if (p.lse) p.lse[((long long)b * p.Hq + head) * p.Sq + q_idx] = -INFINITY;
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (*s_abort) bounded_delay_ns(2000000);
  if (warp == ATT_MMA_WARP) {
    tc_fence_after();
    tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
  }
}

// 5-D map over a [B, S, H, D] view (token stride `row_stride` elements): dims
// {64, S, D/64, H, B}; one box brings a [128 tokens x D] tile as D/64 swizzled 128-byte-row slabs.
static int make_attn_map(CUtensorMap* tm, const void* base, int B, int S, int H, int D, long long row_stride,
                         long long batch_stride, int box_rows) {
  uint64_t dims[5] = {64, (uint64_t)S, (uint64_t)(D / 64), (uint64_t)H, (uint64_t)B};
  uint64_t strides[4] = {(uint64_t)row_stride * 2, 128, (uint64_t)D * 2, (uint64_t)batch_stride * 2};
  uint32_t box[5] = {64, (uint32_t)box_rows, (uint32_t)(D / 64), 1, 1};
  return make_tmap(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, base, dims, strides, box);
}

template <int D, bool MASK>
static int attn_fwd_launch(const AttnFwdParams& p, dim3 grid, cudaStream_t st) {
  static bool set = false;
  if (!set) {
    cudaFuncAttributes fa;
    if (cudaFuncSetAttribute(attn_fwd_kernel<D, MASK>, cudaFuncAttributeMaxDynamicSharedMemorySize, AttnCfg<D>::SMEM_BYTES) != cudaSuccess ||
        cudaFuncGetAttributes(&fa, attn_fwd_kernel<D, MASK>) != cudaSuccess) return -10;
    if (fa.numRegs < ATT_REGS) return -12;
    set = true;
  }
  attn_fwd_kernel<D, MASK><<<grid, ATT_THREADS, AttnCfg<D>::SMEM_BYTES, st>>>(p);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

}  // namespace sx
using namespace sx;

extern "C" int sx_attn_fwd(const SxAttnArgs* a, cudaStream_t st) {
  if (a->D != 64 && a->D != 128) return -1;
  if (a->Hq % a->Hk) return -2;
  if ((a->q_row_stride % 8) || (a->k_row_stride % 8) || (a->v_row_stride % 8) || (a->o_row_stride % 8)) return -3;
  AttnFwdParams p;
  const int v_heads = a->Hk / (a->v_head_div > 0 ? a->v_head_div : 1);
  int rc = make_attn_map(&p.tmQ, a->Q, a->B, a->Sq, a->Hq, a->D, a->q_row_stride, a->q_batch_stride, ATT_BM);
  if (rc) return rc;
  rc = make_attn_map(&p.tmK, a->K, a->B, a->Skv, a->Hk, a->D, a->k_row_stride, a->k_batch_stride, ATT_BN);
  if (rc) return rc;
  rc = make_attn_map(&p.tmV, a->V, a->B, a->Skv, v_heads, a->D, a->v_row_stride, a->v_batch_stride, ATT_BN);
  if (rc) return rc;
  p.O = (__nv_bfloat16*)a->O;
  p.lse = a->lse;
  p.status = a->status;
  p.o_row_stride = a->o_row_stride;
  p.B = a->B; p.Sq = a->Sq; p.Skv = a->Skv; p.Hq = a->Hq; p.Hk = a->Hk;
  p.v_head_div = a->v_head_div > 0 ? a->v_head_div : 1;
  p.causal = a->causal; p.window = a->window;
  p.scale_log2 = a->scale * 1.4426950408889634f;
  p.block_mask = (const uint8_t*)a->block_mask;
  p.bm_batch_stride = a->bm_batch_stride;
  p.bm_head_stride = a->bm_head_stride;
  p.bm_kv_tiles = (a->Skv + ATT_BN - 1) / ATT_BN;
  // Blocks start heaviest first, so that the last ones to start are short: under a causal mask the last pair of query tiles walks the most keys.
  // Heads are next to one another. Then the whole batch where its keys and values stay in L2; otherwise one sequence after another, where the pairs
  // of tiles that run at the same time share what they read. The grid's axes are the three indices themselves (three divisions less in front of a
  // block's first load, 450 cycles); only x holds more than 65535.
  p.pairs = (a->Sq + 2 * ATT_BM - 1) / (2 * ATT_BM);
  const bool batch_first = (long long)a->B * a->Skv * (a->Hk + v_heads) * a->D * 2 <= (64ll << 20);
  p.order = a->B > 65535 ? 2 : p.pairs > 65535 ? 3 : batch_first ? 0 : 1;
  const dim3 grids[4] = {dim3(a->Hq, a->B, p.pairs), dim3(a->Hq, p.pairs, a->B), dim3(a->B, a->Hq, p.pairs), dim3(p.pairs, a->Hq, a->B)};
  const dim3 grid = grids[p.order];
  if (grid.x == 0 || grid.y == 0 || grid.z == 0 || grid.y > 65535 || grid.z > 65535 || (long long)grid.x * grid.y * grid.z > INT_MAX) return -4;
  const bool masked = p.block_mask != nullptr;
  if (a->D == 128) return masked ? attn_fwd_launch<128, true>(p, grid, st) : attn_fwd_launch<128, false>(p, grid, st);
  return masked ? attn_fwd_launch<64, true>(p, grid, st) : attn_fwd_launch<64, false>(p, grid, st);
}
