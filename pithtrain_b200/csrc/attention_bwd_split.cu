// Attention backward that keeps all 24 bits of P and dS, for sm_100a (tcgen05 / TMEM / TMA): head dims 64, 128, 192/128
// (MLA) and 256, any sequence length, with the masks of the forward kernel. It covers what csrc/attention_bwd.cu does
// not (wider heads, lengths that are no multiple of 4), where gradients come from unrounded probabilities:
//   P = hi + mid + lo and dS likewise, three bf16 numbers of 8 bits each (what is left is below 2^-25 of the value), so every
//   product with them is three MMAs into the same fp32 accumulator. S and dP need no split: their operands are bf16.
// Error of the fp32 sums of dV against 64 bits, causal, 64 / 517 / 2048 rows: 5e-7 / 2.6e-6 / 9e-6 (two terms: 2.2e-6 / 3.0e-6 /
// 7.9e-6; fp32 tensor ops: 2.4e-7 / 5.4e-7 / 1.1e-6). At short lengths the terms decide, at long ones that the tensor core cuts
// its fp32 sums off where FMAs round them. The bf16 gradients do not tell the three apart: 1.655e-3 +- 1e-7 each at 3072 rows.
// Two terms did show where the keys share a large common part (it cancels in dQ): 1.6602e-3 against 1.6586e-3 (tensor ops 1.6589e-3).
//
// What bounds the shapes is on-chip memory: at head dim 256 a 128-row dK and dV tile alone fill the 512 TMEM columns, and
// two stationary plus two streamed 128-row tiles do not fit in shared memory. Hence one accumulator per launch and
// 64-row streamed tiles, one kernel with three uses (X stationary, 128 rows; Y streamed, 64 rows):
//   DV : X1 = K           Y1 = Q, Y2 = dO    dV += P^T dO
//   DK : X1 = K, X2 = V   Y1 = Q, Y2 = dO    dK += dS^T Q
//   DQ : X1 = Q, X2 = dO  Y1 = K, Y2 = V     dQ += dS K
//     S = X1 Y1^T, dP = X2 Y2^T -> TMEM (buffers of 64 columns each); P = exp2(S c - lse2), dS = P o (dP - delta);
//     hi and mid go back over S's own columns in TMEM, lo over dP's, and are the A operand of the accumulating MMA (B = Y1 or
//     Y2 read MN-major). With two buffers S and dP of step n+1 run under the exponentials of step n; where two CTAs share an SM
//     (head dims 64 and 128, attn_split_launch) there is one buffer, and the other CTA fills the tensor core meanwhile.
// Recomputing S twice and dP once and splitting costs 14 products of the tile instead of 5, all on the tensor core; the
// tensor-op backward it replaces ran fp32 SIMT products over [heads, S, S] matrices in memory. Measured, causal, DQ + DK + DV, us
// (before: two stages a streamed tile and a fixed order of the MMAs, binary searches for the row bounds, scalar fp32):
//   1 x 2048, 16 heads x 192/128         :  68 +  70 +  54   ( 91 +  81 +  61; tensor ops: about 3 ms)
//   1 x 3072, 16/2 heads x 256           : 202 + 210 + 145   (219 + 217 + 174; tensor ops: about 9 ms)
//   1 x 4093 in 9 documents, 32/4 x 128  : 123 + 143 + 121   (148 + 169 + 150; tensor ops: 21 ms)
//   1 x 3001, 32/4 x 128                 : 234 + 236 + 196   (288 + 289 + 235)
// What is left: 28 MMAs a 64-row step at 64 cycles or more (also where N = 64 should take 32), and the split's arithmetic (without
// it and the exponentials a step takes three quarters of its time).
//
// No atomics: dQ rows belong to one CTA; dK / dV of a query head are written once, directly when there is no GQA group,
// else to per-head fp32 partials that attn_split_group_sum_kernel adds in head order. Results are reproducible.
// Every wait is bounded; on a timeout the roles leave their loops and the status word carries the code.
#include "host_common.h"
#include "ptx.cuh"

namespace pt {

enum : int { ASP_DV = 0, ASP_DK = 1, ASP_DQ = 2 };
constexpr int ASP_XSLAB = 128 * 64 * 2;  // [128 x 64] bf16 swizzle slab
constexpr int ASP_YSLAB = 64 * 64 * 2;   // [64 x 64]

struct AttnSplitArgs {
  int B, Sq, Sk, Hq, Hkv;
  int Sp;                // row pitch of lse2 / delta: Sq rounded up to 4 (their tiles move in 16-byte pieces)
  int causal, q_off;
  int reach;             // keys that a query sees, about: what the host knows of row_lo
  float scale_log2, out_scale;
  const int* row_lo;     // optional [B*Sq]
  const float* lse2;     // [B, Hq, Sp] log2-domain log-sum-exp (+inf for rows that saw no key)
  const float* delta;    // [B, Hq, Sp]
  __nv_bfloat16* out;    // bf16 result (DQ: [B*Sq, Hq*D1]; DK / DV without a group: [B*Sk, Hkv*DA]), or
  float* part;           // fp32 partials [B*Sk, Hq, DA] (DK / DV with a group)
  int* err;
};

template <int D1, int D2, int MODE, bool PAIRED>
struct AttnSplitCfg {
  static constexpr bool HAS_DP = MODE != ASP_DV;
  static constexpr int DA = MODE == ASP_DV ? D2 : D1;     // columns of the accumulator
  static constexpr int X1_BYTES = (D1 / 64) * ASP_XSLAB, X2_BYTES = HAS_DP ? (D2 / 64) * ASP_XSLAB : 0;
  static constexpr int Y1_BYTES = (D1 / 64) * ASP_YSLAB, Y2_BYTES = (D2 / 64) * ASP_YSLAB;
  // PAIRED: two CTAs an SM (attn_split_launch says when), where 256 TMEM columns hold the accumulator and one buffer of S and dP.
  static_assert(!PAIRED || D1 <= 128, "TMEM columns of two CTAs");
  static constexpr int NBUF = PAIRED ? 1 : 2;             // buffers of S and dP (64 columns each)
  static constexpr int T_DP = 64 * NBUF, T_ACC = 128 * NBUF, T_COLS = 256 * NBUF;
  // stages of the streamed tiles: what fits. Where only one of Y2 does, its only reader is the dP product (the scores of the
  // step run meanwhile), or a partner CTA covers the load. (Alone at head dim 128, two of each: 9 to 18 % slower than four and three.)
  static constexpr int NST1 = PAIRED ? (D1 == 64 ? 4 : 2) : D1 + D2 <= 320 ? 4 : (HAS_DP ? 2 : 3);
  static constexpr int NST2 = PAIRED ? (D1 == 64 ? 3 : HAS_DP ? 1 : 2) : D1 + D2 <= 320 ? 3 : (HAS_DP ? 1 : 2);
  // lse2[64] | delta[64] (DV, DK): with each Y1 stage, or one copy that follows the steps where two CTAs share the memory
  static constexpr int STAT_BYTES = (PAIRED ? 1 : NST1) * 512;
  static constexpr int BAR_BYTES = 256;
  static constexpr int SMEM = X1_BYTES + X2_BYTES + NST1 * Y1_BYTES + NST2 * Y2_BYTES + STAT_BYTES + BAR_BYTES;
  static_assert(SMEM <= (PAIRED ? 113 * 1024 : 227 * 1024), "shared memory");
  static_assert(T_ACC + DA <= T_COLS, "TMEM columns");
  static constexpr int THREADS = 10 * 32;
};

template <int D1, int D2, int MODE, bool PAIRED>
__global__ void __launch_bounds__(320, (PAIRED ? 2 : 1))
attn_bwd_split_kernel(const __grid_constant__ CUtensorMap tmX1, const __grid_constant__ CUtensorMap tmX2,
                      const __grid_constant__ CUtensorMap tmY1, const __grid_constant__ CUtensorMap tmY2, const AttnSplitArgs args) {
  using Cfg = AttnSplitCfg<D1, D2, MODE, PAIRED>;
  constexpr bool HAS_DP = Cfg::HAS_DP;
  constexpr int DA = Cfg::DA, NST1 = Cfg::NST1, NST2 = Cfg::NST2, NBUF = Cfg::NBUF;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw;
  if ((smem_u32(smem) & 1023u) != 0) {  // uniform over the CTA
    if (threadIdx.x == 0 && args.err) atomicCAS(args.err, 0, PT_ERR_SMEM_ALIGN);
    return;
  }
  uint8_t* sX1 = smem;
  uint8_t* sX2 = sX1 + Cfg::X1_BYTES;
  uint8_t* sY1 = sX2 + Cfg::X2_BYTES;
  uint8_t* sY2 = sY1 + NST1 * Cfg::Y1_BYTES;
  uint8_t* sStat = sY2 + NST2 * Cfg::Y2_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sStat + Cfg::STAT_BYTES);
  uint64_t* x_full = bars;          // 1
  uint64_t* y1_full = bars + 1;     // NST1 (at most 4)
  uint64_t* y1_empty = bars + 5;    // NST1
  uint64_t* y2_full = bars + 9;     // NST2 (at most 4)
  uint64_t* y2_empty = bars + 13;   // NST2
  uint64_t* s_full = bars + 17;     // 2: S (and dP) of a step are in TMEM
  uint64_t* a_ready = bars + 19;    // 2: compute (8 warps) -> MMA: hi / mid / lo are in TMEM, dP has been read
  uint64_t* acc_done = bars + 21;   // 1
  uint64_t* st_full = bars + 22;    // 1: the single copy of the statistics (PAIRED)
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(bars + 23);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_ptr + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int hq = blockIdx.x % args.Hq, b = blockIdx.x / args.Hq;
  const int hk = hq / (args.Hq / args.Hkv);
  // the tiles with the most work under a causal mask start first: the first key tiles, the last query tiles
  const int tile = MODE == ASP_DQ ? (int)(gridDim.y - 1 - blockIdx.y) : (int)blockIdx.y;
  const int row_base = b * args.Sq, kv_base = b * args.Sk;
  const int x0 = tile * 128;                                   // first row of the stationary tile within the batch entry
  const int x_len = MODE == ASP_DQ ? args.Sq : args.Sk, x_base = MODE == ASP_DQ ? row_base : kv_base;
  const int hx = MODE == ASP_DQ ? hq : hk, hy = MODE == ASP_DQ ? hk : hq;

  // streamed tiles [t_lo, t_lo + N) that share a visible (query, key) pair with the stationary tile
  int t_lo = 0, t_hi;
  if (MODE == ASP_DQ) {
    const int lo = args.row_lo ? max(args.row_lo[row_base + x0], 0) : 0;  // non-decreasing in the row
    const int hi = args.causal ? min(args.Sk - 1, args.q_off + min(x0 + 127, args.Sq - 1)) : args.Sk - 1;
    t_lo = lo / 64;
    t_hi = hi >= lo ? hi / 64 : t_lo - 1;
  } else {
    const int k_last = min(x0 + 127, args.Sk - 1);
    t_hi = (args.Sq + 63) / 64 - 1;
    if (args.causal) {
      const int need = x0 - args.q_off - 63;  // last row of tile i: q_off + 64 i + 63 >= x0
      t_lo = need > 0 ? (need + 63) / 64 : 0;
    }
    if (args.row_lo && t_lo <= t_hi) {
      // the tiles before the first one whose first row has row_lo > k_last: 32 probes a round (each warp for itself), since a
      // binary search is a chain of loads that nothing hides
      int n_t = t_hi - t_lo + 1, first = t_lo;
      t_hi = t_lo - 1;
      while (n_t > 0) {
        const int step = (n_t + 31) / 32;
        const bool seen = lane * step < n_t && args.row_lo[row_base + (first + lane * step) * 64] <= k_last;
        const int c = __popc(__ballot_sync(0xffffffffu, seen));  // the probes that are seen come first
        if (c == 0) break;
        t_hi = first + (c - 1) * step;
        n_t = min(step - 1, first + n_t - 1 - t_hi);
        first = t_hi + 1;
      }
    }
  }
  const int N = t_hi - t_lo + 1;

  // where a row of the result goes: bf16, or the fp32 partial of this query head
  const bool grouped = MODE != ASP_DQ && args.Hq != args.Hkv;
  const long long out_row0 = (long long)(x_base + x0);
  if (N <= 0) {  // uniform over the CTA: nothing visible, the gradient is zero
    for (int i = threadIdx.x; i < 128 * (DA / 8); i += Cfg::THREADS) {
      const int r = i / (DA / 8), c = (i % (DA / 8)) * 8;
      if (x0 + r < x_len) {
        if (grouped) {
          float4* p = reinterpret_cast<float4*>(args.part + ((out_row0 + r) * args.Hq + hq) * DA + c);
          p[0] = make_float4(0.f, 0.f, 0.f, 0.f);
          p[1] = make_float4(0.f, 0.f, 0.f, 0.f);
        } else {
          const int H = MODE == ASP_DQ ? args.Hq : args.Hkv;
          *reinterpret_cast<uint4*>(args.out + ((out_row0 + r) * H + hx) * DA + c) = make_uint4(0u, 0u, 0u, 0u);
        }
      }
    }
    return;
  }

  if (threadIdx.x == 0) {
    mbar_init(x_full, 1);
    for (int s = 0; s < NST1; ++s) { mbar_init(&y1_full[s], 1); mbar_init(&y1_empty[s], 1); }
    for (int s = 0; s < NST2; ++s) { mbar_init(&y2_full[s], 1); mbar_init(&y2_empty[s], 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(&s_full[s], 1); mbar_init(&a_ready[s], 8); }
    mbar_init(acc_done, 1);
    mbar_init(st_full, 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmX1); tma_prefetch_desc(&tmY1); tma_prefetch_desc(&tmY2);
    if (HAS_DP) tma_prefetch_desc(&tmX2);
  }
  if (warp == 1) {
    tmem_alloc(tmem_ptr, Cfg::T_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr;
  const uint32_t tACC = tmem_base + Cfg::T_ACC;  // S: NBUF buffers of 64 columns, then dP, then the accumulator

  if (warp == 0) {
    // ---------------------------------------------------------------- producer
    if (lane == 0) {
      mbar_expect_tx(x_full, Cfg::X1_BYTES + Cfg::X2_BYTES);
#pragma unroll
      for (int db = 0; db < D1 / 64; ++db) tma_load_3d(sX1 + db * ASP_XSLAB, &tmX1, x_full, hx * D1 + 64 * db, x0, b);
      if (HAS_DP) {
#pragma unroll
        for (int db = 0; db < D2 / 64; ++db) tma_load_3d(sX2 + db * ASP_XSLAB, &tmX2, x_full, hx * D2 + 64 * db, x0, b);
      }
      bool ok = true;
      int n1 = 0, n2 = 0, n3 = 0;
      for (int n = 0; n < N && ok; ++n) {
        const int s1 = n % NST1, s2 = n % NST2;
        const int y0 = (t_lo + n) * 64;
        ok = mbar_wait_bounded(&y1_empty[s1], ((n / NST1) & 1) ^ 1, abort_flag, args.err, PT_ERR_TIMEOUT_PRODUCER);
        if (!ok) break;
        constexpr int STATS = MODE == ASP_DQ ? 0 : (MODE == ASP_DK ? 512 : 256);
        mbar_expect_tx(&y1_full[s1], Cfg::Y1_BYTES + (PAIRED ? 0 : STATS));
#pragma unroll
        for (int db = 0; db < D1 / 64; ++db)
          tma_load_3d(sY1 + s1 * Cfg::Y1_BYTES + db * ASP_YSLAB, &tmY1, &y1_full[s1], hy * D1 + 64 * db, y0, b);
        const long long so = ((long long)b * args.Hq + hq) * args.Sp + y0;
        if (MODE != ASP_DQ && !PAIRED) {
          bulk_load_1d(sStat + s1 * 512, args.lse2 + so, 256, &y1_full[s1]);
          if (MODE == ASP_DK) bulk_load_1d(sStat + s1 * 512 + 256, args.delta + so, 256, &y1_full[s1]);
        }
        ++n1;
        ok = mbar_wait_bounded(&y2_empty[s2], ((n / NST2) & 1) ^ 1, abort_flag, args.err, PT_ERR_TIMEOUT_PRODUCER);
        if (!ok) break;
        mbar_expect_tx(&y2_full[s2], Cfg::Y2_BYTES);
#pragma unroll
        for (int db = 0; db < D2 / 64; ++db)
          tma_load_3d(sY2 + s2 * Cfg::Y2_BYTES + db * ASP_YSLAB, &tmY2, &y2_full[s2], hy * D2 + 64 * db, y0, b);
        ++n2;
        if (MODE != ASP_DQ && PAIRED) {
          // the compute warps have read the statistics of step n-1; the scores of step n come after that step's accumulation
          if (n > 0) ok = mbar_wait_bounded(&a_ready[0], (n - 1) & 1, abort_flag, args.err, PT_ERR_TIMEOUT_PRODUCER);
          if (!ok) break;
          mbar_expect_tx(st_full, STATS);
          bulk_load_1d(sStat, args.lse2 + so, 256, st_full);
          if (MODE == ASP_DK) bulk_load_1d(sStat + 256, args.delta + so, 256, st_full);
          ++n3;
        }
      }
      if (*abort_flag) {
        // let copies in flight land before the CTA retires (bounded)
        const uint64_t t0 = globaltimer_ns();
        bool drained = false;
        while (!drained && globaltimer_ns() - t0 < 20000000ull) {
          drained = mbar_try_wait(x_full, 0) && (n3 == 0 || mbar_try_wait(st_full, (n3 - 1) & 1));
          for (int i = 0; i < 4 && drained; ++i) {
            const int c1 = n1 - 1 - i, c2 = n2 - 1 - i;
            if (c1 >= 0 && i < NST1) drained = drained && mbar_try_wait(&y1_full[c1 % NST1], (c1 / NST1) & 1);
            if (c2 >= 0 && i < NST2) drained = drained && mbar_try_wait(&y2_full[c2 % NST2], (c2 / NST2) & 1);
          }
        }
        if (!drained && args.err) atomicCAS(args.err, 0, PT_ERR_TIMEOUT_DRAIN);
      }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA issuer (its MMAs execute in order)
    if (lane == 0) {
      constexpr uint32_t IDESC_S = make_idesc(1, 1, 128, 64, false, false);   // both operands K-major
      constexpr uint32_t IDESC_A = make_idesc(1, 1, 128, DA, false, true);    // A in TMEM, B MN-major
      constexpr uint32_t HI = smem_desc_hi_sw128(1024);
      const uint32_t x1 = smem_desc_lo(smem_u32(sX1), 16), x2 = smem_desc_lo(smem_u32(sX2), 16);
      const uint32_t y1k = smem_desc_lo(smem_u32(sY1), 16), y2k = smem_desc_lo(smem_u32(sY2), 16);
      const uint32_t ym = MODE == ASP_DV ? smem_desc_lo(smem_u32(sY2), ASP_YSLAB) : smem_desc_lo(smem_u32(sY1), ASP_YSLAB);
      // Buffer n % NBUF of S was last read by the accumulation of step n - NBUF (issued earlier by this thread), its dP half by the
      // compute warps of that step (their arrival was awaited before the accumulation).
      // S and dP take turns: two independent accumulators, where one alone waits for its own previous sum (N = 64: 2 to 4 %)
      auto scores = [&](int n) {
        const uint32_t d = tmem_base + (n % NBUF) * 64, yb = y1k + (n % NST1) * (Cfg::Y1_BYTES >> 4);
        const uint32_t yc = y2k + (n % NST2) * (Cfg::Y2_BYTES >> 4);
#pragma unroll
        for (int db = 0; db < D1 / 64; ++db)
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            umma_f16_lh(d, x1 + ((db * ASP_XSLAB + k * 32) >> 4), HI, yb + ((db * ASP_YSLAB + k * 32) >> 4), HI, IDESC_S,
                        (db | k) != 0 ? 1u : 0u);
            if (HAS_DP && db < D2 / 64)
              umma_f16_lh(d + Cfg::T_DP, x2 + ((db * ASP_XSLAB + k * 32) >> 4), HI, yc + ((db * ASP_YSLAB + k * 32) >> 4), HI, IDESC_S,
                          (db | k) != 0 ? 1u : 0u);
          }
        if (HAS_DP) umma_commit(&y2_empty[n % NST2]);
        umma_commit(&s_full[n % NBUF]);
      };
      auto accumulate = [&](int n) {
        const int s1 = n % NST1, s2 = n % NST2;
        const uint32_t yb = ym + (MODE == ASP_DV ? s2 * (Cfg::Y2_BYTES >> 4) : s1 * (Cfg::Y1_BYTES >> 4));
        // columns of the buffer for the k-th 16 streamed rows: hi 8 columns at 16 k, mid at 16 k + 8, lo at 16 k of the dP half
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint32_t a = tmem_base + (n % NBUF) * 64 + k * 16;
          umma_f16_ts_lh(tACC, a, yb + ((k * 2048) >> 4), HI, IDESC_A, (k != 0 || n != 0) ? 1u : 0u);
          umma_f16_ts_lh(tACC, a + 8, yb + ((k * 2048) >> 4), HI, IDESC_A, 1u);
          umma_f16_ts_lh(tACC, a + Cfg::T_DP, yb + ((k * 2048) >> 4), HI, IDESC_A, 1u);
        }
        umma_commit(&y1_empty[s1]);
        if (MODE == ASP_DV) umma_commit(&y2_empty[s2]);
      };
      // Whatever is ready, the scores of the next step (at most NBUF - 1 ahead of the accumulation) first: in a fixed order
      // a late load of step n + 1 holds up the accumulation of step n and with it the stage that the load after it waits for.
      bool ok = mbar_wait_bounded(x_full, 0, abort_flag, args.err, PT_ERR_TIMEOUT_MMA);
      int ns = 0, na = 0;  // steps whose scores, accumulation have been issued
      uint32_t idle = 0;
      uint64_t t0 = 0;
      while (ok && na < N) {
        if (ns < N && ns < na + NBUF && mbar_test_wait(&y1_full[ns % NST1], (ns / NST1) & 1) &&
            (!HAS_DP || mbar_test_wait(&y2_full[ns % NST2], (ns / NST2) & 1))) {
          tc_fence_after();
          scores(ns++);
          idle = 0;
        } else if (na < ns && mbar_test_wait(&a_ready[na % NBUF], (na / NBUF) & 1) &&
                   (MODE != ASP_DV || mbar_test_wait(&y2_full[na % NST2], (na / NST2) & 1))) {
          tc_fence_after();
          accumulate(na++);
          idle = 0;
        } else if ((++idle & 255u) == 0) {  // bounded as in mbar_wait_bounded
          if (*abort_flag) { ok = false; break; }
          const uint64_t now = globaltimer_ns();
          if (idle == 256u) t0 = now;
          if (now - t0 > PT_WAIT_LIMIT_NS) {
            *abort_flag = 1;
            if (args.err) atomicCAS(args.err, 0, PT_ERR_TIMEOUT_MMA);
            ok = false;
          }
        }
      }
      if (ok) umma_commit(acc_done);
    }
  } else {
    // ---------------------------------------------------------------- compute: thread = stationary row, 32 streamed rows
    const int g = (warp - 2) >> 2;            // half of the streamed rows
    const int qd = warp & 3;                  // TMEM lane quarter
    const int r = qd * 32 + lane;
    const int xr = x0 + r;                    // my row within the batch entry: a query (DQ) or a key (DK, DV)
    const bool x_valid = xr < x_len;
    const uint32_t lane_off = static_cast<uint32_t>(qd * 32) << 16;
    float my_lse = INFINITY, my_delta = 0.f;
    // The streamed rows that form visible pairs with my row are a range [my_lo, my_hi]: keys of a query (DQ); queries of a
    // key (DK, DV), because the lower key bounds do not decrease with the query row.
    int my_lo = 0, my_hi = -1;
    if (MODE == ASP_DQ && x_valid) {
      const long long so = ((long long)b * args.Hq + hq) * args.Sp + xr;
      my_lse = args.lse2[so];
      my_delta = args.delta[so];
      my_lo = args.row_lo ? args.row_lo[row_base + xr] : 0;
      my_hi = args.causal ? min(args.Sk - 1, args.q_off + xr) : args.Sk - 1;
    }
    if (MODE != ASP_DQ && x_valid) {
      my_lo = args.causal ? xr - args.q_off : 0;
      my_hi = args.Sq - 1;
    }
    // DK, DV with lower bounds: those of this warp's 32 streamed rows, one a lane, loaded a step ahead
    const bool bounds = MODE != ASP_DQ && args.row_lo != nullptr;
    auto load_bound = [&](int n) {
      const int y = (t_lo + n) * 64 + g * 32 + lane;
      return bounds && n < N && y < args.Sq ? args.row_lo[row_base + y] : 0x7fffffff;
    };
    int bound = load_bound(0);
    bool ok = true;
    for (int n = 0; n < N; ++n) {
      const int y0 = (t_lo + n) * 64 + g * 32;
      int hi_n = my_hi;
      if (bounds) {
        // streamed rows of this step that see my key: the bounds do not decrease, so they are the first c of the 32
        int c = 0;
#pragma unroll
        for (int w = 16; w > 0; w >>= 1)
          if (__shfl_sync(0xffffffffu, bound, c + w - 1) <= xr) c += w;
        if (__shfl_sync(0xffffffffu, bound, c) <= xr) ++c;  // c <= 31 here
        hi_n = min(my_hi, y0 + c - 1);
        bound = load_bound(n + 1);
      }
      int good = 1;
      if (lane == 0) {
        good = mbar_wait_bounded(&s_full[n % NBUF], (n / NBUF) & 1, abort_flag, args.err, PT_ERR_TIMEOUT_EPILOGUE) ? 1 : 0;
        // the statistics that came with Y1, which the S product has already read, are complete, but this thread has to observe it
        if (MODE != ASP_DQ && good)
          good = (PAIRED ? mbar_wait_bounded(st_full, n & 1, abort_flag, args.err, PT_ERR_TIMEOUT_EPILOGUE)
                         : mbar_wait_bounded(&y1_full[n % NST1], (n / NST1) & 1, abort_flag, args.err, PT_ERR_TIMEOUT_EPILOGUE)) ? 1 : 0;
      }
      good = __shfl_sync(0xffffffffu, good, 0);
      if (!good) { ok = false; break; }
      tc_fence_after();
      const uint32_t tS = tmem_base + lane_off + (n % NBUF) * 64 + g * 32;
      // element masks only where a lane needs them (warp-uniform: the stores below are collective)
      const bool masked = __any_sync(0xffffffffu, y0 < my_lo || y0 + 31 > hi_n);
      const float* st = reinterpret_cast<const float*>(sStat + (PAIRED ? 0 : n % NST1) * 512) + g * 32;
      const uint64_t scale2 = f2_pack(args.scale_log2, args.scale_log2), minus1 = f2_pack(-1.f, -1.f);
      constexpr int CH = PAIRED ? 16 : 32;  // streamed rows at a time: two CTAs leave 96 registers a thread
#pragma unroll
      for (int j = 0; j < 32; j += CH) {
        uint32_t sv[CH], dp[CH];
        if constexpr (CH == 32) {
          tmem_ld_32x32(tS, sv);
          if (HAS_DP) tmem_ld_32x32(tS + Cfg::T_DP, dp);
        } else {
          tmem_ld_32x16(tS + j, sv);
          if (HAS_DP) tmem_ld_32x16(tS + j + Cfg::T_DP, dp);
        }
        tmem_ld_wait();
#pragma unroll
        for (int h = 0; h < CH; h += 16) {
          uint32_t hi[8], mid[8], lo[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            // two elements at a time, in packed fp32
            const int c = h + 2 * i, r = j + c;
            const uint64_t l2 = MODE == ASP_DQ ? f2_pack(-my_lse, -my_lse) : f2_pack(-st[r], -st[r + 1]);
            float p0, p1;
            f2_unpack(f2_fma(f2_pack(__uint_as_float(sv[c]), __uint_as_float(sv[c + 1])), scale2, l2), p0, p1);
            p0 = ex2_approx(p0);
            p1 = ex2_approx(p1);
            if (HAS_DP) {
              const uint64_t de = MODE == ASP_DQ ? f2_pack(my_delta, my_delta) : f2_pack(st[64 + r], st[64 + r + 1]);
              const uint64_t d = f2_fma(de, minus1, f2_pack(__uint_as_float(dp[c]), __uint_as_float(dp[c + 1])));
              f2_unpack(f2_mul(f2_pack(p0, p1), d), p0, p1);
            }
            if (masked) {
              p0 = (y0 + r >= my_lo && y0 + r <= hi_n) ? p0 : 0.f;
              p1 = (y0 + r + 1 >= my_lo && y0 + r + 1 <= hi_n) ? p1 : 0.f;
            }
            // rounded, not cut off: cut-off terms all have one sign, which adds to what the tensor core cuts off (1.04e-5 for 9e-6)
            hi[i] = pack_bf16x2(p0, p1);
            const float2 hf = unpack_bf16x2(hi[i]);
            float r0, r1;  // exact: what a rounding leaves fits in fewer bits
            const uint64_t rest = f2_fma(f2_pack(hf.x, hf.y), minus1, f2_pack(p0, p1));
            f2_unpack(rest, r0, r1);
            mid[i] = pack_bf16x2(r0, r1);
            const float2 mf = unpack_bf16x2(mid[i]);
            f2_unpack(f2_fma(f2_pack(mf.x, mf.y), minus1, rest), r0, r1);
            lo[i] = pack_bf16x2(r0, r1);
          }
          // over the columns just read: those 16 of S, and 8 of dP (unused columns in DV), which this warp alone reads
          tmem_st_32x8(tS + j + h, hi);
          tmem_st_32x8(tS + j + h + 8, mid);
          tmem_st_32x8(tS + j + h + Cfg::T_DP, lo);
        }
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&a_ready[n % NBUF]);
    }
    if (ok) {
      int good = 1;
      if (lane == 0) good = mbar_wait_bounded(acc_done, 0, abort_flag, args.err, PT_ERR_TIMEOUT_EPILOGUE) ? 1 : 0;
      good = __shfl_sync(0xffffffffu, good, 0);
      if (good) {
        tc_fence_after();
        const int H = MODE == ASP_DQ ? args.Hq : args.Hkv;
        __nv_bfloat16* orow = args.out + ((out_row0 + r) * H + hx) * DA;
        float* prow = args.part + ((out_row0 + r) * args.Hq + hq) * DA;
#pragma unroll 1
        for (int c = g * 32; c < DA; c += 64) {
          uint32_t v[32];
          tmem_ld_32x32(tACC + lane_off + c, v);
          tmem_ld_wait();
          if (x_valid) {
            if (grouped) {
#pragma unroll
              for (int u = 0; u < 8; ++u)
                *reinterpret_cast<uint4*>(prow + c + 4 * u) = make_uint4(v[4 * u], v[4 * u + 1], v[4 * u + 2], v[4 * u + 3]);
            } else {
              const float sc = args.out_scale;
#pragma unroll
              for (int u = 0; u < 4; ++u) {
                uint4 w;
                w.x = pack_bf16x2(__uint_as_float(v[8 * u + 0]) * sc, __uint_as_float(v[8 * u + 1]) * sc);
                w.y = pack_bf16x2(__uint_as_float(v[8 * u + 2]) * sc, __uint_as_float(v[8 * u + 3]) * sc);
                w.z = pack_bf16x2(__uint_as_float(v[8 * u + 4]) * sc, __uint_as_float(v[8 * u + 5]) * sc);
                w.w = pack_bf16x2(__uint_as_float(v[8 * u + 6]) * sc, __uint_as_float(v[8 * u + 7]) * sc);
                *reinterpret_cast<uint4*>(orow + c + 8 * u) = w;
              }
            }
          }
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, Cfg::T_COLS);
  }
}

// delta = rowsum(dO * O), lse2 = lse * log2(e) (+inf where lse is -inf), both with row pitch Sp; the pad rows get zeros.
// One thread per 8 elements of a (row, head); D is the value head dim.
template <int D>
__global__ void attn_split_pre_kernel(const __nv_bfloat16* __restrict__ out, const __nv_bfloat16* __restrict__ dout,
                                      const float* __restrict__ lse, float* __restrict__ delta, float* __restrict__ lse2,
                                      int B, int Sq, int Sp, int Hq, long long ldo, long long lddo) {
  constexpr int TPR = D / 8;  // threads per (row, head): 8, 16 or 32
  const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long pair = gid / TPR;
  const int part = static_cast<int>(gid % TPR);
  const long long total = (long long)B * Sp * Hq;
  const long long row = pair / Hq;
  const int h = static_cast<int>(pair % Hq);
  const long long bb = row / Sp, r = row % Sp;
  const bool live = pair < total && r < Sq;
  float acc = 0.f;
  if (live) {
    const long long t = bb * Sq + r;
    const uint4 a = *reinterpret_cast<const uint4*>(out + t * ldo + h * D + part * 8);
    const uint4 c = *reinterpret_cast<const uint4*>(dout + t * lddo + h * D + part * 8);
    const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, cw[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 x = unpack_bf16x2(aw[i]), y = unpack_bf16x2(cw[i]);
      acc = fmaf(x.x, y.x, acc);
      acc = fmaf(x.y, y.y, acc);
    }
  }
#pragma unroll
  for (int o = TPR / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (pair < total && part == 0) {
    const long long idx = (bb * Hq + h) * Sp + r;
    delta[idx] = acc;
    const float l = live ? lse[(bb * Hq + h) * Sq + r] : 0.f;
    lse2[idx] = (l == -INFINITY) ? INFINITY : l * 1.4426950408889634f;
  }
}

// out[row, hk, c] = bf16(scale * sum over the group's query heads, in head order, of part[row, hk * group + i, c]).
__global__ void attn_split_group_sum_kernel(const float* __restrict__ part, __nv_bfloat16* __restrict__ out, long long n8,
                                            int group, int D, float scale) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;  // 8 columns of one (row, kv head)
  if (i >= n8) return;
  const int d8 = D / 8;
  const long long rh = i / d8;
  const int c = static_cast<int>(i % d8) * 8;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  for (int x = 0; x < group; ++x) {
    const float4* p = reinterpret_cast<const float4*>(part + (rh * group + x) * D + c);
    const float4 a = p[0], e = p[1];
    acc[0] += a.x; acc[1] += a.y; acc[2] += a.z; acc[3] += a.w;
    acc[4] += e.x; acc[5] += e.y; acc[6] += e.z; acc[7] += e.w;
  }
  uint4 w;
  w.x = pack_bf16x2(acc[0] * scale, acc[1] * scale);
  w.y = pack_bf16x2(acc[2] * scale, acc[3] * scale);
  w.z = pack_bf16x2(acc[4] * scale, acc[5] * scale);
  w.w = pack_bf16x2(acc[6] * scale, acc[7] * scale);
  *reinterpret_cast<uint4*>(out + i * 8) = w;
}

}  // namespace pt

namespace {
using namespace pt;

struct SplitTensors {
  const void *q, *k, *v, *dout;
  long long ldq, ldk, ldv, lddo;
};

template <int D1, int D2, int MODE, bool PAIRED>
int attn_split_launch_as(const SplitTensors& t, const AttnSplitArgs& a, cudaStream_t stream) {
  using Cfg = AttnSplitCfg<D1, D2, MODE, PAIRED>;
  constexpr bool DQ = MODE == ASP_DQ;
  // [B, S, cols] maps: rows past the end of a batch entry read zeros, never the next entry's rows (0 x inf is not 0)
  const uint64_t B = a.B, Sq = a.Sq, Sk = a.Sk;
  CUtensorMap q, k, v, g;  // queries, keys, values, output gradients: 128 stationary or 64 streamed rows
  if (encode_tmap_3d(&q, t.q, TM_BF16, B, Sq, (uint64_t)a.Hq * D1, t.ldq, Sq * t.ldq, 1, DQ ? 128 : 64, 64, TM_SW_128)) return -3;
  if (encode_tmap_3d(&g, t.dout, TM_BF16, B, Sq, (uint64_t)a.Hq * D2, t.lddo, Sq * t.lddo, 1, DQ ? 128 : 64, 64, TM_SW_128)) return -3;
  if (encode_tmap_3d(&k, t.k, TM_BF16, B, Sk, (uint64_t)a.Hkv * D1, t.ldk, Sk * t.ldk, 1, DQ ? 64 : 128, 64, TM_SW_128)) return -3;
  if (encode_tmap_3d(&v, t.v, TM_BF16, B, Sk, (uint64_t)a.Hkv * D2, t.ldv, Sk * t.ldv, 1, DQ ? 64 : 128, 64, TM_SW_128)) return -3;
  if (cudaFuncSetAttribute(attn_bwd_split_kernel<D1, D2, MODE, PAIRED>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM) != cudaSuccess)
    return -4;
  dim3 grid(a.Hq * a.B, ((DQ ? a.Sq : a.Sk) + 127) / 128);
  if (DQ) attn_bwd_split_kernel<D1, D2, MODE, PAIRED><<<grid, Cfg::THREADS, Cfg::SMEM, stream>>>(q, g, k, v, a);
  else attn_bwd_split_kernel<D1, D2, MODE, PAIRED><<<grid, Cfg::THREADS, Cfg::SMEM, stream>>>(k, v, q, g, a);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

// Two CTAs an SM hide each other's steps, loads and stores, but share the tensor core and have one buffer of S and dP and fewer
// stages each. So a CTA has its SM for itself up to one CTA an SM, and beyond that while its range of keys is long and the CTAs of an
// SM are few; many or short ones come in pairs. Whole backward, causal, us, alone / paired:
//   heads x 128, rows           CTAs   one document   4 documents   9          32
//   16/4, 1023                   128    115 / 153      71 / 85       63 / 72
//    8/2, 4093                   256    342 / 554     185 / 222     136 / 144  103 / 97
//   16/4, 2049                   272    216 / 319     127 / 137     111 / 113   89 / 81
//   16/4, 4093                   512    624 / 672     278 / 328     210 / 221  178 / 158
//   64/8, 1023                   512    252 / 242     179 / 173     167 / 149
//   32/4, 4093                  1024   1199 / 1173    513 / 498     375 / 360  306 / 269
// Head dim 64: 98 / 138, 323 / 480, 201 / 274, 525 / 574, 207 / 201, 996 / 994 for one document.
template <int D1, int D2, int MODE>
int attn_split_launch(const SplitTensors& t, const AttnSplitArgs& a, cudaStream_t stream) {
  if constexpr (D1 <= 128) {
    const long long ctas = (long long)a.Hq * a.B * (((MODE == ASP_DQ ? a.Sq : a.Sk) + 127) / 128);
    const long long sms = sm_count();
    if (ctas > (a.reach >= 768 ? 4 * sms : a.reach >= 192 ? 2 * sms : sms)) return attn_split_launch_as<D1, D2, MODE, true>(t, a, stream);
  }
  return attn_split_launch_as<D1, D2, MODE, false>(t, a, stream);
}

template <int D1, int D2>
int attn_split_all(const SplitTensors& t, AttnSplitArgs a, const void* out, const void* lse, float* delta, float* lse2, float* part,
                   void* dq, void* dk, void* dv, long long ldo, float scale, cudaStream_t stream) {
  const long long threads = (long long)a.B * a.Sp * a.Hq * (D2 / 8);
  attn_split_pre_kernel<D2><<<(unsigned)((threads + 255) / 256), 256, 0, stream>>>(
      static_cast<const __nv_bfloat16*>(out), static_cast<const __nv_bfloat16*>(t.dout), static_cast<const float*>(lse), delta, lse2,
      a.B, a.Sq, a.Sp, a.Hq, ldo, t.lddo);
  a.lse2 = lse2;
  a.delta = delta;
  a.part = nullptr;
  a.out = static_cast<__nv_bfloat16*>(dq);
  a.out_scale = scale;
  int rc = attn_split_launch<D1, D2, ASP_DQ>(t, a, stream);
  if (rc) return rc;
  const int group = a.Hq / a.Hkv;
  for (int w = 0; w < 2; ++w) {  // the partials of dK are summed before dV's overwrite them
    void* dst = w == 0 ? dk : dv;
    const int D = w == 0 ? D1 : D2;
    a.out = static_cast<__nv_bfloat16*>(dst);
    a.part = part;
    a.out_scale = w == 0 ? scale : 1.f;
    rc = w == 0 ? attn_split_launch<D1, D2, ASP_DK>(t, a, stream) : attn_split_launch<D1, D2, ASP_DV>(t, a, stream);
    if (rc) return rc;
    if (group > 1) {
      const long long n8 = (long long)a.B * a.Sk * a.Hkv * (D / 8);
      attn_split_group_sum_kernel<<<(unsigned)((n8 + 255) / 256), 256, 0, stream>>>(part, static_cast<__nv_bfloat16*>(dst), n8, group, D,
                                                                                   a.out_scale);
    }
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}
}  // namespace

// Gradients of pt_attn_fwd for (dqk, dv) in {(64,64), (128,128), (192,128), (256,256)} and any Sq, Sk. q, k, v, out, dout: bf16
// token-major with row pitches (elements, multiples of 8, 16-byte aligned bases); lse [B,Hq,Sq] fp32 from the forward.
// delta, lse2: fp32 scratch of B*Hq*Sp + 128 elements each, Sp = Sq rounded up to 4, 16-byte aligned (delta holds the row sums
// of dO*O afterwards, row pitch Sp). part: fp32 scratch [B*Sk, Hq, max(dqk, dv)] when Hq > Hkv, else null. dq / dk / dv
// receive contiguous bf16 results.
// reach: about how many keys a query sees, for the choice between kernels (row_lo lies on the device); Sk if nothing is known.
PT_API int pt_attn_bwd_split_reach(const void* q, const void* k, const void* v, const void* out, const void* dout, const void* lse,
                                   const void* row_lo, void* dq, void* dk, void* dv, void* delta, void* lse2, void* part, int B, int Sq,
                                   int Sk, int Hq, int Hkv, int dqk, int dvd, long long ldq, long long ldk, long long ldv, long long ldo,
                                   long long lddo, float scale, int causal, int q_off, int reach, void* stream_) {
  if (B <= 0 || Sq <= 0 || Sk <= 0 || Hkv <= 0 || Hq % Hkv != 0 || scale <= 0.f) return -2;
  AttnSplitArgs a{};
  a.B = B; a.Sq = Sq; a.Sk = Sk; a.Hq = Hq; a.Hkv = Hkv; a.causal = causal; a.q_off = q_off; a.reach = reach;
  a.Sp = (Sq + 3) & ~3;
  a.scale_log2 = scale * 1.4426950408889634f;
  a.row_lo = static_cast<const int*>(row_lo);
  a.err = device_status_word();
  const SplitTensors t{q, k, v, dout, ldq, ldk, ldv, lddo};
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  float *de = static_cast<float*>(delta), *l2 = static_cast<float*>(lse2), *pa = static_cast<float*>(part);
  if (dqk == 64 && dvd == 64) return attn_split_all<64, 64>(t, a, out, lse, de, l2, pa, dq, dk, dv, ldo, scale, stream);
  if (dqk == 128 && dvd == 128) return attn_split_all<128, 128>(t, a, out, lse, de, l2, pa, dq, dk, dv, ldo, scale, stream);
  if (dqk == 192 && dvd == 128) return attn_split_all<192, 128>(t, a, out, lse, de, l2, pa, dq, dk, dv, ldo, scale, stream);
  if (dqk == 256 && dvd == 256) return attn_split_all<256, 256>(t, a, out, lse, de, l2, pa, dq, dk, dv, ldo, scale, stream);
  return -2;
}

PT_API int pt_attn_bwd_split(const void* q, const void* k, const void* v, const void* out, const void* dout, const void* lse,
                             const void* row_lo, void* dq, void* dk, void* dv, void* delta, void* lse2, void* part, int B, int Sq,
                             int Sk, int Hq, int Hkv, int dqk, int dvd, long long ldq, long long ldk, long long ldv, long long ldo,
                             long long lddo, float scale, int causal, int q_off, void* stream_) {
  return pt_attn_bwd_split_reach(q, k, v, out, dout, lse, row_lo, dq, dk, dv, delta, lse2, part, B, Sq, Sk, Hq, Hkv, dqk, dvd, ldq, ldk, ldv, ldo,
                                 lddo, scale, causal, q_off, Sk, stream_);
}
