// bf16 GEMMs with 2-CTA tcgen05 tiles (cta_group::2): dense products and stacks of equal products.
//
//   D_e[M,N] = A_e * B_e, bf16 in, fp32 accumulate in TMEM. Either operand is K-major (reduction contiguous) or MN-major, so
//   the forward (NT), input-gradient (NN) and weight-gradient (TN) forms read the tensors as they sit in memory.
//   A pair of CTAs (cluster 2x1x1) owns a 256 x 256 output tile: CTA r loads rows [m0 + 128 r, +128) of A and rows
//   [n0 + 128 r, +128) of B (its half of N) with ordinary, non-multicast TMA loads issued in the .cta_group::2 form,
//   whose completion lands on the leader's (CTA 0) mbarrier. The leader's MMA thread issues
//   tcgen05.mma.cta_group::2 (M = 256, N = 256): the pair's tensor cores read both halves of B from both CTAs' shared
//   memory, so each B byte is loaded from L2 once per pair and each shared-memory byte feeds twice the FLOPs of the
//   single-CTA kernel. Each CTA keeps its 128 accumulator rows in its own TMEM and runs its own epilogue.
//
//   per CTA: warp 0 producer, warp 1 MMA (leader only issues; both allocate TMEM), warps 2..5 or 2..9 epilogue.
//   Barriers live at the same shared-memory offset in both CTAs:
//     full[s]       used in CTA 0: leader producer arrives with expect_tx(both CTAs' bytes)
//     empty[s]      in each CTA: one commit of the leader's MMA thread arrives on both copies
//     tmem_full[b]  in each CTA: same
//     tmem_empty[b] used in CTA 0: the epilogue warps of the pair arrive there (remote arrive from CTA 1)
//
// Epilogues:
//   T2_STORE   bf16 through TMA stores: the q/k/v/o projections, lm_head and dense MLPs (ops/gemm.py)
//   T2_FUSED   bf16 of s_e * (alpha * acc + beta * C + diag * I): the products of the Newton-Schulz iteration with the addend,
//              the diagonal, the normalisation and the weight update in them. With `sym` (D symmetric) only the tiles on and
//              above the diagonal are computed, and each is stored a second time, transposed.
//   T2_REDUCE  D += acc in bf16 or fp32 by TMA reduce-add (dense weight gradients)
//   T2_SUM     the same with the sums of an fp32 product: the tensor core cuts its sums off, so every T2_PROMOTE k-blocks they
//              move to registers and are added there with rounding
//
// PTX forms follow the vendored CUTLASS headers (cute/arch/copy_sm100_tma.hpp: SM100_TMA_2SM_LOAD_3D,
// cute/arch/mma_sm100_umma.hpp: SM100_MMA_F16BF16_2x1SM_SS, cute/arch/tmem_allocator_sm100.hpp: Allocator2Sm,
// cutlass/arch/barrier.h: umma_arrive_2x1SM, umma_arrive_2x1SM_sm0).
#include "gemm_skinny.h"
#include "host_common.h"
#include "ptx.cuh"

namespace pt {

constexpr int T2_BM = 128;  // rows per CTA (256 per pair)
constexpr int T2_BN = 256;  // columns per pair; each CTA loads 128 rows of B
constexpr int T2_BK = 64;
constexpr int T2_STAGES = 5;
constexpr int T2_A_BYTES = T2_BM * T2_BK * 2;        // 16 KB
constexpr int T2_B_BYTES = (T2_BN / 2) * T2_BK * 2;  // 16 KB (this CTA's half)
constexpr int T2_STAGE_BYTES = T2_A_BYTES + T2_B_BYTES;
constexpr uint32_t T2_PEER_MASK = 0xFEFFFFFFu;  // clears the pair-rank bit of a shared::cluster address -> CTA 0

enum Gemm2Epi : int { T2_STORE = 0, T2_FUSED = 1, T2_REDUCE = 2, T2_SUM = 3 };

struct Gemm2Args {
  int M, N, K;
  int batch;     // stacked products (dense: 1)
  int sym;       // T2_FUSED: D is symmetric (M == N)
  int out_fp32;  // T2_REDUCE, T2_SUM
  float alpha, beta, diag;
  const float* scale;  // T2_FUSED: one factor per product (null: 1), applied scale_pow times
  int scale_pow;
  const __nv_bfloat16* C;  // T2_FUSED addend, laid out as D (null: none)
  long long ldc, c_stride;
  int* err;
};

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_alloc_2cta(uint32_t* smem_result, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_result)), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_2cta() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_2cta(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// TMA load of this CTA's box; completion bytes go to the mbarrier at the same offset in CTA 0.
__device__ __forceinline__ void tma_load_3d_pair(void* smem_dst, const CUtensorMap* m, uint64_t* bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar) & T2_PEER_MASK), "r"(x), "r"(y), "r"(z)
      : "memory");
}
__device__ __forceinline__ void umma_f16_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                              uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n\t}" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0u)
      : "memory");
}
// Arrive (once the MMAs issued so far have completed) on the barrier at this offset in both CTAs of the pair. One commit for
// both: with one a CTA the tensor pipe lost 20 of 330 ns a k-block (8192^3 1415 -> 1470 TFLOP/s, 8192 x 5120 x 2048 1387 ->
// 1435); one commit for two or three k-blocks gained nothing more and delays the loads.
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
               "h"(static_cast<uint16_t>(3))
               : "memory");
}
// Plain arrive on CTA 0's copy of a barrier (from either CTA).
__device__ __forceinline__ void mbar_arrive_leader(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(smem_u32(bar) & T2_PEER_MASK) : "memory");
}

// Epilogue warps of a CTA: four, one for each 32-row quarter of the accumulator, or eight, the two of a quarter taking its
// 64-column chunks in turn. Eight pay where a short reduction meets an addend (A^2 of 128 x [768, 768]: 102 -> 84 us); elsewhere
// the products of a tile hide four, and eight cost 4 to 5 % (polling beside a power-capped tensor core: A of 128 x [768, 2048] 166
// -> 173 us, B X 246 -> 261).
// T2_SUM: k-blocks that the tensor core sums up before the sum moves to registers. Relative error (2-norm) of [5120, 2048] over
// 3001 rows / [768, 1024] over 1001 and time of the former, cold: never 3.2e-6 / 9.8e-7, every 8 blocks 4.7e-7 / 4.6e-7 76 us, 4
// 2.4e-7 / 2.3e-7 83, 2 1.5e-7 / 1.3e-7 97, 1 1.4e-7 / 1.0e-7 113; the library's fp32 product 5.0e-7 / 2.5e-7, about 1000 us.
constexpr int T2_PROMOTE = 2;
template <int EPI, int EW>
constexpr int t2_slabs() { return EPI == T2_STORE || EW == 8 ? 2 : 4; }  // 4 KB staging slabs of an epilogue warp
template <int EPI, int EW>
constexpr int t2_smem_bytes() { return T2_STAGES * T2_STAGE_BYTES + EW * t2_slabs<EPI, EW>() * 4096 + 256 + 1024; }

// Eight bf16 pairs -> one 128-byte row of a swizzled slab (64 columns).
__device__ __forceinline__ void t2_store_row(uint8_t* rowp, int lane, const float (&v)[64]) {
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    uint4 w;
    w.x = pack_bf16x2(v[8 * j + 0], v[8 * j + 1]);
    w.y = pack_bf16x2(v[8 * j + 2], v[8 * j + 3]);
    w.z = pack_bf16x2(v[8 * j + 4], v[8 * j + 5]);
    w.w = pack_bf16x2(v[8 * j + 6], v[8 * j + 7]);
    *reinterpret_cast<uint4*>(rowp + ((j ^ (lane & 7)) << 4)) = w;
  }
}

template <bool A_MN, bool B_MN, int EPI, int EW>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(64 + 32 * EW, 1)
gemm2cta_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                const __grid_constant__ CUtensorMap tmD, const __grid_constant__ CUtensorMap tmT, const Gemm2Args args) {
  constexpr uint32_t IDESC = make_idesc(1, 1, 2 * T2_BM, T2_BN, A_MN, B_MN);
  constexpr int NSLAB = t2_slabs<EPI, EW>();
  constexpr int SPLIT = EW / 4;  // warps that share a quarter
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* staging = smem + T2_STAGES * T2_STAGE_BYTES;
  uint64_t* full = reinterpret_cast<uint64_t*>(staging + EW * NSLAB * 4096);
  uint64_t* empty = full + T2_STAGES;
  uint64_t* tmem_full = empty + T2_STAGES;
  uint64_t* tmem_empty = tmem_full + 2;
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(tmem_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_ptr + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader = rank == 0;
  const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;
  const int m_tiles = (args.M + 2 * T2_BM - 1) / (2 * T2_BM), n_tiles = (args.N + T2_BN - 1) / T2_BN;
  const bool sym = EPI == T2_FUSED && args.sym;
  const int per_matrix = sym ? m_tiles * (m_tiles + 1) / 2 : m_tiles * n_tiles;
  const int num_tiles = per_matrix * args.batch;
  const int num_kb = (args.K + T2_BK - 1) / T2_BK;
  const int parts = (num_kb + T2_PROMOTE - 1) / T2_PROMOTE;  // T2_SUM: accumulators of a tile

  if (threadIdx.x == 0) {
    for (int s = 0; s < T2_STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&tmem_full[b], 1); mbar_init(&tmem_empty[b], 2 * EW); }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmA); tma_prefetch_desc(&tmB); tma_prefetch_desc(&tmD);
  }
  if (warp == 1) {
    tmem_alloc_2cta(tmem_ptr, 512);
    tmem_relinquish_2cta();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // the peer's barriers exist before anything signals them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr;

  // Tile t of the launch: product e, origin (m0, n0).
  auto tile_origin = [&](int t, int& e, int& m0, int& n0) {
    e = t / per_matrix;
    const int r = t - e * per_matrix;
    int mt, nt;
    if (sym) {
      // columns of the upper triangle one after the other: column nt holds rows 0 .. nt
      nt = 0;
      int left = r;
      while (left > nt) { left -= nt + 1; ++nt; }
      mt = left;
    } else {
      // 8-row supergroups: concurrently running pairs share A rows and B columns in L2
      const int GROUP = 8;
      const int per = GROUP * n_tiles;
      const int gid = r / per, first_m = gid * GROUP;
      const int gsz = min(m_tiles - first_m, GROUP);
      const int local = r - gid * per;
      mt = first_m + local % gsz;
      nt = local / gsz;
    }
    m0 = mt * 2 * T2_BM;
    n0 = nt * T2_BN;
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ producer (both CTAs)
    if (lane == 0) {
      uint32_t it = 0;
      bool ok = true;
      for (int t = pair; t < num_tiles && ok; t += num_pairs) {
        int e, m0, n0;
        tile_origin(t, e, m0, n0);
        m0 += (int)rank * T2_BM;
        n0 += (int)rank * (T2_BN / 2);
        for (int kb = 0; kb < num_kb; ++kb, ++it) {
          const int s = it % T2_STAGES;
          const uint32_t ph = (it / T2_STAGES) & 1;
          ok = mbar_wait_bounded(&empty[s], ph ^ 1, abort_flag, args.err, PT_ERR_TIMEOUT_PRODUCER);
          if (!ok) break;
          if (leader) mbar_expect_tx(&full[s], 2 * T2_STAGE_BYTES);
          uint8_t* sa = smem + s * T2_STAGE_BYTES;
          uint8_t* sb = sa + T2_A_BYTES;
          if (!A_MN) {
            tma_load_3d_pair(sa, &tmA, &full[s], kb * T2_BK, m0, e);
          } else {
#pragma unroll
            for (int j = 0; j < T2_BM / 64; ++j) tma_load_3d_pair(sa + j * (T2_BK * 128), &tmA, &full[s], m0 + 64 * j, kb * T2_BK, e);
          }
          if (!B_MN) {
            tma_load_3d_pair(sb, &tmB, &full[s], kb * T2_BK, n0, e);
          } else {
#pragma unroll
            for (int j = 0; j < T2_BN / 128; ++j) tma_load_3d_pair(sb + j * (T2_BK * 128), &tmB, &full[s], n0 + 64 * j, kb * T2_BK, e);
          }
        }
      }
      if (leader && *abort_flag) {
        // gave up somewhere: let the copies already in flight land before the pair retires (bounded)
        const uint32_t n = it < (uint32_t)T2_STAGES ? it : (uint32_t)T2_STAGES;
        const uint64_t t0 = globaltimer_ns();
        for (uint32_t j = 1; j <= n; ++j) {
          const uint32_t jt = it - j;
          while (!mbar_try_wait(&full[jt % T2_STAGES], (jt / T2_STAGES) & 1)) {
            if (globaltimer_ns() - t0 > 20000000ull) {
              if (args.err) atomicCAS(args.err, 0, PT_ERR_TIMEOUT_DRAIN);
              break;
            }
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (leader CTA only)
    if (leader && lane == 0) {
      uint32_t it = 0, tc = 0;
      bool ok = true;
      for (int item = 0; ok; ++item, ++tc) {
        // an accumulator's work: a tile, or for T2_SUM a tile's next T2_PROMOTE k-blocks
        const int t = pair + (EPI == T2_SUM ? item / parts : item) * num_pairs;
        if (t >= num_tiles) break;
        const int kb0 = EPI == T2_SUM ? (item % parts) * T2_PROMOTE : 0;
        const int kb1 = EPI == T2_SUM ? min(num_kb, kb0 + T2_PROMOTE) : num_kb;
        const int acc = tc & 1;
        ok = mbar_wait_bounded(&tmem_empty[acc], ((tc >> 1) & 1) ^ 1, abort_flag, args.err, PT_ERR_TIMEOUT_MMA);
        if (!ok) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * T2_BN;
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
          const int s = it % T2_STAGES;
          ok = mbar_wait_bounded(&full[s], (it / T2_STAGES) & 1, abort_flag, args.err, PT_ERR_TIMEOUT_MMA);
          if (!ok) break;
          tc_fence_after();
          const uint32_t a_addr = smem_u32(smem + s * T2_STAGE_BYTES);
          const uint32_t b_addr = a_addr + T2_A_BYTES;
#pragma unroll
          for (int k = 0; k < T2_BK / 16; ++k) {
            const uint64_t ad = A_MN ? make_smem_desc_sw128(a_addr + k * 2048, T2_BK * 128, 1024)
                                     : make_smem_desc_sw128(a_addr + k * 32, 16, 1024);
            const uint64_t bd = B_MN ? make_smem_desc_sw128(b_addr + k * 2048, T2_BK * 128, 1024)
                                     : make_smem_desc_sw128(b_addr + k * 32, 16, 1024);
            umma_f16_pair(d_tmem, ad, bd, IDESC, (kb != kb0 || k != 0) ? 1u : 0u);
          }
          umma_commit_pair(&empty[s]);
        }
        if (!ok) break;
        umma_commit_pair(&tmem_full[acc]);
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue (both CTAs, own 128 rows)
    const int q = warp & 3;            // TMEM lane quarter this warp may read
    const int first = (warp - 2) >> 2;  // chunks first, first + SPLIT, ...
    uint8_t* slabs = staging + (warp - 2) * NSLAB * 4096;
    uint32_t tc = 0, slab = 0;
    bool used_tma = false;
    if constexpr (EPI == T2_SUM) {
      // half of the tile's columns in registers, 32 at a time from TMEM
      static_assert(EPI != T2_SUM || EW == 8, "two warps a quarter");
      bool good = true;
      for (int t = pair; t < num_tiles && good; t += num_pairs) {
        int e, m0, n0;
        tile_origin(t, e, m0, n0);
        const int row0 = m0 + (int)rank * T2_BM + q * 32, col0 = n0 + first * (T2_BN / 2);
        float sum[T2_BN / 2];
#pragma unroll
        for (int j = 0; j < T2_BN / 2; ++j) sum[j] = 0.f;
        for (int part = 0; part < parts; ++part, ++tc) {
          const int acc = tc & 1;
          good = mbar_wait_bounded_warp(&tmem_full[acc], (tc >> 1) & 1, abort_flag, args.err, PT_ERR_TIMEOUT_EPILOGUE);
          if (!good) break;
          tc_fence_after();
          const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + acc * T2_BN + first * (T2_BN / 2);
#pragma unroll
          for (int c = 0; c < T2_BN / 32; ++c) {
            uint32_t r[16];
            tmem_ld_32x16(taddr + c * 16, r);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 16; ++j) sum[16 * c + j] += __uint_as_float(r[j]);
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_leader(&tmem_empty[acc]);
        }
        if (!good) break;
        const int cols_per = args.out_fp32 ? 32 : 64;
#pragma unroll
        for (int c = 0; c < T2_BN / 64; ++c) {
          // 32 columns: a slab of fp32, half a slab of bf16
          if (col0 + c * 32 / cols_per * cols_per >= args.N) break;
          uint8_t* st = slabs + (slab % NSLAB) * 4096;
          if (args.out_fp32 || c % 2 == 0) {
            if (lane == 0) tma_store_wait_read<NSLAB - 1>();
            __syncwarp();
          }
          uint8_t* rowp = st + lane * 128;
          if (args.out_fp32) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
              *reinterpret_cast<float4*>(rowp + ((j ^ (lane & 7)) << 4)) =
                  make_float4(sum[32 * c + 4 * j], sum[32 * c + 4 * j + 1], sum[32 * c + 4 * j + 2], sum[32 * c + 4 * j + 3]);
          } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              uint4 w;
              w.x = pack_bf16x2(sum[32 * c + 8 * j], sum[32 * c + 8 * j + 1]);
              w.y = pack_bf16x2(sum[32 * c + 8 * j + 2], sum[32 * c + 8 * j + 3]);
              w.z = pack_bf16x2(sum[32 * c + 8 * j + 4], sum[32 * c + 8 * j + 5]);
              w.w = pack_bf16x2(sum[32 * c + 8 * j + 6], sum[32 * c + 8 * j + 7]);
              *reinterpret_cast<uint4*>(rowp + (((j + (c % 2) * 4) ^ (lane & 7)) << 4)) = w;
            }
            if (c % 2 == 0) continue;
          }
          ++slab;
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            tma_reduce_add_3d(&tmD, st, col0 + c * 32 / cols_per * cols_per, row0, e);  // past the tensor's extent: clipped by TMA
            tma_store_commit();
            used_tma = true;
          }
        }
      }
    } else
    for (int t = pair; t < num_tiles; t += num_pairs, ++tc) {
      int e, m0, n0;
      tile_origin(t, e, m0, n0);
      const int acc = tc & 1;
      const int row0 = m0 + (int)rank * T2_BM + q * 32;
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + acc * T2_BN;
      const int cols_per = EPI == T2_REDUCE && args.out_fp32 ? 32 : 64;
      const int chunks = (min(args.N - n0, T2_BN) + cols_per - 1) / cols_per;
      float sc = 1.f;
      const __nv_bfloat16* cbase = nullptr;
      bool mirror = false;
      uint4 cv[8];
      // addend of chunk cc, four rows of 128 bytes an instruction: lane -> row 4 i + lane / 8, piece lane % 8
      auto load_c = [&](int cc) {
        if (cbase == nullptr) return;
        const int col = cc * 64 + (lane & 7) * 8;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int row = row0 + 4 * i + (lane >> 3);
          cv[i] = make_uint4(0u, 0u, 0u, 0u);
          if (row < args.M && n0 + col < args.N) cv[i] = *reinterpret_cast<const uint4*>(cbase + (long long)row * args.ldc + col);
        }
      };
      if (EPI == T2_FUSED) {
        if (args.scale) {
          const float s = args.scale[e];
          sc = args.scale_pow == 2 ? s * s : s;
        }
        if (args.C) cbase = args.C + (long long)e * args.c_stride + n0;
        mirror = sym && m0 != n0;
        if (first < chunks) load_c(first);  // in flight while the products of this tile finish
      }
      if (!mbar_wait_bounded_warp(&tmem_full[acc], (tc >> 1) & 1, abort_flag, args.err, PT_ERR_TIMEOUT_EPILOGUE)) break;
      tc_fence_after();
      if (SPLIT > 1 && first >= chunks && lane == 0) mbar_arrive_leader(&tmem_empty[acc]);  // a single chunk: nothing for the second warp
#pragma unroll 1
      for (int cc = first; cc < chunks; cc += SPLIT) {
        uint32_t r0[32], r1[32];
        tmem_ld_32x32(taddr + cc * cols_per, r0);
        if (cols_per == 64) tmem_ld_32x32(taddr + cc * 64 + 32, r1);
        tmem_ld_wait();
        if (cc + SPLIT >= chunks) {
          // this warp's part of the accumulator has left TMEM: hand the buffer back to the leader's MMA thread
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_leader(&tmem_empty[acc]);
        }
        uint8_t* st = slabs + (slab % NSLAB) * 4096;
        ++slab;
        if (lane == 0) tma_store_wait_read<NSLAB - 1>();
        __syncwarp();
        if (EPI == T2_REDUCE && args.out_fp32) {
          uint8_t* rowp = st + lane * 128;
#pragma unroll
          for (int j = 0; j < 8; ++j)
            *reinterpret_cast<uint4*>(rowp + ((j ^ (lane & 7)) << 4)) = make_uint4(r0[4 * j], r0[4 * j + 1], r0[4 * j + 2], r0[4 * j + 3]);
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            tma_reduce_add_3d(&tmD, st, n0 + cc * 32, row0, e);
            tma_store_commit();
            used_tma = true;
          }
          continue;
        }
        float v[64];
#pragma unroll
        for (int j = 0; j < 32; ++j) { v[j] = __uint_as_float(r0[j]); v[32 + j] = __uint_as_float(r1[j]); }
        if (EPI == T2_FUSED) {
          const int d = row0 + lane - n0 - cc * 64;  // column of the diagonal in this chunk, if inside
#pragma unroll
          for (int j = 0; j < 64; ++j) v[j] *= args.alpha;
          if (cbase) {
            // through the slab, so that each lane gets its own row
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const int r = 4 * i + (lane >> 3);
              *reinterpret_cast<uint4*>(st + r * 128 + (((lane & 7) ^ (r & 7)) << 4)) = cv[i];
            }
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const uint4 c8 = *reinterpret_cast<const uint4*>(st + lane * 128 + ((j ^ (lane & 7)) << 4));
              const uint32_t w[4] = {c8.x, c8.y, c8.z, c8.w};
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const float2 f = unpack_bf16x2(w[i]);
                v[8 * j + 2 * i] = fmaf(args.beta, f.x, v[8 * j + 2 * i]);
                v[8 * j + 2 * i + 1] = fmaf(args.beta, f.y, v[8 * j + 2 * i + 1]);
              }
            }
            if (cc + SPLIT < chunks) load_c(cc + SPLIT);
          }
          if (args.diag != 0.f) {
#pragma unroll
            for (int j = 0; j < 64; ++j) v[j] += j == d ? args.diag : 0.f;
          }
#pragma unroll
          for (int j = 0; j < 64; ++j) v[j] *= sc;
        }
        t2_store_row(st + lane * 128, lane, v);
        uint8_t* mt = nullptr;
        if (EPI == T2_FUSED && mirror) {
          // the transposed copy: 64 rows (columns of the chunk) x 32 columns (rows of this warp), 64 bytes a row
          mt = slabs + (slab % NSLAB) * 4096;
          ++slab;
          if (lane == 0) tma_store_wait_read<NSLAB - 2>();
          __syncwarp();
#pragma unroll
          for (int j = 0; j < 64; ++j) *reinterpret_cast<__nv_bfloat16*>(mt + j * 64 + lane * 2) = __float2bfloat16(v[j]);
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          // rows or columns past the tensor's extent are clipped by TMA
          if (EPI == T2_REDUCE) tma_reduce_add_3d(&tmD, st, n0 + cc * 64, row0, e);
          else tma_store_3d(&tmD, st, n0 + cc * 64, row0, e);
          tma_store_commit();
          if (EPI == T2_FUSED && mt) {
            tma_store_3d(&tmT, mt, row0, n0 + cc * 64, e);
            tma_store_commit();
          }
          used_tma = true;
        }
      }
    }
    if (lane == 0 && used_tma) tma_store_wait_all<0>();
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // both CTAs are done with TMEM and with each other's barriers
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_2cta(tmem_base, 512);
  }
}

// One operand: a stack of row-major matrices [rows, cols], pitch ld, `stride` elements apart.
struct T2Mat {
  const void* p;
  long long rows, cols, ld, stride;
};

// D_e = A_e B_e for args.batch products. A is [M, K] (or [K, M] with A_MN), B [N, K] (or [K, N] with B_MN), D [M, N].
template <bool A_MN, bool B_MN, int EPI, int EW = 4>
int t2_launch(const T2Mat& A, const T2Mat& B, const T2Mat& D, Gemm2Args& a, cudaStream_t stream) {
  CUtensorMap tmA, tmB, tmD, tmT;
  const int mn_rows = T2_BK, mn_cols = 64;
  if (encode_tmap_3d(&tmA, A.p, TM_BF16, a.batch, A.rows, A.cols, A.ld, A.stride, 1, A_MN ? mn_rows : T2_BM, A_MN ? mn_cols : T2_BK, TM_SW_128)) return -3;
  if (encode_tmap_3d(&tmB, B.p, TM_BF16, a.batch, B.rows, B.cols, B.ld, B.stride, 1, B_MN ? mn_rows : T2_BN / 2, B_MN ? mn_cols : T2_BK, TM_SW_128)) return -3;
  const bool f32 = (EPI == T2_REDUCE || EPI == T2_SUM) && a.out_fp32;
  if (encode_tmap_3d(&tmD, D.p, f32 ? TM_F32 : TM_BF16, a.batch, D.rows, D.cols, D.ld, D.stride, 1, 32, f32 ? 32 : 64, TM_SW_128)) return -3;
  tmT = tmD;
  if (EPI == T2_FUSED && a.sym && encode_tmap_3d(&tmT, D.p, TM_BF16, a.batch, D.rows, D.cols, D.ld, D.stride, 1, 64, 32, TM_SW_NONE)) return -3;
  a.err = device_status_word();
  auto kern = gemm2cta_kernel<A_MN, B_MN, EPI, EW>;
  constexpr int smem = t2_smem_bytes<EPI, EW>();
  static SmemLimit limit;
  if (limit.set(kern, smem) != cudaSuccess) return -4;
  const long long m_tiles = (a.M + 2 * T2_BM - 1) / (2 * T2_BM), n_tiles = (a.N + T2_BN - 1) / T2_BN;
  const long long tiles = a.batch * (EPI == T2_FUSED && a.sym ? m_tiles * (m_tiles + 1) / 2 : m_tiles * n_tiles);
  if (tiles > 0x3fffffffLL) return -2;
  long long pairs = sm_count() / 2;
  if (pairs > tiles) pairs = tiles;
  kern<<<(unsigned)(2 * pairs), 64 + 32 * EW, smem, stream>>>(tmA, tmB, tmD, tmT, a);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

inline Gemm2Args t2_args(int M, int N, int K, int batch) {
  Gemm2Args a;
  a.M = M; a.N = N; a.K = K; a.batch = batch; a.sym = 0; a.out_fp32 = 0;
  a.alpha = 1.f; a.beta = 0.f; a.diag = 0.f;
  a.scale = nullptr; a.scale_pow = 1; a.C = nullptr; a.ldc = 0; a.c_stride = 0; a.err = nullptr;
  return a;
}

}  // namespace pt

// x [M, K], w [N, K] bf16 row-major with pitches lda / ldb, out [M, N] bf16 with pitch ldd; K a multiple of 8.
PT_API int pt_gemm2cta_nt(const void* x, const void* w, void* out, int M, int N, int K, long long lda, long long ldb,
                          long long ldd, void* stream_) {
  using namespace pt;
  if (M <= 0 || N <= 0 || K <= 0 || K % 8 != 0) return -2;
  if (gemm_skinny_better(M, N, K)) return gemm_skinny_nt(x, w, out, M, N, K, lda, ldb, ldd, static_cast<cudaStream_t>(stream_));
  Gemm2Args a = t2_args(M, N, K, 1);
  return t2_launch<false, false, T2_STORE>({x, M, K, lda, lda * M}, {w, N, K, ldb, ldb * N}, {out, M, N, ldd, ldd * M}, a,
                                           static_cast<cudaStream_t>(stream_));
}

extern "C" int pt_gemm_bf16(const void* A, const void* B, void* D, int mode, int M, int N, int K, int a_mn, int b_mn, long long a_rows,
                            long long a_cols, long long lda, long long b_rows, long long b_cols, long long ldb, long long d_rows, long long ldd,
                            const int* offs, int num_groups, int b_group_rows, long long d_group_stride, int out_fp32, int accumulate,
                            int use_tma_store, int epi, int bn, int max_ctas, const int* a_idx, int a_idx_div, long long a_idx_len, void* stream_);

// Pairs cut the rows of D into 256, the single-CTA kernel of csrc/gemm.cu into 128: just past a whole number of pair tiles it can need
// a wave less, which counts while the waves are few. Cold cache, us, pair / single, waves: input gradients: 1025 rows of [2048, 4096]
// 31 / 23 (2 / 1), 3329: 54 / 51 (4 / 3), 4609: 68 / 66 (5 / 4), 6913: 90 / 93 (7 / 6); 4609 rows of [10944, 2048] 182 / 148 (3 / 2);
// fp32 weight gradients of 4096 rows: [1032, 4096] 55 / 38 (2 / 1), [4616, 4096] 133 / 127 (5 / 4), [2056, 10944] 162 / 162 (6 / 5).
namespace {
bool fewer_waves_alone(long long rows, long long cols) {
  using namespace pt;
  const long long n_tiles = (cols + T2_BN - 1) / T2_BN, sms = sm_count(), slots = sms / 2 > 0 ? sms / 2 : 1;
  const long long pairs = ((rows + 2 * T2_BM - 1) / (2 * T2_BM) * n_tiles + slots - 1) / slots;
  const long long alone = ((rows + T2_BM - 1) / T2_BM * n_tiles + sms - 1) / sms;
  return alone < pairs && pairs <= 5;
}
}  // namespace

// dy [M, N], w [N, K] -> out [M, K] bf16, reduction over N (input gradient of a dense layer). K a multiple of 8.
// Reductions below 512 and products of fewer waves there take the single-CTA kernel: the launch of the pair costs what its tiles save (64 and 128 columns 9 us for
// 11, from 512 on even or behind: csrc/gemm.cu 40, here 35 at 512 rows of [5120, 2048]).
PT_API int pt_dense_nn(const void* dy, const void* w, void* out, int M, int K, int N, long long lda, long long ldb, long long ldd,
                       void* stream_) {
  using namespace pt;
  if (M <= 0 || N <= 0 || K <= 0 || K % 8 != 0) return -2;
  if (N < 512 || fewer_waves_alone(M, K))
    return pt_gemm_bf16(dy, w, out, 0, M, K, N, 0, 1, M, N, lda, N, K, ldb, M, ldd, nullptr, 0, 0, 0, 0, 0, 1, 2, 0, 0, nullptr, 1, 0, stream_);
  Gemm2Args a = t2_args(M, K, N, 1);
  return t2_launch<false, true, T2_STORE>({dy, M, N, lda, lda * M}, {w, N, K, ldb, ldb * N}, {out, M, K, ldd, ldd * M}, a,
                                          static_cast<cudaStream_t>(stream_));
}

// dy [M, N], x [M, K] -> D [N, K] += dy^T x in fp32 or bf16 (weight gradient of a dense layer). N and K multiples of 8.
// fp32_sums: the error of an fp32 product, at about half the rate. Other reductions below 1024 rows, and products of fewer waves
// there, take the single-CTA kernel
// ([5120, 2048] into fp32, single / pair: 64 rows 24 / 28 us, 512 rows 31 / 32, 2048 rows 57 / 51). Launches that add to the same
// elements are ordered by the caller, as for pt_gemm_bf16.
PT_API int pt_dense_tn(const void* dy, const void* x, void* D, int out_fp32, int fp32_sums, int N, int K, int M, long long lda,
                       long long ldb, long long ldd, void* stream_) {
  using namespace pt;
  if (M <= 0 || N <= 0 || K <= 0 || N % 8 != 0 || K % 8 != 0) return -2;
  if (!fp32_sums && (M < 1024 || fewer_waves_alone(N, K)))
    return pt_gemm_bf16(dy, x, D, 0, N, K, M, 1, 1, M, N, lda, M, K, ldb, N, ldd, nullptr, 0, 0, 0, out_fp32, 1, 1, 2, 0, 0, nullptr, 1, 0,
                        stream_);
  Gemm2Args a = t2_args(N, K, M, 1);
  a.out_fp32 = out_fp32;
  const T2Mat tA{dy, M, N, lda, lda * M}, tB{x, M, K, ldb, ldb * M}, tD{D, N, K, ldd, ldd * N};
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  return fp32_sums ? t2_launch<true, true, T2_SUM, 8>(tA, tB, tD, a, stream) : t2_launch<true, true, T2_REDUCE>(tA, tB, tD, a, stream);
}

// Orthogonalisation of Muon's updates: `steps` >= 1 quintic Newton-Schulz steps X <- (s_i (bA + cA^2 + aI)) X, A = X X^T, on a stack
// Y [E, r, c] (bf16, contiguous, r and c multiples of 8), starting from s_e Y_e with the factors s [E] (fp32). Y
// keeps its orientation: a wide one takes A = Y Y^T and B Y, a tall one A = Y^T Y and Y B, B being symmetric. The first step's
// normalisation goes into the epilogues (A by s^2, B by s). Scratch: Z and Z2 like Y (Z2 may be Y itself),
// A and B [E, min, min].
// The last product updates weights: outs[i] holds the next counts[i] matrices, w = decay * w + alpha * X (decay 0: w = alpha * X).
//
// Bound by the tensor cores. Both Gram products are symmetric, so a third (three tiles a side) to 7/16 (eight) of their tiles
// need not be computed, and the addend, diagonal, scaling and weight update ride in the epilogues instead of in passes of
// their own. Five steps, library batched products with separate passes / here: 128 x [768, 2048] 3627 -> 2734 us, 64 x [1408, 2048]
// 7767 -> 4539, 64 x [2880, 2880] 41.5 -> 28.8 ms, 32 x [256, 512] 300 -> 184, one [2048, 4096] 575 -> 555 (36 tiles for 74 pairs).
PT_API int pt_muon_orthogonalize(const void* Y, void* Z, void* Z2, void* A, void* B, const float* s, int E, int r, int c, int steps,
                                 const long long* outs, const int* counts, int n_outs, float decay, float alpha, void* stream_) {
  using namespace pt;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (E <= 0 || r <= 0 || c <= 0) return 0;
  if (r % 8 != 0 || c % 8 != 0 || steps < 1) return -2;
  const bool wide = r <= c;
  const int m = wide ? r : c;
  const float ka = 3.4445f, kb = -4.7750f, kc = 2.0315f;
  const long long yy = (long long)r * c, mm = (long long)m * m;
  const T2Mat tA{A, m, m, m, mm}, tB{B, m, m, m, mm};
  const void* X = Y;
  for (int it = 0; it < steps; ++it) {
    const T2Mat tX{X, r, c, c, yy};
    Gemm2Args g = t2_args(m, m, wide ? c : r, E);
    g.sym = 1;
    if (it == 0) { g.scale = s; g.scale_pow = 2; }
    int rc = wide ? t2_launch<false, false, T2_FUSED>(tX, tX, tA, g, stream) : t2_launch<true, true, T2_FUSED>(tX, tX, tA, g, stream);
    if (rc) return rc;
    g = t2_args(m, m, m, E);
    g.sym = 1; g.alpha = kc; g.beta = kb; g.diag = ka;
    g.C = static_cast<const __nv_bfloat16*>(A); g.ldc = m; g.c_stride = mm;
    if (it == 0) g.scale = s;
    rc = t2_launch<false, false, T2_FUSED, 8>(tA, tA, tB, g, stream);
    if (rc) return rc;
    if (it < steps - 1) {
      g = t2_args(r, c, m, E);
      void* next = it % 2 == 0 ? Z : Z2;
      const T2Mat tN{next, r, c, c, yy};
      rc = wide ? t2_launch<false, true, T2_STORE>(tB, tX, tN, g, stream) : t2_launch<false, false, T2_STORE>(tX, tB, tN, g, stream);
      if (rc) return rc;
      X = next;
      continue;
    }
    long long first = 0;
    for (int i = 0; i < n_outs; ++i) {
      if (counts[i] <= 0) continue;
      g = t2_args(r, c, m, counts[i]);
      g.alpha = alpha; g.beta = decay;
      void* w = reinterpret_cast<void*>(outs[i]);
      if (decay != 0.f) { g.C = static_cast<const __nv_bfloat16*>(w); g.ldc = c; g.c_stride = yy; }
      T2Mat xi = tX, bi = tB;
      xi.p = static_cast<const __nv_bfloat16*>(X) + first * yy;
      bi.p = static_cast<const __nv_bfloat16*>(B) + first * mm;
      const T2Mat tW{w, r, c, c, yy};
      rc = wide ? t2_launch<false, true, T2_FUSED, 8>(bi, xi, tW, g, stream) : t2_launch<false, false, T2_FUSED, 8>(xi, bi, tW, g, stream);
      if (rc) return rc;
      first += counts[i];
    }
    if (first != E) return -2;
  }
  return 0;
}
