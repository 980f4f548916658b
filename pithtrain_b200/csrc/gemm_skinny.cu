// out[M, N] = x[M, K] w[N, K]^T in bf16 for few rows of x (a decode step, a short prompt). Bound by one pass over w, which the
// 256-wide tiles of csrc/gemm_2cta.cu leave to 8 to 40 SMs. Here w is the 128-row operand of the tensor core and the rows of x
// are its columns, and the K range of a tile is split over a cluster of CTAs, two of them on an SM: each sums its share in TMEM, puts it
// into its shared memory, and the CTAs of the cluster add one another's shares up, each for a part of the rows, in rank order
// and fp32 (one launch, no workspace, the same sums in every run).
#include <cooperative_groups.h>

#include "gemm_skinny.h"
#include "host_common.h"
#include "ptx.cuh"

namespace pt {
namespace cg = cooperative_groups;

constexpr int SK_BW = 128, SK_BK = 64, SK_THREADS = 192, SK_MAX_SPLIT = 8, SK_RING = 96 * 1024;
constexpr int SK_SMEM = SK_RING + 1024 + 256;
// A CTA of a cluster that waits for tensor memory holds its cluster up, so two kernels of clusters that share an SM and its tensor
// memory could wait for one another for good. The other one, csrc/gemm_2cta.cu, takes more shared memory than this one leaves.

struct SkinnyArgs {
  __nv_bfloat16* out;
  long long ldd;
  int M, N, K, split;
  int* err;
};

// TN: rows of x in a tile (columns of the accumulator).
template <int TN>
__global__ void __launch_bounds__(SK_THREADS, 2)
gemm_skinny_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const SkinnyArgs args) {
  constexpr int W_BYTES = SK_BW * SK_BK * 2, STAGE = W_BYTES + TN * SK_BK * 2, STAGES = SK_RING / STAGE;
  static_assert(TN * SK_BW * 4 <= SK_RING, "the shares of a tile take the ring's place");
  constexpr uint32_t IDESC = make_idesc(1, 1, SK_BW, TN, false, false);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + SK_RING);
  uint64_t* empty = full + STAGES;
  uint64_t* done = empty + STAGES;
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(done + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_ptr + 1);
  float* share = reinterpret_cast<float*>(smem);  // [TN][SK_BW], once the ring has been read

  cg::cluster_group cluster = cg::this_cluster();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)cluster.block_rank(), split = args.split;
  const int n0 = (int)(blockIdx.x / split) * SK_BW, m0 = (int)blockIdx.y * TN;
  const int num_kb = (args.K + SK_BK - 1) / SK_BK;
  const int kb0 = num_kb * rank / split, kb1 = num_kb * (rank + 1) / split;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    mbar_init(done, 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmW); tma_prefetch_desc(&tmX);
  }
  if (warp == 1) {
    tmem_alloc(tmem_ptr, TN);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_ptr;

  if (warp == 0) {
    if (lane == 0) {
      int it = 0;
      for (int kb = kb0; kb < kb1; ++kb, ++it) {
        const int s = it % STAGES;
        if (!mbar_wait_bounded(&empty[s], ((it / STAGES) & 1) ^ 1, abort_flag, args.err, PT_ERR_TIMEOUT_PRODUCER)) break;
        mbar_expect_tx(&full[s], STAGE);
        tma_load_2d(smem + s * STAGE, &tmW, &full[s], kb * SK_BK, n0);
        tma_load_2d(smem + s * STAGE + W_BYTES, &tmX, &full[s], kb * SK_BK, m0);
      }
      // What is still on its way lands before the ring is given another use or the block ends (bounded); the tensor core has
      // waited for all of it unless something gave up.
      const uint64_t t0 = globaltimer_ns();
      for (int j = 1; j <= it && j <= STAGES; ++j)
        while (!mbar_try_wait(&full[(it - j) % STAGES], ((it - j) / STAGES) & 1)) {
          if (globaltimer_ns() - t0 > PT_WAIT_LIMIT_NS) {
            if (args.err) atomicCAS(args.err, 0, PT_ERR_TIMEOUT_DRAIN);
            break;
          }
        }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      int it = 0;
      bool ok = true;
      for (int kb = kb0; kb < kb1; ++kb, ++it) {
        const int s = it % STAGES;
        ok = mbar_wait_bounded(&full[s], (it / STAGES) & 1, abort_flag, args.err, PT_ERR_TIMEOUT_MMA);
        if (!ok) break;
        tc_fence_after();
        const uint32_t w_addr = smem_u32(smem + s * STAGE), x_addr = w_addr + W_BYTES;
#pragma unroll
        for (int k = 0; k < SK_BK / 16; ++k)
          umma_f16(tmem, make_smem_desc_sw128(w_addr + k * 32, 16, 1024), make_smem_desc_sw128(x_addr + k * 32, 16, 1024), IDESC,
                   (it != 0 || k != 0) ? 1u : 0u);
        umma_commit(&empty[s]);
      }
      umma_commit(done);
    }
  }
  __syncwarp();
  // Everybody waits for the accumulator; its rows (features) are the lanes, 32 to a warp, its columns the rows of x.
  const bool good = mbar_wait_bounded(done, 0, abort_flag, args.err, PT_ERR_TIMEOUT_EPILOGUE);
  const bool whole = __syncthreads_and(good);
  tc_fence_after();
  if (whole && warp >= 2) {
    const int q = warp & 3, n = n0 + 32 * q + lane;
#pragma unroll 1
    for (int c0 = 0; c0 < TN; c0 += 32) {
      uint32_t v[32];
      tmem_ld_32x32(tmem + (static_cast<uint32_t>(32 * q) << 16) + c0, v);
      tmem_ld_wait();
      if (split == 1) {
#pragma unroll
        for (int i = 0; i < 32; ++i)
          if (m0 + c0 + i < args.M && n < args.N) args.out[(long long)(m0 + c0 + i) * args.ldd + n] = __float2bfloat16(__uint_as_float(v[i]));
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) share[(c0 + i) * SK_BW + 32 * q + lane] = __uint_as_float(v[i]);
      }
    }
    tc_fence_before();
  }
  if (split > 1) {
    cluster.sync();
    const int c1 = min(TN * (rank + 1) / split, args.M - m0), n = n0 + 4 * lane;
    for (int c = TN * rank / split + warp; whole && c < c1; c += SK_THREADS / 32) {
      float4 part[SK_MAX_SPLIT];
#pragma unroll
      for (int r = 0; r < SK_MAX_SPLIT; ++r)
        if (r < split) part[r] = *reinterpret_cast<const float4*>(cluster.map_shared_rank(share, r) + c * SK_BW + 4 * lane);
      float4 s = part[0];
#pragma unroll
      for (int r = 1; r < SK_MAX_SPLIT; ++r)
        if (r < split) { s.x += part[r].x; s.y += part[r].y; s.z += part[r].z; s.w += part[r].w; }
      __nv_bfloat16* o = args.out + (long long)(m0 + c) * args.ldd + n;
      if (n + 4 <= args.N) {
        *reinterpret_cast<uint2*>(o) = make_uint2(pack_bf16x2(s.x, s.y), pack_bf16x2(s.z, s.w));
      } else {
        const float e[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (n + i < args.N) o[i] = __float2bfloat16(e[i]);
      }
    }
    cluster.sync();  // nobody leaves while its share is read
  }
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, TN);
}

template <int TN>
static int skinny_launch(const void* x, const void* w, SkinnyArgs a, long long lda, long long ldb, cudaStream_t stream) {
  CUtensorMap tmW, tmX;
  if (encode_tmap_2d(&tmW, w, TM_BF16, a.N, a.K, ldb, SK_BW, SK_BK, TM_SW_128)) return -3;
  if (encode_tmap_2d(&tmX, x, TM_BF16, a.M, a.K, lda, TN, SK_BK, TM_SW_128)) return -3;
  static SmemLimit smem;
  if (smem.set(gemm_skinny_kernel<TN>, SK_SMEM) != cudaSuccess) return -4;
  const int n_tiles = (a.N + SK_BW - 1) / SK_BW, m_tiles = (a.M + TN - 1) / TN, num_kb = (a.K + SK_BK - 1) / SK_BK;
  // As many CTAs as are resident at once (two an SM, a few left over where clusters do not fit), two k-blocks or more for each.
  int split = (int)(sm_count() * 2LL * 7 / 8 / ((long long)n_tiles * m_tiles));
  if (split > SK_MAX_SPLIT) split = SK_MAX_SPLIT;
  if (split > num_kb / 2) split = num_kb / 2;
  if (split < 1) split = 1;
  a.split = split;
  a.err = device_status_word();
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(n_tiles * split), (unsigned)m_tiles);
  cfg.blockDim = dim3(SK_THREADS);
  cfg.dynamicSmemBytes = SK_SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = (unsigned)split;
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, gemm_skinny_kernel<TN>, tmW, tmX, a) == cudaSuccess ? 0 : -5;
}

// A 256-wide pair tile takes 8.5 us + 0.3 us for each k-block of its chain, however few tiles there are; here the chain is split, but
// w and x are read by 128-row tiles. Measured, cold cache, pair -> this, us:
//   N x K            64 rows        128            256            512            1024           4096
//   5120 x 2048      19.5 -> 15.2   19.5 -> 17.3   20.5 -> 18.4   21.4 -> 23.6   30.7 -> 39.9
//   2048 x 4096      29.6 -> 15.2   29.7 -> 18.4   29.5 -> 19.4   29.6 -> 20.5   29.7 -> 27.6
//   2048 x 10944     60.4 -> 20.5   60.3 -> 23.5   60.4 -> 25.5   60.4 -> 32.8   62.4 -> 51.2
//   128 x 2048       19.4 -> 10.2   18.5 -> 12.5   19.3 -> 13.2   19.5 -> 12.3   19.3 -> 13.2   19.3 -> 18.4
//   9496 x 2048      20.5 -> 17.3   21.4 -> 19.4   21.5 -> 25.5   30.8 -> 41.0
//   512 x 512                       13.3 -> 11.2   13.2 -> 12.3   13.2 -> 12.3   13.2 -> 12.3   13.3 -> 16.4
//   151936 x 2048    122 -> 116     126 -> 134     132 -> 246
// So: always up to 64 rows; up to 128 while the tiles are one wave; beyond that while each tile's chain can be split and is
// long against the number of tiles.
bool gemm_skinny_better(int M, int N, int K) {
  const long long tiles = ((N + SK_BW - 1) / SK_BW) * ((M + 127LL) / 128);
  const int num_kb = (K + SK_BK - 1) / SK_BK, sms = sm_count();
  if (M <= 64) return true;
  if (M <= 128) return tiles <= sms * 7 / 4;
  return num_kb >= 16 && tiles <= 2 * num_kb && tiles <= sms * 7 / 8;
}

int gemm_skinny_nt(const void* x, const void* w, void* out, int M, int N, int K, long long lda, long long ldb, long long ldd, cudaStream_t stream) {
  if (ldd % 8 != 0 || reinterpret_cast<uintptr_t>(out) % 16 != 0) return -3;
  SkinnyArgs a{static_cast<__nv_bfloat16*>(out), ldd, M, N, K, 1, nullptr};
  return M <= 64 ? skinny_launch<64>(x, w, a, lda, ldb, stream) : skinny_launch<128>(x, w, a, lda, ldb, stream);
}

}  // namespace pt
