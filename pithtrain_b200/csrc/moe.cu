// MoE routing and data-movement kernels, all sized from device-side counts (no host sync):
//   router_topk  : softmax -> top-k (-> renormalise) or top-k -> softmax, fwd + bwd
//   route_count / route_place : stable counting sort of (token, slot) pairs by local expert into a
//                  16-row-aligned grouped layout: offs[E+1], row_of_slot, slot_of_row
//   gather_rows  : build the expert-sorted activation matrix (pad rows zeroed)
//   combine      : out[t] = residual[t] + sum_j w[t,j] * y[row_of_slot[t,j]]   (gather-reduce, no atomics)
//   swiglu fwd / fused backward (also emits routing-weight grads and the weight-scaled activation
//                  that the down-projection wgrad consumes)
// These replace the reference's Triton scatter kernels and compiled stage-5 region
// (pithtrain/operators/token_scatter.py:38-153, pithtrain/models/qwen3_moe.py:81-89,229-245,
// pithtrain/operators/silu_mul.py:28-87, pithtrain/operators/clamped_swiglu.py:18-89).
#include <cooperative_groups.h>

#include "elementwise.cuh"
#include <mutex>

#include "host_common.h"
#include "no_alloc.h"
#include "ptx.cuh"

namespace pt {

// ----------------------------------------------------------------------------------------------
// Router: one warp per token, E <= 512 experts (E/32 values per lane), k <= 16.
// mode 0: p = softmax(logits); pick top-k of p; w = p[idx] (/ sum if renorm) * scale
// mode 1: pick top-k of logits; w = softmax over the k picked logits * scale   (GPT-OSS)
// ----------------------------------------------------------------------------------------------
constexpr int MAX_EPL = 16;  // experts per lane

template <typename T>
__device__ __forceinline__ float ld_as_float(const T* p);
template <>
__device__ __forceinline__ float ld_as_float<float>(const float* p) { return *p; }
template <>
__device__ __forceinline__ float ld_as_float<__nv_bfloat16>(const __nv_bfloat16* p) { return __bfloat162float(*p); }

// GIVEN: the experts are handed in through topk_idx (a router replay) and only their weights are computed; mode 0. A pick
// outside [0, E) has no weight: it reads as NaN.
template <typename T, bool GIVEN>
__global__ void __launch_bounds__(256)
router_topk_fwd_kernel(const T* __restrict__ logits, float* __restrict__ probs,
                       int* __restrict__ topk_idx, float* __restrict__ topk_w, int n, int E, int k,
                       int mode, int renorm, float scale) {
  const int lane = threadIdx.x & 31;
  const int tok = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (tok >= n) return;
  const int epl = (E + 31) / 32;
  float v[MAX_EPL];
  float mx = -INFINITY;
#pragma unroll
  for (int j = 0; j < MAX_EPL; ++j) {
    int e = lane + 32 * j;
    v[j] = (j < epl && e < E) ? ld_as_float(logits + (size_t)tok * E + e) : -INFINITY;
    mx = fmaxf(mx, v[j]);
  }
  mx = warp_max(mx);
  if (mode == 0) {
    float s = 0.f;
#pragma unroll
    for (int j = 0; j < MAX_EPL; ++j) {
      // a replay takes the place of a library softmax, whose exponential is right to the last bits
      v[j] = (v[j] == -INFINITY) ? 0.f : GIVEN ? exp_compensated(v[j] - mx) : __expf(v[j] - mx);
      s += v[j];
    }
    s = warp_sum(s);
    float inv = 1.f / s;
#pragma unroll
    for (int j = 0; j < MAX_EPL; ++j) {
      int e = lane + 32 * j;
      v[j] *= inv;
      if (j < epl && e < E && probs) probs[(size_t)tok * E + e] = v[j];
      if (!(j < epl && e < E)) v[j] = -1.f;  // never selected
    }
  }
  float picked_w[16];
  int picked_i[16];
  float wsum = 0.f;
  if constexpr (GIVEN) {
    for (int t = 0; t < k; ++t) {
      const int e = topk_idx[(size_t)tok * k + t];
      float mine = 0.f;
#pragma unroll
      for (int j = 0; j < MAX_EPL; ++j) if (j == (e >> 5)) mine = v[j];
      const float p = __shfl_sync(0xffffffffu, mine, e & 31);
      picked_w[t] = (e >= 0 && e < E) ? p : NAN;
      picked_i[t] = e;
      wsum += picked_w[t];
    }
  } else {
    // iterative arg-max; ties resolve to the lowest expert index
    for (int t = 0; t < k; ++t) {
      float best = -INFINITY;
      int bi = 0x7fffffff;
#pragma unroll
      for (int j = 0; j < MAX_EPL; ++j) {
        int e = lane + 32 * j;
        if (j < epl && e < E && (v[j] > best)) { best = v[j]; bi = e; }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        float ob = __shfl_xor_sync(0xffffffffu, best, o);
        int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
      }
      if (mode == 0 && bi == 0x7fffffff) {  // a row of NaN scores has no order: the first k experts, weight NaN
        bi = t;
        best = NAN;
      }
      picked_w[t] = best;
      picked_i[t] = bi;
      wsum += best;
      if ((bi & 31) == lane) {
#pragma unroll
        for (int j = 0; j < MAX_EPL; ++j) if (j == (bi >> 5)) v[j] = -INFINITY;
      }
    }
  }
  if (mode == 1) {
    // softmax over the k selected logits (picked_w[0] is the maximum)
    float s = 0.f;
    const float top = picked_w[0];
    for (int t = 0; t < k; ++t) { picked_w[t] = __expf(picked_w[t] - top); s += picked_w[t]; }
    for (int t = 0; t < k; ++t) picked_w[t] = picked_w[t] / s * scale;
  } else {
    float mul = renorm ? scale / wsum : scale;
    for (int t = 0; t < k; ++t) picked_w[t] *= mul;
  }
  if (lane == 0) {
    for (int t = 0; t < k; ++t) {
      if (!GIVEN) topk_idx[(size_t)tok * k + t] = picked_i[t];
      topk_w[(size_t)tok * k + t] = picked_w[t];
    }
  }
}

// d_logits from d_topk_w (and an optional dense d_probs, e.g. from a load-balance loss).
template <typename T>
__global__ void __launch_bounds__(256)
router_topk_bwd_kernel(const float* __restrict__ probs, const int* __restrict__ topk_idx,
                       const float* __restrict__ topk_w, const float* __restrict__ d_topk_w,
                       const float* __restrict__ d_probs, T* __restrict__ d_logits, int n, int E,
                       int k, int mode, int renorm, float scale) {
  const int lane = threadIdx.x & 31;
  const int tok = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (tok >= n) return;
  const int epl = (E + 31) / 32;
  float dp[MAX_EPL];
#pragma unroll
  for (int j = 0; j < MAX_EPL; ++j) {
    int e = lane + 32 * j;
    dp[j] = (mode == 0 && d_probs && j < epl && e < E) ? d_probs[(size_t)tok * E + e] : 0.f;
  }
  if (mode == 0) {
    // w_j = scale * p_j / s (renorm) or scale * p_j
    float s = 0.f, dot = 0.f;
    for (int t = 0; t < k; ++t) {
      float w = topk_w[(size_t)tok * k + t], dw = d_topk_w[(size_t)tok * k + t];
      int e = topk_idx[(size_t)tok * k + t];
      if (e >= 0 && e < E) s += probs[(size_t)tok * E + e];  // a replayed pick may be out of range
      dot += dw * w;
    }
    for (int t = 0; t < k; ++t) {
      int e = topk_idx[(size_t)tok * k + t];
      float dw = d_topk_w[(size_t)tok * k + t];
      float g = renorm ? (dw * scale - dot) / s : dw * scale;
      if ((e & 31) == lane) {
#pragma unroll
        for (int j = 0; j < MAX_EPL; ++j) if (j == (e >> 5)) dp[j] += g;
      }
    }
    float pd = 0.f;
    float p[MAX_EPL];
#pragma unroll
    for (int j = 0; j < MAX_EPL; ++j) {
      int e = lane + 32 * j;
      p[j] = (j < epl && e < E) ? probs[(size_t)tok * E + e] : 0.f;
      pd += p[j] * dp[j];
    }
    pd = warp_sum(pd);
#pragma unroll
    for (int j = 0; j < MAX_EPL; ++j) {
      int e = lane + 32 * j;
      if (j < epl && e < E) d_logits[(size_t)tok * E + e] = (T)(p[j] * (dp[j] - pd));
    }
  } else {
    float dot = 0.f;
    for (int t = 0; t < k; ++t) dot += d_topk_w[(size_t)tok * k + t] * topk_w[(size_t)tok * k + t];
#pragma unroll
    for (int j = 0; j < MAX_EPL; ++j) dp[j] = 0.f;
    for (int t = 0; t < k; ++t) {
      int e = topk_idx[(size_t)tok * k + t];
      float w = topk_w[(size_t)tok * k + t], dw = d_topk_w[(size_t)tok * k + t];
      // w = scale * softmax  ->  dlogit = w * (dw - sum(dw * w) / scale)
      float g = w * (dw - dot / scale);
      if ((e & 31) == lane) {
#pragma unroll
        for (int j = 0; j < MAX_EPL; ++j) if (j == (e >> 5)) dp[j] += g;
      }
    }
#pragma unroll
    for (int j = 0; j < MAX_EPL; ++j) {
      int e = lane + 32 * j;
      if (j < epl && e < E) d_logits[(size_t)tok * E + e] = (T)dp[j];
    }
  }
}

// ----------------------------------------------------------------------------------------------
// Stable counting sort by expert. One CTA per expert scans all slots in order, so ranks inside a
// group follow slot order: deterministic, no atomics. eids < 0 or >= E are skipped.
// ----------------------------------------------------------------------------------------------
constexpr int ROUTE_THREADS = 512;

__global__ void __launch_bounds__(ROUTE_THREADS)
route_count_kernel(const int* __restrict__ eids, const int* __restrict__ n_ptr, int n_max, int E,
                   int* __restrict__ counts) {
  __shared__ float red[32];
  const int e = blockIdx.x;
  const int n = n_ptr ? min(*n_ptr, n_max) : n_max;
  int c = 0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) c += (eids[i] == e);
  float tot = block_sum((float)c, red);
  if (threadIdx.x == 0) counts[e] = (int)(tot + 0.5f);
}

__global__ void __launch_bounds__(ROUTE_THREADS)
route_place_kernel(const int* __restrict__ eids, const int* __restrict__ n_ptr, int n_max, int E,
                   int align, const int* __restrict__ counts, int* __restrict__ offs,
                   int* __restrict__ row_of_slot, int* __restrict__ slot_of_row, int r_cap,
                   int* __restrict__ err) {
  __shared__ int warp_tot[ROUTE_THREADS / 32];
  __shared__ int base_sh;
  const int e = blockIdx.x;
  const int n = n_ptr ? min(*n_ptr, n_max) : n_max;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  if (threadIdx.x == 0) {
    int b = 0;
    for (int j = 0; j < e; ++j) b += (counts[j] + align - 1) / align * align;
    base_sh = b;
    offs[e] = b;
    if (e == E - 1) {
      int end = b + (counts[e] + align - 1) / align * align;
      offs[E] = end;
      if (end > r_cap && err) atomicCAS(err, 0, PT_ERR_CAPACITY);
    }
  }
  __syncthreads();
  int base = base_sh;
  const int my_rows = (counts[e] + align - 1) / align * align;
  if (base + my_rows > r_cap) return;  // overflow reported by the last block
  int running = 0;
  for (int start = 0; start < n; start += blockDim.x) {
    int i = start + threadIdx.x;
    bool hit = (i < n) && (eids[i] == e);
    unsigned m = __ballot_sync(0xffffffffu, hit);
    int before = __popc(m & ((1u << lane) - 1));
    if (lane == 0) warp_tot[w] = __popc(m);
    __syncthreads();
    int woff = 0, tot = 0;
    for (int j = 0; j < nw; ++j) { int t = warp_tot[j]; if (j < w) woff += t; tot += t; }
    if (hit) {
      int r = base + running + woff + before;
      row_of_slot[i] = r;
      slot_of_row[r] = i;
    }
    running += tot;
    __syncthreads();
  }
  // pad rows of this group
  for (int r = base + counts[e] + threadIdx.x; r < base + my_rows; r += blockDim.x) slot_of_row[r] = -1;
}

// Slots that were skipped (eid < 0) get row -1; rows past offs[E] get slot -1.
__global__ void route_fill_kernel(const int* __restrict__ eids, const int* __restrict__ n_ptr,
                                  int n_max, int E, const int* __restrict__ offs,
                                  int* __restrict__ row_of_slot, int* __restrict__ slot_of_row,
                                  int r_cap) {
  const int n = n_ptr ? min(*n_ptr, n_max) : n_max;
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n_max) {
    if (i >= n || eids[i] < 0 || eids[i] >= E) row_of_slot[i] = -1;
  }
  int end = min(offs[E], r_cap);
  if (i < r_cap && i >= end) slot_of_row[i] = -1;
}

// ----------------------------------------------------------------------------------------------
// gather_rows: dst[r] = src[idx[r] / div]  (zero row when idx[r] < 0). One warp per row, 16B vectors.
// ----------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
gather_rows_kernel(const __nv_bfloat16* __restrict__ src, const int* __restrict__ idx, int div,
                   __nv_bfloat16* __restrict__ dst, const int* __restrict__ n_rows_ptr,
                   int n_rows_max, int H, long long src_stride) {
  const int n_rows = n_rows_ptr ? min(*n_rows_ptr, n_rows_max) : n_rows_max;
  const int lane = threadIdx.x & 31;
  const int wpb = blockDim.x >> 5;
  for (int r = blockIdx.x * wpb + (threadIdx.x >> 5); r < n_rows; r += gridDim.x * wpb) {
    int s = idx[r];
    uint4* d = reinterpret_cast<uint4*>(dst + (size_t)r * H);
    if (s < 0) {
      for (int c = lane; c < H / 8; c += 32) d[c] = make_uint4(0, 0, 0, 0);
    } else {
      const uint4* p = reinterpret_cast<const uint4*>(src + (size_t)(s / div) * src_stride);
      for (int c = lane; c < H / 8; c += 32) d[c] = p[c];
    }
  }
}

// ----------------------------------------------------------------------------------------------
// embedding gradient: grad[ids[r]] += dy[r], fp32 from bf16. Bound by the rows of dy once and the touched rows of grad twice. A warp
// has 256 columns of EB_ROWS rows that follow one another, 8 columns a lane in two four-wide reductions, which the L2 performs, so
// that equal ids need no order; those of neighbours (padding) are added up first, since reductions of one address wait for one
// another. An id outside the table is recorded and skipped.
// ----------------------------------------------------------------------------------------------
constexpr int EB_ROWS = 8;

__global__ void __launch_bounds__(256)
embedding_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const long long* __restrict__ ids, float* __restrict__ grad, int n, int H,
                     long long V, int* __restrict__ err) {
  const int lane = threadIdx.x & 31, warps = blockDim.x >> 5, slices = (H + 255) / 256;
  const long long items = (long long)((n + EB_ROWS - 1) / EB_ROWS) * slices;
  for (long long item = (long long)blockIdx.x * warps + (threadIdx.x >> 5); item < items; item += (long long)gridDim.x * warps) {
    const int r0 = (int)(item / slices) * EB_ROWS, c = (int)(item % slices) * 256 + lane * 8;
    long long mine = lane < EB_ROWS && r0 + lane < n ? ids[r0 + lane] : -1;
    if (mine < 0 || mine >= V) {
      if (lane < EB_ROWS && r0 + lane < n) atomicCAS(err, 0, PT_ERR_BOUNDS);
      mine = -1;
    }
    uint4 row[EB_ROWS];
#pragma unroll
    for (int i = 0; i < EB_ROWS; ++i)
      if (r0 + i < n && c < H) row[i] = *reinterpret_cast<const uint4*>(dy + (size_t)(r0 + i) * H + c);
    float sum[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    long long id = __shfl_sync(0xffffffffu, mine, 0);
#pragma unroll
    for (int i = 0; i < EB_ROWS; ++i) {
      const long long next = i + 1 < EB_ROWS ? __shfl_sync(0xffffffffu, mine, (i + 1) % EB_ROWS) : -1;
      if (id >= 0 && c < H) {
        float v[8];
        load8(reinterpret_cast<const __nv_bfloat16*>(&row[i]), v);
#pragma unroll
        for (int e = 0; e < 8; ++e) sum[e] += v[e];
        if (next != id) {
          float* g = grad + (size_t)id * H + c;
          asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(g), "f"(sum[0]), "f"(sum[1]), "f"(sum[2]), "f"(sum[3]) : "memory");
          asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(g + 4), "f"(sum[4]), "f"(sum[5]), "f"(sum[6]), "f"(sum[7]) : "memory");
#pragma unroll
          for (int e = 0; e < 8; ++e) sum[e] = 0.f;
        }
      }
      id = next;
    }
  }
}

// ----------------------------------------------------------------------------------------------
// combine: out[t] = (res ? res[t] : 0) + sum_{j<k, row>=0} (w ? w[t,j] : 1) * y[row_of_slot[t*k+j]]
// fp32 accumulation in slot order, in one of two kernels (pt_combine says when).
// ----------------------------------------------------------------------------------------------
// A warp a token, one row after the other: for many tokens of few or short rows.
__global__ void __launch_bounds__(256)
combine_warp_kernel(const __nv_bfloat16* __restrict__ y, const int* __restrict__ row_of_slot, const float* __restrict__ w,
                    const __nv_bfloat16* __restrict__ res, __nv_bfloat16* __restrict__ out, const int* __restrict__ n_ptr, int n_max,
                    int k, int H) {
  const int n = n_ptr ? min(*n_ptr, n_max) : n_max;
  const int lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  for (int t = blockIdx.x * warps + (threadIdx.x >> 5); t < n; t += gridDim.x * warps) {
    for (int c0 = lane * 8; c0 < H; c0 += 256) {
      float acc[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] = 0.f;
      if (res) load8(res + (size_t)t * H + c0, acc);
      for (int j = 0; j < k; ++j) {
        const int r = row_of_slot[(size_t)t * k + j];
        if (r < 0) continue;
        const float f = w ? w[(size_t)t * k + j] : 1.f;
        float v[8];
        load8(y + (size_t)r * H + c0, v);
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[e] += f * v[e];
      }
      store8(out + (size_t)t * H + c0, acc);
    }
  }
}

// The ring. Bound by the bytes of the rows, if enough of them are on their way: a row is contiguous, so
// one warp of the block fetches rows by bulk copies into a ring in shared memory, four rows of a token to a stage, a lane to a
// row; the other warps add them up, a thread 8 columns wide. Rows in flight then cost shared memory and no registers. A block
// has a run of tokens that follow one another, so that a load of 32 indices is several tokens' worth and is asked for one load
// ahead. Tokens of more than CB_COLS columns are walked in slices of equal width, one after the other.
// ----------------------------------------------------------------------------------------------
constexpr int CB_ROWS = 4, CB_STAGES = 8, CB_COLS = 4096;

__global__ void __launch_bounds__(CB_COLS / 8 + 32)
combine_kernel(const __nv_bfloat16* __restrict__ y, const int* __restrict__ row_of_slot, const float* __restrict__ w,
               const __nv_bfloat16* __restrict__ res, __nv_bfloat16* __restrict__ out, const int* __restrict__ n_ptr, int n_max,
               int k, int H, int slices, int W, int stages, int* __restrict__ err) {
  extern __shared__ __align__(128) uint8_t ring[];
  __shared__ uint64_t full[CB_STAGES], empty[CB_STAGES];
  __shared__ float weight_of[CB_STAGES][CB_ROWS];
  __shared__ int present[CB_STAGES][CB_ROWS];
  __shared__ int abort_flag;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, adders = (blockDim.x >> 5) - 1;
  if (threadIdx.x == 0) {
    for (int i = 0; i < stages; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], adders); }
    abort_flag = 0;
    mbar_fence_init();
  }
  __syncthreads();
  const int n = n_ptr ? min(*n_ptr, n_max) : n_max;
  const long long items = (long long)n * slices;
  const size_t row_bytes = (size_t)W * 2;
  int stage = 0;
  uint32_t phase = 0;
  const long long first = items * blockIdx.x / gridDim.x, last = items * (blockIdx.x + 1) / gridDim.x;
  if (warp == adders) {
    int id = -1, next_id = -1;  // slots base + lane, base + 32 + lane
    float f = 1.f, next_f = 1.f;
    const long long slots = (long long)n * k;
    long long base = 0, armed = 0;
    auto fetch = [&](long long slot, int& i, float& v) {
      i = slot < slots ? row_of_slot[slot] : -1;
      v = slot < slots && w ? w[slot] : 1.f;
    };
    bool ok = true;
    for (long long item = first; ok && item < last; ++item) {
      const int s = (int)(item / n), c0 = s * W;
      const long long t = item - (long long)s * n;
      const uint32_t bytes = (uint32_t)min(W, H - c0) * 2;
      if (item == first || t == 0) {
        base = t * k;
        fetch(base + lane, id, f);
        fetch(base + 32 + lane, next_id, next_f);
      }
      for (int j0 = 0; j0 < k; j0 += CB_ROWS) {
        if (t * k + j0 - base >= 32) {
          base += 32;
          id = next_id;
          f = next_f;
          fetch(base + 32 + lane, next_id, next_f);
        }
        ok = mbar_wait_bounded_warp(&empty[stage], phase ^ 1, &abort_flag, err, PT_ERR_TIMEOUT_PRODUCER);
        if (!ok) break;
        const int at = (int)(t * k + j0 - base) + lane;  // below 64 in the lanes that count
        const int near = __shfl_sync(0xffffffffu, id, at & 31), far = __shfl_sync(0xffffffffu, next_id, at & 31);
        const float near_f = __shfl_sync(0xffffffffu, f, at & 31), far_f = __shfl_sync(0xffffffffu, next_f, at & 31);
        const int row = lane >= min(CB_ROWS, k - j0) ? -1 : at < 32 ? near : far;
        if (lane < CB_ROWS) {
          weight_of[stage][lane] = at < 32 ? near_f : far_f;
          present[stage][lane] = row >= 0;
        }
        const uint32_t rows = __popc(__ballot_sync(0xffffffffu, row >= 0));
        __syncwarp();
        if (lane == 0) mbar_expect_tx(&full[stage], rows * bytes);
        __syncwarp();
        if (row >= 0) bulk_load_1d(ring + (stage * CB_ROWS + lane) * row_bytes, y + (size_t)row * H + c0, bytes, &full[stage]);
        ++armed;
        if (++stage == stages) { stage = 0; phase ^= 1; }
      }
    }
    if (!ok) {  // the copies that are still on their way end before the block does
      for (int back = 0; back < stages && back < armed; ++back) {
        if (--stage < 0) { stage = stages - 1; phase ^= 1; }
        const uint64_t t0 = globaltimer_ns();
        while (!mbar_try_wait(&full[stage], phase) && globaltimer_ns() - t0 < PT_WAIT_LIMIT_NS) {}
      }
    }
    return;
  }
  const int c = threadIdx.x * 8;
  for (long long item = first; item < last; ++item) {
    const int s = (int)(item / n), c0 = s * W;
    const long long t = item - (long long)s * n;
    const bool in = c < min(W, H - c0);
    const size_t at = (size_t)t * H + c0 + c;
    float acc[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e] = 0.f;
    if (res && in) load8(res + at, acc);
    for (int j0 = 0; j0 < k; j0 += CB_ROWS) {
      if (!mbar_wait_bounded(&full[stage], phase, &abort_flag, err, PT_ERR_TIMEOUT_EPILOGUE)) return;
#pragma unroll
      for (int u = 0; u < CB_ROWS; ++u) {
        if (!in || !present[stage][u]) continue;
        const float f = weight_of[stage][u];
        float v[8];
        load8(reinterpret_cast<const __nv_bfloat16*>(ring + (stage * CB_ROWS + u) * row_bytes) + c, v);
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[e] += f * v[e];
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[stage]);
      if (++stage == stages) { stage = 0; phase ^= 1; }
    }
    if (in) store8(out + at, acc);
  }
}

// ----------------------------------------------------------------------------------------------
// SwiGLU. gu is [R, 2I]: gate = cols [0,I), up = cols [I,2I) (interleaved = 0) or gate = even cols,
// up = odd cols (interleaved = 1, GPT-OSS). limit > 0 enables the clamped form
//   gc = min(g, limit), uc = clamp(u, +-limit), act = (uc + 1) * gc * sigmoid(alpha * gc).
// Plain form: act = silu(g) * u.
// ----------------------------------------------------------------------------------------------
__device__ __forceinline__ void swiglu_point(float g, float u, float alpha, float limit, float& act,
                                             float& dact_dg, float& dact_du) {
  if (limit > 0.f) {
    float gc = fminf(g, limit), uc = fminf(fmaxf(u, -limit), limit);
    float sg = 1.f / (1.f + __expf(-alpha * gc));
    float glu = gc * sg;
    act = (uc + 1.f) * glu;
    float dglu = sg + alpha * gc * sg * (1.f - sg);
    dact_dg = (g <= limit) ? (uc + 1.f) * dglu : 0.f;
    dact_du = (u >= -limit && u <= limit) ? glu : 0.f;
  } else {
    float sg = 1.f / (1.f + __expf(-g));
    act = g * sg * u;
    dact_dg = u * (sg + g * sg * (1.f - sg));
    dact_du = g * sg;
  }
}

__global__ void __launch_bounds__(256)
swiglu_fwd_kernel(const __nv_bfloat16* __restrict__ gu, __nv_bfloat16* __restrict__ act,
                  const int* __restrict__ n_rows_ptr, int n_rows_max, int I, int interleaved,
                  float alpha, float limit) {
  const int n_rows = n_rows_ptr ? min(*n_rows_ptr, n_rows_max) : n_rows_max;
  const int vec_per_row = I / 8;
  const long long total = (long long)n_rows * vec_per_row;
  for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < total;
       v += (long long)gridDim.x * blockDim.x) {
    int r = (int)(v / vec_per_row), c = (int)(v % vec_per_row) * 8;
    float g[8], u[8], o[8];
    const __nv_bfloat16* row = gu + (size_t)r * 2 * I;
    if (!interleaved) {
      load8(row + c, g);
      load8(row + I + c, u);
    } else {
      float a[8], b[8];
      load8(row + 2 * c, a);
      load8(row + 2 * c + 8, b);
#pragma unroll
      for (int e = 0; e < 4; ++e) { g[e] = a[2 * e]; u[e] = a[2 * e + 1]; g[e + 4] = b[2 * e]; u[e + 4] = b[2 * e + 1]; }
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) { float dg, du; swiglu_point(g[e], u[e], alpha, limit, o[e], dg, du); }
    store8(act + (size_t)r * I + c, o);
  }
}

// Backward with optional per-row routing weight. One warp per row.
//   dact_in      : gradient w.r.t. the (unweighted) activation            [R, I]
//   row_w        : per-row routing weight (nullable -> 1)                  [R]
//   dgu          : out, gradient w.r.t. gu = row_w * dact_in * d act/d gu  [R, 2I]
//   act_scaled   : out (nullable), row_w * act  — wgrad operand of the down projection
//   d_row_w      : out (nullable), <dact_in, act>
__global__ void __launch_bounds__(256)
swiglu_bwd_kernel(const __nv_bfloat16* __restrict__ gu, const __nv_bfloat16* __restrict__ dact_in,
                  const float* __restrict__ row_w, __nv_bfloat16* __restrict__ dgu,
                  __nv_bfloat16* __restrict__ act_scaled, float* __restrict__ d_row_w,
                  const int* __restrict__ n_rows_ptr, int n_rows_max, int I, int interleaved,
                  float alpha, float limit, const int* __restrict__ slot_of_row) {
  const int n_rows = n_rows_ptr ? min(*n_rows_ptr, n_rows_max) : n_rows_max;
  const int lane = threadIdx.x & 31;
  const int wpb = blockDim.x >> 5;
  for (int r = blockIdx.x * wpb + (threadIdx.x >> 5); r < n_rows; r += gridDim.x * wpb) {
    // with slot_of_row, row_w and d_row_w are indexed by the row's (token, slot) index instead of the row
    const int widx = slot_of_row ? slot_of_row[r] : r;
    const float wt = row_w ? (widx >= 0 ? row_w[widx] : 0.f) : 1.f;
    const __nv_bfloat16* row = gu + (size_t)r * 2 * I;
    __nv_bfloat16* drow = dgu + (size_t)r * 2 * I;
    float dot = 0.f;
    for (int c = lane * 8; c < I; c += 256) {
      float g[8], u[8], d[8], a[8], dg[8], du[8];
      if (!interleaved) {
        load8(row + c, g);
        load8(row + I + c, u);
      } else {
        float x[8], y[8];
        load8(row + 2 * c, x);
        load8(row + 2 * c + 8, y);
#pragma unroll
        for (int e = 0; e < 4; ++e) { g[e] = x[2 * e]; u[e] = x[2 * e + 1]; g[e + 4] = y[2 * e]; u[e + 4] = y[2 * e + 1]; }
      }
      load8(dact_in + (size_t)r * I + c, d);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        float pg, pu;
        swiglu_point(g[e], u[e], alpha, limit, a[e], pg, pu);
        dot += d[e] * a[e];
        dg[e] = wt * d[e] * pg;
        du[e] = wt * d[e] * pu;
        a[e] *= wt;
      }
      if (!interleaved) {
        store8(drow + c, dg);
        store8(drow + I + c, du);
      } else {
        float x[8], y[8];
#pragma unroll
        for (int e = 0; e < 4; ++e) { x[2 * e] = dg[e]; x[2 * e + 1] = du[e]; y[2 * e] = dg[e + 4]; y[2 * e + 1] = du[e + 4]; }
        store8(drow + 2 * c, x);
        store8(drow + 2 * c + 8, y);
      }
      if (act_scaled) store8(act_scaled + (size_t)r * I + c, a);
    }
    if (d_row_w) {
      dot = warp_sum(dot);
      if (lane == 0 && widx >= 0) d_row_w[widx] = dot;
    }
  }
}


// ----------------------------------------------------------------------------------------------
// Per-expert biases on expert-sorted rows (GPT-OSS). Takes the role of the reference's
// pithtrain/operators/indexed_bias_add.py (forward :54-83, segmented bias gradient :20-51).
//   indexed_bias_add: out[r] = x[r] + bias[group(r)], group(r) found by binary search in offs; one warp per row.
//   row_bias_dot:     dw[slot_of_row[r]] += <x[r], bias[group(r)]>, fp32: what a bias behind the routing weight adds to that
//                     weight's gradient. One warp per row; as tensor ops it was three fp32 passes over the rows.
//   segment_sum:      out[g, c] = sum over rows of group g of x[r, c] * (row_w ? row_w[r] : 1), fp32, no atomics: one CTA per
//                     (group, 64-column slab); its eight warps split the rows, four in flight each, and are added in a fixed
//                     order (deterministic). One thread per column pair walked a chain of rows / 2 loads (two
//                     calls of 256 rows x 2880 and x 5760 in 32 groups: 202 -> 78 us).
// ----------------------------------------------------------------------------------------------
__device__ __forceinline__ int group_of_row(const int* __restrict__ offs, int E, int r) {
  int lo = 0, hi = E - 1;  // largest g with offs[g] <= r (rows past offs[E] map to the last group)
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (offs[mid] <= r) lo = mid; else hi = mid - 1;
  }
  return lo;
}

__global__ void __launch_bounds__(256)
indexed_bias_add_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ bias,
                        const int* __restrict__ offs, int E, __nv_bfloat16* __restrict__ out,
                        const int* __restrict__ n_rows_ptr, int n_rows_max, int H) {
  const int n_rows = n_rows_ptr ? min(*n_rows_ptr, n_rows_max) : n_rows_max;
  const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
  for (int r = blockIdx.x * wpb + (threadIdx.x >> 5); r < n_rows; r += gridDim.x * wpb) {
    const int g = group_of_row(offs, E, r);
    const uint4* xr = reinterpret_cast<const uint4*>(x + (size_t)r * H);
    const uint4* br = reinterpret_cast<const uint4*>(bias + (size_t)g * H);
    uint4* orow = reinterpret_cast<uint4*>(out + (size_t)r * H);
    for (int c = lane; c < H / 8; c += 32) {
      const uint4 a = xr[c], b = br[c];
      const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, bw[4] = {b.x, b.y, b.z, b.w};
      uint32_t o[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 u = unpack_bf16x2(aw[i]), v = unpack_bf16x2(bw[i]);
        o[i] = pack_bf16x2(u.x + v.x, u.y + v.y);
      }
      orow[c] = make_uint4(o[0], o[1], o[2], o[3]);
    }
  }
}

__global__ void __launch_bounds__(256)
row_bias_dot_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ bias, const int* __restrict__ offs, int E,
                    const int* __restrict__ slot_of_row, float* __restrict__ dw, const int* __restrict__ n_rows_ptr, int n_rows_max, int H) {
  const int n_rows = n_rows_ptr ? min(*n_rows_ptr, n_rows_max) : n_rows_max;
  const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
  for (int r = blockIdx.x * wpb + (threadIdx.x >> 5); r < n_rows; r += gridDim.x * wpb) {
    const int slot = slot_of_row[r];
    if (slot < 0) continue;  // a pad row
    const __nv_bfloat16 *xr = x + (size_t)r * H, *br = bias + (size_t)group_of_row(offs, E, r) * H;
    float acc = 0.f;
    for (int c = lane * 8; c < H; c += 256) {
      float a[8], b[8];
      load8(xr + c, a);
      load8(br + c, b);
#pragma unroll
      for (int i = 0; i < 8; ++i) acc = fmaf(a[i], b[i], acc);
    }
    acc = warp_sum(acc);
    if (lane == 0) dw[slot] += acc;  // a slot has one row
  }
}

constexpr int SEG_WARPS = 8;
template <typename T>
__global__ void __launch_bounds__(32 * SEG_WARPS)
segment_sum_kernel(const T* __restrict__ x, const float* __restrict__ row_w, const int* __restrict__ offs,
                   float* __restrict__ out, int H) {
  __shared__ float2 red[SEG_WARPS][32];
  const int g = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = (blockIdx.y * 32 + lane) * 2;
  const int r0 = offs[g], r1 = offs[g + 1];
  float2 acc[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) acc[u] = make_float2(0.f, 0.f);
  if (c < H) {
    for (int r = r0 + warp; r < r1; r += 4 * SEG_WARPS) {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int q = r + u * SEG_WARPS;
        if (q < r1) {
          float2 v;
          if constexpr (sizeof(T) == 2) v = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(x + (size_t)q * H + c));
          else v = *reinterpret_cast<const float2*>(x + (size_t)q * H + c);
          const float w = row_w ? row_w[q] : 1.f;
          acc[u].x = fmaf(v.x, w, acc[u].x);
          acc[u].y = fmaf(v.y, w, acc[u].y);
        }
      }
    }
  }
  red[warp][lane] = make_float2((acc[0].x + acc[1].x) + (acc[2].x + acc[3].x), (acc[0].y + acc[1].y) + (acc[2].y + acc[3].y));
  __syncthreads();
  if (warp == 0 && c < H) {
    float2 s = red[0][lane];
#pragma unroll
    for (int i = 1; i < SEG_WARPS; ++i) { s.x += red[i][lane].x; s.y += red[i][lane].y; }
    *reinterpret_cast<float2*>(out + (size_t)g * H + c) = s;
  }
}

// out[t, j] = (t + j * stride) mod E: one launch for the five tensor operations of a balanced replay.
template <typename T>
__global__ void __launch_bounds__(256) balanced_replay_kernel(T* __restrict__ out, long long total, int k, int E, int stride) {
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  if (i < total) out[i] = (T)((i / k + (i % k) * stride) % E);
}

}  // namespace pt

using namespace pt;

static inline int grid_for(long long work_items, int per_block, int cap_mult = 8) {
  long long g = (work_items + per_block - 1) / per_block;
  long long cap = (long long)sm_count() * cap_mult;
  if (g > cap) g = cap;
  return g < 1 ? 1 : (int)g;
}

PT_API int pt_router_topk_fwd(const void* logits, int logits_fp32, float* probs, int* topk_idx,
                              float* topk_w, int n, int E, int k, int mode, int renorm, float scale,
                              void* stream_) {
  cudaStream_t st = (cudaStream_t)stream_;
  if (n <= 0) return 0;
  if (E > 32 * MAX_EPL || k > 16 || k > E) return -1;
  int grid = (n + 7) / 8;
  if (logits_fp32)
    router_topk_fwd_kernel<float, false><<<grid, 256, 0, st>>>((const float*)logits, probs, topk_idx, topk_w, n, E, k, mode, renorm, scale);
  else
    router_topk_fwd_kernel<__nv_bfloat16, false><<<grid, 256, 0, st>>>((const __nv_bfloat16*)logits, probs, topk_idx, topk_w, n, E, k, mode, renorm, scale);
  return (int)cudaGetLastError();
}

// Weights of given picks (int32 [n, k]): w = softmax(logits)[idx] (/ their sum if renorm) * scale; probs [n, E] is written.
// pt_router_topk_bwd with mode 0 differentiates it.
PT_API int pt_router_given_fwd(const void* logits, int logits_fp32, float* probs, const int* idx, float* w, int n, int E, int k, int renorm,
                               float scale, void* stream_) {
  cudaStream_t st = (cudaStream_t)stream_;
  if (n <= 0) return 0;
  if (E > 32 * MAX_EPL || k > 16 || k <= 0) return -1;
  const int grid = (n + 7) / 8;
  int* picks = const_cast<int*>(idx);  // read only
  if (logits_fp32)
    router_topk_fwd_kernel<float, true><<<grid, 256, 0, st>>>((const float*)logits, probs, picks, w, n, E, k, 0, renorm, scale);
  else
    router_topk_fwd_kernel<__nv_bfloat16, true><<<grid, 256, 0, st>>>((const __nv_bfloat16*)logits, probs, picks, w, n, E, k, 0, renorm, scale);
  return (int)cudaGetLastError();
}

// out: int32 or int64 [n, k]; E / k == 0 (more slots than experts) gives all slots of a token the same expert.
PT_API int pt_balanced_replay(void* out, int is_int64, int n, int k, int E, void* stream_) {
  if (n <= 0) return 0;
  if (k <= 0 || E <= 0) return -2;
  const long long total = (long long)n * k;
  const unsigned grid = (unsigned)((total + 255) / 256);
  if (is_int64) balanced_replay_kernel<long long><<<grid, 256, 0, (cudaStream_t)stream_>>>((long long*)out, total, k, E, E / k);
  else balanced_replay_kernel<int><<<grid, 256, 0, (cudaStream_t)stream_>>>((int*)out, total, k, E, E / k);
  return (int)cudaGetLastError();
}

PT_API int pt_router_topk_bwd(const float* probs, const int* topk_idx, const float* topk_w,
                              const float* d_topk_w, const float* d_probs, void* d_logits,
                              int dlogits_fp32, int n, int E, int k, int mode, int renorm,
                              float scale, void* stream_) {
  cudaStream_t st = (cudaStream_t)stream_;
  if (n <= 0) return 0;
  if (E > 32 * MAX_EPL || k > 16) return -1;
  int grid = (n + 7) / 8;
  if (dlogits_fp32)
    router_topk_bwd_kernel<float><<<grid, 256, 0, st>>>(probs, topk_idx, topk_w, d_topk_w, d_probs, (float*)d_logits, n, E, k, mode, renorm, scale);
  else
    router_topk_bwd_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>(probs, topk_idx, topk_w, d_topk_w, d_probs, (__nv_bfloat16*)d_logits, n, E, k, mode, renorm, scale);
  return (int)cudaGetLastError();
}

// ----------------------------------------------------------------------------------------------
// Routing sort in one launch: a cluster of eight CTAs, 256 warps, each with a run of consecutive slots.
//   count: every warp counts the experts of its run in shared memory; a CTA's warps are summed up in slot order
//   scan : the CTAs read one another's totals (distributed shared memory); group offsets by a block scan, in every CTA alike
//   place: every warp walks its run in slot order; match.any groups the lanes of one expert, so a slot's row is
//          offs[e] + (slots of e in earlier runs) + (earlier slots of e in this run)
// The result is the same stable order as the per-expert kernels above. Bound by the chain of its phases, not by its 8 bytes a
// slot: histogram, scan, placement and pad rows as four launches took 15 us on the device at 64 x 8 slots and 128 experts (21.5 at
// 4096 x 8, 134 at 65536 x 8) and 16 us of launches, this 5.4 (10, 79) and 5.
// ----------------------------------------------------------------------------------------------
constexpr int RS_CTAS = 8, RS_WARPS = 32;
constexpr int RS_MAX_E = 1024;  // one expert a thread in the scan

__global__ void __cluster_dims__(RS_CTAS, 1, 1) __launch_bounds__(RS_WARPS * 32)
route_sort_kernel(const int* __restrict__ eids, const int* __restrict__ n_ptr, int n_max, int E, int align, int* __restrict__ offs,
                  int* __restrict__ row_of_slot, int* __restrict__ slot_of_row, int r_cap, int* __restrict__ err) {
  extern __shared__ int sh[];  // [RS_WARPS][E] counts, then rows before each warp's run; [E] totals of this CTA; [E] first rows
  __shared__ int warp_sum[RS_WARPS];
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  int* hist = sh;
  int* tot = sh + RS_WARPS * E;
  int* base = tot + E;
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const int n = n_ptr ? max(0, min(*n_ptr, n_max)) : n_max;
  const int warps = RS_CTAS * RS_WARPS;
  const int run_len = ((n_max + warps - 1) / warps + 31) / 32 * 32;
  const long long begin64 = (long long)(rank * RS_WARPS + w) * run_len;
  const int begin = (int)min(begin64, (long long)n_max);
  const int hard_end = (int)min(begin64 + run_len, (long long)n_max), end = min(hard_end, n);

  for (int i = tid; i < RS_WARPS * E; i += blockDim.x) hist[i] = 0;
  __syncthreads();
  int* mine = hist + w * E;
  for (int i = begin + lane; i < end; i += 32) {
    const int e = eids[i];
    if (e >= 0 && e < E) atomicAdd(&mine[e], 1);
  }
  __syncthreads();
  if (tid < E) {
    int run = 0;
    for (int v = 0; v < RS_WARPS; ++v) {
      const int c = hist[v * E + tid];
      hist[v * E + tid] = run;
      run += c;
    }
    tot[tid] = run;
  }
  cluster.sync();
  int before = 0, all = 0;
  if (tid < E) {
    for (int r = 0; r < RS_CTAS; ++r) {
      const int c = cluster.map_shared_rank(tot, r)[tid];
      before += r < rank ? c : 0;
      all += c;
    }
  }
  cluster.sync();  // nobody leaves while its totals are read
  const int padded = (all + align - 1) / align * align;  // 0 for threads past the experts
  int incl = padded;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int up = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += up;
  }
  if (lane == 31) warp_sum[w] = incl;
  __syncthreads();
  int before_warp = 0, rows = 0;
  for (int v = 0; v < RS_WARPS; ++v) {
    before_warp += v < w ? warp_sum[v] : 0;
    rows += warp_sum[v];
  }
  const int first = before_warp + incl - padded;
  const bool fits = rows <= r_cap;
  if (rank == 0) {
    if (tid < E) offs[tid] = first;
    if (tid == 0) {
      offs[E] = rows;
      if (!fits && err) atomicCAS(err, 0, PT_ERR_CAPACITY);
    }
  }
  if (tid < E) {
    base[tid] = first + before;
    if (fits && tid % RS_CTAS == rank)
      for (int r = first + all; r < first + padded; ++r) slot_of_row[r] = -1;  // pad rows of the group
  }
  __syncthreads();
  // rows past the last group; without room for the groups, all of them
  for (int r = (fits ? rows : 0) + rank * (int)blockDim.x + tid; r < r_cap; r += RS_CTAS * (int)blockDim.x) slot_of_row[r] = -1;
  for (int i0 = begin; i0 < hard_end; i0 += 32) {
    const int i = i0 + lane;
    const int e = i < end ? eids[i] : -1;
    const bool valid = fits && e >= 0 && e < E;
    const unsigned peers = __match_any_sync(0xffffffffu, valid ? e : -1);
    const int earlier = __popc(peers & ((1u << lane) - 1));
    const int ahead = valid ? mine[e] : 0;
    __syncwarp();
    if (valid) {
      const int r = base[e] + ahead + earlier;
      row_of_slot[i] = r;
      slot_of_row[r] = i;
      if (earlier == 0) mine[e] = ahead + __popc(peers);
    } else if (i < hard_end) {
      row_of_slot[i] = -1;
    }
    __syncwarp();
  }
}

// Stable sort of n slots by expert id into groups aligned to `align` rows: offs [E+1], row_of_slot [n_max], slot_of_row [r_cap].
// Up to 1024 experts one launch; beyond, the per-expert kernels (3 launches, counts [E] scratch, counts_len >= E).
PT_API int pt_route_sort(const int* eids, const int* n_ptr, int n_max, int E, int align,
                         int* counts, long long counts_len, int* offs, int* row_of_slot, int* slot_of_row, int r_cap,
                         void* stream_) {
  cudaStream_t st = (cudaStream_t)stream_;
  if (E <= 0 || n_max < 0 || align <= 0 || r_cap < 0) return -1;
  if (E <= RS_MAX_E) {
    const int smem = (RS_WARPS + 2) * E * (int)sizeof(int);
    static SmemLimit limit;
    if (const cudaError_t e = limit.set(route_sort_kernel, (RS_WARPS + 2) * RS_MAX_E * (int)sizeof(int))) return (int)e;
    route_sort_kernel<<<RS_CTAS, RS_WARPS * 32, smem, st>>>(eids, n_ptr, n_max, E, align, offs, row_of_slot, slot_of_row, r_cap, device_status_word());
    return (int)cudaGetLastError();
  }
  if (counts == nullptr || counts_len < E) return -1;
  route_count_kernel<<<E, ROUTE_THREADS, 0, st>>>(eids, n_ptr, n_max, E, counts);
  route_place_kernel<<<E, ROUTE_THREADS, 0, st>>>(eids, n_ptr, n_max, E, align, counts, offs,
                                                  row_of_slot, slot_of_row, r_cap, device_status_word());
  int m = n_max > r_cap ? n_max : r_cap;
  route_fill_kernel<<<(m + 255) / 256, 256, 0, st>>>(eids, n_ptr, n_max, E, offs, row_of_slot, slot_of_row, r_cap);
  return (int)cudaGetLastError();
}

// ----------------------------------------------------------------------------------------------
// Routing sort for callers that must not allocate (declaration and contract: no_alloc.h).
// ----------------------------------------------------------------------------------------------
// Per-expert counters of the no-allocation variant. In host code this name is only a handle for
// the runtime, not a device address: the address comes from cudaGetSymbolAddress below.
static __device__ __align__(256) int g_route_counts_scratch[PT_ROUTE_SORT_NOALLOC_MAX_EXPERTS];

namespace {
constexpr int kNoAllocMaxDevices = 64;
int* g_route_counts_addr[kNoAllocMaxDevices] = {nullptr};
std::mutex g_route_counts_mu;

// Device address of the scratch on the current device; resolved once per device.
int route_counts_scratch(int** out) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  if (dev < 0 || dev >= kNoAllocMaxDevices) return -1;
  std::lock_guard<std::mutex> lk(g_route_counts_mu);
  if (!g_route_counts_addr[dev]) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_route_counts_scratch);
    if (e != cudaSuccess) {
      fprintf(stderr, "[pithtrain_b200] cudaGetSymbolAddress(route counters) failed on device %d: %s\n", dev,
              cudaGetErrorString(e));
      return (int)e;
    }
    g_route_counts_addr[dev] = static_cast<int*>(p);
  }
  *out = g_route_counts_addr[dev];
  return 0;
}
}  // namespace

PT_API int pt_route_sort_noalloc(const int* eids, int n, int E, int align, int* offs, int* row_of_slot,
                                 int* slot_of_row, int r_cap, void* stream_) {
  cudaStream_t st = (cudaStream_t)stream_;
  if (E <= 0 || n < 0 || align <= 0 || r_cap < 0 || !eids || !offs || !row_of_slot || !slot_of_row) return -1;
  if (E > PT_ROUTE_SORT_NOALLOC_MAX_EXPERTS) {
    fprintf(stderr, "[pithtrain_b200] pt_route_sort_noalloc: %d experts exceed the static scratch (max %d)\n", E,
            PT_ROUTE_SORT_NOALLOC_MAX_EXPERTS);
    return -2;
  }
  int* counts = nullptr;
  int rc = route_counts_scratch(&counts);
  if (rc != 0) return rc;
  // every counter in [0, E) is overwritten by the count kernel, nothing has to be cleared first
  route_count_kernel<<<E, ROUTE_THREADS, 0, st>>>(eids, nullptr, n, E, counts);
  route_place_kernel<<<E, ROUTE_THREADS, 0, st>>>(eids, nullptr, n, E, align, counts, offs, row_of_slot,
                                                  slot_of_row, r_cap, nullptr);
  int m = n > r_cap ? n : r_cap;
  if (m > 0)
    route_fill_kernel<<<(m + 255) / 256, 256, 0, st>>>(eids, nullptr, n, E, offs, row_of_slot, slot_of_row, r_cap);
  return (int)cudaGetLastError();
}

PT_API int pt_gather_rows(const void* src, const int* idx, int div, void* dst, const int* n_rows_ptr,
                          int n_rows_max, int H, long long src_stride, void* stream_) {
  cudaStream_t st = (cudaStream_t)stream_;
  if (n_rows_max <= 0) return 0;
  if (H % 8 != 0) return -1;
  gather_rows_kernel<<<grid_for(n_rows_max, 8, 16), 256, 0, st>>>((const __nv_bfloat16*)src, idx, div,
      (__nv_bfloat16*)dst, n_rows_ptr, n_rows_max, H, src_stride);
  return (int)cudaGetLastError();
}

// Cold cache, us, 2048 columns into 32000 rows: a conversion of dy and an indexed addition of one element a thread -> here (one row a
// warp, without adding up neighbours -> here): 4096 random ids 77 -> 21 (21), 256: 15 -> 8; 4096 times one id 77 -> 18 (150), 16384: 309
// -> 51 (533); 700 of every 1024 rows one id, 16384 rows 312 -> 53 (192). What is left to the L2's queue: two ids at random,
// 16384 rows of 64 columns 48 -> 53 (90).
PT_API int pt_embedding_bwd(const void* dy, const long long* ids, float* grad, int n, int H, long long V, void* stream_) {
  if (n <= 0 || H <= 0) return 0;
  if (H % 8 != 0) return -1;
  embedding_bwd_kernel<<<grid_for((long long)((n + EB_ROWS - 1) / EB_ROWS) * ((H + 255) / 256), 8, 8), 256, 0, (cudaStream_t)stream_>>>((const __nv_bfloat16*)dy, ids, grad, n, H, V, device_status_word());
  return (int)cudaGetLastError();
}

PT_API int pt_combine(const void* y, const int* row_of_slot, const float* w, const void* res, void* out,
                      const int* n_ptr, int n_max, int k, int H, void* stream_) {
  cudaStream_t st = (cudaStream_t)stream_;
  if (n_max <= 0) return 0;
  if (H % 8 != 0) return -1;
  // Many tokens of few or short rows have more row loads than the ring's copies are worth: a warp a token asks for its row with all
  // lanes, and there are warps enough. Measured, cold cache, us, ring / warp a token:
  //   columns x k    1536 tokens   2560        4096        6144        12288       32768
  //   512 x 1         9 / 8        10 / 8      10 / 8      12 / 8      16 / 11     31 / 17
  //   2048 x 1       12 / 12       14 / 12     18 / 13     24 / 14     39 / 23     92 / 51
  //   256 x 2         8 / 8        10 / 8      10 / 8      12 / 8      14 / 10     25 / 16
  //   2048 x 2       12 / 18       14 / 18     19 / 18     25 / 21     43 / 35    100 / 80
  //   4096 x 2       14 / 26       18 / 27     25 / 29     33 / 33     57 / 63    139 / 150
  //   1536 x 3       12 / 19       14 / 19     18 / 21     23 / 21     37 / 35     82 / 80
  //   512 x 4         9 / 12       10 / 12     12 / 12     14 / 12     21 / 18     39 / 38
  //   1024 x 4       10 / 16       12 / 17     14 / 18     18 / 18     29 / 31     64 / 70
  //   256 x 8        10 / 12       12 / 12     12 / 12     14 / 12     23 / 18     41 / 37
  //   512 x 8        11 / 16       12 / 16     14 / 16     18 / 18     27 / 29     59 / 65
  //   256 x 16       12 / 16       15 / 16     16 / 16     20 / 18     33 / 29     68 / 62
  const long long cols = (long long)k * H;
  const bool short_rows = (k <= 3 && cols <= 1024 && n_max >= 1536) ||
                          (k == 1   ? n_max >= 2560
                           : k == 2 ? n_max > 3072 && (cols <= 4608 || H > CB_COLS)
                                    : n_max > 4096 && (cols <= (k == 3 ? 4608 : 3072) || H <= 256));
  if (short_rows) {
    combine_warp_kernel<<<grid_for(n_max, 8, 16), 256, 0, st>>>((const __nv_bfloat16*)y, row_of_slot, w, (const __nv_bfloat16*)res, (__nv_bfloat16*)out,
                                                                n_ptr, n_max, k, H);
    return (int)cudaGetLastError();
  }
  const int pieces = H / 8, W = (pieces + (pieces + 511) / 512 - 1) / ((pieces + 511) / 512) * 8, slices = (H + W - 1) / W;
  const int adders = (W / 8 + 31) / 32;
  // Some sixteen adding warps an SM, in two to sixteen blocks, share 200 KB of rings: 3 to 8 stages each. Rows wider than the 2048
  // columns of eight warps are better left whole (two blocks of twelve warps and 4 stages for 2880 columns: 70 us for 12288 tokens
  // of 4, as two slices of six warps 84). Measured, cold cache, us; before: one thread for 8 columns of a token with four loads in
  // flight up to 3072 tokens, one warp a token above that:
  //   columns x k       64 tokens   1024      2048      3072      4096      8192      12288
  //   2048 x 8          12 -> 10    25 -> 16  39 -> 23  51 -> 31  57 -> 37  100 -> 61 109 -> 88
  //   2048 x 4           9 -> 8     16 -> 12  25 -> 16  33 -> 21  34 -> 25  59 -> 38   66 -> 51
  //   2880 x 4          10 -> 8     21 -> 14  33 -> 20  45 -> 25  47 -> 30  84 -> 49   90 -> 70
  //    512 x 8          11 -> 8     12 -> 10  17 -> 13  18 -> 15  19 -> 16  33 -> 23   37 -> 31
  const int blocks = adders > 8 ? 2 : (16 + adders / 2) / adders;
  const int stage_bytes = CB_ROWS * W * 2, room = 200 * 1024 / blocks / stage_bytes, stages = room < CB_STAGES ? room : CB_STAGES;
  static SmemLimit limit;
  if (const cudaError_t e = limit.set(combine_kernel, 100 * 1024)) return (int)e;
  combine_kernel<<<grid_for((long long)n_max * slices, 1, blocks), adders * 32 + 32, stages * stage_bytes, st>>>(
      (const __nv_bfloat16*)y, row_of_slot, w, (const __nv_bfloat16*)res, (__nv_bfloat16*)out, n_ptr, n_max, k, H, slices, W, stages,
      device_status_word());
  return (int)cudaGetLastError();
}

PT_API int pt_swiglu_fwd(const void* gu, void* act, const int* n_rows_ptr, int n_rows_max, int I,
                         int interleaved, float alpha, float limit, void* stream_) {
  cudaStream_t st = (cudaStream_t)stream_;
  if (n_rows_max <= 0) return 0;
  if (I % 8 != 0) return -1;
  swiglu_fwd_kernel<<<grid_for((long long)n_rows_max * (I / 8), 256, 16), 256, 0, st>>>(
      (const __nv_bfloat16*)gu, (__nv_bfloat16*)act, n_rows_ptr, n_rows_max, I, interleaved, alpha, limit);
  return (int)cudaGetLastError();
}

PT_API int pt_swiglu_bwd(const void* gu, const void* dact, const float* row_w, void* dgu,
                         void* act_scaled, float* d_row_w, const int* n_rows_ptr, int n_rows_max,
                         int I, int interleaved, float alpha, float limit, const int* slot_of_row, void* stream_) {
  cudaStream_t st = (cudaStream_t)stream_;
  if (n_rows_max <= 0) return 0;
  if (I % 8 != 0) return -1;
  swiglu_bwd_kernel<<<grid_for(n_rows_max, 8, 16), 256, 0, st>>>((const __nv_bfloat16*)gu,
      (const __nv_bfloat16*)dact, row_w, (__nv_bfloat16*)dgu, (__nv_bfloat16*)act_scaled, d_row_w,
      n_rows_ptr, n_rows_max, I, interleaved, alpha, limit, slot_of_row);
  return (int)cudaGetLastError();
}

// out[r] = x[r] + bias[group(r)] for the first n rows (device-side count optional); x, bias, out bf16, H % 8 == 0;
// out may alias x.
PT_API int pt_indexed_bias_add(const void* x, const void* bias, const int* offs, int E, void* out, const int* n_rows_ptr,
                               int n_rows_max, int H, void* stream_) {
  cudaStream_t st = (cudaStream_t)stream_;
  if (n_rows_max <= 0) return 0;
  if (H % 8 != 0 || E <= 0) return -1;
  indexed_bias_add_kernel<<<grid_for(n_rows_max, 8, 16), 256, 0, st>>>((const __nv_bfloat16*)x, (const __nv_bfloat16*)bias,
                                                                       offs, E, (__nv_bfloat16*)out, n_rows_ptr, n_rows_max, H);
  return (int)cudaGetLastError();
}

// dw[slot_of_row[r]] += <x[r], bias[group(r)]> for the first n rows (device-side count optional); x, bias bf16, dw fp32, H % 8 == 0.
PT_API int pt_row_bias_dot(const void* x, const void* bias, const int* offs, int E, const int* slot_of_row, float* dw, const int* n_rows_ptr,
                           int n_rows_max, int H, void* stream_) {
  cudaStream_t st = (cudaStream_t)stream_;
  if (n_rows_max <= 0) return 0;
  if (H % 8 != 0 || E <= 0) return -1;
  row_bias_dot_kernel<<<grid_for(n_rows_max, 8, 16), 256, 0, st>>>((const __nv_bfloat16*)x, (const __nv_bfloat16*)bias, offs, E, slot_of_row, dw,
                                                                   n_rows_ptr, n_rows_max, H);
  return (int)cudaGetLastError();
}

// out[g, :] = sum of rows [offs[g], offs[g+1]) of x (bf16 when x_fp32 == 0, else fp32), optionally weighted per row;
// out fp32 [E, H], H even.
PT_API int pt_segment_sum(const void* x, int x_fp32, const float* row_w, const int* offs, int E, float* out, int H,
                          void* stream_) {
  cudaStream_t st = (cudaStream_t)stream_;
  if (E <= 0 || H <= 0) return 0;
  if (H % 2 != 0) return -1;
  const dim3 grid(E, (H / 2 + 31) / 32);
  if (x_fp32) segment_sum_kernel<float><<<grid, 32 * SEG_WARPS, 0, st>>>((const float*)x, row_w, offs, out, H);
  else segment_sum_kernel<__nv_bfloat16><<<grid, 32 * SEG_WARPS, 0, st>>>((const __nv_bfloat16*)x, row_w, offs, out, H);
  return (int)cudaGetLastError();
}
