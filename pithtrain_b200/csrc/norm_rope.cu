// RMSNorm (with fused residual add) and fused per-head QK-RMSNorm + rotary embedding, forward and
// backward. Memory-bound kernels: one 16-byte vector per thread per access, each tensor read once.
// They replace the Inductor-generated stage-1 region of the reference
// (pithtrain/models/qwen3_moe.py:156-168,188-202).
#include "elementwise.cuh"
#include "host_common.h"

namespace pt {

constexpr int NORM_THREADS = 256;

// y = (x [+ res]) * rstd * w ; optionally writes h = x + res and rstd.
template <int VPT>
__global__ void __launch_bounds__(NORM_THREADS)
rmsnorm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ res,
                   const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ y,
                   __nv_bfloat16* __restrict__ h_out, float* __restrict__ rstd_out, int n_rows,
                   int H, float eps, int w_plus_one) {
  __shared__ float red[32];
  const int nvec = H / 8;
  for (int row = blockIdx.x; row < n_rows; row += gridDim.x) {
    const __nv_bfloat16* xr = x + (size_t)row * H;
    float v[VPT][8];
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      int c = threadIdx.x + i * NORM_THREADS;
      if (c < nvec) {
        load8(xr + c * 8, v[i]);
        if (res) {
          float r[8];
          load8(res + (size_t)row * H + c * 8, r);
#pragma unroll
          for (int e = 0; e < 8; ++e) v[i][e] += r[e];
          if (h_out) {
            // round to bf16 first so the norm sees exactly the stored residual stream
            store8(h_out + (size_t)row * H + c * 8, v[i]);
            load8(h_out + (size_t)row * H + c * 8, v[i]);
          }
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) ss += v[i][e] * v[i][e];
      }
    }
    ss = block_sum(ss, red);
    float rstd = rsqrtf(ss / H + eps);
    if (threadIdx.x == 0 && rstd_out) rstd_out[row] = rstd;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      int c = threadIdx.x + i * NORM_THREADS;
      if (c < nvec) {
        float wv[8], o[8];
        load8(w + c * 8, wv);
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] = v[i][e] * rstd * (w_plus_one ? (1.f + wv[e]) : wv[e]);
        store8(y + (size_t)row * H + c * 8, o);
      }
    }
  }
}

// dx = rstd * (w*dy - xhat * mean(w*dy*xhat)) [+ dh_extra]; dw partial per CTA (fp32). Bound by the rows of its three inputs and its
// output; a row's loads are asked for while the row before it is summed up and stored. With the residual's gradient, cold cache, us,
// before (loads of a row, sum, load of dh_extra, store) -> now: 4096 x 2048 23 -> 20, 8192 x 2048 36 -> 29, 4096 x 2880 46 -> 28,
// 4096 x 7168 91 -> 68, 3001 x 512 15 -> 11.
template <int VPT>
__global__ void __launch_bounds__(NORM_THREADS)
rmsnorm_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ dh_extra,
                   const __nv_bfloat16* __restrict__ h, const __nv_bfloat16* __restrict__ w,
                   const float* __restrict__ rstd_in, __nv_bfloat16* __restrict__ dx,
                   float* __restrict__ dw_partial, int n_rows, int H, int w_plus_one) {
  __shared__ float red[32];
  const int nvec = H / 8;
  float dw[VPT][8];
  uint4 wv[VPT], hv[VPT], gv[VPT], ev[VPT];
  float rstd = 0.f;
  auto fetch = [&](int row) {
    if (row >= n_rows) return;
    rstd = rstd_in[row];
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int c = threadIdx.x + i * NORM_THREADS;
      if (c >= nvec) continue;
      const size_t at = (size_t)row * H + c * 8;
      hv[i] = *reinterpret_cast<const uint4*>(h + at);
      gv[i] = *reinterpret_cast<const uint4*>(dy + at);
      if (dh_extra) ev[i] = *reinterpret_cast<const uint4*>(dh_extra + at);
    }
  };
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
#pragma unroll
    for (int e = 0; e < 8; ++e) dw[i][e] = 0.f;
    const int c = threadIdx.x + i * NORM_THREADS;
    if (c < nvec) wv[i] = *reinterpret_cast<const uint4*>(w + c * 8);
  }
  fetch(blockIdx.x);
  for (int row = blockIdx.x; row < n_rows; row += gridDim.x) {
    const float r = rstd;
    float xh[VPT][8], g[VPT][8];
    uint4 extra[VPT];
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      int c = threadIdx.x + i * NORM_THREADS;
      if (c < nvec) {
        float wf[8];
        load8(reinterpret_cast<const __nv_bfloat16*>(&hv[i]), xh[i]);
        load8(reinterpret_cast<const __nv_bfloat16*>(&gv[i]), g[i]);
        load8(reinterpret_cast<const __nv_bfloat16*>(&wv[i]), wf);
        extra[i] = ev[i];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          xh[i][e] *= r;
          dw[i][e] += g[i][e] * xh[i][e];
          g[i][e] *= (w_plus_one ? (1.f + wf[e]) : wf[e]);
          dot += g[i][e] * xh[i][e];
        }
      }
    }
    fetch(row + gridDim.x);
    dot = block_sum(dot, red) / H;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      int c = threadIdx.x + i * NORM_THREADS;
      if (c < nvec) {
        float o[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] = r * (g[i][e] - xh[i][e] * dot);
        if (dh_extra) {
          float ex[8];
          load8(reinterpret_cast<const __nv_bfloat16*>(&extra[i]), ex);
#pragma unroll
          for (int e = 0; e < 8; ++e) o[e] += ex[e];
        }
        store8(dx + (size_t)row * H + c * 8, o);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    int c = threadIdx.x + i * NORM_THREADS;
    if (c < nvec) {
      float* p = dw_partial + (size_t)blockIdx.x * H + c * 8;
#pragma unroll
      for (int e = 0; e < 8; ++e) p[e] = dw[i][e];
    }
  }
}

// ----------------------------------------------------------------------------------------------
// Fused per-head RMSNorm (optional) + rotate-half RoPE for q and k, reading the fused qkv GEMM output.
// A head of D elements is handled by D/16 lanes: lane `sub` owns elements [8 sub, 8 sub + 8) of the first
// half and their rotation partners in the second half, so every access is a 16-byte vector and the pair
// (i, i + D/2) never leaves the lane. A warp covers 32 / (D/16) heads. D in {64, 128}: PAIRS = D / 64.
// ----------------------------------------------------------------------------------------------
template <int LPH>
__device__ __forceinline__ float group_sum(float v) {
#pragma unroll
  for (int o = LPH / 2; o >= 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <int PAIRS>
__global__ void __launch_bounds__(256)
qk_norm_rope_fwd_kernel(const __nv_bfloat16* __restrict__ qkv, __nv_bfloat16* __restrict__ q_out,
                        __nv_bfloat16* __restrict__ k_out, const __nv_bfloat16* __restrict__ qw,
                        const __nv_bfloat16* __restrict__ kw, const __nv_bfloat16* __restrict__ cosb,
                        const __nv_bfloat16* __restrict__ sinb, const int* __restrict__ pos,
                        float* __restrict__ rstd_q, float* __restrict__ rstd_k, int n_tokens, int S,
                        int Hq, int Hkv, long long qkv_stride, float eps, int w_plus_one, int rot_dim) {
  constexpr int D = PAIRS * 64, HALF = D / 2, LPH = D / 16, HPW = 32 / LPH;
  const int lane = threadIdx.x & 31, sub = lane % LPH, i0 = sub * 8;
  const int heads = Hq + Hkv;
  const long long total = (long long)n_tokens * heads;
  const long long item = ((long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * HPW + lane / LPH;
  const bool live = item < total;
  const long long it = live ? item : total - 1;
  const int tok = (int)(it / heads), hd = (int)(it % heads);
  const bool is_q = hd < Hq;
  const __nv_bfloat16* src = qkv + (size_t)tok * qkv_stride + (size_t)hd * D;  // k heads follow q heads
  __nv_bfloat16* dst = is_q ? q_out + ((size_t)tok * Hq + hd) * D : k_out + ((size_t)tok * Hkv + (hd - Hq)) * D;
  const __nv_bfloat16* wn = is_q ? qw : kw;
  const int p = pos ? pos[tok] : (tok % S);
  float a[8], b[8];
  load8(src + i0, a);
  load8(src + HALF + i0, b);
  float ss = 0.f;
#pragma unroll
  for (int e = 0; e < 8; ++e) ss += a[e] * a[e] + b[e] * b[e];
  float rstd = 1.f;
  if (wn) {
    ss = group_sum<LPH>(ss);
    rstd = rsqrtf(ss / D + eps);
    if (live && sub == 0) {
      if (is_q) rstd_q[(size_t)tok * Hq + hd] = rstd;
      else rstd_k[(size_t)tok * Hkv + (hd - Hq)] = rstd;
    }
  }
  float wa[8], wb[8], c[8], sn[8];
  if (wn) {
    load8(wn + i0, wa);
    load8(wn + HALF + i0, wb);
  }
  const bool rotate = rot_dim == D;
  if (rotate) {
    load8(cosb + (size_t)p * D + i0, c);
    load8(sinb + (size_t)p * D + i0, sn);
  }
  float oa[8], ob[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    float na = a[e] * rstd, nb = b[e] * rstd;
    if (wn) {
      float x = wa[e], y = wb[e];
      if (w_plus_one) { x += 1.f; y += 1.f; }
      na *= x; nb *= y;
    }
    // round like the unfused path (norm output is bf16 before the rotation)
    na = __bfloat162float(__float2bfloat16(na));
    nb = __bfloat162float(__float2bfloat16(nb));
    oa[e] = rotate ? na * c[e] - nb * sn[e] : na;
    ob[e] = rotate ? nb * c[e] + na * sn[e] : nb;
  }
  if (live) {
    store8(dst + i0, oa);
    store8(dst + HALF + i0, ob);
  }
}

// Sum of v over the lanes that hold the same channels of a warp's heads.
template <int LPH>
__device__ __forceinline__ float across_groups(float v) {
#pragma unroll
  for (int o = 16; o >= LPH; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

struct RopeBwdArgs {
  const __nv_bfloat16 *qkv, *cosb, *sinb;
  const int* pos;
  __nv_bfloat16* dqkv;
  long long qkv_stride, dqkv_stride;
  int n, S, w_plus_one;
};

// One group of heads of one kind (q or k): grp counts groups of HPW heads among the n * H of that kind, head0 is the kind's place
// in the packed row. ka, kb collect the norm weight's gradient for my channels.
template <int D>
__device__ __forceinline__ void rope_bwd_group(const RopeBwdArgs& a, long long grp, int H, int head0, const __nv_bfloat16* __restrict__ grad,
                                               const __nv_bfloat16* __restrict__ wn, const float* __restrict__ rstd_in, float (&ka)[8], float (&kb)[8]) {
  constexpr int HALF = D / 2, LPH = D / 16, HPW = 32 / LPH;
  const int lane = threadIdx.x & 31, i0 = lane % LPH * 8;
  const long long total = (long long)a.n * H, item = grp * HPW + lane / LPH;
  const bool live = item < total;
  const long long it = live ? item : total - 1;  // a spare group repeats the last head and stores nothing
  const int tok = total <= 0x7fffffffLL ? (int)it / H : (int)(it / H), hd = (int)(it - (long long)tok * H);
  const __nv_bfloat16* src = a.qkv + (size_t)tok * a.qkv_stride + (size_t)(head0 + hd) * D;
  const int p = a.pos ? a.pos[tok] : tok % a.S;
  float ga[8], gb[8], c[8], sn[8], da[8], db[8];
  load8(grad + (size_t)it * D + i0, ga);
  load8(grad + (size_t)it * D + HALF + i0, gb);
  load8(a.cosb + (size_t)p * D + i0, c);
  load8(a.sinb + (size_t)p * D + i0, sn);
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    da[e] = ga[e] * c[e] + gb[e] * sn[e];
    db[e] = gb[e] * c[e] - ga[e] * sn[e];
  }
  if (wn) {
    float xa[8], xb[8], wa[8], wb[8];
    load8(src + i0, xa);
    load8(src + HALF + i0, xb);
    load8(wn + i0, wa);
    load8(wn + HALF + i0, wb);
    const float rstd = rstd_in[it], one = a.w_plus_one ? 1.f : 0.f;
    float dot = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      xa[e] *= rstd; xb[e] *= rstd;
      const float ta = da[e] * xa[e], tb = db[e] * xb[e];
      if (live) { ka[e] += ta; kb[e] += tb; }
      const float sa = wa[e] + one, sb = wb[e] + one;
      dot += ta * sa + tb * sb;
      da[e] *= sa; db[e] *= sb;
    }
    dot = group_sum<LPH>(dot) / D;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      da[e] = rstd * (da[e] - xa[e] * dot);
      db[e] = rstd * (db[e] - xb[e] * dot);
    }
  }
  if (live) {
    __nv_bfloat16* dst = a.dqkv + (size_t)tok * a.dqkv_stride + (size_t)(head0 + hd) * D;
    store8(dst + i0, da);
    store8(dst + HALF + i0, db);
  }
}

// dqkv from dq, dk, dv (null: zeros); dw_partial [gridDim.x, 2 * D]: sums of the q and k weight gradients of this block.
// Bound by instructions first (conversions, two rotations' worth of products on 16 channels a lane), then by memory traffic, and
// at small sizes by its tail. So a warp's heads are all of one kind (no selects between q and k, v is a plain copy), and heads are
// counted in 32 bits when they fit. The weight sums are folded over the head groups of a warp by shuffles and over the warps in
// shared memory: fp32 atomics there are a compare-and-swap loop, and 32 lane groups on one address held a block for 15 us.
// Measured (32 / 4 heads of 128), with the copy of dv that used to be a launch: 4096 tokens 66 -> 43 us (52 with kinds mixed in a
// warp), 512 tokens 31 -> 9.6. Two blocks an SM: three (85 registers) measured 52, four 43 and 13.
template <int PAIRS>
__global__ void __launch_bounds__(256, 2)
qk_norm_rope_bwd_kernel(RopeBwdArgs a, const __nv_bfloat16* __restrict__ dq, const __nv_bfloat16* __restrict__ dk, const __nv_bfloat16* __restrict__ dv,
                        const __nv_bfloat16* __restrict__ qw, const __nv_bfloat16* __restrict__ kw, const float* __restrict__ rstd_q,
                        const float* __restrict__ rstd_k, float* __restrict__ dw_partial, int Hq, int Hkv) {
  constexpr int D = PAIRS * 64, HALF = D / 2, LPH = D / 16, HPW = 32 / LPH;
  __shared__ float acc[8][2 * D];  // weight-gradient sums of each warp: q scales then k scales
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, i0 = lane % LPH * 8;
  const long long gq = ((long long)a.n * Hq + HPW - 1) / HPW, gk = ((long long)a.n * Hkv + HPW - 1) / HPW;
  float dwq_a[8], dwq_b[8], dwk_a[8], dwk_b[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) dwq_a[e] = dwq_b[e] = dwk_a[e] = dwk_b[e] = 0.f;
  for (long long grp = (long long)blockIdx.x * 8 + wib; grp < gq + 2 * gk; grp += (long long)gridDim.x * 8) {
    if (grp < gq) {
      rope_bwd_group<D>(a, grp, Hq, 0, dq, qw, rstd_q, dwq_a, dwq_b);
    } else if (grp < gq + gk) {
      rope_bwd_group<D>(a, grp - gq, Hkv, Hq, dk, kw, rstd_k, dwk_a, dwk_b);
    } else {
      const long long item = (grp - gq - gk) * HPW + lane / LPH;
      if (item < (long long)a.n * Hkv) {
        const long long tok = item / Hkv;
        __nv_bfloat16* dst = a.dqkv + (size_t)tok * a.dqkv_stride + (size_t)(Hq + Hkv + (item - tok * Hkv)) * D;
        const uint4 zero = make_uint4(0, 0, 0, 0);
        *reinterpret_cast<uint4*>(dst + i0) = dv ? *reinterpret_cast<const uint4*>(dv + (size_t)item * D + i0) : zero;
        *reinterpret_cast<uint4*>(dst + HALF + i0) = dv ? *reinterpret_cast<const uint4*>(dv + (size_t)item * D + HALF + i0) : zero;
      }
    }
  }
  if (qw && dw_partial) {
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float s[4] = {across_groups<LPH>(dwq_a[e]), across_groups<LPH>(dwq_b[e]), across_groups<LPH>(dwk_a[e]), across_groups<LPH>(dwk_b[e])};
      if (lane < LPH) {
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[wib][j * HALF + i0 + e] = s[j];
      }
    }
    __syncthreads();
    for (int cidx = threadIdx.x; cidx < 2 * D; cidx += blockDim.x) {
      float t = 0.f;
#pragma unroll
      for (int w = 0; w < 8; ++w) t += acc[w][cidx];
      dw_partial[(size_t)blockIdx.x * 2 * D + cidx] = t;
    }
  }
}

// out[i] = i - start of the document that row i lies in: document s holds cu[s + 1] - cu[s] rows, one after the other from row 0;
// rows past the last one count on. One launch for the slices, casts, differences, scan and repetition of the tensor-op form.
__global__ void __launch_bounds__(256) packed_positions_kernel(const int* __restrict__ cu, int n_cu, long long* __restrict__ out, long long S) {
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  if (i >= S) return;
  const long long first = cu[0];
  int a = 1, z = n_cu;  // first boundary beyond row i
  while (a < z) {
    const int mid = (a + z) >> 1;
    if (cu[mid] - first <= i) a = mid + 1; else z = mid;
  }
  out[i] = i - cu[min(a - 1, n_cu - 2)];
}

}  // namespace pt

using namespace pt;

PT_API int pt_rmsnorm_fwd(const void* x, const void* res, const void* w, void* y, void* h_out,
                          float* rstd, int n_rows, int H, float eps, int w_plus_one, void* stream_) {
  cudaStream_t st = (cudaStream_t)stream_;
  if (n_rows <= 0) return 0;
  if (H % 8 != 0 || H > 8 * NORM_THREADS * 4) return -1;
  int vpt = (H / 8 + NORM_THREADS - 1) / NORM_THREADS;
  int grid = n_rows < sm_count() * 8 ? n_rows : sm_count() * 8;
#define LAUNCH(V)                                                                                     \
  rmsnorm_fwd_kernel<V><<<grid, NORM_THREADS, 0, st>>>(                                               \
      (const __nv_bfloat16*)x, (const __nv_bfloat16*)res, (const __nv_bfloat16*)w, (__nv_bfloat16*)y, \
      (__nv_bfloat16*)h_out, rstd, n_rows, H, eps, w_plus_one)
  switch (vpt) { case 1: LAUNCH(1); break; case 2: LAUNCH(2); break; case 3: LAUNCH(3); break; default: LAUNCH(4); }
#undef LAUNCH
  return (int)cudaGetLastError();
}

// dw_partial must hold [grid, H] floats where grid = pt_rmsnorm_bwd_grid(n_rows).
PT_API int pt_rmsnorm_bwd_grid(int n_rows) {
  int g = sm_count() * 4;
  return n_rows < g ? (n_rows > 0 ? n_rows : 1) : g;
}
PT_API int pt_rmsnorm_bwd(const void* dy, const void* dh_extra, const void* h, const void* w,
                          const float* rstd, void* dx, float* dw_partial, int n_rows, int H,
                          int w_plus_one, void* stream_) {
  cudaStream_t st = (cudaStream_t)stream_;
  if (n_rows <= 0) return 0;
  if (H % 8 != 0 || H > 8 * NORM_THREADS * 4) return -1;
  int vpt = (H / 8 + NORM_THREADS - 1) / NORM_THREADS;
  int grid = pt_rmsnorm_bwd_grid(n_rows);
#define LAUNCH(V)                                                                                 \
  rmsnorm_bwd_kernel<V><<<grid, NORM_THREADS, 0, st>>>(                                           \
      (const __nv_bfloat16*)dy, (const __nv_bfloat16*)dh_extra, (const __nv_bfloat16*)h,          \
      (const __nv_bfloat16*)w, rstd, (__nv_bfloat16*)dx, dw_partial, n_rows, H, w_plus_one)
  switch (vpt) { case 1: LAUNCH(1); break; case 2: LAUNCH(2); break; case 3: LAUNCH(3); break; default: LAUNCH(4); }
#undef LAUNCH
  return (int)cudaGetLastError();
}

PT_API int pt_qk_norm_rope_fwd(const void* qkv, void* q_out, void* k_out, const void* qw,
                               const void* kw, const void* cosb, const void* sinb, const int* pos,
                               float* rstd_q, float* rstd_k, int n_tokens, int S, int Hq, int Hkv,
                               int D, long long qkv_stride, float eps, int w_plus_one, void* stream_) {
  cudaStream_t st = (cudaStream_t)stream_;
  if (n_tokens <= 0) return 0;
  if (D != 64 && D != 128) return -1;
  const int heads_per_warp = 32 / (D / 16);
  long long warps = ((long long)n_tokens * (Hq + Hkv) + heads_per_warp - 1) / heads_per_warp;
  int grid = (int)((warps + 7) / 8);
  if (D == 128)
    qk_norm_rope_fwd_kernel<2><<<grid, 256, 0, st>>>((const __nv_bfloat16*)qkv, (__nv_bfloat16*)q_out, (__nv_bfloat16*)k_out,
        (const __nv_bfloat16*)qw, (const __nv_bfloat16*)kw, (const __nv_bfloat16*)cosb, (const __nv_bfloat16*)sinb, pos,
        rstd_q, rstd_k, n_tokens, S, Hq, Hkv, qkv_stride, eps, w_plus_one, D);
  else
    qk_norm_rope_fwd_kernel<1><<<grid, 256, 0, st>>>((const __nv_bfloat16*)qkv, (__nv_bfloat16*)q_out, (__nv_bfloat16*)k_out,
        (const __nv_bfloat16*)qw, (const __nv_bfloat16*)kw, (const __nv_bfloat16*)cosb, (const __nv_bfloat16*)sinb, pos,
        rstd_q, rstd_k, n_tokens, S, Hq, Hkv, qkv_stride, eps, w_plus_one, D);
  return (int)cudaGetLastError();
}

PT_API int pt_qk_norm_rope_bwd_grid(int n_tokens, int Hq, int Hkv, int D) {
  const long long want = ((long long)n_tokens * (Hq + 2 * Hkv) * (D / 16) + 255) / 256, cap = sm_count() * 4;
  return (int)(want < 1 ? 1 : want < cap ? want : cap);
}
// dw_partial: [grid, 2*D] floats (q weight grads then k weight grads per row); may be null when qw is null. dv may be null (zeros).
PT_API int pt_qk_norm_rope_bwd(const void* dq, const void* dk, const void* dv, const void* qkv, void* dqkv,
                               const void* qw, const void* kw, const void* cosb, const void* sinb,
                               const int* pos, const float* rstd_q, const float* rstd_k,
                               float* dw_partial, int n_tokens, int S, int Hq, int Hkv, int D,
                               long long qkv_stride, long long dqkv_stride, int w_plus_one, void* stream_) {
  cudaStream_t st = (cudaStream_t)stream_;
  if (n_tokens <= 0) return 0;
  if (D != 64 && D != 128) return -1;
  const int grid = pt_qk_norm_rope_bwd_grid(n_tokens, Hq, Hkv, D);
  const RopeBwdArgs a{(const __nv_bfloat16*)qkv, (const __nv_bfloat16*)cosb, (const __nv_bfloat16*)sinb, pos, (__nv_bfloat16*)dqkv,
                      qkv_stride, dqkv_stride, n_tokens, S, w_plus_one};
#define LAUNCH(P) qk_norm_rope_bwd_kernel<P><<<grid, 256, 0, st>>>(a, (const __nv_bfloat16*)dq, (const __nv_bfloat16*)dk, (const __nv_bfloat16*)dv, \
    (const __nv_bfloat16*)qw, (const __nv_bfloat16*)kw, rstd_q, rstd_k, dw_partial, Hq, Hkv)
  if (D == 128) LAUNCH(2);
  else LAUNCH(1);
#undef LAUNCH
  return (int)cudaGetLastError();
}

// ----------------------------------------------------------------------------------------------
// dst[c] += sum_g part[g, c]: finishes the per-block partial sums of a weight gradient (RMSNorm scale,
// QK-norm scales) and accumulates into the gradient buffer in one launch.
// ----------------------------------------------------------------------------------------------
namespace pt {
// A latency problem, not a bandwidth one (G = 592 partial rows of 128..2048 columns, 0.3..5 MB, all in L2): with one thread
// per column every thread walked a serial chain of G / 4 loads and only H / 128 blocks ran. Here a block owns 32 columns
// and its 32 warps split the rows, eight loads in flight each, so the chain is ceil(G / 256) long.
constexpr int COLSUM_WARPS = 32;
template <typename T>
__global__ void __launch_bounds__(32 * COLSUM_WARPS)
colsum_accumulate_kernel(const float* __restrict__ part, int G, int ld, int H, T* __restrict__ dst, T* __restrict__ dst2, int split) {
  __shared__ float red[COLSUM_WARPS][33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + lane;
  float acc[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i] = 0.f;
  if (c < H) {
    for (int g = warp; g < G; g += 8 * COLSUM_WARPS) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int r = g + i * COLSUM_WARPS;
        if (r < G) acc[i] += part[(size_t)r * ld + c];
      }
    }
  }
  red[warp][lane] = ((acc[0] + acc[1]) + (acc[2] + acc[3])) + ((acc[4] + acc[5]) + (acc[6] + acc[7]));
  __syncthreads();
  // warp w finishes column w of the block: lane l brings the sum of row group l
  float v = red[lane][warp];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int cc = blockIdx.x * 32 + warp;
  T* d = cc < split ? dst + cc : dst2 + (cc - split);
  if (lane == 0 && cc < H) *d = (T)((float)*d + v);
}
}  // namespace pt

// part: G rows of pitch ld floats; columns [0, H) of it are summed into dst[0:H).
PT_API int pt_colsum_accumulate(const float* part, int G, int ld, int H, void* dst, int dst_fp32, void* stream_) {
  cudaStream_t st = (cudaStream_t)stream_;
  if (G <= 0 || H <= 0) return 0;
  const int grid = (H + 31) / 32, threads = 32 * pt::COLSUM_WARPS;
  if (dst_fp32) pt::colsum_accumulate_kernel<float><<<grid, threads, 0, st>>>(part, G, ld, H, (float*)dst, nullptr, H);
  else pt::colsum_accumulate_kernel<__nv_bfloat16><<<grid, threads, 0, st>>>(part, G, ld, H, (__nv_bfloat16*)dst, nullptr, H);
  return (int)cudaGetLastError();
}

// Columns [0, H) into dst0 and [H, 2 H) into dst1: the q and k norms of a layer in one launch.
PT_API int pt_colsum_accumulate_pair(const float* part, int G, int ld, int H, void* dst0, void* dst1, int dst_fp32, void* stream_) {
  cudaStream_t st = (cudaStream_t)stream_;
  if (G <= 0 || H <= 0) return 0;
  const int grid = (2 * H + 31) / 32, threads = 32 * pt::COLSUM_WARPS;
  if (dst_fp32) pt::colsum_accumulate_kernel<float><<<grid, threads, 0, st>>>(part, G, ld, 2 * H, (float*)dst0, (float*)dst1, H);
  else pt::colsum_accumulate_kernel<__nv_bfloat16><<<grid, threads, 0, st>>>(part, G, ld, 2 * H, (__nv_bfloat16*)dst0, (__nv_bfloat16*)dst1, H);
  return (int)cudaGetLastError();
}

// cu: int32 [n_cu], n_cu >= 2; out: int64 [S].
PT_API int pt_packed_positions(const int* cu, int n_cu, long long* out, long long S, void* stream_) {
  if (S <= 0) return 0;
  if (n_cu < 2 || S > 0x7fffffffLL) return -2;
  packed_positions_kernel<<<(unsigned)((S + 255) / 256), 256, 0, (cudaStream_t)stream_>>>(cu, n_cu, out, S);
  return (int)cudaGetLastError();
}
