// The elementwise passes of an attention layer whose q projection also emits an output gate (bf16 in and out, fp32 inside):
//   pre  : packed rows [q0 | gate0 | q1 | gate1 | ... | k | v] -> q, k (per-head RMSNorm with weight 1 + w, then rotate-half RoPE on
//          the first R channels) and v, each contiguous. The gate is read where it lies.
//   post : out * sigmoid(gate).
// The tensor-op form split, copied, normalised, rotated (six elementwise operations and two concatenations for each of q and
// k) and gated in passes of its own, each rounding to bf16. Bound by memory traffic: every element is read and written once
// each way. D / 8 lanes hold a head, 8 channels a lane, so a channel's rotation partner is R / 16 lanes away; rstd is kept for
// the backward, which recomputes the normalised value from the packed row.
// Measured with the passes they replace: a Qwen3.5 layer (16 / 2 heads of 256) at 3072 positions, forward
// and backward 850 -> 160 us of device time; two layers (one Gated DeltaNet) at 2 x 3072 positions 22.2 -> 20.8 ms a step.
#include "elementwise.cuh"
#include "host_common.h"

namespace pt {
namespace gattn {

struct Args {
  const __nv_bfloat16 *qkv, *qw, *kw, *cosb, *sinb;  // cos, sin: [n, R]
  float* rstd;                                      // [n, Hq + Hk]
  long long stride;                                 // elements between rows of qkv (and of dqkv)
  int n, Hq, Hk, R;
  float eps;
};

template <int LPH>
__device__ __forceinline__ float group_sum(float v) {
#pragma unroll
  for (int o = LPH / 2; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Lane holding the rotation partner of my channels; mine if I am not rotated. half = R / 16 lanes.
__device__ __forceinline__ int partner_of(int lane, int sub, int half) { return sub < half ? lane + half : sub < 2 * half ? lane - half : lane; }

template <int D>
__global__ void __launch_bounds__(256) pre_fwd_kernel(Args a, __nv_bfloat16* __restrict__ q, __nv_bfloat16* __restrict__ k, __nv_bfloat16* __restrict__ v) {
  constexpr int LPH = D / 8, HPW = 32 / LPH;
  const int lane = threadIdx.x & 31, sub = lane % LPH, half = a.R / 16, partner = partner_of(lane, sub, half);
  const int heads = a.Hq + 2 * a.Hk;
  const long long total = (long long)a.n * heads, warps = (long long)gridDim.x * 8;
  const bool narrow = total <= 0x7fffffffLL;  // a 64-bit division costs more than the head's arithmetic
  for (long long base = ((long long)blockIdx.x * 8 + (threadIdx.x >> 5)) * HPW; base < total; base += warps * HPW) {
    const long long item = base + lane / LPH;
    const bool live = item < total;
    const long long it = live ? item : total - 1;  // a spare group repeats the last head and stores nothing
    const int tok = narrow ? (int)it / heads : (int)(it / heads), hd = (int)(it - (long long)tok * heads);
    const bool is_q = hd < a.Hq, is_v = hd >= a.Hq + a.Hk;
    const __nv_bfloat16* src = a.qkv + tok * a.stride + (long long)(is_q ? 2 * hd : a.Hq + hd) * D + sub * 8;
    float x[8];
    load8(src, x);
    float ss = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) ss += x[e] * x[e];
    ss = group_sum<LPH>(ss);
    float y[8];
    if (!is_v) {
      const float r = rsqrtf(ss / D + a.eps);
      float w[8];
      load8((is_q ? a.qw : a.kw) + sub * 8, w);
#pragma unroll
      for (int e = 0; e < 8; ++e) y[e] = x[e] * r * (1.f + w[e]);
      if (live && sub == 0) a.rstd[(long long)tok * (a.Hq + a.Hk) + hd] = r;
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) y[e] = x[e];
    }
    float o[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) o[e] = __shfl_sync(0xffffffffu, y[e], partner);
    if (!is_v && sub < 2 * half) {
      float c[8], s[8];
      load8(a.cosb + (long long)tok * a.R + sub * 8, c);
      load8(a.sinb + (long long)tok * a.R + sub * 8, s);
#pragma unroll
      for (int e = 0; e < 8; ++e) y[e] = y[e] * c[e] + (sub < half ? -o[e] : o[e]) * s[e];
    }
    if (live) {
      __nv_bfloat16* dst = is_q ? q + ((long long)tok * a.Hq + hd) * D
                                : is_v ? v + ((long long)tok * a.Hk + hd - a.Hq - a.Hk) * D : k + ((long long)tok * a.Hk + hd - a.Hq) * D;
      store8(dst + sub * 8, y);
    }
  }
}

// One group of heads of one kind (q or k) on the way back; place: elements from the start of a packed row to the kind's first
// head, pitch: between its heads, rs0: its first column of rstd. wsum collects the norm weight's gradient for my channels.
template <int D>
__device__ __forceinline__ void bwd_group(const Args& a, long long grp, int H, long long place, int pitch, int rs0, const __nv_bfloat16* __restrict__ grad,
                                          const __nv_bfloat16* __restrict__ wn, __nv_bfloat16* __restrict__ dqkv, float (&wsum)[8]) {
  constexpr int LPH = D / 8, HPW = 32 / LPH;
  const int lane = threadIdx.x & 31, sub = lane % LPH, half = a.R / 16, partner = partner_of(lane, sub, half);
  const long long total = (long long)a.n * H, item = grp * HPW + lane / LPH;
  const bool live = item < total, rot = sub < 2 * half;
  const long long it = live ? item : total - 1;
  const int tok = total <= 0x7fffffffLL ? (int)it / H : (int)(it / H), hd = (int)(it - (long long)tok * H);
  const long long at = tok * a.stride + place + (long long)hd * pitch + sub * 8;
  float y[8], t[8], x[8], w[8];
  load8(grad + it * D + sub * 8, y);
  load8(a.qkv + at, x);
  const float r = a.rstd[(long long)tok * (a.Hq + a.Hk) + rs0 + hd];
#pragma unroll
  for (int e = 0; e < 8; ++e) t[e] = 0.f;
  if (rot) {
    float c[8], s[8];
    load8(a.cosb + (long long)tok * a.R + sub * 8, c);
    load8(a.sinb + (long long)tok * a.R + sub * 8, s);
#pragma unroll
    for (int e = 0; e < 8; ++e) { t[e] = y[e] * s[e]; y[e] *= c[e]; }
  }
  // transposed rotation: the first half gets + the partner's g sin, the second half - it
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const float o = __shfl_sync(0xffffffffu, t[e], partner);
    if (rot) y[e] += sub < half ? o : -o;
  }
  load8(wn + sub * 8, w);
  float dot = 0.f;
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    x[e] *= r;
    if (live) wsum[e] += y[e] * x[e];
    y[e] *= 1.f + w[e];
    dot += y[e] * x[e];
  }
  dot = group_sum<LPH>(dot) / D;
#pragma unroll
  for (int e = 0; e < 8; ++e) y[e] = r * (y[e] - x[e] * dot);
  if (live) store8(dqkv + at, y);
}

// dqkv from dq, dk, dv [n, heads, D] and the gate's gradient [n, Hq, D]; part [gridDim.x, 2 * D]: sums for the q and k weights.
// A warp's heads are all of one kind, so the copies of dv and the gate's gradient do none of the arithmetic of the others: 3072 tokens,
// 16 / 2 heads of 256: 90 us with kinds mixed, 60 with two blocks an SM, 42 with four.
template <int D>
__global__ void __launch_bounds__(256, 4) pre_bwd_kernel(Args a, const __nv_bfloat16* __restrict__ dq, const __nv_bfloat16* __restrict__ dk,
                                                      const __nv_bfloat16* __restrict__ dv, const __nv_bfloat16* __restrict__ dgate,
                                                      __nv_bfloat16* __restrict__ dqkv, float* __restrict__ part) {
  constexpr int LPH = D / 8, HPW = 32 / LPH;
  __shared__ float acc[8][2 * D];  // weight sums of each warp
  const int lane = threadIdx.x & 31, sub = lane % LPH;
  const long long gq = ((long long)a.n * a.Hq + HPW - 1) / HPW, gk = ((long long)a.n * a.Hk + HPW - 1) / HPW;
  float wq[8], wk[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) wq[e] = wk[e] = 0.f;
  for (long long grp = (long long)blockIdx.x * 8 + (threadIdx.x >> 5); grp < 2 * (gq + gk); grp += (long long)gridDim.x * 8) {
    if (grp < gq) {
      bwd_group<D>(a, grp, a.Hq, 0, 2 * D, 0, dq, a.qw, dqkv, wq);
    } else if (grp < gq + gk) {
      bwd_group<D>(a, grp - gq, a.Hk, 2LL * a.Hq * D, D, a.Hq, dk, a.kw, dqkv, wk);
    } else {
      const bool gate = grp < 2 * gq + gk;
      const int H = gate ? a.Hq : a.Hk;
      const long long item = (grp - (gate ? gq + gk : 2 * gq + gk)) * HPW + lane / LPH;
      if (item < (long long)a.n * H) {
        const long long tok = item / H, hd = item - tok * H;
        const long long at = tok * a.stride + (gate ? hd * 2 * D + D : (2LL * a.Hq + a.Hk + hd) * D) + sub * 8;
        *reinterpret_cast<uint4*>(dqkv + at) = *reinterpret_cast<const uint4*>((gate ? dgate : dv) + item * D + sub * 8);
      }
    }
  }
  // folded over the warp's heads by shuffles, over the warps in shared memory: fp32 atomics there are a compare-and-swap loop
#pragma unroll
  for (int e = 0; e < 8; ++e) {
#pragma unroll
    for (int o = 16; o >= LPH; o >>= 1) {
      wq[e] += __shfl_xor_sync(0xffffffffu, wq[e], o);
      wk[e] += __shfl_xor_sync(0xffffffffu, wk[e], o);
    }
    if (lane < LPH) {
      acc[threadIdx.x >> 5][sub * 8 + e] = wq[e];
      acc[threadIdx.x >> 5][D + sub * 8 + e] = wk[e];
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 2 * D; i += 256) {
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) t += acc[w][i];
    part[(long long)blockIdx.x * 2 * D + i] = t;
  }
}

__device__ __forceinline__ float sigmoid(float x) { return 1.f / (1.f + __expf(-x)); }

// o, y, dy, d_o, dgate: [n, H, D] contiguous; gate: head h of row t at gate + t * stride + h * 2 * D.
__global__ void __launch_bounds__(256) post_fwd_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ gate, long long stride,
                                                       __nv_bfloat16* __restrict__ y, long long nvec, int H, int D) {
  const int hv = D / 8, rv = H * hv;
  for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < nvec; i += (long long)gridDim.x * 256) {
    const long long tok = i / rv;
    const int in = (int)(i % rv);
    float f[8], g[8];
    load8(o + i * 8, f);
    load8(gate + tok * stride + (long long)(in / hv) * 2 * D + in % hv * 8, g);
#pragma unroll
    for (int e = 0; e < 8; ++e) f[e] *= sigmoid(g[e]);
    store8(y + i * 8, f);
  }
}

__global__ void __launch_bounds__(256) post_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ o,
                                                       const __nv_bfloat16* __restrict__ gate, long long stride, __nv_bfloat16* __restrict__ d_o,
                                                       __nv_bfloat16* __restrict__ dgate, long long nvec, int H, int D) {
  const int hv = D / 8, rv = H * hv;
  for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < nvec; i += (long long)gridDim.x * 256) {
    const long long tok = i / rv;
    const int in = (int)(i % rv);
    float d[8], f[8], g[8];
    load8(dy + i * 8, d);
    load8(o + i * 8, f);
    load8(gate + tok * stride + (long long)(in / hv) * 2 * D + in % hv * 8, g);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float s = sigmoid(g[e]);
      g[e] = d[e] * f[e] * s * (1.f - s);
      d[e] *= s;
    }
    store8(d_o + i * 8, d);
    store8(dgate + i * 8, g);
  }
}

}  // namespace gattn
}  // namespace pt

using namespace pt;

static inline int gattn_blocks(long long items, int per_block, int per_sm) {
  const long long want = (items + per_block - 1) / per_block, cap = (long long)sm_count() * per_sm;
  return (int)(want < 1 ? 1 : want < cap ? want : cap);
}
static bool gattn_ok(int n, int Hq, int Hk, int D, int R, long long stride) {
  return n > 0 && Hq > 0 && Hk > 0 && (D == 64 || D == 128 || D == 256) && R > 0 && R % 16 == 0 && R <= D && stride % 8 == 0 &&
         stride >= 2LL * (Hq + Hk) * D;
}

PT_API int pt_gated_attn_pre_fwd(const void* qkv, const void* qw, const void* kw, const void* cosb, const void* sinb, void* q, void* k, void* v,
                                 float* rstd, int n, int Hq, int Hk, int D, int R, long long stride, float eps, void* stream_) {
  if (!gattn_ok(n, Hq, Hk, D, R, stride)) return -2;
  cudaStream_t st = (cudaStream_t)stream_;
  const gattn::Args a{(const __nv_bfloat16*)qkv, (const __nv_bfloat16*)qw, (const __nv_bfloat16*)kw, (const __nv_bfloat16*)cosb,
                      (const __nv_bfloat16*)sinb, rstd, stride, n, Hq, Hk, R, eps};
  const int grid = gattn_blocks((long long)n * (Hq + 2 * Hk), 8 * 256 / D, 16);
#define LAUNCH(DD) gattn::pre_fwd_kernel<DD><<<grid, 256, 0, st>>>(a, (__nv_bfloat16*)q, (__nv_bfloat16*)k, (__nv_bfloat16*)v)
  if (D == 64) LAUNCH(64);
  else if (D == 128) LAUNCH(128);
  else LAUNCH(256);
#undef LAUNCH
  return (int)cudaGetLastError();
}

// Rows of the partial weight gradients ([rows, 2 * D] fp32).
PT_API int pt_gated_attn_parts(int n, int Hq, int Hk, int D) { return gattn_blocks((long long)n * 2 * (Hq + Hk), 8 * 256 / D, 4); }

PT_API int pt_gated_attn_pre_bwd(const void* dq, const void* dk, const void* dv, const void* dgate, const void* qkv, const void* qw, const void* kw,
                                 const void* cosb, const void* sinb, const float* rstd, void* dqkv, float* part, int n, int Hq, int Hk, int D,
                                 int R, long long stride, void* stream_) {
  if (!gattn_ok(n, Hq, Hk, D, R, stride)) return -2;
  cudaStream_t st = (cudaStream_t)stream_;
  const gattn::Args a{(const __nv_bfloat16*)qkv, (const __nv_bfloat16*)qw, (const __nv_bfloat16*)kw, (const __nv_bfloat16*)cosb,
                      (const __nv_bfloat16*)sinb, const_cast<float*>(rstd), stride, n, Hq, Hk, R, 0.f};
  const int grid = pt_gated_attn_parts(n, Hq, Hk, D);
#define LAUNCH(DD) gattn::pre_bwd_kernel<DD><<<grid, 256, 0, st>>>(a, (const __nv_bfloat16*)dq, (const __nv_bfloat16*)dk, (const __nv_bfloat16*)dv, (const __nv_bfloat16*)dgate, (__nv_bfloat16*)dqkv, part)
  if (D == 64) LAUNCH(64);
  else if (D == 128) LAUNCH(128);
  else LAUNCH(256);
#undef LAUNCH
  return (int)cudaGetLastError();
}

PT_API int pt_gated_attn_post_fwd(const void* o, const void* gate, long long stride, void* y, int n, int H, int D, void* stream_) {
  if (n <= 0 || H <= 0 || D % 8 != 0 || stride % 8 != 0) return -2;
  const long long nvec = (long long)n * H * D / 8;
  gattn::post_fwd_kernel<<<gattn_blocks(nvec, 256, 16), 256, 0, (cudaStream_t)stream_>>>((const __nv_bfloat16*)o, (const __nv_bfloat16*)gate, stride,
                                                                                       (__nv_bfloat16*)y, nvec, H, D);
  return (int)cudaGetLastError();
}

PT_API int pt_gated_attn_post_bwd(const void* dy, const void* o, const void* gate, long long stride, void* d_o, void* dgate, int n, int H, int D,
                                  void* stream_) {
  if (n <= 0 || H <= 0 || D % 8 != 0 || stride % 8 != 0) return -2;
  const long long nvec = (long long)n * H * D / 8;
  gattn::post_bwd_kernel<<<gattn_blocks(nvec, 256, 16), 256, 0, (cudaStream_t)stream_>>>((const __nv_bfloat16*)dy, (const __nv_bfloat16*)o,
                                                                                       (const __nv_bfloat16*)gate, stride, (__nv_bfloat16*)d_o,
                                                                                       (__nv_bfloat16*)dgate, nvec, H, D);
  return (int)cudaGetLastError();
}
