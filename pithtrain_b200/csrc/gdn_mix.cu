// The elementwise passes of a Gated DeltaNet layer around its delta rule, forward and backward (bf16 in and out, fp32 inside):
//   conv  : causal depthwise convolution over the positions (4 taps) -> SiLU -> per-head l2 norm of q and k, written per
//           value head (q and k heads repeated), v as it is. The tensor-op form was a depthwise convolution over transposed
//           views, a SiLU, two transposing copies, two normalisations and two repeats.
//   gnorm : rmsnorm(o) * w * silu(z) per head.
// Bound by memory traffic. A warp holds one 128-channel head of one position, 4 channels a lane (eight would halve the
// instructions, but the backward then needs 182 registers and one block fills an SM). In conv a warp walks CT consecutive
// positions with the convolution window in registers, so x is read (1 + 3 / CT) times; the backward recomputes the activation
// from x, and the weight gradients leave as one row of partial sums per block of positions.
// Measured with the passes they replace, two Qwen3.5 layers (one Gated DeltaNet), 2 x 3072 positions: 29.4 -> 23.7 ms a step.
#include "elementwise.cuh"
#include "host_common.h"

namespace pt {
namespace gdn {

constexpr int D = 128, CT = 32, WARPS = 8;  // channels of a head, positions per warp, warps per block

__device__ __forceinline__ float sigmoid(float x) { return 1.f / (1.f + __expf(-x)); }
__device__ __forceinline__ void ld4b(const __nv_bfloat16* p, float (&f)[4]) {
  const uint2 r = *reinterpret_cast<const uint2*>(p);
  f[0] = __uint_as_float(r.x << 16); f[1] = __uint_as_float(r.x & 0xffff0000u);
  f[2] = __uint_as_float(r.y << 16); f[3] = __uint_as_float(r.y & 0xffff0000u);
}
__device__ __forceinline__ void st4b(__nv_bfloat16* p, const float (&f)[4]) {
  __nv_bfloat162 lo = __floats2bfloat162_rn(f[0], f[1]), hi = __floats2bfloat162_rn(f[2], f[3]);
  *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
}
// Row t of x (my 4 channels); zeros outside the sequence.
__device__ __forceinline__ void ld_row(const __nv_bfloat16* x, int t, int S, long long ld, float (&o)[4]) {
  if (t >= 0 && t < S) ld4b(x + (long long)t * ld, o);
  else o[0] = o[1] = o[2] = o[3] = 0.f;
}

struct ConvArgs {
  const __nv_bfloat16 *x, *w;  // x [B, S, (2 nk + nv) * 128], w [(2 nk + nv) * 128, 4]
  int B, S, nk, nv;
};
// Taps of my 4 channels: t[j][c] = w[ch + c][j].
__device__ __forceinline__ void ld_taps(const __nv_bfloat16* w, int ch, float (&t)[4][4]) {
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    float r[4];
    ld4b(w + (size_t)(ch + c) * 4, r);
#pragma unroll
    for (int j = 0; j < 4; ++j) t[j][c] = r[j];
  }
}

// One warp per (head, block of CT positions, batch entry); head < nk: q, < 2 nk: k, else v.
__global__ void __launch_bounds__(32 * WARPS) conv_fwd_kernel(const ConvArgs p, __nv_bfloat16* __restrict__ q, __nv_bfloat16* __restrict__ k,
                                                              __nv_bfloat16* __restrict__ v) {
  const int heads = 2 * p.nk + p.nv, rep = p.nv / p.nk;
  const int hd = blockIdx.x * WARPS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (hd >= heads) return;
  const int b = blockIdx.z, t0 = blockIdx.y * CT, t1 = min(t0 + CT, p.S);
  const int ch = hd * D + lane * 4;
  const long long ld = (long long)heads * D;
  const __nv_bfloat16* x = p.x + (long long)b * p.S * ld + ch;
  float w[4][4], win[3][4];
  ld_taps(p.w, ch, w);
#pragma unroll
  for (int i = 0; i < 3; ++i) ld_row(x, t0 - 3 + i, p.S, ld, win[i]);
  const bool norm = hd < 2 * p.nk;
#pragma unroll 4
  for (int t = t0; t < t1; ++t) {
    float cur[4], y[4], ss = 0.f;
    ld4b(x + (long long)t * ld, cur);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const float pre = fmaf(w[0][c], win[0][c], fmaf(w[1][c], win[1][c], fmaf(w[2][c], win[2][c], w[3][c] * cur[c])));
      y[c] = pre * sigmoid(pre);
      ss = fmaf(y[c], y[c], ss);
      win[0][c] = win[1][c]; win[1][c] = win[2][c]; win[2][c] = cur[c];
    }
    const long long row = ((long long)b * p.S + t) * p.nv;
    if (!norm) {  // uniform over the warp
      st4b(v + (row + hd - 2 * p.nk) * D + lane * 4, y);
    } else {
      const float inv = 1.f / fmaxf(sqrtf(warp_sum(ss)), 1e-12f);
#pragma unroll
      for (int c = 0; c < 4; ++c) y[c] *= inv;
      __nv_bfloat16* o = (hd < p.nk ? q : k) + (row + (long long)(hd < p.nk ? hd : hd - p.nk) * rep) * D + lane * 4;
      for (int i = 0; i < rep; ++i) st4b(o + i * D, y);
    }
  }
}

__global__ void __launch_bounds__(32 * WARPS) conv_bwd_kernel(const ConvArgs p, const __nv_bfloat16* __restrict__ dq,
                                                              const __nv_bfloat16* __restrict__ dk, const __nv_bfloat16* __restrict__ dv,
                                                              __nv_bfloat16* __restrict__ dx, float* __restrict__ dw_part) {
  const int heads = 2 * p.nk + p.nv, rep = p.nv / p.nk;
  const int hd = blockIdx.x * WARPS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (hd >= heads) return;
  const int b = blockIdx.z, t0 = blockIdx.y * CT;
  const int ch = hd * D + lane * 4;
  const long long ld = (long long)heads * D;
  const __nv_bfloat16* x = p.x + (long long)b * p.S * ld + ch;
  __nv_bfloat16* dxp = dx + (long long)b * p.S * ld + ch;
  float w[4][4], win[3][4], dp[3][4], dw[4][4];
  ld_taps(p.w, ch, w);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    ld_row(x, t0 - 3 + i, p.S, ld, win[i]);
#pragma unroll
    for (int c = 0; c < 4; ++c) dp[i][c] = 0.f;
  }
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int c = 0; c < 4; ++c) dw[j][c] = 0.f;
  const bool norm = hd < 2 * p.nk;
  const int own = min(t0 + CT, p.S);  // my positions are [t0, own); three more give the gradients that reach back into them
  const __nv_bfloat16* g = norm ? (hd < p.nk ? dq + (long long)hd * rep * D : dk + (long long)(hd - p.nk) * rep * D)
                                : dv + (long long)(hd - 2 * p.nk) * D;
  g += (long long)b * p.S * p.nv * D + lane * 4;
  const long long gld = (long long)p.nv * D;
  const int copies = norm ? rep : 1;
#pragma unroll 2
  for (int t = t0; t < own + 3; ++t) {
    float cur[4], d[4];
    ld_row(x, t, p.S, ld, cur);
    ld_row(g, t, p.S, gld, d);
    for (int i = 1; i < copies; ++i) {
      float e[4];
      ld_row(g + i * D, t, p.S, gld, e);
#pragma unroll
      for (int c = 0; c < 4; ++c) d[c] += e[c];
    }
    float pre[4], sg[4], ss = 0.f, dot = 0.f;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      pre[c] = fmaf(w[0][c], win[0][c], fmaf(w[1][c], win[1][c], fmaf(w[2][c], win[2][c], w[3][c] * cur[c])));
      sg[c] = sigmoid(pre[c]);
      const float y = pre[c] * sg[c];
      ss = fmaf(y, y, ss);
      dot = fmaf(y, d[c], dot);
    }
    if (norm) {
      // z = y / n: dy = (dz - z <z, dz>) / n; a norm under the floor is a constant divisor
      ss = warp_sum(ss);
      dot = warp_sum(dot);
      const float n = sqrtf(ss), inv = 1.f / fmaxf(n, 1e-12f), f = n > 1e-12f ? dot * inv * inv : 0.f;
#pragma unroll
      for (int c = 0; c < 4; ++c) d[c] = (d[c] - pre[c] * sg[c] * f) * inv;
    }
    float o[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      d[c] *= sg[c] * (1.f + pre[c] * (1.f - sg[c]));
      if (t < own) {
        dw[0][c] = fmaf(d[c], win[0][c], dw[0][c]);
        dw[1][c] = fmaf(d[c], win[1][c], dw[1][c]);
        dw[2][c] = fmaf(d[c], win[2][c], dw[2][c]);
        dw[3][c] = fmaf(d[c], cur[c], dw[3][c]);
      }
      // position t - 3 is complete: taps 3 .. 0 meet the gradients of positions t - 3 .. t
      o[c] = fmaf(w[3][c], dp[0][c], fmaf(w[2][c], dp[1][c], fmaf(w[1][c], dp[2][c], w[0][c] * d[c])));
      dp[0][c] = dp[1][c]; dp[1][c] = dp[2][c]; dp[2][c] = d[c];
      win[0][c] = win[1][c]; win[1][c] = win[2][c]; win[2][c] = cur[c];
    }
    if (t - 3 >= t0) st4b(dxp + (long long)(t - 3) * ld, o);
  }
  float* o = dw_part + ((long long)b * gridDim.y + blockIdx.y) * ld * 4 + (long long)ch * 4;
#pragma unroll
  for (int c = 0; c < 4; ++c) *reinterpret_cast<float4*>(o + 4 * c) = make_float4(dw[0][c], dw[1][c], dw[2][c], dw[3][c]);
}

__global__ void __launch_bounds__(32 * WARPS) gnorm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ z,
                                                               const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ out,
                                                               long long rows, float eps) {
  const int lane = threadIdx.x & 31;
  float wv[4];
  ld4b(w + lane * 4, wv);
  const long long step = (long long)gridDim.x * WARPS;
#pragma unroll 2
  for (long long r = (long long)blockIdx.x * WARPS + (threadIdx.x >> 5); r < rows; r += step) {
    float a[4], g[4], ss = 0.f;
    ld4b(x + r * D + lane * 4, a);
    ld4b(z + r * D + lane * 4, g);
#pragma unroll
    for (int c = 0; c < 4; ++c) ss = fmaf(a[c], a[c], ss);
    const float rstd = rsqrtf(warp_sum(ss) / D + eps);
#pragma unroll
    for (int c = 0; c < 4; ++c) a[c] = a[c] * rstd * wv[c] * (g[c] * sigmoid(g[c]));
    st4b(out + r * D + lane * 4, a);
  }
}

__global__ void __launch_bounds__(32 * WARPS) gnorm_bwd_kernel(const __nv_bfloat16* __restrict__ dout, const __nv_bfloat16* __restrict__ x,
                                                               const __nv_bfloat16* __restrict__ z, const __nv_bfloat16* __restrict__ w,
                                                               __nv_bfloat16* __restrict__ dx, __nv_bfloat16* __restrict__ dz,
                                                               float* __restrict__ dw_part, long long rows, float eps) {
  __shared__ float red[WARPS][D];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float wv[4], dw[4] = {0.f, 0.f, 0.f, 0.f};
  ld4b(w + lane * 4, wv);
  const long long step = (long long)gridDim.x * WARPS;
#pragma unroll 2
  for (long long r = (long long)blockIdx.x * WARPS + warp; r < rows; r += step) {
    float a[4], g[4], d[4], ss = 0.f, dot = 0.f;
    ld4b(x + r * D + lane * 4, a);
    ld4b(z + r * D + lane * 4, g);
    ld4b(dout + r * D + lane * 4, d);
#pragma unroll
    for (int c = 0; c < 4; ++c) ss = fmaf(a[c], a[c], ss);
    const float rstd = rsqrtf(warp_sum(ss) / D + eps);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const float sg = sigmoid(g[c]), sl = g[c] * sg;
      a[c] *= rstd;
      const float dn = d[c] * sl;  // gradient of xhat * w
      dw[c] = fmaf(dn, a[c], dw[c]);
      g[c] = d[c] * a[c] * wv[c] * (sg * (1.f + g[c] * (1.f - sg)));
      d[c] = dn * wv[c];
      dot = fmaf(d[c], a[c], dot);
    }
    dot = warp_sum(dot) / D;
#pragma unroll
    for (int c = 0; c < 4; ++c) a[c] = rstd * (d[c] - a[c] * dot);
    st4b(dx + r * D + lane * 4, a);
    st4b(dz + r * D + lane * 4, g);
  }
#pragma unroll
  for (int c = 0; c < 4; ++c) red[warp][lane * 4 + c] = dw[c];
  __syncthreads();
  if (threadIdx.x < D) {
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < WARPS; ++i) s += red[i][threadIdx.x];
    dw_part[(long long)blockIdx.x * D + threadIdx.x] = s;
  }
}

}  // namespace gdn
}  // namespace pt

using namespace pt;

// x [B, S, (2 nk + nv) * 128] bf16 contiguous, w [(2 nk + nv) * 128, 4]; q, k, v [B, S, nv, 128]; nv a multiple of nk. All
// pointers 16-byte aligned.
PT_API int pt_gdn_conv_fwd(const void* x, const void* w, void* q, void* k, void* v, int B, int S, int nk, int nv, void* stream_) {
  if (B <= 0 || S <= 0 || nk <= 0 || nv <= 0 || nv % nk != 0 || B > 65535 || S > 65535 * gdn::CT) return -2;
  const gdn::ConvArgs a{static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(w), B, S, nk, nv};
  const dim3 grid((2 * nk + nv + gdn::WARPS - 1) / gdn::WARPS, (S + gdn::CT - 1) / gdn::CT, B);
  gdn::conv_fwd_kernel<<<grid, 32 * gdn::WARPS, 0, static_cast<cudaStream_t>(stream_)>>>(
      a, static_cast<__nv_bfloat16*>(q), static_cast<__nv_bfloat16*>(k), static_cast<__nv_bfloat16*>(v));
  return (int)cudaGetLastError();
}

// Rows of dw_part: one per (batch entry, block of positions), (2 nk + nv) * 128 * 4 floats each, laid out like w.
PT_API int pt_gdn_conv_parts(int B, int S) { return B * ((S + gdn::CT - 1) / gdn::CT); }
PT_API int pt_gdn_conv_bwd(const void* x, const void* w, const void* dq, const void* dk, const void* dv, void* dx, float* dw_part, int B, int S,
                           int nk, int nv, void* stream_) {
  if (B <= 0 || S <= 0 || nk <= 0 || nv <= 0 || nv % nk != 0 || B > 65535 || S > 65535 * gdn::CT) return -2;
  const gdn::ConvArgs a{static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(w), B, S, nk, nv};
  const dim3 grid((2 * nk + nv + gdn::WARPS - 1) / gdn::WARPS, (S + gdn::CT - 1) / gdn::CT, B);
  gdn::conv_bwd_kernel<<<grid, 32 * gdn::WARPS, 0, static_cast<cudaStream_t>(stream_)>>>(
      a, static_cast<const __nv_bfloat16*>(dq), static_cast<const __nv_bfloat16*>(dk), static_cast<const __nv_bfloat16*>(dv),
      static_cast<__nv_bfloat16*>(dx), dw_part);
  return (int)cudaGetLastError();
}

// x, z, out [rows, 128] bf16 contiguous
PT_API int pt_gdn_gnorm_fwd(const void* x, const void* z, const void* w, void* out, long long rows, float eps, void* stream_) {
  if (rows <= 0) return 0;
  const long long need = (rows + gdn::WARPS - 1) / gdn::WARPS, cap = (long long)sm_count() * 16;
  gdn::gnorm_fwd_kernel<<<(unsigned)(need < cap ? need : cap), 32 * gdn::WARPS, 0, static_cast<cudaStream_t>(stream_)>>>(
      static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(z), static_cast<const __nv_bfloat16*>(w),
      static_cast<__nv_bfloat16*>(out), rows, eps);
  return (int)cudaGetLastError();
}
PT_API int pt_gdn_gnorm_parts(long long rows) {
  const long long need = (rows + gdn::WARPS - 1) / gdn::WARPS, cap = (long long)sm_count() * 8;
  return (int)(need < cap ? (need > 0 ? need : 1) : cap);
}
// dw_part [pt_gdn_gnorm_parts(rows), 128] fp32
PT_API int pt_gdn_gnorm_bwd(const void* dout, const void* x, const void* z, const void* w, void* dx, void* dz, float* dw_part, long long rows,
                            float eps, void* stream_) {
  if (rows <= 0) return 0;
  gdn::gnorm_bwd_kernel<<<pt_gdn_gnorm_parts(rows), 32 * gdn::WARPS, 0, static_cast<cudaStream_t>(stream_)>>>(
      static_cast<const __nv_bfloat16*>(dout), static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(z),
      static_cast<const __nv_bfloat16*>(w), static_cast<__nv_bfloat16*>(dx), static_cast<__nv_bfloat16*>(dz), dw_part, rows, eps);
  return (int)cudaGetLastError();
}
