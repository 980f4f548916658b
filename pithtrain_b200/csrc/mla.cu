// Query / key / value assembly of multi-head latent attention, forward and backward, one pass each:
//   q [n, Hq, dn + dr] and the up-projected latent kv [n, Hq, dn + dv] with one shared rotary key k_pe [n, dr] become
//   q' = (q_nope, rope(q_pe)), k' = (k_nope, rope(k_pe) for every head), v, each contiguous [n, Hq, d] as the attention
//   kernels read them. The tensor-op form was two de-interleaving copies, two rotations of four operations each, an expand, two
//   concatenations and a copy of v, and as much again backward. Bound by memory traffic; a block owns a token, every access is
//   16 bytes. The rotary dims arrive as (x0, y0, x1, y1, ..) pairs and leave as (x.., y..) halves; rotated in fp32, rounded once.
#include "elementwise.cuh"
#include "host_common.h"
#include "ptx.cuh"

namespace pt {
namespace mla {

struct Args {
  const __nv_bfloat16 *q, *kpe, *kv;  // row pitches ldq, ldk, ldkv
  long long ldq, ldk, ldkv;
  const __nv_bfloat16 *cosb, *sinb;   // [rows, dr]
  const int* pos;                     // optional [n]; else row % S
  int n, S, H, dn, dr, dv, rows;
  int* err;
};

// Row of the rotary tables for token t, counted from their end if negative. A position outside them is recorded and reads as
// row 0 (false): its rotated values are NaN.
__device__ __forceinline__ bool table_row(const Args& p, int t, long long& row) {
  const int pos = p.pos ? p.pos[t] : t % p.S;
  row = pos < 0 ? pos + p.rows : pos;
  if (row >= 0 && row < p.rows) return true;
  if (threadIdx.x == 0 && p.err) atomicCAS(p.err, 0, PT_ERR_BOUNDS);
  row = 0;
  return false;
}
__device__ __forceinline__ void spoil(float (&a)[8], float (&b)[8]) {
#pragma unroll
  for (int e = 0; e < 8; ++e) a[e] = b[e] = NAN;
}

// 16 interleaved values -> 8 of the first and 8 of the second half, rotated; i0 = 8 j is the first pair
__device__ __forceinline__ void rotate(const __nv_bfloat16* src, const __nv_bfloat16* c, const __nv_bfloat16* s, int i0, int half,
                                       float (&o1)[8], float (&o2)[8]) {
  float a[8], b[8], c1[8], c2[8], s1[8], s2[8];
  load8(src + 2 * i0, a);
  load8(src + 2 * i0 + 8, b);
  load8(c + i0, c1); load8(c + half + i0, c2);
  load8(s + i0, s1); load8(s + half + i0, s2);
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const float x = e < 4 ? a[2 * e] : b[2 * e - 8], y = e < 4 ? a[2 * e + 1] : b[2 * e - 7];
    o1[e] = x * c1[e] - y * s1[e];
    o2[e] = y * c2[e] + x * s2[e];
  }
}
// its transpose: gradients of the halves -> 16 interleaved gradients
__device__ __forceinline__ void rotate_back(const __nv_bfloat16* g, const __nv_bfloat16* c, const __nv_bfloat16* s, int i0, int half,
                                            float (&lo)[8], float (&hi)[8]) {
  float g1[8], g2[8], c1[8], c2[8], s1[8], s2[8];
  load8(g + i0, g1); load8(g + half + i0, g2);
  load8(c + i0, c1); load8(c + half + i0, c2);
  load8(s + i0, s1); load8(s + half + i0, s2);
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const float x = g1[e] * c1[e] + g2[e] * s2[e], y = g2[e] * c2[e] - g1[e] * s1[e];
    if (e < 4) { lo[2 * e] = x; lo[2 * e + 1] = y; }
    else { hi[2 * e - 8] = x; hi[2 * e - 7] = y; }
  }
}
__device__ __forceinline__ void copy8(__nv_bfloat16* d, const __nv_bfloat16* s) { *reinterpret_cast<uint4*>(d) = *reinterpret_cast<const uint4*>(s); }

__global__ void __launch_bounds__(256) fwd_kernel(const Args p, __nv_bfloat16* __restrict__ qo, __nv_bfloat16* __restrict__ ko,
                                                  __nv_bfloat16* __restrict__ vo) {
  const int t = blockIdx.x, half = p.dr / 2, d = p.dn + p.dr;
  const __nv_bfloat16 *q = p.q + t * p.ldq, *kv = p.kv + t * p.ldkv, *kpe = p.kpe + t * p.ldk;
  long long row;
  const bool known = table_row(p, t, row);
  const __nv_bfloat16 *c = p.cosb + row * p.dr, *s = p.sinb + row * p.dr;
  __nv_bfloat16 *qt = qo + (long long)t * p.H * d, *kt = ko + (long long)t * p.H * d, *vt = vo + (long long)t * p.H * p.dv;
  const int nn = p.dn / 8, nv = p.dv / 8, nr = p.dr / 16;
  for (int i = threadIdx.x; i < p.H * nn; i += blockDim.x) {
    const int h = i / nn, x = (i - h * nn) * 8;
    copy8(qt + h * d + x, q + h * d + x);
    copy8(kt + h * d + x, kv + h * (p.dn + p.dv) + x);
  }
  for (int i = threadIdx.x; i < p.H * nv; i += blockDim.x) {
    const int h = i / nv, x = (i - h * nv) * 8;
    copy8(vt + h * p.dv + x, kv + h * (p.dn + p.dv) + p.dn + x);
  }
  for (int i = threadIdx.x; i < p.H * nr; i += blockDim.x) {
    const int h = i / nr, i0 = (i - h * nr) * 8;
    float a[8], b[8];
    rotate(q + h * d + p.dn, c, s, i0, half, a, b);
    if (!known) spoil(a, b);
    store8(qt + h * d + p.dn + i0, a);
    store8(qt + h * d + p.dn + half + i0, b);
    rotate(kpe, c, s, i0, half, a, b);
    if (!known) spoil(a, b);
    store8(kt + h * d + p.dn + i0, a);
    store8(kt + h * d + p.dn + half + i0, b);
  }
}

__global__ void __launch_bounds__(256) bwd_kernel(const Args p, const __nv_bfloat16* __restrict__ gq, const __nv_bfloat16* __restrict__ gk,
                                                  const __nv_bfloat16* __restrict__ gv, __nv_bfloat16* __restrict__ dq,
                                                  __nv_bfloat16* __restrict__ dkpe, __nv_bfloat16* __restrict__ dkv) {
  extern __shared__ float part[];  // [H][dr]: the heads' gradients of the shared rotary key
  const int t = blockIdx.x, half = p.dr / 2, d = p.dn + p.dr;
  long long row;
  const bool known = table_row(p, t, row);
  const __nv_bfloat16 *c = p.cosb + row * p.dr, *s = p.sinb + row * p.dr;
  const __nv_bfloat16 *qt = gq + (long long)t * p.H * d, *kt = gk + (long long)t * p.H * d, *vt = gv + (long long)t * p.H * p.dv;
  __nv_bfloat16 *dqt = dq + (long long)t * p.H * d, *dkvt = dkv + (long long)t * p.H * (p.dn + p.dv);
  const int nn = p.dn / 8, nv = p.dv / 8, nr = p.dr / 16;
  for (int i = threadIdx.x; i < p.H * nr; i += blockDim.x) {
    const int h = i / nr, i0 = (i - h * nr) * 8;
    float lo[8], hi[8];
    rotate_back(qt + h * d + p.dn, c, s, i0, half, lo, hi);
    if (!known) spoil(lo, hi);
    store8(dqt + h * d + p.dn + 2 * i0, lo);
    store8(dqt + h * d + p.dn + 2 * i0 + 8, hi);
    rotate_back(kt + h * d + p.dn, c, s, i0, half, lo, hi);
    if (!known) spoil(lo, hi);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      part[h * p.dr + 2 * i0 + e] = lo[e];
      part[h * p.dr + 2 * i0 + 8 + e] = hi[e];
    }
  }
  for (int i = threadIdx.x; i < p.H * nn; i += blockDim.x) {
    const int h = i / nn, x = (i - h * nn) * 8;
    copy8(dqt + h * d + x, qt + h * d + x);
    copy8(dkvt + h * (p.dn + p.dv) + x, kt + h * d + x);
  }
  for (int i = threadIdx.x; i < p.H * nv; i += blockDim.x) {
    const int h = i / nv, x = (i - h * nv) * 8;
    copy8(dkvt + h * (p.dn + p.dv) + p.dn + x, vt + h * p.dv + x);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < p.dr; i += blockDim.x) {
    float a = 0.f;
    for (int h = 0; h < p.H; ++h) a += part[h * p.dr + i];
    dkpe[(long long)t * p.dr + i] = __float2bfloat16(a);
  }
}

inline bool valid(const Args& a) {
  return a.n > 0 && a.H > 0 && a.S > 0 && a.rows > 0 && a.dn > 0 && a.dv > 0 && a.dr > 0 && a.dn % 8 == 0 && a.dv % 8 == 0 && a.dr % 16 == 0 &&
         a.H * a.dr * 4 <= 48 * 1024;
}

}  // namespace mla
}  // namespace pt

using namespace pt;

// q [n, H (dn + dr)], kpe [n, dr], kv [n, H (dn + dv)] bf16 with row pitches (elements, multiples of 8, 16-byte aligned bases); cosb,
// sinb [rows, dr] bf16; pos int32 [n] or null (then row % S). Outputs contiguous. dn, dv multiples of 8, dr of 16.
PT_API int pt_mla_fwd(const void* q, const void* kpe, const void* kv, long long ldq, long long ldk, long long ldkv, const void* cosb,
                      const void* sinb, const int* pos, void* qo, void* ko, void* vo, int n, int S, int H, int dn, int dr, int dv,
                      int rows, void* stream_) {
  using B = __nv_bfloat16;
  const mla::Args a{static_cast<const B*>(q), static_cast<const B*>(kpe), static_cast<const B*>(kv), ldq, ldk, ldkv, static_cast<const B*>(cosb),
                    static_cast<const B*>(sinb), pos, n, S, H, dn, dr, dv, rows, device_status_word()};
  if (!mla::valid(a)) return -2;
  mla::fwd_kernel<<<n, 256, 0, static_cast<cudaStream_t>(stream_)>>>(a, static_cast<B*>(qo), static_cast<B*>(ko), static_cast<B*>(vo));
  return (int)cudaGetLastError();
}

// Gradients gq, gk, gv of the outputs (contiguous) -> dq [n, H (dn + dr)], dkpe [n, dr], dkv [n, H (dn + dv)], contiguous.
PT_API int pt_mla_bwd(const void* gq, const void* gk, const void* gv, const void* cosb, const void* sinb, const int* pos, void* dq, void* dkpe,
                      void* dkv, int n, int S, int H, int dn, int dr, int dv, int rows, void* stream_) {
  using B = __nv_bfloat16;
  const mla::Args a{nullptr, nullptr, nullptr, 0, 0, 0, static_cast<const B*>(cosb), static_cast<const B*>(sinb), pos, n, S, H, dn, dr, dv, rows,
                    device_status_word()};
  if (!mla::valid(a)) return -2;
  mla::bwd_kernel<<<n, 256, H * dr * 4, static_cast<cudaStream_t>(stream_)>>>(
      a, static_cast<const B*>(gq), static_cast<const B*>(gk), static_cast<const B*>(gv), static_cast<B*>(dq), static_cast<B*>(dkpe),
      static_cast<B*>(dkv));
  return (int)cudaGetLastError();
}
