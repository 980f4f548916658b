// Gated delta rule (Gated DeltaNet) for bf16 q, k, v with head dims 128: the whole chunked evaluation in six kernels, forward
// and backward, chunk C = 64. (csrc/gdr.cu holds only the pass over the chunks, for the other dtypes and head dims.)
//
//   per chunk, b = cumulative log gate, D_ij = exp(b_i - b_j) for j <= i, qs = q / sqrt(dk):
//     A = strict_lower(beta_i <k_i, k_j> D_ij)     T = (I + A)^-1     u = T (beta v)     w = T (beta e^b k)
//     P = lower(<qs_i, k_j> D_ij)
//   across chunks:  v' = u - w S      S+ = e^{b_last} S + (e^{b_last - b} k)^T v'
//     o = (e^b qs) S + P v'
//
//   gdr_chunk_fwd   (chunks x heads)            : b, P, T, u, w
//   gdr_scan_fwd    (heads x 4 value slices)    : v', and the entry state of every chunk
//   gdr_out         (chunks x heads x 2 halves) : o
//   gdr_dvp         (chunks x heads)            : P^T do, what the outputs ask of v'
//   gdr_scan_bwd    (heads x 4 value slices)    : dv', and the gradient of every chunk's exit state
//   gdr_chunk_bwd   (chunks x heads)            : dq, dk, dv, dg, dbeta
//
// All arithmetic is fp32 FMA on fp32 values (q, k, v and do are bf16 and enter exactly), as in the tensor-op form: splitting
// operands over tensor-core products was not taken because the state recurrence carries every rounding to the end of the
// sequence. 5.8 M FMA per chunk and head forward, 12 M backward; two to an instruction they keep the FMA pipe 38 to 55 % busy.
// What bounds the kernels is the shared memory that the operands come from (63 to 82 % of its pipe) and the wait for it. Two
// things follow. Only the products that need the running state stay in the sequential kernels (w S and k^T v' forward); and every
// product reads its operands from shared memory in 16-byte pieces, 8 to 11 FMA per piece, tiles padded to 132 or 68 columns so
// that the eight threads of a phase hit different banks. The sequential kernels prefetch the next chunk with cp.async.
//
// A product phase of a chunk kernel has eight warps and nothing beside it, so what it needs is fetched before it: tiles by
// cp.async under the phase in front, rows of q, k and v into registers.
// Measured, 1 x 3072, 32 heads (48 chunks): chunk_fwd 211, scan_fwd 291, out 136, dvp 49, scan_bwd 397, chunk_bwd 816 us; with
// plain loads between the phases out took 242 and chunk_bwd 1122 (issue slots 28 %, waits for global memory 2.7 per issue; now
// 42 % and 0.3). The tensor-op form with the recurrence kernels of csrc/gdr.cu took about 8 ms for the two directions.
// The sums of a row or column are made in a fixed order: results are reproducible.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "elementwise.cuh"
#include "host_common.h"
#include "ptx.cuh"

namespace pt {
namespace gdr {

constexpr int C = 64, D = 128, LD = 132, LS = 68, VS = 32, LV = 36, NT = 256;
constexpr int T64 = C * LD;    // floats of a padded [64 x 128] tile
constexpr int LK = 136;        // bf16 row pitch of the prefetched q / k tiles

struct Args {
  const __nv_bfloat16 *q, *k, *v;      // [B, S, H, 128], element strides below
  long long q_b, q_s, q_h, k_b, k_s, k_h, v_b, v_s, v_h;
  const float *g, *beta;               // [B, S, H]
  float *gc;                           // [BH, N, 64] cumulative log gates
  float *P, *T;                        // [BH, N, 64, 64]
  float *u, *w, *vn;                   // [BH, N, 64, 128]
  float *st;                           // [BH, N, 128, 128] entry states
  __nv_bfloat16* o;                    // [B, S, H, 128]
  // backward
  const __nv_bfloat16* d_o;            // [B, S, H, 128]
  float *dvn;                          // [BH, N, 64, 128]: P^T do, then dv' (in place)
  float *dst;                          // [BH, N, 128, 128] gradients of the exit states
  __nv_bfloat16 *dq, *dk, *dv;         // [B, S, H, 128]
  float *dg, *dbeta;                   // [B, S, H]
  int B, S, H, N;
  float scale;
};

__device__ __forceinline__ float exp_c(float x) { return exp_compensated(x); }

// Two fp32 FMAs in one instruction (fma.rn.f32x2, same rounding as two fmaf): half the issue slots beside the loads.
typedef uint64_t f2;
struct Pair2 { f2 lo, hi; };  // a 16-byte piece as two packed pairs
__device__ __forceinline__ Pair2 ld2(const float* p) {
  const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
  return Pair2{v.x, v.y};
}
__device__ __forceinline__ float sum2(f2 v) {
  float a, b;
  f2_unpack(v, a, b);
  return a + b;
}
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float a, float b, float c, float d) { *reinterpret_cast<float4*>(p) = make_float4(a, b, c, d); }
__device__ __forceinline__ float4 bf4(uint2 r) {
  return make_float4(__uint_as_float(r.x << 16), __uint_as_float(r.x & 0xffff0000u), __uint_as_float(r.y << 16), __uint_as_float(r.y & 0xffff0000u));
}
__device__ __forceinline__ uint2 pack4(float a, float b, float c, float d) {
  __nv_bfloat162 lo = __floats2bfloat162_rn(a, b), hi = __floats2bfloat162_rn(c, d);
  return make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
}
__device__ __forceinline__ void cp16(void* dst, const void* src, int bytes) {  // bytes = 16, or 0 to fill with zeros
  const uint32_t s = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int K>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(K) : "memory"); }

// Thread layout of every 64-row product: ti = tid / 16, tj = tid % 16; rows ti + 16 r (r < 4). Columns of a 64-column result:
// tj + 16 c (c < 4); of a 128-column result: 4 tj + 64 h + e, index x = 4 h + e (h < 2, e < 4).

// acc[r][c] += sum_d A[ti + 16 r][d] * B[tj + 16 c][d] (even and odd d in the two halves of a packed sum)
__device__ __forceinline__ void mm_nt64(const float* A, const float* B, float (&acc)[4][4]) {
  const int ti = threadIdx.x >> 4, tj = threadIdx.x & 15;
  f2 s[4][4];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) s[r][c] = 0ull;
#pragma unroll 2
  for (int d = 0; d < D; d += 4) {
    Pair2 a[4], b[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) a[r] = ld2(A + (ti + 16 * r) * LD + d);
#pragma unroll
    for (int c = 0; c < 4; ++c) b[c] = ld2(B + (tj + 16 * c) * LD + d);
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) s[r][c] = f2_fma(a[r].hi, b[c].hi, f2_fma(a[r].lo, b[c].lo, s[r][c]));
  }
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[r][c] += sum2(s[r][c]);
}
// acc[0..8) += a * (p, q): four packed FMAs
__device__ __forceinline__ void fma8(float a, const Pair2& p, const Pair2& q, f2 (&acc)[4]) {
  const f2 aa = f2_pack(a, a);
  acc[0] = f2_fma(aa, p.lo, acc[0]);
  acc[1] = f2_fma(aa, p.hi, acc[1]);
  acc[2] = f2_fma(aa, q.lo, acc[2]);
  acc[3] = f2_fma(aa, q.hi, acc[3]);
}
// m += x * p, n += y * p for a piece p of four
__device__ __forceinline__ void fma4x2(float x, float y, const Pair2& p, f2 (&m)[2], f2 (&n)[2]) {
  const f2 xx = f2_pack(x, x), yy = f2_pack(y, y);
  m[0] = f2_fma(xx, p.lo, m[0]); m[1] = f2_fma(xx, p.hi, m[1]);
  n[0] = f2_fma(yy, p.lo, n[0]); n[1] = f2_fma(yy, p.hi, n[1]);
}
__device__ __forceinline__ void pack8(const float (&a)[4][8], f2 (&s)[4][4]) {
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int x = 0; x < 4; ++x) s[r][x] = f2_pack(a[r][2 * x], a[r][2 * x + 1]);
}
__device__ __forceinline__ void unpack8(const f2 (&s)[4][4], float (&a)[4][8]) {
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int x = 0; x < 4; ++x) f2_unpack(s[r][x], a[r][2 * x], a[r][2 * x + 1]);
}
// acc[r][x] += sum_{j < K} A[ti + 16 r][j] * B[j][col x]; pitches LA and LB
template <int K, int LA, int LB>
__device__ __forceinline__ void mm_nn(const float* A, const float* B, float (&acc)[4][8]) {
  const int ti = threadIdx.x >> 4, tj = threadIdx.x & 15;
  f2 s[4][4];
  pack8(acc, s);
#pragma unroll 2
  for (int j = 0; j < K; j += 4) {
    float4 a[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) a[r] = ld4(A + (ti + 16 * r) * LA + j);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const Pair2 p = ld2(B + (j + e) * LB + 4 * tj), q = ld2(B + (j + e) * LB + 4 * tj + 64);
#pragma unroll
      for (int r = 0; r < 4; ++r) fma8(e == 0 ? a[r].x : e == 1 ? a[r].y : e == 2 ? a[r].z : a[r].w, p, q, s[r]);
    }
  }
  unpack8(s, acc);
}
// acc[r][x] += sum_{j < 64} A[j][ti + 16 r] * B[j][col x]; A pitch LS, B pitch LD
__device__ __forceinline__ void mm_tn(const float* A, const float* B, float (&acc)[4][8]) {
  const int ti = threadIdx.x >> 4, tj = threadIdx.x & 15;
  f2 s[4][4];
  pack8(acc, s);
#pragma unroll 4
  for (int j = 0; j < C; ++j) {
    const Pair2 p = ld2(B + j * LD + 4 * tj), q = ld2(B + j * LD + 4 * tj + 64);
#pragma unroll
    for (int r = 0; r < 4; ++r) fma8(A[j * LS + ti + 16 * r], p, q, s[r]);
  }
  unpack8(s, acc);
}
// A [128 x 128] tile whose rows are read as columns of a 128-column result: row d lies at physical row state_row(d), so that
// the threads tj of a phase read neighbouring physical rows (tj + 16 x).
__device__ __forceinline__ int state_row(int d) { return ((d & 63) >> 2) + 16 * ((d & 3) + 4 * (d >> 6)); }
// acc[r][x] += sum_v A[ti + 16 r][v] * St[col x][v]
__device__ __forceinline__ void mm_nt128(const float* A, const float* St, float (&acc)[4][8]) {
  const int ti = threadIdx.x >> 4, tj = threadIdx.x & 15;
  f2 s[4][8];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int x = 0; x < 8; ++x) s[r][x] = 0ull;
#pragma unroll 1
  for (int v = 0; v < D; v += 4) {
    Pair2 a[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) a[r] = ld2(A + (ti + 16 * r) * LD + v);
#pragma unroll
    for (int x = 0; x < 8; ++x) {
      const Pair2 b = ld2(St + (tj + 16 * x) * LD + v);
#pragma unroll
      for (int r = 0; r < 4; ++r) s[r][x] = f2_fma(a[r].hi, b.hi, f2_fma(a[r].lo, b.lo, s[r][x]));
    }
  }
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int x = 0; x < 8; ++x) acc[r][x] += sum2(s[r][x]);
}
template <int R, int X>
__device__ __forceinline__ void zero(float (&a)[R][X]) {
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int x = 0; x < X; ++x) a[r][x] = 0.f;
}
// Sum over the 16 threads tj of a row (all get it).
__device__ __forceinline__ float row_sum(float v) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// [64 x 128] bf16 rows of one head -> fp32 tile, each row times rs[i] (null: 1); rows past the sequence are zero. All loads are
// in flight before the first is used: between two products nothing else hides their latency.
__device__ __forceinline__ void load_bf16(float* dst, const __nv_bfloat16* src, long long pitch, int rows, const float* rs) {
  constexpr int IT = C * (D / 8) / NT;
  uint4 x[IT];
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int i = threadIdx.x + it * NT, r = i >> 4;
    x[it] = make_uint4(0u, 0u, 0u, 0u);
    if (r < rows) x[it] = *reinterpret_cast<const uint4*>(src + r * pitch + (i & 15) * 8);
  }
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int i = threadIdx.x + it * NT, r = i >> 4, c = (i & 15) * 8;
    const float f = rs ? rs[r] : 1.f;
    const float4 a = bf4(make_uint2(x[it].x, x[it].y)), b = bf4(make_uint2(x[it].z, x[it].w));
    st4(dst + r * LD + c, a.x * f, a.y * f, a.z * f, a.w * f);
    st4(dst + r * LD + c + 4, b.x * f, b.y * f, b.z * f, b.w * f);
  }
}
// fp32 [64 x 128] and [64 x 64] -> padded tiles, asynchronously (cp_commit / cp_wait by the caller)
__device__ __forceinline__ void load_f32(float* dst, const float* src) {
#pragma unroll
  for (int it = 0; it < C * (D / 4) / NT; ++it) {
    const int i = threadIdx.x + it * NT;
    cp16(dst + (i >> 5) * LD + (i & 31) * 4, src + i * 4, 16);
  }
}
__device__ __forceinline__ void load_sq(float* dst, const float* src) {
#pragma unroll
  for (int it = 0; it < C * (C / 4) / NT; ++it) {
    const int i = threadIdx.x + it * NT;
    cp16(dst + (i >> 4) * LS + (i & 15) * 4, src + i * 4, 16);
  }
}
// result rows ti + 16 r, 8 columns -> fp32 [64 x 128]
__device__ __forceinline__ void store_f32(float* dst, const float (&a)[4][8]) {
  const int ti = threadIdx.x >> 4, tj = threadIdx.x & 15;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    st4(dst + (ti + 16 * r) * D + 4 * tj, a[r][0], a[r][1], a[r][2], a[r][3]);
    st4(dst + (ti + 16 * r) * D + 4 * tj + 64, a[r][4], a[r][5], a[r][6], a[r][7]);
  }
}
__device__ __forceinline__ void store_tile(float* dst, const float (&a)[4][8]) {
  const int ti = threadIdx.x >> 4, tj = threadIdx.x & 15;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    st4(dst + (ti + 16 * r) * LD + 4 * tj, a[r][0], a[r][1], a[r][2], a[r][3]);
    st4(dst + (ti + 16 * r) * LD + 4 * tj + 64, a[r][4], a[r][5], a[r][6], a[r][7]);
  }
}
// 8 columns of a bf16 row [.., 128]
__device__ __forceinline__ void store_bf16_row(__nv_bfloat16* row, const float (&a)[8]) {
  const int tj = threadIdx.x & 15;
  *reinterpret_cast<uint2*>(row + 4 * tj) = pack4(a[0], a[1], a[2], a[3]);
  *reinterpret_cast<uint2*>(row + 4 * tj + 64) = pack4(a[4], a[5], a[6], a[7]);
}

struct Where {
  int n, bh, b, h, s0, rows;  // chunk, (batch, head), first position and live rows of the chunk
};
__device__ __forceinline__ Where where(const Args& p, int n, int bh) {
  Where x;
  x.n = n; x.bh = bh; x.b = bh / p.H; x.h = bh % p.H; x.s0 = n * C;
  x.rows = min(C, p.S - x.s0);
  return x;
}

// T = (I + A)^-1 of a strictly lower A [64 x 64] in shared memory (pitch LS), by blocks: the four 16 x 16 diagonal blocks by
// substitution, then T21 = -T22 A21 T11 for 32- and 64-blocks. The upper right quarter of A is scratch.
__device__ __forceinline__ void unit_lower_inverse(float* A, float* T) {
  const int tid = threadIdx.x;
  for (int i = tid; i < C * LS; i += NT) T[i] = 0.f;
  __syncthreads();
  if (tid < 64) {
    const int b0 = (tid >> 4) * 16, c = tid & 15;
    float x[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      float s = i == c ? 1.f : 0.f;
#pragma unroll
      for (int k = 0; k < i; ++k) s = fmaf(-A[(b0 + i) * LS + b0 + k], x[k], s);
      x[i] = s;
      T[(b0 + i) * LS + b0 + c] = s;
    }
  }
  __syncthreads();
  float* tmp = A + 32;  // [32 x 32] at rows 0..31, columns 32..63
  {
    float s[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {  // pair h of 16-blocks: rows 32 h + 16 .. , columns 32 h ..
      const int i = tid >> 4, j = tid & 15, r0 = 32 * h + 16, c0 = 32 * h;
      s[h] = 0.f;
#pragma unroll
      for (int k = 0; k < 16; ++k) s[h] = fmaf(A[(r0 + i) * LS + c0 + k], T[(c0 + k) * LS + c0 + j], s[h]);
    }
    const int i = tid >> 4, j = tid & 15;
    tmp[i * LS + j] = s[0];
    tmp[(16 + i) * LS + j] = s[1];
  }
  __syncthreads();
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int i = tid >> 4, j = tid & 15, r0 = 32 * h + 16, c0 = 32 * h;
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < 16; ++k) s = fmaf(T[(r0 + i) * LS + r0 + k], tmp[(16 * h + k) * LS + j], s);
    T[(r0 + i) * LS + c0 + j] = -s;
  }
  __syncthreads();
  const int i = tid >> 3, j0 = (tid & 7) * 4;
  {
    float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
    for (int k = 0; k < 32; ++k) {
      const float a = A[(32 + i) * LS + k];
      const float4 t = ld4(T + k * LS + j0);
      s[0] = fmaf(a, t.x, s[0]); s[1] = fmaf(a, t.y, s[1]); s[2] = fmaf(a, t.z, s[2]); s[3] = fmaf(a, t.w, s[3]);
    }
    st4(tmp + i * LS + j0, s[0], s[1], s[2], s[3]);
  }
  __syncthreads();
  {
    float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
    for (int k = 0; k < 32; ++k) {
      const float a = T[(32 + i) * LS + 32 + k];
      const float4 t = ld4(tmp + k * LS + j0);
      s[0] = fmaf(-a, t.x, s[0]); s[1] = fmaf(-a, t.y, s[1]); s[2] = fmaf(-a, t.z, s[2]); s[3] = fmaf(-a, t.w, s[3]);
    }
    st4(T + (32 + i) * LS + j0, s[0], s[1], s[2], s[3]);
  }
  __syncthreads();
}

constexpr int CHUNK_FWD_SMEM = (2 * T64 + 2 * C * LS + 3 * C) * 4;

__global__ void __launch_bounds__(NT) gdr_chunk_fwd_kernel(const Args p) {
  extern __shared__ __align__(16) float sm[];
  float *K = sm, *X = K + T64, *A = X + T64, *T = A + C * LS, *gc = T + C * LS, *be = gc + C, *f = be + C;
  const Where x = where(p, blockIdx.x, blockIdx.y);
  const int tid = threadIdx.x, ti = tid >> 4, tj = tid & 15;
  if (tid < 32) {  // cumulative log gates of 64 positions: two per lane
    const int i0 = 2 * tid;
    const long long o = ((long long)x.b * p.S + x.s0) * p.H + x.h;
    const float g0 = i0 < x.rows ? p.g[o + (long long)i0 * p.H] : 0.f, g1 = i0 + 1 < x.rows ? p.g[o + (long long)(i0 + 1) * p.H] : 0.f;
    float run = g0 + g1;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const float y = __shfl_up_sync(0xffffffffu, run, d);
      if (tid >= d) run += y;
    }
    gc[i0 + 1] = run;
    gc[i0] = run - g1;
    be[i0] = i0 < x.rows ? p.beta[o + (long long)i0 * p.H] : 0.f;
    be[i0 + 1] = i0 + 1 < x.rows ? p.beta[o + (long long)(i0 + 1) * p.H] : 0.f;
    float* go = p.gc + ((long long)x.bh * p.N + x.n) * C;
    go[i0] = gc[i0];
    go[i0 + 1] = gc[i0 + 1];
  }
  load_bf16(K, p.k + x.b * p.k_b + x.s0 * p.k_s + x.h * p.k_h, p.k_s, x.rows, nullptr);
  load_bf16(X, p.q + x.b * p.q_b + x.s0 * p.q_s + x.h * p.q_h, p.q_s, x.rows, nullptr);
  __syncthreads();
  const long long sq = ((long long)x.bh * p.N + x.n) * C * C;
  {
    float kk[4][4], qk[4][4];
    zero(kk);
    zero(qk);
    mm_nt64(K, K, kk);
    mm_nt64(X, K, qk);
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int i = ti + 16 * r, j = tj + 16 * c;
        const float dec = j <= i ? exp_c(gc[i] - gc[j]) : 0.f;
        A[i * LS + j] = j < i ? be[i] * kk[r][c] * dec : 0.f;
        p.P[sq + i * C + j] = j <= i ? qk[r][c] * p.scale * dec : 0.f;
      }
  }
  if (tid < C) f[tid] = be[tid] * exp_c(gc[tid]);
  __syncthreads();
  unit_lower_inverse(A, T);
  for (int i = tid; i < C * (C / 4); i += NT)
    reinterpret_cast<float4*>(p.T + sq)[i] = ld4(T + (i >> 4) * LS + (i & 15) * 4);
  load_bf16(X, p.v + x.b * p.v_b + x.s0 * p.v_s + x.h * p.v_h, p.v_s, x.rows, be);
  for (int i = tid; i < C * (D / 4); i += NT) {
    const int r = i >> 5;
    float* kp = K + r * LD + (i & 31) * 4;
    const float4 a = ld4(kp);
    st4(kp, a.x * f[r], a.y * f[r], a.z * f[r], a.w * f[r]);
  }
  __syncthreads();
  const long long ch = ((long long)x.bh * p.N + x.n) * C * D;
  float acc[4][8];
  zero(acc);
  mm_nn<C, LS, LD>(T, X, acc);
  store_f32(p.u + ch, acc);
  zero(acc);
  mm_nn<C, LS, LD>(T, K, acc);
  store_f32(p.w + ch, acc);
}

// ---------------------------------------------------------------------------------------------- sequential, forward
constexpr int SCAN_FWD_SMEM = (2 * T64 + 2 * C * LV + D * LV + C * LV + 2 * C) * 4 + 2 * C * LK * 2;

__global__ void __launch_bounds__(NT) gdr_scan_fwd_kernel(const Args p) {
  extern __shared__ __align__(16) float sm[];
  float *W = sm, *U = W + 2 * T64, *S = U + 2 * C * LV, *V = S + D * LV, *G = V + C * LV;
  __nv_bfloat16* Kb = reinterpret_cast<__nv_bfloat16*>(G + 2 * C);
  const int bh = blockIdx.x, vs = blockIdx.y * VS, tid = threadIdx.x;
  const __nv_bfloat16* kh = p.k + (bh / p.H) * p.k_b + (bh % p.H) * p.k_h;
  auto fetch = [&](int n, int s) {
    const long long ch = ((long long)bh * p.N + n) * C * D;
    for (int i = tid; i < C * (D / 4); i += NT) cp16(W + s * T64 + (i >> 5) * LD + (i & 31) * 4, p.w + ch + i * 4, 16);
    for (int i = tid; i < C * (VS / 4); i += NT) cp16(U + s * C * LV + (i >> 3) * LV + (i & 7) * 4, p.u + ch + (i >> 3) * D + vs + (i & 7) * 4, 16);
    for (int i = tid; i < C * (D / 8); i += NT) {
      const int r = i >> 4, t = n * C + r;
      cp16(Kb + s * C * LK + r * LK + (i & 15) * 8, kh + (long long)min(t, p.S - 1) * p.k_s + (i & 15) * 8, t < p.S ? 16 : 0);
    }
    if (tid < C / 4) cp16(G + s * C + tid * 4, p.gc + ((long long)bh * p.N + n) * C + tid * 4, 16);
  };
  for (int i = tid; i < D * LV; i += NT) S[i] = 0.f;
  fetch(0, 0);
  cp_commit();
  const int r8 = tid >> 3, c4 = (tid & 7) * 4;  // v': rows r8, r8 + 32; state: rows 4 r8 .. 4 r8 + 3
  for (int n = 0; n < p.N; ++n) {
    const int s = n & 1;
    if (n + 1 < p.N) fetch(n + 1, s ^ 1);
    cp_commit();
    cp_wait<1>();
    __syncthreads();
    float* so = p.st + ((long long)bh * p.N + n) * D * D + vs;
    for (int i = tid; i < D * (VS / 4); i += NT)
      *reinterpret_cast<float4*>(so + (i >> 3) * D + (i & 7) * 4) = ld4(S + (i >> 3) * LV + (i & 7) * 4);
    const float* Ws = W + s * T64;
    f2 m0[2] = {0ull, 0ull}, m1[2] = {0ull, 0ull};
#pragma unroll 4
    for (int d = 0; d < D; d += 4) {
      const float4 x = ld4(Ws + r8 * LD + d), y = ld4(Ws + (r8 + 32) * LD + d);
      const float xa[4] = {x.x, x.y, x.z, x.w}, ya[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) fma4x2(xa[e], ya[e], ld2(S + (d + e) * LV + c4), m0, m1);
    }
    float a0[4], a1[4];
    f2_unpack(m0[0], a0[0], a0[1]); f2_unpack(m0[1], a0[2], a0[3]);
    f2_unpack(m1[0], a1[0], a1[1]); f2_unpack(m1[1], a1[2], a1[3]);
    const float* Gs = G + s * C;
    const float gl = Gs[C - 1], a = exp_c(gl);
    float* vo = p.vn + ((long long)bh * p.N + n) * C * D + vs + c4;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = r8 + 32 * h;
      const float4 u = ld4(U + s * C * LV + r * LV + c4);
      const float* m = h ? a1 : a0;
      const float4 v = make_float4(u.x - m[0], u.y - m[1], u.z - m[2], u.w - m[3]);
      *reinterpret_cast<float4*>(vo + r * D) = v;
      const float f = exp_c(gl - Gs[r]);
      st4(V + r * LV + c4, v.x * f, v.y * f, v.z * f, v.w * f);
    }
    __syncthreads();
    f2 acc[4][2];
    const __nv_bfloat16* Ks = Kb + s * C * LK + 4 * r8;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float4 t = ld4(S + (4 * r8 + e) * LV + c4);
      acc[e][0] = f2_pack(a * t.x, a * t.y);
      acc[e][1] = f2_pack(a * t.z, a * t.w);
    }
#pragma unroll 8
    for (int j = 0; j < C; ++j) {
      const float4 k = bf4(*reinterpret_cast<const uint2*>(Ks + j * LK));
      const Pair2 v = ld2(V + j * LV + c4);
      fma4x2(k.x, k.y, v, acc[0], acc[1]);
      fma4x2(k.z, k.w, v, acc[2], acc[3]);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) *reinterpret_cast<ulonglong2*>(S + (4 * r8 + e) * LV + c4) = make_ulonglong2(acc[e][0], acc[e][1]);
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------------------------- outputs
// o = (e^b qs) S + P v' for 64 of the 128 value columns: rows ti + 16 r, columns 4 tj + e of the half.
constexpr int LH = 68;  // pitch of the half-width tiles
constexpr int OUT_SMEM = (T64 + C * LS + D * LH + C * LH + C) * 4;

__global__ void __launch_bounds__(NT) gdr_out_kernel(const Args p) {
  extern __shared__ __align__(16) float sm[];
  float *Q = sm, *P = Q + T64, *S = P + C * LS, *V = S + D * LH, *f = V + C * LH;
  const Where x = where(p, blockIdx.x, blockIdx.y);
  const int tid = threadIdx.x, ti = tid >> 4, tj = tid & 15, v0 = blockIdx.z * 64;
  const long long id = (long long)x.bh * p.N + x.n;
#pragma unroll
  for (int it = 0; it < D * 16 / NT; ++it) {
    const int i = tid + it * NT;
    cp16(S + (i >> 4) * LH + (i & 15) * 4, p.st + id * D * D + (i >> 4) * D + v0 + (i & 15) * 4, 16);
  }
#pragma unroll
  for (int it = 0; it < C * 16 / NT; ++it) {
    const int i = tid + it * NT;
    cp16(V + (i >> 4) * LH + (i & 15) * 4, p.vn + id * C * D + (i >> 4) * D + v0 + (i & 15) * 4, 16);
  }
  load_sq(P, p.P + id * C * C);
  cp_commit();
  if (tid < C) f[tid] = p.scale * exp_c(p.gc[id * C + tid]);
  __syncthreads();
  load_bf16(Q, p.q + x.b * p.q_b + x.s0 * p.q_s + x.h * p.q_h, p.q_s, x.rows, f);
  cp_wait<0>();
  __syncthreads();
  f2 s2[4][2];
#pragma unroll
  for (int r = 0; r < 4; ++r) s2[r][0] = s2[r][1] = 0ull;
  auto product = [&](const float* A, int la, const float* B, int K) {
#pragma unroll 2
    for (int j = 0; j < K; j += 4) {
      float4 a[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) a[r] = ld4(A + (ti + 16 * r) * la + j);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const Pair2 b = ld2(B + (j + e) * LH + 4 * tj);
#pragma unroll
        for (int r = 0; r < 4; r += 2) {
          const float y = e == 0 ? a[r].x : e == 1 ? a[r].y : e == 2 ? a[r].z : a[r].w;
          const float z = e == 0 ? a[r + 1].x : e == 1 ? a[r + 1].y : e == 2 ? a[r + 1].z : a[r + 1].w;
          fma4x2(y, z, b, s2[r], s2[r + 1]);
        }
      }
    }
  };
  product(Q, LD, S, D);
  product(P, LS, V, C);
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int i = ti + 16 * r;
    float o[4];
    f2_unpack(s2[r][0], o[0], o[1]);
    f2_unpack(s2[r][1], o[2], o[3]);
    if (i < x.rows)
      *reinterpret_cast<uint2*>(p.o + (((long long)x.b * p.S + x.s0 + i) * p.H + x.h) * D + v0 + 4 * tj) = pack4(o[0], o[1], o[2], o[3]);
  }
}

// ---------------------------------------------------------------------------------------------- backward
constexpr int DVP_SMEM = (T64 + C * LS) * 4;

__global__ void __launch_bounds__(NT) gdr_dvp_kernel(const Args p) {
  extern __shared__ __align__(16) float sm[];
  float *X = sm, *P = X + T64;
  const Where x = where(p, blockIdx.x, blockIdx.y);
  const long long id = (long long)x.bh * p.N + x.n;
  load_sq(P, p.P + id * C * C);
  cp_commit();
  load_bf16(X, p.d_o + (((long long)x.b * p.S + x.s0) * p.H + x.h) * D, (long long)p.H * D, x.rows, nullptr);
  cp_wait<0>();
  __syncthreads();
  float acc[4][8];
  zero(acc);
  mm_tn(P, X, acc);
  store_f32(p.dvn + id * C * D, acc);
}

// dv' = P^T do + (e^{b_last - b} k) dS;  dS <- e^{b_last} dS + (e^b qs)^T do - w^T dv'
constexpr int SCAN_BWD_SMEM = (2 * T64 + 2 * C * LV + D * LV + 2 * C * LV + 2 * C) * 4 + 4 * C * LK * 2 + 2 * C * VS * 2;

__global__ void __launch_bounds__(NT) gdr_scan_bwd_kernel(const Args p) {
  extern __shared__ __align__(16) float sm[];
  float *W = sm, *U = W + 2 * T64, *S = U + 2 * C * LV, *V = S + D * LV, *O = V + C * LV, *G = O + C * LV;
  __nv_bfloat16 *Kb = reinterpret_cast<__nv_bfloat16*>(G + 2 * C), *Qb = Kb + 2 * C * LK, *Ob = Qb + 2 * C * LK;
  const int bh = blockIdx.x, vs = blockIdx.y * VS, tid = threadIdx.x, b = bh / p.H, h = bh % p.H;
  const __nv_bfloat16 *kh = p.k + b * p.k_b + h * p.k_h, *qh = p.q + b * p.q_b + h * p.q_h;
  const __nv_bfloat16* oh = p.d_o + ((long long)b * p.S * p.H + h) * D + vs;
  auto fetch = [&](int n, int s) {
    const long long ch = ((long long)bh * p.N + n) * C * D;
    for (int i = tid; i < C * (D / 4); i += NT) cp16(W + s * T64 + (i >> 5) * LD + (i & 31) * 4, p.w + ch + i * 4, 16);
    for (int i = tid; i < C * (VS / 4); i += NT) cp16(U + s * C * LV + (i >> 3) * LV + (i & 7) * 4, p.dvn + ch + (i >> 3) * D + vs + (i & 7) * 4, 16);
    for (int i = tid; i < C * (D / 8); i += NT) {
      const int r = i >> 4, t = n * C + r, z = t < p.S ? 16 : 0;
      const long long tc = min(t, p.S - 1);
      cp16(Kb + s * C * LK + r * LK + (i & 15) * 8, kh + tc * p.k_s + (i & 15) * 8, z);
      cp16(Qb + s * C * LK + r * LK + (i & 15) * 8, qh + tc * p.q_s + (i & 15) * 8, z);
    }
    for (int i = tid; i < C * (VS / 8); i += NT) {
      const int r = i >> 2, t = n * C + r;
      cp16(Ob + s * C * VS + r * VS + (i & 3) * 8, oh + (long long)min(t, p.S - 1) * p.H * D + (i & 3) * 8, t < p.S ? 16 : 0);
    }
    if (tid < C / 4) cp16(G + s * C + tid * 4, p.gc + ((long long)bh * p.N + n) * C + tid * 4, 16);
  };
  for (int i = tid; i < D * LV; i += NT) S[i] = 0.f;
  fetch(p.N - 1, 0);
  cp_commit();
  const int r8 = tid >> 3, c4 = (tid & 7) * 4;
  for (int m = 0; m < p.N; ++m) {
    const int n = p.N - 1 - m, s = m & 1;
    if (m + 1 < p.N) fetch(n - 1, s ^ 1);
    cp_commit();
    cp_wait<1>();
    __syncthreads();
    float* so = p.dst + ((long long)bh * p.N + n) * D * D + vs;
    for (int i = tid; i < D * (VS / 4); i += NT)
      *reinterpret_cast<float4*>(so + (i >> 3) * D + (i & 7) * 4) = ld4(S + (i >> 3) * LV + (i & 7) * 4);
    const float* Gs = G + s * C;
    const float gl = Gs[C - 1], a = exp_c(gl);
    f2 m0[2] = {0ull, 0ull}, m1[2] = {0ull, 0ull};
    const __nv_bfloat16* Ks = Kb + s * C * LK;
#pragma unroll 4
    for (int d = 0; d < D; d += 4) {
      const float4 x = bf4(*reinterpret_cast<const uint2*>(Ks + r8 * LK + d)), y = bf4(*reinterpret_cast<const uint2*>(Ks + (r8 + 32) * LK + d));
      const float xa[4] = {x.x, x.y, x.z, x.w}, ya[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) fma4x2(xa[e], ya[e], ld2(S + (d + e) * LV + c4), m0, m1);
    }
    float a0[4], a1[4];
    f2_unpack(m0[0], a0[0], a0[1]); f2_unpack(m0[1], a0[2], a0[3]);
    f2_unpack(m1[0], a1[0], a1[1]); f2_unpack(m1[1], a1[2], a1[3]);
    float* vo = p.dvn + ((long long)bh * p.N + n) * C * D + vs + c4;
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
      const int r = r8 + 32 * hh;
      const float4 u = ld4(U + s * C * LV + r * LV + c4);
      const float* mm = hh ? a1 : a0;
      const float f = exp_c(gl - Gs[r]);
      const float4 v = make_float4(fmaf(f, mm[0], u.x), fmaf(f, mm[1], u.y), fmaf(f, mm[2], u.z), fmaf(f, mm[3], u.w));
      *reinterpret_cast<float4*>(vo + r * D) = v;
      st4(V + r * LV + c4, -v.x, -v.y, -v.z, -v.w);
      const float q = p.scale * exp_c(Gs[r]);
      const float4 o = bf4(*reinterpret_cast<const uint2*>(Ob + s * C * VS + r * VS + c4));
      st4(O + r * LV + c4, o.x * q, o.y * q, o.z * q, o.w * q);
    }
    __syncthreads();
    f2 acc[4][2];
    const __nv_bfloat16* Qs = Qb + s * C * LK + 4 * r8;
    const float* Ws = W + s * T64 + 4 * r8;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float4 t = ld4(S + (4 * r8 + e) * LV + c4);
      acc[e][0] = f2_pack(a * t.x, a * t.y);
      acc[e][1] = f2_pack(a * t.z, a * t.w);
    }
#pragma unroll 4
    for (int j = 0; j < C; ++j) {
      const float4 k = bf4(*reinterpret_cast<const uint2*>(Qs + j * LK)), w = ld4(Ws + j * LD);
      const Pair2 o = ld2(O + j * LV + c4), v = ld2(V + j * LV + c4);
      fma4x2(k.x, k.y, o, acc[0], acc[1]);
      fma4x2(k.z, k.w, o, acc[2], acc[3]);
      fma4x2(w.x, w.y, v, acc[0], acc[1]);
      fma4x2(w.z, w.w, v, acc[2], acc[3]);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) *reinterpret_cast<ulonglong2*>(S + (4 * r8 + e) * LV + c4) = make_ulonglong2(acc[e][0], acc[e][1]);
    __syncthreads();
  }
}

constexpr int CHUNK_BWD_SMEM = (4 * T64 + D * LD + 16 * C + 6 * C + 32) * 4;

__global__ void __launch_bounds__(NT, 1) gdr_chunk_bwd_kernel(const Args p) {
  extern __shared__ __align__(16) float sm[];
  float *X = sm, *Y = X + T64, *Z = Y + T64, *W = Z + T64, *St = W + T64;
  float *red = St + D * LD, *gc = red + 16 * C, *be = gc + C, *dgr = be + C, *dgcol = dgr + C, *dbe = dgcol + C, *eg = dbe + C, *wred = eg + C;
  float *K = St, *Q = St + T64;  // after the state products
  const Where x = where(p, blockIdx.x, blockIdx.y);
  const int tid = threadIdx.x, ti = tid >> 4, tj = tid & 15;
  const long long id = (long long)x.bh * p.N + x.n;
  const __nv_bfloat16 *kp = p.k + x.b * p.k_b + x.s0 * p.k_s + x.h * p.k_h, *qp = p.q + x.b * p.q_b + x.s0 * p.q_s + x.h * p.q_h;
  const __nv_bfloat16* vp = p.v + x.b * p.v_b + x.s0 * p.v_s + x.h * p.v_h;
  const long long row0 = ((long long)x.b * p.S + x.s0) * p.H + x.h;  // (position, head) index of row 0; rows are H apart
#pragma unroll
  for (int it = 0; it < D * (D / 4) / NT; ++it) {
    const int i = tid + it * NT;
    cp16(St + state_row(i >> 5) * LD + (i & 31) * 4, p.st + id * D * D + i * 4, 16);
  }
  load_f32(Y, p.dvn + id * C * D);
  cp_commit();
  load_f32(Z, p.vn + id * C * D);  // first read after the next barrier but one
  cp_commit();
  if (tid < C) {
    gc[tid] = p.gc[id * C + tid];
    be[tid] = tid < x.rows ? p.beta[row0 + (long long)tid * p.H] : 0.f;
    eg[tid] = exp_c(gc[tid]);
  }
  load_bf16(X, p.d_o + row0 * D, (long long)p.H * D, x.rows, nullptr);
  cp_wait<1>();
  __syncthreads();
  const float gl = gc[C - 1];
  // my 4 rows x 8 columns of q, k or v in bf16 (zero past the sequence): fetched before a product, read after it
  auto fetch8 = [&](const __nv_bfloat16* base, long long pitch, uint2 (&o)[4][2]) {
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int i = ti + 16 * r;
      o[r][0] = o[r][1] = make_uint2(0u, 0u);
      if (i < x.rows) {
        o[r][0] = *reinterpret_cast<const uint2*>(base + i * pitch + 4 * tj);
        o[r][1] = *reinterpret_cast<const uint2*>(base + i * pitch + 4 * tj + 64);
      }
    }
  };
  auto row8 = [&](const uint2 (&raw)[2], float (&o)[8]) {
    const float4 a = bf4(raw[0]), c = bf4(raw[1]);
    o[0] = a.x; o[1] = a.y; o[2] = a.z; o[3] = a.w; o[4] = c.x; o[5] = c.y; o[6] = c.z; o[7] = c.w;
  };
  uint2 raw[4][2], raw2[4][2];
  float dq[4][8], dk[4][8], acc[4][8];
  float db_row[4] = {0.f, 0.f, 0.f, 0.f}, dbeta_row[4] = {0.f, 0.f, 0.f, 0.f};  // gradients of b_i and beta_i, rows ti + 16 r
  float dlast = 0.f;                                                            // my share of the gradient of b_last

  // dq from the state: (do S^T) e^b scale;  dw = -dv' S^T
  fetch8(qp, p.q_s, raw);
  zero(dq);
  mm_nt128(X, St, dq);
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int i = ti + 16 * r;
    float t[8], s = 0.f;
    row8(raw[r], t);
    const float f = p.scale * eg[i];
#pragma unroll
    for (int c = 0; c < 8; ++c) { dq[r][c] *= f; s = fmaf(dq[r][c], t[c], s); }
    db_row[r] += row_sum(s);
  }
  zero(acc);
  mm_nt128(Y, St, acc);
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 8; ++c) acc[r][c] = -acc[r][c];
  store_tile(W, acc);
  __syncthreads();
  // the exit-state gradient takes the state's place; <dS, S> on the way: d e^{b_last}
  {
    float s = 0.f;
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
      constexpr int IT = D * (D / 4) / NT / 2;
      float4 g[IT];
#pragma unroll
      for (int it = 0; it < IT; ++it) g[it] = reinterpret_cast<const float4*>(p.dst + id * D * D)[tid + (it + h * IT) * NT];
#pragma unroll
      for (int it = 0; it < IT; ++it) {
        const int i = tid + (it + h * IT) * NT;
        float* q4 = St + state_row(i >> 5) * LD + (i & 31) * 4;
        const float4 a = ld4(q4);
        s = fmaf(a.x, g[it].x, s); s = fmaf(a.y, g[it].y, s); s = fmaf(a.z, g[it].z, s); s = fmaf(a.w, g[it].w, s);
        *reinterpret_cast<float4*>(q4) = g[it];
      }
    }
    dlast = s * exp_c(gl);
  }
  fetch8(kp, p.k_s, raw);
  cp_wait<0>();  // v'
  __syncthreads();
  // dk from the state update: (v' dS^T) e^{b_last - b}
  zero(dk);
  mm_nt128(Z, St, dk);
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int i = ti + 16 * r;
    float t[8], s = 0.f;
    row8(raw[r], t);
    const float f = exp_c(gl - gc[i]);
#pragma unroll
    for (int c = 0; c < 8; ++c) { dk[r][c] *= f; s = fmaf(dk[r][c], t[c], s); }
    dlast += s;
    db_row[r] -= row_sum(s);
  }
  __syncthreads();  // St is free
  load_bf16(K, kp, p.k_s, x.rows, nullptr);
  load_bf16(Q, qp, p.q_s, x.rows, nullptr);
  // dP = lower(do v'^T); b_i and b_j through D_ij; E = dP D
  float e4[4][4], col[4], pij[4][4];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) pij[r][c] = p.P[id * C * C + (ti + 16 * r) * C + tj + 16 * c];
  zero(e4);
  mm_nt64(X, Z, e4);
#pragma unroll
  for (int c = 0; c < 4; ++c) col[c] = 0.f;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int i = ti + 16 * r;
    float s = 0.f;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int j = tj + 16 * c;
      const float t = j <= i ? e4[r][c] * pij[r][c] : 0.f;
      s += t;
      col[c] += t;
      e4[r][c] = j <= i ? e4[r][c] * exp_c(gc[i] - gc[j]) * p.scale : 0.f;
    }
    db_row[r] += row_sum(s);
  }
  __syncthreads();  // X and Z have been read; K and Q are complete
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) X[(ti + 16 * r) * LS + tj + 16 * c] = e4[r][c];
  load_sq(Z, p.T + id * C * C);  // first read after these two products
  cp_commit();
  __syncthreads();
  mm_nn<C, LS, LD>(X, K, dq);
  mm_tn(X, Q, dk);
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int i = ti + 16 * r;
    if (i < x.rows) store_bf16_row(p.dq + (row0 + (long long)i * p.H) * D, dq[r]);
  }
  // through T: dRv = T^T dv', dRk = T^T dw
  fetch8(vp, p.v_s, raw2);  // raw still holds my rows of k
  cp_wait<0>();
  __syncthreads();
  zero(acc);
  mm_tn(Z, Y, acc);
  zero(dq);
  mm_tn(Z, W, dq);  // dq's registers hold dRk from here
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int i = ti + 16 * r;
    float t[8], s = 0.f, o[8];
    row8(raw2[r], t);
#pragma unroll
    for (int c = 0; c < 8; ++c) { s = fmaf(acc[r][c], t[c], s); o[c] = be[i] * acc[r][c]; }
    if (i < x.rows) store_bf16_row(p.dv + (row0 + (long long)i * p.H) * D, o);
    row8(raw[r], t);
    float sk = 0.f;
    const float f = be[i] * eg[i];
#pragma unroll
    for (int c = 0; c < 8; ++c) { sk = fmaf(dq[r][c], t[c], sk); dk[r][c] = fmaf(f, dq[r][c], dk[r][c]); }
    sk = row_sum(sk);
    dbeta_row[r] += row_sum(s) + eg[i] * sk;
    db_row[r] += f * sk;
  }
  __syncthreads();  // X, Z, Y, W have been read
  load_f32(Y, p.u + id * C * D);
  load_f32(W, p.w + id * C * D);
  cp_commit();
  store_tile(X, acc);
  store_tile(Z, dq);
  // dA = -strict_lower(dRv u^T + dRk w^T); A = beta_i kk D
  float kk[4][4];
  zero(kk);
  mm_nt64(K, K, kk);  // under the fetch of u and w
  cp_wait<0>();
  __syncthreads();
  zero(e4);
  mm_nt64(X, Y, e4);
  mm_nt64(Z, W, e4);
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int i = ti + 16 * r;
    float s = 0.f;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int j = tj + 16 * c;
      const float dec = j < i ? exp_c(gc[i] - gc[j]) : 0.f;
      const float t = -e4[r][c] * kk[r][c] * dec;  // d beta_i
      s += t;
      col[c] += be[i] * t;
      e4[r][c] = j < i ? -e4[r][c] * be[i] * dec : 0.f;
    }
    s = row_sum(s);
    dbeta_row[r] += s;
    db_row[r] += be[i] * s;
  }
  __syncthreads();  // X has been read
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) X[(ti + 16 * r) * LS + tj + 16 * c] = e4[r][c];
#pragma unroll
  for (int c = 0; c < 4; ++c) red[ti * C + tj + 16 * c] = col[c];
  if (tj == 0) {
#pragma unroll
    for (int r = 0; r < 4; ++r) { dgr[ti + 16 * r] = db_row[r]; dbe[ti + 16 * r] = dbeta_row[r]; }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) dlast += __shfl_xor_sync(0xffffffffu, dlast, o);
  if ((tid & 31) == 0) wred[tid >> 5] = dlast;
  __syncthreads();
  mm_nn<C, LS, LD>(X, K, dk);
  mm_tn(X, K, dk);
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int i = ti + 16 * r;
    if (i < x.rows) store_bf16_row(p.dk + (row0 + (long long)i * p.H) * D, dk[r]);
  }
  if (tid < C) {
    float s = 0.f;
    for (int t = 0; t < 16; ++t) s += red[t * C + tid];
    dgcol[tid] = s;
  }
  __syncthreads();
  if (tid < 32) {  // dg_t = sum_{i >= t} db_i: two positions per lane, suffix sums
    float last = 0.f;
#pragma unroll
    for (int i = 0; i < NT / 32; ++i) last += wred[i];
    const int i0 = 2 * tid;
    const float b0 = dgr[i0] - dgcol[i0], b1 = dgr[i0 + 1] - dgcol[i0 + 1] + (tid == 31 ? last : 0.f);
    float run = b0 + b1;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const float y = __shfl_down_sync(0xffffffffu, run, d);
      if (tid + d < 32) run += y;
    }
    if (i0 < x.rows) {
      p.dg[row0 + (long long)i0 * p.H] = run;
      p.dbeta[row0 + (long long)i0 * p.H] = dbe[i0];
    }
    if (i0 + 1 < x.rows) {
      p.dg[row0 + (long long)(i0 + 1) * p.H] = run - b0;
      p.dbeta[row0 + (long long)(i0 + 1) * p.H] = dbe[i0 + 1];
    }
  }
}

template <typename F>
bool allow_smem(F f, int bytes) {
  return cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess;
}

}  // namespace gdr
}  // namespace pt

using namespace pt;

// q, k, v: bf16 [B, S, H, 128] with element strides (batch, position, head), multiples of 8, bases 16-byte aligned; g, beta fp32
// [B, S, H] contiguous; o bf16 [B, S, H, 128]. N = ceil(S / 64). Kept for the backward: gc [B*H, N, 64], P and T
// [B*H, N, 64, 64], u, w, vn [B*H, N, 64, 128], st [B*H, N, 128, 128], all fp32.
PT_API int pt_gdr_fwd(const void* q, const void* k, const void* v, const long long* strides, const float* g, const float* beta, float* gc,
                      float* P, float* T, float* u, float* w, float* vn, float* st, void* o, int B, int S, int H, float scale,
                      void* stream_) {
  using namespace pt::gdr;
  if (B <= 0 || S <= 0 || H <= 0 || (long long)B * H > 65535) return -2;
  Args a{};
  a.q = static_cast<const __nv_bfloat16*>(q); a.k = static_cast<const __nv_bfloat16*>(k); a.v = static_cast<const __nv_bfloat16*>(v);
  a.q_b = strides[0]; a.q_s = strides[1]; a.q_h = strides[2];
  a.k_b = strides[3]; a.k_s = strides[4]; a.k_h = strides[5];
  a.v_b = strides[6]; a.v_s = strides[7]; a.v_h = strides[8];
  a.g = g; a.beta = beta; a.gc = gc; a.P = P; a.T = T; a.u = u; a.w = w; a.vn = vn; a.st = st;
  a.o = static_cast<__nv_bfloat16*>(o);
  a.B = B; a.S = S; a.H = H; a.N = (S + C - 1) / C; a.scale = scale;
  cudaStream_t s = static_cast<cudaStream_t>(stream_);
  if (!allow_smem(gdr_chunk_fwd_kernel, CHUNK_FWD_SMEM) || !allow_smem(gdr_scan_fwd_kernel, SCAN_FWD_SMEM) ||
      !allow_smem(gdr_out_kernel, OUT_SMEM))
    return -4;
  gdr_chunk_fwd_kernel<<<dim3(a.N, B * H), NT, CHUNK_FWD_SMEM, s>>>(a);
  gdr_scan_fwd_kernel<<<dim3(B * H, D / VS), NT, SCAN_FWD_SMEM, s>>>(a);
  gdr_out_kernel<<<dim3(a.N, B * H, 2), NT, OUT_SMEM, s>>>(a);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

// Gradients of pt_gdr_fwd: d_o bf16 [B, S, H, 128] contiguous; dvn [B*H, N, 64, 128] and dst [B*H, N, 128, 128] are fp32 scratch;
// dq, dk, dv bf16 [B, S, H, 128], dg, dbeta fp32 [B, S, H] are written.
PT_API int pt_gdr_bwd(const void* q, const void* k, const void* v, const long long* strides, const float* beta, const float* gc, const float* P,
                      const float* T, const float* u, const float* w, const float* vn, const float* st, const void* d_o, float* dvn,
                      float* dst, void* dq, void* dk, void* dv, float* dg, float* dbeta, int B, int S, int H, float scale, void* stream_) {
  using namespace pt::gdr;
  if (B <= 0 || S <= 0 || H <= 0 || (long long)B * H > 65535) return -2;
  Args a{};
  a.q = static_cast<const __nv_bfloat16*>(q); a.k = static_cast<const __nv_bfloat16*>(k); a.v = static_cast<const __nv_bfloat16*>(v);
  a.q_b = strides[0]; a.q_s = strides[1]; a.q_h = strides[2];
  a.k_b = strides[3]; a.k_s = strides[4]; a.k_h = strides[5];
  a.v_b = strides[6]; a.v_s = strides[7]; a.v_h = strides[8];
  a.beta = beta; a.gc = const_cast<float*>(gc); a.P = const_cast<float*>(P); a.T = const_cast<float*>(T);
  a.u = const_cast<float*>(u); a.w = const_cast<float*>(w); a.vn = const_cast<float*>(vn); a.st = const_cast<float*>(st);
  a.d_o = static_cast<const __nv_bfloat16*>(d_o); a.dvn = dvn; a.dst = dst;
  a.dq = static_cast<__nv_bfloat16*>(dq); a.dk = static_cast<__nv_bfloat16*>(dk); a.dv = static_cast<__nv_bfloat16*>(dv);
  a.dg = dg; a.dbeta = dbeta;
  a.B = B; a.S = S; a.H = H; a.N = (S + C - 1) / C; a.scale = scale;
  cudaStream_t s = static_cast<cudaStream_t>(stream_);
  if (!allow_smem(gdr_dvp_kernel, DVP_SMEM) || !allow_smem(gdr_scan_bwd_kernel, SCAN_BWD_SMEM) || !allow_smem(gdr_chunk_bwd_kernel, CHUNK_BWD_SMEM))
    return -4;
  gdr_dvp_kernel<<<dim3(a.N, B * H), NT, DVP_SMEM, s>>>(a);
  gdr_scan_bwd_kernel<<<dim3(B * H, D / VS), NT, SCAN_BWD_SMEM, s>>>(a);
  gdr_chunk_bwd_kernel<<<dim3(a.N, B * H), NT, CHUNK_BWD_SMEM, s>>>(a);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}
