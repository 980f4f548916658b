// Fused cross-entropy over bf16 logits: per-row online softmax, per-token loss, and the logits are
// overwritten in place by d loss / d logits = softmax - onehot (zero for ignored rows), so the
// [tokens, vocab] matrix is materialised exactly once. Same contract as the reference's Triton
// kernel (pithtrain/operators/cross_entropy.py:15-125).
#include "elementwise.cuh"
#include "host_common.h"
#include "ptx.cuh"

namespace pt {

// Exponentials are 2^((v - max) log2(e) - c), two of them in two packed instructions and one each of the special function unit, so
// that the two passes over a row (39 M logits: 17 us of that unit) fit beside its read and write. c is 0 in the sum and log2(sum)
// in the gradient. The maximum is taken off first: v log2(e) - max log2(e) costs as much, but the second product overflows for
// the lowest bf16 value, a common mask, and from 1e9 on is rounded by whole numbers.
constexpr float LOG2E = 1.4426950408889634f;

__device__ __forceinline__ float max8(const uint4& v) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
  const __nv_bfloat162 a = __hmax2(__hmax2(h[0], h[1]), __hmax2(h[2], h[3]));
  return fmaxf(__low2float(a), __high2float(a));
}
// What is subtracted for the maximum m: of minus infinities alone (a masked stretch), a finite number below every other logit.
__device__ __forceinline__ float below(float m) { return fmaxf(m, -3.4028234e38f); }
__device__ __forceinline__ float exp1(float v, float m, float c) { return ex2_approx(fmaf(v - m, LOG2E, -c)); }
template <bool C>  // without c: it is 0
__device__ __forceinline__ void exp8(const uint4& v, float m, float c, float (&e)[8]) {
  const uint32_t q[4] = {v.x, v.y, v.z, v.w};
  const uint64_t m2 = f2_pack(-m, -m), c2 = f2_pack(-c, -c), log2e2 = f2_pack(LOG2E, LOG2E);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 p = unpack_bf16x2(q[i]);
    const uint64_t d = f2_add(f2_pack(p.x, p.y), m2);
    float a, b;
    f2_unpack(C ? f2_fma(d, log2e2, c2) : f2_mul(d, log2e2), a, b);
    e[2 * i] = ex2_approx(a);
    e[2 * i + 1] = ex2_approx(b);
  }
}
__device__ __forceinline__ void minus_one_at(float (&e)[8], int c, long long label) {
  if (c != label >> 3) return;
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if (i == (label & 7)) e[i] -= 1.f;
}
// Stops the compiler from carrying a vector's fp32 form from one pass to the next.
__device__ __forceinline__ void keep_packed(uint4& v) { asm volatile("" : "+r"(v.x), "+r"(v.y), "+r"(v.z), "+r"(v.w)); }

// A block of T threads to a row. NV > 0: the row is held in registers, NV vectors of 8 columns a thread. NV = 0: it is read
// twice, the first time with a running maximum. The reductions of a row leave its warps idle, so small blocks beat wide ones as
// long as all rows of an SM have 1536 threads or more; with 8 vectors a thread (55 us for 9496 columns, 150 for 32000) they have
// too few, and a ring of rows in shared memory (50 us) pays for its waits.
template <int T, int NV>
__global__ void __launch_bounds__(T, (NV > 2 ? 1536 : 2048) / T)
cross_entropy_kernel(__nv_bfloat16* __restrict__ logits, const long long* __restrict__ labels, float* __restrict__ loss, int V,
                     long long ld, int ignore_index) {
  __shared__ float red[32];
  const int row = blockIdx.x, tid = threadIdx.x, nvec = V / 8;
  __nv_bfloat16* x = logits + (size_t)row * ld;
  uint4* xv = reinterpret_cast<uint4*>(x);
  const long long label = labels[row];
  const int rest = nvec * 8 + tid;  // a column past the last whole vector, in the first V % 8 threads
  if (label == ignore_index) {
    for (int c = tid; c < nvec; c += T) xv[c] = make_uint4(0, 0, 0, 0);
    if (rest < V) x[rest] = __float2bfloat16(0.f);
    if (tid == 0) loss[row] = 0.f;
    return;
  }
  const float last = rest < V ? __bfloat162float(x[rest]) : -INFINITY;
  const float xl = tid == 0 ? __bfloat162float(x[label]) : 0.f;
  uint4 raw[NV > 0 ? NV : 1];
  float m = last, s = 0.f, gm;  // gm: maximum of the row, later what is subtracted for it
  if (NV > 0) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c = tid + i * T;
      raw[i] = c < nvec ? xv[c] : make_uint4(0xff80ff80u, 0xff80ff80u, 0xff80ff80u, 0xff80ff80u);  // -inf
    }
#pragma unroll
    for (int i = 0; i < NV; ++i) m = fmaxf(m, max8(raw[i]));
    gm = below(block_max(m, red));
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      keep_packed(raw[i]);
      float e[8];
      exp8<false>(raw[i], gm, 0.f, e);
      s += ((e[0] + e[1]) + (e[2] + e[3])) + ((e[4] + e[5]) + (e[6] + e[7]));
    }
  } else {
    m = below(m);
#pragma unroll 4
    for (int c = tid; c < nvec; c += T) {
      const uint4 v = xv[c];
      const float up = fmaxf(m, max8(v));
      float e[8];
      exp8<false>(v, up, 0.f, e);
      s = s * exp1(m, up, 0.f) + (((e[0] + e[1]) + (e[2] + e[3])) + ((e[4] + e[5]) + (e[6] + e[7])));
      m = up;
    }
    gm = block_max(m, red);
    s *= exp1(m, gm, 0.f);
  }
  s += exp1(last, gm, 0.f);
  const float gs = block_sum(s, red);
  // x[label] was read ahead of the barriers above, it is written after them. The logarithm of the loss is taken in 64 bits: the fast one
  // is off by 3e-7 on average.
  const float log2_sum = __log2f(gs);
  auto gradient = [&](const uint4& v, int c) {
    float e[8];
    exp8<true>(v, gm, log2_sum, e);
    minus_one_at(e, c, label);
    store8(x + c * 8, e);
  };
  if (NV > 0) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      keep_packed(raw[i]);
      if (tid + i * T < nvec) gradient(raw[i], tid + i * T);
    }
  } else {
#pragma unroll 4
    for (int c = tid; c < nvec; c += T) gradient(xv[c], c);
  }
  if (rest < V) x[rest] = __float2bfloat16(exp1(last, gm, log2_sum) - (rest == label ? 1.f : 0.f));
  if (tid == 0) loss[row] = (float)((double)gm - xl + log((double)gs));
}

// x *= s[0] over a flat bf16 buffer (s on the device).
__global__ void scale_bf16_kernel(__nv_bfloat16* __restrict__ x, const float* __restrict__ s, long long nvec) {
  const float sc = *s;
  if (sc == 1.f) return;  // a summed loss: nothing to change
  for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < nvec; v += (long long)gridDim.x * blockDim.x) {
    float f[8];
    load8(x + v * 8, f);
#pragma unroll
    for (int e = 0; e < 8; ++e) f[e] *= sc;
    store8(x + v * 8, f);
  }
}

}  // namespace pt

using namespace pt;

PT_API int pt_cross_entropy(void* logits, const long long* labels, float* loss, int n, int V,
                            long long ld, int ignore_index, void* stream_) {
  cudaStream_t st = (cudaStream_t)stream_;
  if (n <= 0) return 0;
  if (ld % 8 != 0) return -1;
  auto launch = [&](auto kernel, int threads) {
    kernel<<<n, threads, 0, st>>>((__nv_bfloat16*)logits, labels, loss, V, ld, ignore_index);
    return (int)cudaGetLastError();
  };
  // Cold cache, us, before (1024 threads and two reads for every row) -> now, and one read and one write at 6.5 TB/s. 4096 rows:
  // 1000 columns 37 -> 12 (3), 4096: 44 -> 18 (10), 8192: 53 -> 31 (21), 9496: 61 -> 42 (24), 12288: 63 -> 45 (31), 15520: 74 -> 59 (39).
  // 2048 rows: 20000 columns 46 -> 37 (25), 32000: 60 -> 51 (40), 50304: 87 -> 86 (63), 151936: 265 -> 252 (192); the last four read
  // their rows twice, up to 32768 columns by 512 threads (by 1024: 47 and 57 us) where there are more rows than SMs.
  const int nvec = V / 8;
  if (nvec <= 128 * 2) return launch(cross_entropy_kernel<128, 2>, 128);
  if (nvec <= 128 * 4) return launch(cross_entropy_kernel<128, 4>, 128);
  if (nvec <= 256 * 4) return launch(cross_entropy_kernel<256, 4>, 256);
  if (nvec <= 512 * 3) return launch(cross_entropy_kernel<512, 3>, 512);
  if (nvec <= 512 * 4) return launch(cross_entropy_kernel<512, 4>, 512);
  // A row alone on its SM wants all the loads it can have on their way: 32000 columns, 1 to 148 rows, 512 / 1024 threads 12.3 / 10.2.
  if (nvec <= 4096 && n > sm_count()) return launch(cross_entropy_kernel<512, 0>, 512);
  return launch(cross_entropy_kernel<1024, 0>, 1024);
}

PT_API int pt_scale_bf16(void* x, const float* s, long long numel, void* stream_) {
  cudaStream_t st = (cudaStream_t)stream_;
  if (numel <= 0) return 0;
  if (numel % 8 != 0) return -1;
  long long nvec = numel / 8;
  long long g = (nvec + 255) / 256, cap = (long long)sm_count() * 16;
  scale_bf16_kernel<<<(int)(g < cap ? g : cap), 256, 0, st>>>((__nv_bfloat16*)x, s, nvec);
  return (int)cudaGetLastError();
}
