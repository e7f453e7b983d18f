// fp32 numbers as sums of 16-bit terms for the tensor cores, and the bounded waits of the kernels that use them.
#pragma once
#include <cuda_bf16.h>

#include "gnr_tc.cuh"

namespace {

// Split<0>: the fp32 network (mlp_mode 0).  An fp32 number is EXACTLY the sum of three bf16 numbers (8 + 8 + 8
// significand bits; bf16 has the exponent range of fp32), x = h + m + l with |m| <= 2^-8 |x|, |l| <= 2^-16 |x| up to
// rounding.  A product of two such sums needs six of the nine partial products, hh, hm, mh, mm, hl, lh: what is left out
// is below 2^-24 of the product, i.e. below the rounding of one fp32 multiplication.  Partial products of 16-bit terms
// are exact, sums are fp32 in tensor memory.
// Split<1>: mlp_mode 1.  Activations as fp16 hi + lo (about 22 bits), weights as one fp16.
// TA x TW terms of activations and weights; PRODUCTS partial products in the order they are added, the leading one last.
template <int MODE>
struct Split;

// sin and cos to within 7.1e-8 (rms 1.7e-8, i.e. little more than the rounding of the result) for |x| <= 1000.  Cody and
// Waite's argument reduction (Software Manual for the Elementary Functions, 1980): the multiple of pi/2 nearest to x is
// taken off in two steps (pi/2 as the sum of two floats; the fused multiply-adds round once).  What is left,
// |r| <= pi/4, goes into the Taylor polynomials up to r^9 and r^10 (next terms: 2e-9 and 1e-10), and the quadrant picks
// and signs them.
__device__ __forceinline__ void sincos_short(float x, float& s, float& c) {
  const float m = fmaf(x, 0.636619772f, 12582912.0f);  // 1.5 x 2^23: the low bits of m are the quadrant
  const float k = m - 12582912.0f;
  const int q = __float_as_int(m);
  float r = fmaf(-k, 1.57079637f, x);
  r = fmaf(-k, -4.37113883e-8f, r);
  const float z = r * r;
  float sp = fmaf(z, 2.75573192e-6f, -1.98412698e-4f);
  sp = fmaf(sp, z, 8.33333333e-3f);
  sp = fmaf(sp, z, -1.66666667e-1f);
  const float sr = fmaf(sp, z * r, r);
  float cp = fmaf(z, -2.75573192e-7f, 2.48015873e-5f);
  cp = fmaf(cp, z, -1.38888889e-3f);
  cp = fmaf(cp, z, 4.16666667e-2f);
  cp = fmaf(cp, z, -0.5f);
  const float cr = fmaf(cp, z, 1.0f);
  const float a = (q & 1) ? cr : sr, b = (q & 1) ? sr : cr;
  s = __int_as_float(__float_as_int(a) ^ ((q & 2) << 30));
  c = __int_as_float(__float_as_int(b) ^ (((q + 1) & 2) << 30));
}

template <>
struct Split<0> {
  static constexpr int TA = 3, TW = 3, PRODUCTS = 6;
  static constexpr uint32_t kFormat = (1u << 7) | (1u << 10);  // A and B bf16
  __host__ __device__ static constexpr int a(int i) { return i == 0 ? 2 : i == 1 ? 0 : i == 2 ? 1 : i == 3 ? 1 : 0; }
  __host__ __device__ static constexpr int w(int i) { return i == 0 ? 0 : i == 1 ? 2 : i == 2 ? 1 : i == 3 ? 0 : i == 4 ? 1 : 0; }
  // two numbers -> three packed pairs (`x` in the low halves)
  __device__ static __forceinline__ uint32_t pack(float x, float y) {
    uint32_t d;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(y), "f"(x));
    return d;
  }
  __device__ static __forceinline__ void split(float x, float y, uint32_t (&t)[TA]) {
    t[0] = pack(x, y);
    x -= __uint_as_float(t[0] << 16);
    y -= __uint_as_float(t[0] & 0xffff0000u);
    t[1] = pack(x, y);
    x -= __uint_as_float(t[1] << 16);
    y -= __uint_as_float(t[1] & 0xffff0000u);
    t[2] = pack(x, y);
  }
  // one weight -> its term t as 16 bits; `x` becomes the remainder
  __device__ static __forceinline__ uint16_t term(float& x) {
    const __nv_bfloat16 b = __float2bfloat16_rn(x);
    x -= __bfloat162float(b);
    return __bfloat16_as_ushort(b);
  }
  // three values -> one K step of layer 1: v, sin v, sin 2v, cos v, cos 2v of each, and a zero
  __device__ static __forceinline__ void encode(const float (&v)[3], float (&x)[16]) {
    // one test for all six angles of the warp's rows, so that the short form has no branches between them; where it fails
    // every value still takes the form that its own size asks for (a sample's bits do not depend on its neighbours)
    const bool large = !(fabsf(v[0]) <= 500.0f && fabsf(v[1]) <= 500.0f && fabsf(v[2]) <= 500.0f);
    if (__any_sync(0xffffffffu, large)) {
#pragma unroll 1
      for (int i = 0; i < 3; ++i) {
        const float u = i == 0 ? v[0] : i == 1 ? v[1] : v[2];
        float s1, c1, s2, c2;
        if (fabsf(u) <= 500.0f) {
          sincos_short(u, s1, c1);
          sincos_short(2.0f * u, s2, c2);
        } else {
          sincosf(u, &s1, &c1);
          sincosf(2.0f * u, &s2, &c2);
        }
#pragma unroll
        for (int e = 0; e < 3; ++e)
          if (e == i) {
            x[5 * e] = u;
            x[5 * e + 1] = s1;
            x[5 * e + 2] = s2;
            x[5 * e + 3] = c1;
            x[5 * e + 4] = c2;
          }
      }
    } else {
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        x[5 * i] = v[i];
        sincos_short(v[i], x[5 * i + 1], x[5 * i + 3]);
        sincos_short(2.0f * v[i], x[5 * i + 2], x[5 * i + 4]);
      }
    }
    x[15] = 0.0f;
  }
};

template <>
struct Split<1> {
  static constexpr int TA = 2, TW = 1, PRODUCTS = 2;
  static constexpr uint32_t kFormat = 0u;  // A and B fp16
  __host__ __device__ static constexpr int a(int i) { return i == 0 ? 1 : 0; }
  __host__ __device__ static constexpr int w(int) { return 0; }
  __device__ static __forceinline__ void split(float x, float y, uint32_t (&t)[TA]) {
    t[0] = pack_h2(x, y);
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&t[0]));
    t[1] = pack_h2(x - f.x, y - f.y);
  }
  __device__ static __forceinline__ uint16_t term(float& x) {
    const __half h = __float2half_rn(x);
    x -= __half2float(h);
    return __half_as_ushort(h);
  }
  // (one hardware sine and cosine, then the double-angle identities)
  __device__ static __forceinline__ void encode(const float (&v)[3], float (&x)[16]) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      float s, c;
      sincos_reduced(v[i], s, c);
      x[5 * i] = v[i];
      x[5 * i + 1] = s;
      x[5 * i + 2] = 2.0f * s * c;
      x[5 * i + 3] = c;
      x[5 * i + 4] = 1.0f - 2.0f * s * s;
    }
    x[15] = 0.0f;
  }
};

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32"
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_st4(uint32_t taddr, const uint32_t (&v)[4]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};\n" ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]),
               "r"(v[3])
               : "memory");
}
__device__ __forceinline__ void mbar_init(uint32_t mbar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(mbar), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint32_t mbar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(mbar) : "memory");
}

// All lanes of a warp wait together (bounded); false if the wait ran out or another role gave up.
__device__ __forceinline__ bool warp_wait(uint32_t mbar, uint32_t parity, volatile int* abort_flag, int32_t* status, uint32_t limit) {
  bool ok = false;
  for (uint32_t it = 0; it < limit; ++it) {
    ok = mbar_try_wait(mbar, parity);
    if (ok || *abort_flag) break;
    if (it > 64) __nanosleep(64);
  }
  if (__all_sync(0xffffffffu, ok)) return true;
  if ((threadIdx.x & 31) == 0) {
    *abort_flag = 1;
    atomicExch(status + GNR_ST_WAIT_EXPIRED, 1);
  }
  return false;
}

}  // namespace
