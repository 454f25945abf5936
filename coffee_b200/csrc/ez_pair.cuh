// Two values of the field precision worked on by one instruction, and the
// branch-free correctly rounded quotients and roots of the flat kernels.
//
// Every operation of the EZ update on a component of E is also done on the
// same component of B (the derivatives, the curl and divergence, the dot
// products with the curls, the Runge-Kutta update, the dissipation), so the
// kernels hold (E_a, B_a) as a pair.  In FP32 a pair is one 64-bit register
// pair and each operation one packed instruction (fma.rn.f32x2 and its kin),
// which rounds each half as the scalar operation does.  In FP64 a pair is two
// scalars.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace coffee {

template <typename T> struct Pair;
template <> struct Pair<float> { unsigned long long v; };
template <> struct Pair<double> { double a, b; };

__device__ __forceinline__ Pair<float> pk(float a, float b) {
  Pair<float> p;
  asm("mov.b64 %0, {%1, %2};" : "=l"(p.v) : "f"(a), "f"(b));
  return p;
}
__device__ __forceinline__ Pair<double> pk(double a, double b) { return {a, b}; }
__device__ __forceinline__ float first(Pair<float> p) {
  float a, b;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(p.v));
  return a;
}
__device__ __forceinline__ float second(Pair<float> p) {
  float a, b;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(p.v));
  return b;
}
__device__ __forceinline__ double first(Pair<double> p) { return p.a; }
__device__ __forceinline__ double second(Pair<double> p) { return p.b; }
template <typename T>
__device__ __forceinline__ Pair<T> both(T x) { return pk(x, x); }

// x y + z, x y, x + y, x - y of both halves, each rounded once
__device__ __forceinline__ Pair<float> pfma(Pair<float> x, Pair<float> y, Pair<float> z) {
  Pair<float> r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(x.v), "l"(y.v), "l"(z.v));
  return r;
}
__device__ __forceinline__ Pair<float> pmul(Pair<float> x, Pair<float> y) {
  Pair<float> r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(x.v), "l"(y.v));
  return r;
}
__device__ __forceinline__ Pair<float> padd(Pair<float> x, Pair<float> y) {
  Pair<float> r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(x.v), "l"(y.v));
  return r;
}
__device__ __forceinline__ Pair<float> psub(Pair<float> x, Pair<float> y) {
  Pair<float> r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(x.v), "l"(y.v));
  return r;
}
__device__ __forceinline__ Pair<double> pfma(Pair<double> x, Pair<double> y, Pair<double> z) {
  return {__fma_rn(x.a, y.a, z.a), __fma_rn(x.b, y.b, z.b)};
}
__device__ __forceinline__ Pair<double> pmul(Pair<double> x, Pair<double> y) {
  return {__dmul_rn(x.a, y.a), __dmul_rn(x.b, y.b)};
}
__device__ __forceinline__ Pair<double> padd(Pair<double> x, Pair<double> y) {
  return {__dadd_rn(x.a, y.a), __dadd_rn(x.b, y.b)};
}
__device__ __forceinline__ Pair<double> psub(Pair<double> x, Pair<double> y) {
  return {__dsub_rn(x.a, y.a), __dsub_rn(x.b, y.b)};
}
// the single operations the pairs are mixed with
__device__ __forceinline__ float sfma(float x, float y, float z) { return __fmaf_rn(x, y, z); }
__device__ __forceinline__ double sfma(double x, double y, double z) { return __fma_rn(x, y, z); }
__device__ __forceinline__ float smul(float x, float y) { return __fmul_rn(x, y); }
__device__ __forceinline__ double smul(double x, double y) { return __dmul_rn(x, y); }

// a pair from shared memory: 32-bit address plus a compile-time offset
template <typename T, int OFF>
__device__ __forceinline__ Pair<T> ldsp(uint32_t a) {
  Pair<T> p;
  if constexpr (sizeof(T) == 4)
    asm volatile("ld.shared.b64 %0, [%1+%2];\n" : "=l"(p.v) : "r"(a), "n"(OFF));
  else
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2+%3];\n"
                 : "=d"(p.a), "=d"(p.b) : "r"(a), "n"(OFF));
  return p;
}

// a . b of two vectors of pairs: the first product rounded, the other two
// fused into the sum
template <typename T>
__device__ __forceinline__ Pair<T> pdot3(const Pair<T> a[3], const Pair<T> b[3]) {
  return pfma(a[2], b[2], pfma(a[1], b[1], pmul(a[0], b[0])));
}

// ---- correctly rounded quotients and roots without branches -------------
// The IEEE division and square root of the CUDA compiler take a branch per
// operation for operands near the ends of the range, so a point's eleven
// quotients and two roots run one after the other.  Here they are straight
// line code that overlaps, correct for operands in the middle of the range;
// a `Guard` notes anything outside it and the caller then recomputes the
// point with the IEEE operations.
//
// Reciprocal y = RN(1/b): the hardware approximation and one Newton step;
// quotient: q = a y and the correction q + (a - b q) y with the exact residual
// (P. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. Res. Dev. 34(1), 1990).  Square root: the coupled iteration of the same paper
// for g -> sqrt(x), h -> 1/(2 sqrt(x)), with the residual x - g g exact at the
// end.  Numerators are scaled by 2^64 first, so that their residuals are
// exact however small they are (FP32); a quotient below 2^-124 is left to the
// IEEE division, whose rounding of it is to a subnormal number.
// Compared with the IEEE operations on the GPU (tests/cuda/pair_check.cu): every FP32
// reciprocal and root mantissa, 6e8 FP32 quotients beside rounding boundaries and 2e8
// random ones, 3e8 roots, 1e8 FP64 quotients and 6e7 roots: no difference, but for -0 / b,
// which is +0 here.  The FP64 reciprocal of the one mantissa that is all ones is an ulp
// off (as the paper says), and then quotients within 2^-53 of a boundary are, too.
template <typename T> struct MidRange;
template <> struct MidRange<float> {
  static constexpr float den_max = 1073741824.0f;             // 2^30
  static constexpr float num_max = 1.2676506002282294e30f;    // 2^100
  static constexpr float root_scale = 18446744073709551616.0f, root_back = 2.3283064365386963e-10f;
  static constexpr float root_min = 2.5849394142282115e-26f;  // 2^-85
};
template <> struct MidRange<double> {
  static constexpr double den_max = 3.273390607896142e150;     // 2^500
  static constexpr double num_max = 1.0715086071862673e301;    // 2^1000
  static constexpr double root_scale = 1.0, root_back = 1.0;
  static constexpr double root_min = 1.183052186166774e-271;   // 2^-900
};

// What a point's straight-line arithmetic met: the smallest key of its small
// operands (see key()) and whether a large or undefined one was among them.
template <typename T> struct Guard {
  uint32_t kmin = 0xFFFFFFFFu;
  bool large = false;
  __device__ __forceinline__ bool bad() const;
  // note that x must be at most `m` (false for a NaN, too)
  __device__ __forceinline__ void below(T x, T m) { large = large || !(x < m); }
  __device__ __forceinline__ void above(T x, T m) { large = large || !(x > m); }
  // Key of a value: drops the sign, sends zero to the largest value and is
  // below the threshold exactly for the nonzero values below 2^-124 (FP32)
  // or 2^-900 (FP64).
  __device__ __forceinline__ static uint32_t key(float x) {
    const uint32_t b = __float_as_uint(x);
    return b + b - 1u;
  }
  __device__ __forceinline__ static uint32_t key(double x) {
    const uint32_t h = (uint32_t)__double2hiint(x);
    return ((h + h) | (__double2loint(x) != 0 ? 1u : 0u)) - 1u;
  }
  __device__ __forceinline__ void small(T x) { kmin = min(kmin, key(x)); }
  __device__ __forceinline__ void small(Pair<T> p) {
    kmin = min(kmin, min(key(first(p)), key(second(p))));
  }
};
template <> __device__ __forceinline__ bool Guard<float>::bad() const {
  return large || kmin < 0x02FFFFFEu;
}
template <> __device__ __forceinline__ bool Guard<double>::bad() const {
  return large || kmin < 0x0F600000u;
}

__device__ __forceinline__ float rcp_seed(float b) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(b));
  return y;
}
__device__ __forceinline__ double rcp_seed(double b) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
  // 2^-20 -> 2^-40 -> 2^-53: the last step is the caller's
  double e = __fma_rn(-b, y, 1.0);
  y = __fma_rn(e, y, y);
  e = __fma_rn(-b, y, 1.0);
  return __fma_rn(e, y, y);
}
// RN(1/b), b in the middle of the range
template <typename T>
__device__ __forceinline__ T rcp_mid(T b) {
  const T y = rcp_seed(b);
  return sfma(sfma(-b, y, (T)1), y, y);
}
// a / b with y = RN(1/b) formed on the host: the quotient rounded as the division
// rounds it (for a quotient and residual in the range of normal numbers), three
// operations instead of the division's ten and a branch.
template <typename T>
__device__ __forceinline__ T div_const(T a, T b, T y) {
  const T q = smul(a, y);
  return sfma(sfma(-b, q, a), y, q);
}
// a / b for both halves, with nb = -b and y = RN(1/b)
__device__ __forceinline__ Pair<float> pdiv_mid(Pair<float> a, Pair<float> nb, Pair<float> y,
                                                Guard<float>& g) {
  const Pair<float> as = pmul(a, both(18446744073709551616.0f));  // 2^64
  Pair<float> q = pmul(as, y);
  q = pfma(pfma(nb, q, as), y, q);
  q = pmul(q, both(5.421010862427522e-20f));  // 2^-64
  g.small(q);
  return q;
}
__device__ __forceinline__ Pair<double> pdiv_mid(Pair<double> a, Pair<double> nb, Pair<double> y,
                                                 Guard<double>& g) {
  Pair<double> q = pmul(a, y);
  q = pfma(pfma(nb, q, a), y, q);
  g.small(a);
  return q;
}

__device__ __forceinline__ float rsqrt_seed(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ double rsqrt_seed(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}
// RN(sqrt(x)), x in the middle of the range
template <typename T>
__device__ __forceinline__ T sqrt_mid(T x) {
  const T y = rsqrt_seed(x);
  T g = smul(x, y), h = smul(y, (T)0.5);
#pragma unroll
  for (int it = 0; it < (sizeof(T) == 8 ? 2 : 1); ++it) {
    const T r = sfma(-h, g, (T)0.5);
    g = sfma(g, r, g);
    h = sfma(h, r, h);
  }
  return sfma(sfma(-g, g, x), h, g);
}

// sqrt(x) for a small or large x, to be added to a number of at least TINY:
// scaled by 2^64 (FP32), so that the residual is exact for every x > 0, and with
// a floor under x (2^-149, or 2^-900) whose root vanishes in that sum as 0 does.
template <typename T>
__device__ __forceinline__ T sqrt_floor(T x) {
  x = smul(x, MidRange<T>::root_scale);
  return smul(sqrt_mid(x > MidRange<T>::root_min ? x : MidRange<T>::root_min),
              MidRange<T>::root_back);
}

}  // namespace coffee
