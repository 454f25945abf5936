// The straight-line quotients and roots of coffee_b200/csrc/ez_pair.cuh and the
// division by 12 of ez_kernels.cuh (pd1_4) against the IEEE operations, on the GPU.
// Prints one line per check, "<name> <values compared> <values that differ>".
#include <cstdint>
#include <cstdio>

#include "ez_kernels.cuh"

using namespace coffee;

__device__ unsigned long long g_n, g_bad;

struct Rng {  // splitmix64
  uint64_t s;
  __device__ uint64_t next() {
    uint64_t z = (s += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
  }
  __device__ int below(int n) { return (int)(next() % (uint64_t)n); }
  // a float / double of a random mantissa and an exponent in [lo, hi)
  __device__ float f32(int lo, int hi) {
    return __uint_as_float(((uint32_t)(lo + below(hi - lo) + 127) << 23) | (uint32_t)(next() >> 41));
  }
  __device__ double f64(int lo, int hi) {
    return __longlong_as_double(((long long)(lo + below(hi - lo) + 1023) << 52) |
                                (long long)(next() >> 12));
  }
  template <typename T> __device__ T of(int lo, int hi) {
    if constexpr (sizeof(T) == 4) return f32(lo, hi);
    else return f64(lo, hi);
  }
};

__device__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b); }
__device__ bool same(double a, double b) {
  return __double_as_longlong(a) == __double_as_longlong(b);
}
__device__ void count(long long n, long long bad) {
  atomicAdd(&g_n, (unsigned long long)n);
  atomicAdd(&g_bad, (unsigned long long)bad);
}
__device__ long long thread_id() { return blockIdx.x * (long long)blockDim.x + threadIdx.x; }
__device__ long long threads() { return gridDim.x * (long long)blockDim.x; }

// every FP32 mantissa, at a few exponents inside the range
__global__ void reciprocals() {
  const int e[5] = {-23, -1, 0, 7, 29};
  long long n = 0, bad = 0;
  for (long long m = thread_id(); m < 5LL << 23; m += threads()) {
    const float b = __uint_as_float(((uint32_t)(e[m >> 23] + 127) << 23) | (uint32_t)(m & 0x7FFFFF));
    bad += !same(rcp_mid(b), __fdiv_rn(1.0f, b));
    ++n;
  }
  count(n, bad);
}
__global__ void roots() {
  const int e[6] = {-84, -41, 0, 1, 60, 99};
  long long n = 0, bad = 0;
  for (long long m = thread_id(); m < 6LL << 23; m += threads()) {
    const float x = __uint_as_float(((uint32_t)(e[m >> 23] + 127) << 23) | (uint32_t)(m & 0x7FFFFF));
    bad += !same(sqrt_mid(x), __fsqrt_rn(x));
    ++n;
  }
  count(n, bad);
}
__device__ double ieee_sqrt(double x) { return __dsqrt_rn(x); }
__device__ float ieee_sqrt(float x) { return __fsqrt_rn(x); }
__device__ double ieee_div(double a, double b) { return __ddiv_rn(a, b); }
__device__ float ieee_div(float a, float b) { return __fdiv_rn(a, b); }

// random roots, and sqrt_floor in the sum it is made for (any x >= 0, plus 1e-7)
template <typename T>
__global__ void random_roots(int per) {
  Rng r{(uint64_t)thread_id() * 977 + 5};
  long long bad = 0;
  constexpr int lo = sizeof(T) == 4 ? -84 : -800, hi = sizeof(T) == 4 ? 99 : 800;
  for (int q = 0; q < per; ++q) {
    const T x = r.of<T>(lo, hi);
    bad += !same(sqrt_mid(x), ieee_sqrt(x));
    // any exponent down to the subnormal numbers, and zero
    const T y = r.below(50) == 0 ? (T)0
                : sizeof(T) == 4 ? (T)__uint_as_float((uint32_t)(r.next() >> 33) % 0x52000000u)
                                 : (T)r.f64(-1000, 200);
    bad += !same((T)(sqrt_floor(y) + (T)1e-7), (T)(ieee_sqrt(y) + (T)1e-7));
  }
  count(2LL * per, bad);
}

// Quotients: where the guard accepts the operands the quotient is the IEEE one.
// Divisors and numerators over the whole range and beyond it, at the guard's
// thresholds, and quotients whose exact value lies within a few units of the
// divisor's last place of a rounding boundary.
template <typename T>
__global__ void quotients(int per, int near_boundary) {
  Rng r{(uint64_t)thread_id() * 1315423911ull + (uint64_t)near_boundary};
  long long n = 0, bad = 0;
  constexpr bool F = sizeof(T) == 4;
  constexpr int eb = F ? 30 : 500;
  for (int q = 0; q < per; ++q) {
    T b = r.of<T>(F ? -24 : -37, eb + 2);  // (the kernels' divisors are at least TINY)
    if (r.below(64) == 0) b = MidRange<T>::den_max;
    T a;
    if (near_boundary) {
      // the numerator of a quotient half a unit above t, give or take 3 units
      const T t = r.of<T>(F ? -90 : -300, F ? 30 : 300);
      T half;
      if constexpr (F) half = (__uint_as_float(__float_as_uint(t) + 1) - t) * 0.5f;
      else half = (__longlong_as_double(__double_as_longlong(t) + 1) - t) * 0.5;
      const T hi = smul(t, b);
      a = hi + sfma(half, b, sfma(t, b, -hi));
      const int d = r.below(7) - 3;
      if constexpr (F) a = __uint_as_float(__float_as_uint(a) + d);
      else a = __longlong_as_double(__double_as_longlong(a) + d);
    } else {
      a = r.of<T>(F ? -126 : -1000, F ? 127 : 1000);
      const int k = r.below(64);
      if (k == 0) a = MidRange<T>::num_max;
      if (k == 1) a = b * (F ? (T)4.70197740328915e-38 : (T)1.183052186166774e-271);  // 2^-124, 2^-900
      if (k == 2) a = (T)0;
    }
    if (r.next() & 1) a = -a;
    Guard<T> g;
    g.below(b, MidRange<T>::den_max);
    g.below(xa::mul(a, a), MidRange<T>::num_max);
    const T y = rcp_mid(b);
    const Pair<T> p = pdiv_mid(both(a), both(-b), both(y), g);
    g.below(xa::mul(first(p), first(p)), MidRange<T>::num_max);  // (as the kernels' E^2)
    if (g.bad()) continue;
    ++n;
    const T want = ieee_div(a, b);
    bad += !(same(first(p), second(p)) && (same(first(p), want) || (a == (T)0 && first(p) == want)));
    // and the quotient by a constant
    if constexpr (!F) continue;
    if (fabs(a) > (T)1e-20 && fabs(a) < (T)1e20) bad += !same(div_const(a, b, ieee_div((T)1, b)), want);
  }
  count(n, bad);
}

// t / 12 for every FP32 bit pattern that the guard accepts; a zero t gives +0.
__global__ void twelfths() {
  long long n = 0, bad = 0;
  for (long long u = thread_id(); u < 1LL << 32; u += threads()) {
    const float t = __uint_as_float((uint32_t)u);
    if (!(fabsf(t) <= 3.4e38f)) continue;
    Guard<float> g, h;
    // t from its four terms: (t - 8 * 0 + 8 * -0) - 0
    const Pair<float> p = pd1_4<true>(both(t), both(0.0f), both(-0.0f), both(0.0f), 0.0f, g);
    const float s = sd1_4<true>(t, 0.0f, -0.0f, 0.0f, 0.0f, h);
    if (g.bad() != h.bad() || g.bad() != (t != 0.0f && fabsf(t) < 4.70197740328915e-38f)) ++bad;
    if (g.bad()) continue;
    ++n;
    const float want = t == 0.0f ? 0.0f : __fdiv_rn(t, 12.0f);
    bad += !(same(first(p), want) && same(second(p), want) && same(s, want));
  }
  count(n, bad);
}

template <typename F>
static int check(const char* name, F&& launch) {
  const unsigned long long zero = 0;
  unsigned long long n, bad;
  cudaMemcpyToSymbol(g_n, &zero, sizeof zero);
  cudaMemcpyToSymbol(g_bad, &zero, sizeof zero);
  launch();
  const cudaError_t e = cudaDeviceSynchronize();
  if (e != cudaSuccess) {
    printf("%s %s\n", name, cudaGetErrorString(e));
    return 1;
  }
  cudaMemcpyFromSymbol(&n, g_n, sizeof n);
  cudaMemcpyFromSymbol(&bad, g_bad, sizeof bad);
  printf("%s %llu %llu\n", name, n, bad);
  return 0;
}

int main() {
  const int B = 148 * 8, T = 256;
  int rc = 0;
  rc |= check("reciprocals", [&] { reciprocals<<<B, T>>>(); });
  rc |= check("roots", [&] { roots<<<B, T>>>(); });
  rc |= check("roots_f32", [&] { random_roots<float><<<B, T>>>(500); });
  rc |= check("roots_f64", [&] { random_roots<double><<<B, T>>>(100); });
  rc |= check("quotients_f32", [&] { quotients<float><<<B, T>>>(1000, 0); });
  rc |= check("quotients_near_f32", [&] { quotients<float><<<B, T>>>(2000, 1); });
  rc |= check("quotients_f64", [&] { quotients<double><<<B, T>>>(200, 0); });
  rc |= check("quotients_near_f64", [&] { quotients<double><<<B, T>>>(200, 1); });
  rc |= check("twelfths", [&] { twelfths<<<B, T>>>(); });
  return rc;
}
