// Kernels of the GR force-free solver in Cartesian Kerr-Schild coordinates
// (reference src/algorithms/field_solver_gr_EZ.cu, metric
// src/algorithms/metric_cks_impl.hpp).
//
// sim_data's E holds the densitised displacement D; the curl acts on the
// constitutive fields E = alpha D_i + sqrt(gamma) (beta x B)_i and
// H = alpha B_i - sqrt(gamma) (beta x D)_i.  A stage is two launches: one
// writes E and H over the whole grid (the reference's get_Ed / get_Hd), the
// other does the LSRK update, the clamps and, in the last stage, both
// absorbing layers in one pass over the update box, reading the current
// buffer and writing the other one.  Near the horizon the metric comes from
// a table evaluated once per solver in FP64 (gr_metric_kernel); elsewhere it
// is evaluated per point in field precision, as the reference does, but
// once per point and launch (the reference calls get_r inside every metric
// component, about forty times per point).
#pragma once

#include "axisym_kernels.cuh"
#include "ez_common.cuh"
#include "ez_pair.cuh"

namespace coffee {

template <typename T>
struct GrConst {
  int d[3];                 // dims
  int lo[3], hi[3];         // update box
  int g[3];                 // guards
  T lower[3], delta[3], inv_delta[3];
  T a, dt, tau, inv_tau, ko_c;
  int calc_current, divB_clean, clean_ep, check_egb;
  int absorbing;
  T xl[3], xh[3];           // outer layer edges (boundary.cu:43-54)
  T pmlscale, sigpml;
  T r1, r2, dd;             // inner layer: 0.7 r_H, 0.01 r_H, 0.2 r_H (:617-621)
  int nb_lo[3], nb_n[3];    // the near-horizon box of the metric table (grid indices)
};

// Reciprocals and roots of the metric: the straight-line ones of ez_pair.cuh
// (the IEEE operations' range branches would run the metric's eight roots and
// quotients one after another), with the ends of the range made harmless.
template <typename T>
__device__ __forceinline__ T metric_rcp(T x) {
  // an overflowed denominator (r beyond 1e9) has the reciprocal 0
  const T y = rcp_seed(x);
  return x < (sizeof(T) == 4 ? (T)1e37 : (T)1e300) ? sfma(sfma(-x, y, (T)1), y, y) : (T)0;
}
template <typename T>
__device__ __forceinline__ T metric_sqrt(T x) {
  constexpr T lo = sizeof(T) == 4 ? (T)1e-30 : (T)1e-60, hi = sizeof(T) == 4 ? (T)1e37 : (T)1e300;
  return x < hi ? sqrt_mid(x > lo ? x : lo) : ::sqrt(x);
}

// r of the Kerr-Schild coordinates (metric_cks_impl.hpp:17-24)
template <typename T>
__device__ __forceinline__ T cks_r(T a, T x, T y, T z, T tiny = Tiny<T>::v) {
  const T R2 = x * x + y * y + z * z;
  const T q = R2 - a * a;
  T s = q * q + T(4) * (a * z) * (a * z);
  if (s < tiny) s = tiny;
  return metric_sqrt((q + metric_sqrt(s)) * T(0.5));
}

// sqrt(gamma) = sqrt(1 + 2 r^3 / (r^4 + a^2 z^2)) (:77-83)
template <typename T>
__device__ __forceinline__ T cks_sqrt_gamma(T a, T x, T y, T z) {
  const T r = cks_r(a, x, y, z);
  T den = r * r * r * r + a * a * z * z;
  if (den < Tiny<T>::v) den = Tiny<T>::v;
  return metric_sqrt(T(1) + T(2) * r * r * r * metric_rcp(den));
}

// The Kerr-Schild metric at one point (metric_cks_impl.hpp:13-181): gamma_ij =
// delta_ij + H l_i l_j, gamma^ij = delta_ij - H/(1+H) l_i l_j, beta^i = H/(1+H)
// l_i, alpha = 1/sqrt(1+H), sqrt(gamma) = sqrt(1+H), with H = 2 r^3 / (r^4 +
// a^2 z^2) and l = ((r x + a y)/(r^2 + a^2), (r y - a x)/(r^2 + a^2), z/r).
// Eight numbers instead of the eighteen components of the metric and its
// inverse: fewer registers in kernels that have too few, and an index is
// lowered or raised by a dot product and three fused multiply-adds.
// Evaluated in precision T with the TINY floors of the field precision TF.
template <typename T, typename TF = T>
struct Cks {
  T r, H, hb, alpha, sg;  // hb = H / (1 + H)
  T l[3];

  Cks() = default;
  __device__ __forceinline__ Cks(T a, T x, T y, T z) {
    constexpr T tiny = (T)Tiny<TF>::v;
    r = cks_r(a, x, y, z, tiny);
    const T r2 = r * r, aa = a * a;
    T den = r2 * r2 + aa * z * z;
    if (den < tiny) den = tiny;
    T ar = aa + r2;
    if (ar < tiny) ar = tiny;
    const T iar = metric_rcp(ar);
    l[0] = (r * x + a * y) * iar;
    l[1] = (r * y - a * x) * iar;
    l[2] = z * metric_rcp(r);
    H = T(2) * r2 * r * metric_rcp(den);
    derive();
  }
  // alpha, sqrt(gamma) and H / (1 + H) from H
  __device__ __forceinline__ void derive() {
    const T gam = T(1) + H;
    sg = metric_sqrt(gam);
    alpha = metric_rcp(sg);
    hb = H * metric_rcp(gam);
  }
  __device__ __forceinline__ T beta(int i) const { return hb * l[i]; }
  __device__ __forceinline__ T along(const T* v) const {
    return l[0] * v[0] + l[1] * v[1] + l[2] * v[2];
  }
  __device__ __forceinline__ void lower(const T* v, T* o) const {
    const T q = H * along(v);
#pragma unroll
    for (int i = 0; i < 3; ++i) o[i] = v[i] + q * l[i];
  }
  // of both vectors of a pair
  __device__ __forceinline__ void lower(const Pair<T> v[3], Pair<T> o[3]) const {
    const Pair<T> L[3] = {both(l[0]), both(l[1]), both(l[2])};
    const Pair<T> q = pmul(both(H), pdot3(L, v));
#pragma unroll
    for (int i = 0; i < 3; ++i) o[i] = pfma(q, L[i], v[i]);
  }
};

template <typename T>
__device__ __forceinline__ T gr_pos(const GrConst<T>& c, int a, int n) {
  return c.lower[a] + c.delta[a] * (T)(n - c.g[a]);
}

// The near-horizon metric table.  Within a box of half-width kNearRH r_H
// around the hole the metric is evaluated once per solver in FP64 (at the
// grid's coordinates in the field precision, where the reference evaluates
// it) and rounded to the field precision: there the field-precision formula
// loses digits (r from sqrt((q + sqrt(q^2 + 4 a^2 z^2)) / 2) with
// q = R^2 - a^2 cancels inside the horizon, giving FP32 errors of 1e-5 in r
// and the shift against 1e-7 outside 1.5 r_H).  Elsewhere it is evaluated in
// the field precision per point, as the reference does.  kMetricComps
// components, component q of table point t at m[q * nt + t]: r, H, l_1..3,
// alpha, sqrt(gamma).
constexpr int kMetricComps = 7;
constexpr double kNearRH = 3.0;

template <typename T>
__device__ __forceinline__ long long near_index(const GrConst<T>& c, int i, int j, int k) {
  const int a = i - c.nb_lo[0], b = j - c.nb_lo[1], e = k - c.nb_lo[2];
  if ((unsigned)a >= (unsigned)c.nb_n[0] || (unsigned)b >= (unsigned)c.nb_n[1] ||
      (unsigned)e >= (unsigned)c.nb_n[2])
    return -1;
  return a + (long long)c.nb_n[0] * (b + (long long)c.nb_n[1] * e);
}

template <typename T>
__global__ void gr_metric_kernel(const __grid_constant__ GrConst<T> c, T* __restrict__ m,
                                 T* __restrict__ sg) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int k = blockIdx.z * blockDim.z + threadIdx.z;
  if (i >= c.d[0] || j >= c.d[1] || k >= c.d[2]) return;
  const long long o = i + (long long)c.d[0] * (j + (long long)c.d[1] * k);
  const Cks<double, T> q((double)c.a, (double)gr_pos(c, 0, i), (double)gr_pos(c, 1, j),
                         (double)gr_pos(c, 2, k));
  // sqrt(gamma) of every point: the divergence stencil (div4,
  // field_solver_gr_EZ.cu:44-86) weights each neighbour by it
  sg[o] = (T)q.sg;
  const long long t = near_index(c, i, j, k);
  if (t < 0) return;
  const long long nt = (long long)c.nb_n[0] * c.nb_n[1] * c.nb_n[2];
  const double v[kMetricComps] = {q.r, q.H, q.l[0], q.l[1], q.l[2], q.alpha, q.sg};
#pragma unroll
  for (int a = 0; a < kMetricComps; ++a) m[a * nt + t] = (T)v[a];
}

// The metric at grid point (i, j, k) with coordinates (x, y, z): from the
// table inside the near-horizon box, else evaluated here.
template <typename T>
__device__ __forceinline__ Cks<T> metric_at(const GrConst<T>& c, const T* __restrict__ m,
                                            int i, int j, int k, T x, T y, T z) {
  const long long t = near_index(c, i, j, k);
  if (t < 0) return Cks<T>(c.a, x, y, z);
  const long long nt = (long long)c.nb_n[0] * c.nb_n[1] * c.nb_n[2];
  Cks<T> q;
  q.r = __ldg(m + t);
  q.H = __ldg(m + nt + t);
#pragma unroll
  for (int a = 0; a < 3; ++a) q.l[a] = __ldg(m + (2 + a) * nt + t);
  q.alpha = __ldg(m + 5 * nt + t);
  q.sg = __ldg(m + 6 * nt + t);
  q.hb = q.H * q.alpha * q.alpha;
  return q;
}

// E = alpha D + sqrt(gamma) beta x B and H = alpha B - sqrt(gamma) beta x D
// (lowered D, B) at one point, stored at offset o of eh[0..5]
// (kernel_compute_E_gr / kernel_compute_H_gr, field_solver_gr_EZ.cu:88-186).
// Every kernel that writes D and B at a point also writes E and H there
// through this function, so they are computed the same way everywhere.
template <typename T>
__device__ __forceinline__ void gr_eh_store(const Cks<T>& m, const Pair<T> db[3],
                                            const F7<T>& eh, const uint32_t o) {
  Pair<T> low[3];
  m.lower(db, low);
  const T sh = m.sg * m.hb;  // sqrt(gamma) beta = sh l
  const Pair<T> L[3] = {both(m.l[0]), both(m.l[1]), both(m.l[2])};
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const int b = (a + 1) % 3, c = (a + 2) % 3;
    // (l x D, l x B)_a
    const Pair<T> x = pfma(L[b], db[c], pmul(both(-m.l[c]), db[b]));
    eh.p[a][o] = sfma(sh, second(x), smul(m.alpha, first(low[a])));
    eh.p[3 + a][o] = sfma(-sh, first(x), smul(m.alpha, second(low[a])));
  }
}

// E and H over the whole grid (guards included): once per call of the
// solver, for both field buffers; afterwards every stage and KO pass writes
// E and H of the points it updates (ehout), so the next kernel finds those
// of its input.  eh[0..2] = E, eh[3..5] = H.
// GUARDS: only the points outside the update box (the first stage writes E and
// H of the others).
template <typename T, bool GUARDS>
__global__ void __launch_bounds__(256) gr_eh_kernel(const __grid_constant__ GrConst<T> c,
                                                    const F7<T> u, const F7<T> eh,
                                                    const T* __restrict__ mt) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int k = blockIdx.z * blockDim.z + threadIdx.z;
  if (i >= c.d[0] || j >= c.d[1] || k >= c.d[2]) return;
  if (GUARDS && i >= c.lo[0] && i < c.hi[0] && j >= c.lo[1] && j < c.hi[1] && k >= c.lo[2] &&
      k < c.hi[2])
    return;
  const uint32_t o = (uint32_t)i + (uint32_t)c.d[0] * ((uint32_t)j + (uint32_t)c.d[1] * (uint32_t)k);
  Pair<T> db[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) db[a] = pk(__ldg(u.p[a] + o), __ldg(u.p[3 + a] + o));
  const Cks<T> m =
      metric_at(c, mt, i, j, k, gr_pos(c, 0, i), gr_pos(c, 1, j), gr_pos(c, 2, k));
  gr_eh_store(m, db, eh, o);
}

// clean_epar / check_eGTb with the 3-metric (kernel_clean_epar_gr,
// kernel_check_eGTb_gr, field_solver_gr_EZ.cu:422-521)
// Lowering is linear, so the lowered D after the cleaning is that of before
// minus the same multiple of the lowered B.
template <typename T>
__device__ __forceinline__ void gr_clamps(const GrConst<T>& c, const Cks<T>& m, Pair<T> db[3]) {
  if (!c.clean_ep && !c.check_egb) return;
  Pair<T> low[3];
  m.lower(db, low);
  T D[3] = {first(db[0]), first(db[1]), first(db[2])};
  const T B[3] = {second(db[0]), second(db[1]), second(db[2])};
  T Dd[3] = {first(low[0]), first(low[1]), first(low[2])};
  const T Bd[3] = {second(low[0]), second(low[1]), second(low[2])};
  const T B2 = B[0] * Bd[0] + B[1] * Bd[1] + B[2] * Bd[2];
  if (c.clean_ep) {
    const T q =
        fdiv(D[0] * Bd[0] + D[1] * Bd[1] + D[2] * Bd[2], B2 < Tiny<T>::v ? Tiny<T>::v : B2);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      D[a] -= q * B[a];
      Dd[a] -= q * Bd[a];
    }
  }
  if (c.check_egb) {
    T D2 = D[0] * Dd[0] + D[1] * Dd[1] + D[2] * Dd[2];
    if (D2 < Tiny<T>::v) D2 = Tiny<T>::v;
    if (D2 > B2) {
      const T s = sqrt(fdiv(B2, D2));
#pragma unroll
      for (int a = 0; a < 3; ++a) D[a] *= s;
    }
  }
#pragma unroll
  for (int a = 0; a < 3; ++a) db[a] = pk(D[a], B[a]);
}

// Outer layer at the six faces (kernel_boundary_absorbing_thread,
// src/algorithms/boundary.cu:17-79), then the inner layer inside 0.7 r_H and
// the zeroed core inside 0.01 r_H (kernel_absorbing_inner,
// field_solver_gr_EZ.cu:610-701); both blend towards the start-of-step
// values n.
template <typename T>
__device__ __noinline__ V7<T> gr_absorb(const GrConst<T>& c, V7<T> v, V7<T> n, T x, T y, T z,
                                        T r) {
  const T pos[3] = {x, y, z};
  bool outside = false;
  T sig = T(0);
  for (int a = 0; a < 3; ++a) {
    outside = outside || pos[a] > c.xh[a] || pos[a] < c.xl[a];
    sig += cyl_pmlsigma(pos[a], c.xl[a], c.xh[a], c.pmlscale, c.sigpml);
  }
  if (outside && sig > Tiny<T>::v) {
    const T e = exp(-sig);
    const T f = (T(1) - e) / sig;
    for (int a = 0; a < 6; ++a) v.v[a] = e * n.v[a] + f * (v.v[a] - n.v[a]);
  }
  if (r < c.r1) {
    const T q = (c.r1 - r) / c.dd;
    const T s = c.sigpml * q * q * q * c.dt;
    if (s > Tiny<T>::v) {
      const T e = exp(-s);
      const T f = (T(1) - e) / s;
      for (int a = 0; a < 6; ++a) v.v[a] = e * n.v[a] + f * (v.v[a] - n.v[a]);
    }
  }
  if (r < c.r2)
    for (int a = 0; a < 6; ++a) v.v[a] = T(0);
  return v;
}

// One LSRK stage of the GR solver (kernel_rk_step1_gr + kernel_rk_step2_gr,
// field_solver_gr_EZ.cu:188-420, then the clamps and, in the last stage,
// the absorbing layers: order of :876-893).  u: D, B, P of the current
// buffer; eh: E, H of the same buffer.
// Minimum resident 256-thread CTAs per SM of the stage and KO kernels: bound by the
// latency of their stencil loads, they want warps until spilling costs more.  Stage with
// 4 / 5 / 6, us: 64^3 19.1 / 20.3 / 21.5, 128^3 129 / 131 / 130, 192^3 399 / 402 / 396,
// 256^3 910 / 915 / 910; KO 14.7 / 15.4 / 18.0, 86 / 84 / 88, 258 / 250 / 255, 586 / 569
// / 577.
#ifndef COFFEE_GR_STAGE_MIN_BLOCKS
#define COFFEE_GR_STAGE_MIN_BLOCKS 4
#endif
#ifndef COFFEE_GR_KO_MIN_BLOCKS
#define COFFEE_GR_KO_MIN_BLOCKS 5
#endif
// The stage at one point, given its stencil values through fetch(q, ax,
// n): array q (0-2 E, 3-5 H, 6-8 D, 9-11 B, 12 P, 13 sqrt(gamma)) at offset
// n = -2, -1, 1, 2 along axis ax from the point, and own(q), array q at the
// point (read where the values are first needed, which keeps them out of
// the registers of the stencil sums).  Both stage kernels (global stencil
// loads, shared-memory tiles) run this code, so their arithmetic is the
// same.
template <typename T, bool FIRST, typename Metric, typename Fetch, typename Own>
__device__ __forceinline__ void gr_stage_point(const GrConst<T>& c, Metric&& metric, const T x,
                                               const T y, const T z, const uint32_t o,
                                               Fetch&& f, Own&& own,
                                               const F7<T>& out, const F7<T>& du,
                                               const F7<T>& un, const F5<T>& aux, const T As,
                                               const T Bs, const int flags,
                                               const F7<T>& ehout) {
  using I0 = std::integral_constant<int, 0>;
  using I1 = std::integral_constant<int, 1>;
  using I2 = std::integral_constant<int, 2>;
  using QP = std::integral_constant<int, 12>;
  using QS = std::integral_constant<int, 13>;
  // diff1_4 of the pair (E_q, H_q) along an axis, times 12 / inv_delta.  1 / 12 goes
  // with the 1 / sqrt(gamma) of a whole curl or divergence: its terms cancel, and
  // 1 / 12 rounded into inv_delta of each axis would change their ratio where the
  // spacings differ (P of such a run 1% farther from 64 bits)
  auto d1 = [&](auto qc, auto ac) {
    constexpr int q = decltype(qc)::value;
    using H = std::integral_constant<int, q + 3>;
    auto v = [&](int n) { return pk(f(qc, ac, n), f(H{}, ac, n)); };
    Pair<T> t = psub(v(-2), v(2));
    t = pfma(v(-1), both((T)-8), t);
    return pfma(v(1), both((T)8), t);
  };
  const T* w = c.inv_delta;
  // the curls and divergences before their 1 / sqrt(gamma) factor: the
  // metric is evaluated after the stencil sums, so that its values do not
  // take registers while those are formed (the same operations either way)
  Pair<T> rot[3];  // (rot E, rot H)
  rot[0] = pfma(d1(I2{}, I1{}), both(w[1]), pmul(d1(I1{}, I2{}), both(-w[2])));
  rot[1] = pfma(d1(I0{}, I2{}), both(w[2]), pmul(d1(I2{}, I0{}), both(-w[0])));
  rot[2] = pfma(d1(I1{}, I0{}), both(w[0]), pmul(d1(I0{}, I1{}), both(-w[1])));
  // div4 (:44-86): each neighbour weighted by sqrt(gamma) there (the
  // per-solver table; the reference evaluates it at the shifted coordinates)
  Pair<T> dvg = both((T)0);  // (div D, div B)
  static_for<3>([&](auto ac) {
    constexpr int ax = decltype(ac)::value;
    using QD = std::integral_constant<int, 6 + ax>;
    using QB = std::integral_constant<int, 9 + ax>;
    auto v = [&](int n) { return pk(f(QD{}, ac, n), f(QB{}, ac, n)); };
    Pair<T> t = pmul(v(-2), both(f(QS{}, ac, -2)));
    t = pfma(v(-1), both(T(-8) * f(QS{}, ac, -1)), t);
    t = pfma(v(1), both(T(8) * f(QS{}, ac, 1)), t);
    t = pfma(v(2), both(-f(QS{}, ac, 2)), t);
    dvg = pfma(t, both(w[ax]), dvg);
  });
  T Pd[3];
  static_for<3>([&](auto ac) {
    constexpr int ax = decltype(ac)::value;
    const T t = sfma(f(QP{}, ac, -1), (T)-8, f(QP{}, ac, -2) - f(QP{}, ac, 2));
    Pd[ax] = sfma(f(QP{}, ac, 1), (T)8, t) * (w[ax] * T(1.0 / 12.0));
  });
  const Cks<T> m = metric();
  const T igms = metric_rcp(m.sg), igms12 = igms * T(1.0 / 12.0);
#pragma unroll
  for (int a = 0; a < 3; ++a) rot[a] = pmul(rot[a], both(igms12));
  dvg = pmul(dvg, both(igms12));
  const T divD = first(dvg), divB = second(dvg);
  Pair<T> db[3];  // (D, B)
#pragma unroll
  for (int a = 0; a < 3; ++a) db[a] = pk(own(6 + a), own(9 + a));
  T P = own(12);
  T J[3] = {T(0), T(0), T(0)};
  if (c.calc_current) {
    Pair<T> low[3];
    m.lower(db, low);
    T B2 = second(pdot3(db, low));
    if (B2 < Tiny<T>::v) B2 = Tiny<T>::v;
    const Pair<T> lr = pdot3(low, rot);  // (D . rot E, B . rot H)
    const T Jp = second(lr) - first(lr);
    const T e[3] = {own(0), own(1), own(2)};
    const T b[3] = {second(low[0]), second(low[1]), second(low[2])};
    const T iB2 = fdiv(T(1), B2), s = divD * igms;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const int a1 = (a + 1) % 3, a2 = (a + 2) % 3;
      J[a] = (s * (e[a1] * b[a2] - e[a2] * b[a1]) + Jp * second(db[a])) * iB2;
    }
  }
  // beta . grad P = hb (l . grad P), and -alpha P^i + beta^i div B as a
  // multiple of l^i and of P_i
  const T lP = m.hb * m.along(Pd);
  const T kl = m.alpha * lP + m.hb * divB;
  // r0 = 5, del = 1 (:276-278): 0.5 (1 - tanh(r - 5)) = 1 / (1 + exp(2 (r - 5)))
  const T shape = c.divB_clean ? T(1) / (T(1) + exp(T(2) * (m.r - T(5)))) : T(0);
  const T dt = c.dt;
  if (flags & AX_WRITE_UN) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      un.p[a][o] = first(db[a]);
      un.p[3 + a][o] = second(db[a]);
    }
  }
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const T clean = c.divB_clean ? kl * m.l[a] - m.alpha * Pd[a] : T(0);
    Pair<T> d = pmul(pk(second(rot[a]) - J[a], sfma(clean, shape, -first(rot[a]))), both(dt));
    if constexpr (!FIRST) d = pfma(pk(du.p[a][o], du.p[3 + a][o]), both(As), d);
    du.p[a][o] = first(d);
    du.p[3 + a][o] = second(d);
    db[a] = pfma(d, both(Bs), db[a]);
  }
  {
    T d = dt * (lP - m.alpha * divB) - div_const(m.alpha * P, c.tau, c.inv_tau);
    if constexpr (!FIRST) d = sfma(du.p[6][o], As, d);
    du.p[6][o] = d;
    P = sfma(d, Bs, P);
  }
  if (flags & AX_AUX) {
    aux.p[0][o] = J[0];
    aux.p[1][o] = J[1];
    aux.p[2][o] = J[2];
    aux.p[3][o] = divD;
    aux.p[4][o] = divB;
  }
  gr_clamps(c, m, db);
  const bool in_layer = x > c.xh[0] || x < c.xl[0] || y > c.xh[1] || y < c.xl[1] ||
                        z > c.xh[2] || z < c.xl[2] || m.r < c.r1;
  if ((flags & AX_LAST) && c.absorbing && in_layer) {
    V7<T> w, n;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      w.v[a] = first(db[a]);
      w.v[3 + a] = second(db[a]);
    }
    w.v[6] = P;
#pragma unroll
    for (int a = 0; a < 6; ++a) n.v[a] = un.p[a][o];
    n.v[6] = T(0);
    w = gr_absorb(c, w, n, x, y, z, m.r);
#pragma unroll
    for (int a = 0; a < 3; ++a) db[a] = pk(w.v[a], w.v[3 + a]);
  }
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    out.p[a][o] = first(db[a]);
    out.p[3 + a][o] = second(db[a]);
  }
  out.p[6][o] = P;
  if (ehout.p[0]) gr_eh_store(m, db, ehout, o);
}

template <typename T, bool FIRST>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? COFFEE_GR_STAGE_MIN_BLOCKS : 3) gr_stage_kernel(const __grid_constant__ GrConst<T> c,
                                                       const F7<T> u, const F7<T> eh,
                                                       const F7<T> out, const F7<T> du,
                                                       const F7<T> un, const F5<T> aux,
                                                       const T* __restrict__ mt,
                                                       const T* __restrict__ sgt, const T As,
                                                       const T Bs, const int flags,
                                                       const F7<T> ehout) {
  const int i = c.lo[0] + blockIdx.x * blockDim.x + threadIdx.x;
  const int j = c.lo[1] + blockIdx.y * blockDim.y + threadIdx.y;
  const int k = c.lo[2] + blockIdx.z * blockDim.z + threadIdx.z;
  if (i >= c.hi[0] || j >= c.hi[1] || k >= c.hi[2]) return;
  const uint32_t sy = (uint32_t)c.d[0], sz = sy * (uint32_t)c.d[1];
  const uint32_t o = (uint32_t)i + sy * (uint32_t)j + sz * (uint32_t)k;
  const T x = gr_pos(c, 0, i), y = gr_pos(c, 1, j), z = gr_pos(c, 2, k);
  auto metric = [&]() { return metric_at(c, mt, i, j, k, x, y, z); };
  // the array pointers straight from the kernel parameters (a local array
  // of them would take registers this kernel does not have); 32-bit element
  // offsets (gr_check), so an address is one wide multiply-add, and the x
  // neighbours are immediate offsets from the point's own address
  auto fetch = [&](auto qc, auto ac, int n) {
    constexpr int q = decltype(qc)::value, ax = decltype(ac)::value;
    const T* p;
    if constexpr (q < 6) p = eh.p[q];
    else if constexpr (q < 13) p = u.p[q - 6];
    else p = sgt;
    if constexpr (ax == 0) return __ldg(p + o + n);
    else return __ldg(p + (uint32_t)(o + (uint32_t)n * (ax == 1 ? sy : sz)));
  };
  auto own = [&](int q) { return __ldg((q < 6 ? eh.p[q] : u.p[q - 6]) + o); };
  gr_stage_point<T, FIRST>(c, metric, x, y, z, o, fetch, own, out, du, un, aux, As, Bs, flags,
                           ehout);
}

// The same stage streamed along z through shared memory (FP32; opt-in with
// COFFEE_GR_TILED=1).  A CTA owns a 32 x 8 column of points and a chunk of
// z planes; each plane of the 14 stencil arrays (E, H, D, B, P,
// sqrt(gamma)) with its 2-point x / y halo is copied by cp.async into a ring
// of kGrRing planes ahead of the one computed, and the z neighbours of the
// point's own column of the 8 arrays that are differentiated along z (E_x,
// E_y, H_x, H_y, D_z, B_z, P, sqrt(gamma)) are kept in a register window of
// planes k-2 .. k+2.  The per-point global stencil loads of gr_stage_kernel
// become one coalesced copy per array and plane, but the metric, the
// near-horizon table and the per-point reads and writes of dU, the
// start-of-step copy, J and E, H keep the kernel latency-bound, and the
// registers and shared memory of the tiles leave too few warps to hide it.
// Measured at 256^3 (the Wald run): 5 slots and one CTA per SM 2.50 ms per
// stage, 4 slots and two CTAs per SM 1.61 ms, the per-point gr_stage_kernel
// 1.09 ms, which stays the default.
#ifndef COFFEE_GR_TILE_RING
#define COFFEE_GR_TILE_RING 4
#endif
#ifndef COFFEE_GR_TILE_MINB
#define COFFEE_GR_TILE_MINB 2
#endif
// ring slots: planes k .. k+2, PF = kGrRing - 4 planes in flight, the spare
constexpr int kGrTX = 32, kGrTY = 8, kGrRing = COFFEE_GR_TILE_RING, kGrArrays = 14;
constexpr int kGrPF = kGrRing - 4;
static_assert(kGrPF == 0 || kGrPF == 1, "a ring of 4 or 5 planes");
constexpr int kGrSX = kGrTX + 4, kGrSP = kGrSX * (kGrTY + 4);
#ifndef COFFEE_GR_KCHUNK
#define COFFEE_GR_KCHUNK 64
#endif

__host__ __device__ constexpr size_t gr_tile_smem_bytes() {
  return (size_t)kGrRing * kGrArrays * kGrSP * sizeof(float);
}

// window slot of array q (only the 8 arrays differentiated along z)
template <int Q>
__device__ __forceinline__ constexpr int gr_wslot() {
  return Q == 0 ? 0 : Q == 1 ? 1 : Q == 3 ? 2 : Q == 4 ? 3 : Q == 8 ? 4 : Q == 11 ? 5 : Q == 12 ? 6 : 7;
}

template <bool FIRST>
__global__ void __launch_bounds__(kGrTX * kGrTY, COFFEE_GR_TILE_MINB) gr_stage_tile_kernel(
    const __grid_constant__ GrConst<float> c, const F7<float> u, const F7<float> eh,
    const F7<float> out, const F7<float> du, const F7<float> un, const F5<float> aux,
    const float* __restrict__ mt, const float* __restrict__ sgt, const float As, const float Bs,
    const int flags, const F7<float> ehout, const int kchunk) {
  constexpr int NT = kGrTX * kGrTY, NLOAD = (kGrSP + NT - 1) / NT;
  constexpr int WQ[8] = {0, 1, 3, 4, 8, 11, 12, 13};  // the window's arrays
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float* ring = reinterpret_cast<float*>(smem_raw);  // [kGrRing][kGrArrays][kGrSP]
  const uint32_t rbase = smem_u32(smem_raw);
  const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * kGrTX + tx;
  const int i = c.lo[0] + blockIdx.x * kGrTX + tx;
  const int j = c.lo[1] + blockIdx.y * kGrTY + ty;
  const int k0 = c.lo[2] + blockIdx.z * kchunk;
  const int k1 = min(k0 + kchunk, c.hi[2]);
  const bool active = i < c.hi[0] && j < c.hi[1];
  const long long sy = c.d[0], sz = (long long)c.d[0] * c.d[1];
  const float* arr[kGrArrays] = {eh.p[0], eh.p[1], eh.p[2], eh.p[3], eh.p[4],
                                 eh.p[5], u.p[0],  u.p[1],  u.p[2],  u.p[3],
                                 u.p[4],  u.p[5],  u.p[6],  sgt};
  // this thread's copies of a plane: tile point e -> shared slot, global offset
  const int gx0 = c.lo[0] + (int)blockIdx.x * kGrTX - 2, gy0 = c.lo[1] + (int)blockIdx.y * kGrTY - 2;
  int soff[NLOAD];
  long long goff[NLOAD];
  bool lv[NLOAD];
#pragma unroll
  for (int m = 0; m < NLOAD; ++m) {
    const int e = tid + m * NT, r = e / kGrSX, cl = e - r * kGrSX;
    lv[m] = e < kGrSP && gx0 + cl < c.d[0] && gy0 + r < c.d[1];
    soff[m] = e;
    goff[m] = (long long)(gy0 + r) * sy + gx0 + cl;
  }
  const int kend = k1 + 2;  // planes [k0 - 2, k1 + 2) are read
  auto slot_of = [&](int kp) { return (kp - k0) % kGrRing; };
  auto issue = [&](int kp) {
    if (kp < kend) {
      const uint32_t sb = rbase + (uint32_t)(slot_of(kp) * kGrArrays * kGrSP) * 4u;
#pragma unroll
      for (int m = 0; m < NLOAD; ++m) {
        if (!lv[m]) continue;
        const long long g = (long long)kp * sz + goff[m];
#pragma unroll
        for (int q = 0; q < kGrArrays; ++q)
          cp_async<4>(sb + (uint32_t)(q * kGrSP + soff[m]) * 4u, arr[q] + g);
      }
    }
    cp_async_commit();
  };
#pragma unroll 1
  for (int p = 0; p < 3 + kGrPF; ++p) issue(k0 + p);

  const int own = (ty + 2) * kGrSX + tx + 2;
  const long long ocol = (long long)j * sy + i;
  // window: w[s][q'] = array WQ[q'] at (i, j, k - 2 + s)
  float w[5][8];
  if (active) {
#pragma unroll
    for (int s2 = 0; s2 < 4; ++s2)
#pragma unroll
      for (int q = 0; q < 8; ++q) w[s2][q] = arr[WQ[q]][(long long)(k0 - 2 + s2) * sz + ocol];
  }
#pragma unroll 1
  for (int k = k0; k < k1; ++k) {
    cp_async_wait<kGrPF>();  // planes up to k + 2 have landed
    __syncthreads();
    issue(k + 3 + kGrPF);    // into the slot of plane k - 1
    if (active) {
      const float* cs = ring + slot_of(k) * kGrArrays * kGrSP;
      const float* c2 = ring + slot_of(k + 2) * kGrArrays * kGrSP;
#pragma unroll
      for (int q = 0; q < 8; ++q) w[4][q] = c2[WQ[q] * kGrSP + own];
      auto fetch = [&](auto qc, auto ac, int n) -> float {
        constexpr int q = decltype(qc)::value, ax = decltype(ac)::value;
        if constexpr (ax == 2) return w[2 + n][gr_wslot<q>()];
        else if constexpr (ax == 0) return cs[q * kGrSP + own + n];
        else return cs[q * kGrSP + own + n * kGrSX];
      };
      auto ownv = [&](int q) { return cs[q * kGrSP + own]; };
      const float x = gr_pos(c, 0, i), y = gr_pos(c, 1, j), z = gr_pos(c, 2, k);
      auto metric = [&]() { return metric_at(c, mt, i, j, k, x, y, z); };
      gr_stage_point<float, FIRST>(c, metric, x, y, z, (uint32_t)(k * sz + ocol), fetch, ownv, out,
                                   du, un, aux, As, Bs, flags, ehout);
#pragma unroll
      for (int s2 = 0; s2 < 4; ++s2)
#pragma unroll
        for (int q = 0; q < 8; ++q) w[s2][q] = w[s2 + 1][q];
    }
  }
  cp_async_wait<0>();
}

// Kreiss-Oliger pass (kernel_KO_step1_gr / _step2_gr, :523-608, with the
// 3D 6th difference of finite_diff.h:84-92), then the clamps (:895-900).
template <typename T>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? COFFEE_GR_KO_MIN_BLOCKS : 2) gr_ko_kernel(const __grid_constant__ GrConst<T> c,
                                                    const F7<T> u, const F7<T> out,
                                                    const T* __restrict__ mt,
                                                    const F7<T> ehout) {
  const int i = c.lo[0] + blockIdx.x * blockDim.x + threadIdx.x;
  const int j = c.lo[1] + blockIdx.y * blockDim.y + threadIdx.y;
  const int k = c.lo[2] + blockIdx.z * blockDim.z + threadIdx.z;
  if (i >= c.hi[0] || j >= c.hi[1] || k >= c.hi[2]) return;
  const uint32_t sy = (uint32_t)c.d[0], sz = sy * (uint32_t)c.d[1];
  const uint32_t o = (uint32_t)i + sy * (uint32_t)j + sz * (uint32_t)k;
  auto at = [&](const T* p, int ax, int n) {
    if (ax == 0) return __ldg(p + o + n);
    return __ldg(p + (uint32_t)(o + (uint32_t)n * (ax == 1 ? sy : sz)));
  };
  // the 6th differences, one chain per axis from one end to the other, where the
  // running sum stays below 10 fields (as sph_ko_point)
  Pair<T> db[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const T *pd = u.p[a], *pb = u.p[3 + a];
    Pair<T> t[3];
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
      t[ax] = pk(at(pd, ax, -3), at(pb, ax, -3));
#pragma unroll
      for (int n = 1; n < 7; ++n)
        t[ax] = pfma(pk(at(pd, ax, n - 3), at(pb, ax, n - 3)), both(diff6<T>(n)), t[ax]);
    }
    db[a] = pfma(padd(padd(t[0], t[1]), t[2]), both(c.ko_c), pk(__ldg(pd + o), __ldg(pb + o)));
  }
  T P;
  {
    const T* p = u.p[6];
    T t[3];
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
      t[ax] = at(p, ax, -3);
#pragma unroll
      for (int n = 1; n < 7; ++n) t[ax] = sfma(at(p, ax, n - 3), diff6<T>(n), t[ax]);
    }
    P = sfma(t[0] + t[1] + t[2], c.ko_c, __ldg(p + o));
  }
  const Cks<T> m =
      metric_at(c, mt, i, j, k, gr_pos(c, 0, i), gr_pos(c, 1, j), gr_pos(c, 2, k));
  gr_clamps(c, m, db);
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    out.p[a][o] = first(db[a]);
    out.p[3 + a][o] = second(db[a]);
  }
  out.p[6][o] = P;
  if (ehout.p[0]) gr_eh_store(m, db, ehout, o);
}

}  // namespace coffee
