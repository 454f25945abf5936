// Kernels of the two 2D axisymmetric EZ solvers: log-spherical (x = ln r,
// y = theta; reference src/algorithms/field_solver_EZ_spherical.cu) and
// cylindrical (x = R, y = z; src/algorithms/field_solver_EZ_cylindrical.cu).
//
// Both run on one plane of (d0 x d1) points stored as the flat solver's
// arrays (i fastest).  A stage is one launch over the update box
// [guard - shift, dims - guard + shift) of axes 0 and 1 that reads the
// current buffer and writes the other one (the reference's rk_step1 ->
// rk_step2 -> clamps -> point boundaries, with no intermediate arrays); the
// non-local axis boundaries are written by the threads that own their source
// points.  These grids are small enough (a few million points) that the
// stencil neighbours of a warp are served from L1/L2; the kernels read
// global memory directly.
#pragma once

#include "coffee_b200.h"
#include "ez_common.cuh"
#include "ez_pair.cuh"

namespace coffee {

enum AxiFlags { AX_LAST = 1, AX_AUX = 2, AX_WRITE_UN = 4 };

// CTAs of 256 threads kept resident per SM (bounds the registers per thread;
// the kernels are latency-bound on their stencil loads, so more warps help,
// until spilling costs more).  Measured, us a step: log-spherical 2048 x 1024 with 8
// (32 registers) / 6 / 5 / 4: 554 / 496 / 506 / 522, 512 x 256 67 / 66 / 63 / 55; FP64
// with 8 / 6 / 5 / 4 / 3: 1748 / 1203 / 987 / 893 / 984.  Four batched runs (whose
// parameters come from shared memory) with 4 (64) / 5 / 6: 863 / 832 / 809, the persistent
// launch 1038 / 1056 / 1086; FP64 with 5 / 4 / 3 / 2: 1532 / 1425 / 1487 / 1711.
// Cylindrical 1024 x 2048, stage and KO with 4 (64) and 4 / 3 and 5 / 5 and 3: 449 / 492
// / 459; FP64 772 / 809 / 855.
#ifndef COFFEE_SPH_MIN_BLOCKS
#define COFFEE_SPH_MIN_BLOCKS 6
#endif
#ifndef COFFEE_SPH_MIN_BLOCKS_F64
#define COFFEE_SPH_MIN_BLOCKS_F64 4
#endif
#ifndef COFFEE_SPH_BATCH_MIN_BLOCKS_F64
#define COFFEE_SPH_BATCH_MIN_BLOCKS_F64 4
#endif
#ifndef COFFEE_SPH_BATCH_MIN_BLOCKS
#define COFFEE_SPH_BATCH_MIN_BLOCKS 5
#endif
#ifndef COFFEE_CYL_STAGE_MIN_BLOCKS
#define COFFEE_CYL_STAGE_MIN_BLOCKS 4
#endif
#ifndef COFFEE_CYL_KO_MIN_BLOCKS
#define COFFEE_CYL_KO_MIN_BLOCKS 4
#endif
template <typename T>
constexpr int kSphMinBlocks = sizeof(T) == 4 ? COFFEE_SPH_MIN_BLOCKS : COFFEE_SPH_MIN_BLOCKS_F64;
template <typename T>
constexpr int kSphBatchMinBlocks =
    sizeof(T) == 4 ? COFFEE_SPH_BATCH_MIN_BLOCKS : COFFEE_SPH_BATCH_MIN_BLOCKS_F64;
constexpr int kCylStageMinBlocks = COFFEE_CYL_STAGE_MIN_BLOCKS;
constexpr int kCylKoMinBlocks = COFFEE_CYL_KO_MIN_BLOCKS;

// Load of a field value.  NC: through the read-only data path (__ldg), for
// kernels in which nothing writes the array; otherwise a plain load, as the
// persistent batch kernel needs: it reads in one phase what other CTAs wrote
// in an earlier phase of the same launch, which the read-only path does not
// promise to see.
template <bool NC, typename T>
__device__ __forceinline__ T ldf(const T* p) {
  if constexpr (NC) return __ldg(p);
  else return *p;
}

// ---- parameter block of the log-spherical solver ------------------------
template <typename T>
struct SphConst {
  int d0, d1;
  int lo0, hi0, lo1, hi1;  // update box
  int axis_lo, axis_hi;    // theta = 0 / theta = pi rows, -1 if not on the grid
  int g0, g1;              // guards: x_i = x0 + dx * (i - g0), y_j = y0 + dy * (j - g1)
  T dx, dy, inv_dx, inv_dy, x0, y0;
  T dt, ch2, tau, inv_tau, gam_dt, ko_c;
  int calc_current, edotb, divB_clean, clean_ep, check_egb, ko_geometry;
  T radius, b0, omega;
  T tp_start, tp_end, dw0, nT, thp1, thp2;
  T tp_start1, tp_end1, dw1, nT1, thp11, thp21;
  int absorbing;
  T xh, rh, pmllen, sigpml;
  const T* rt;  // r_i = exp(x_i), i in [0, d0)
  const T* st;  // sin(theta_j), j in [0, d1)
  const T* ct;  // cos(theta_j)
};

// ---- parameter block of the cylindrical solver --------------------------
template <typename T>
struct CylConst {
  int d0, d1;
  int lo0, hi0, lo1, hi1;
  int axis_col;  // the R = 0 column, -1 if not on the grid
  int g0, g1;    // guards: R_i = R0 + dR * (i - g0), z_j = z0 + dz * (j - g1)
  T dR, dz, inv_dR, inv_dz, R0, z0;
  T dt, ch2, tau, inv_tau, ko_c;
  int clean_ep, check_egb;
  T radius, b0, omega;
  T tp_start, tp_end, dw0, th1, th2;  // wpert window in theta (precomputed)
  int absorbing;
  T xh, xl, yh, yl, pmlscale, sigpml;
};

// The four weights of diff1_4 (src/algorithms/finite_diff.h:14-19) and the seven of
// the 6th difference.
template <typename T>
__device__ __forceinline__ constexpr T diff4(int k) {
  return T(k == 0 ? 1 : k == 1 ? -8 : k == 2 ? 8 : -1);
}
template <typename T>
__device__ __forceinline__ constexpr T diff6(int k) {
  return T(k == 0 || k == 6 ? 1 : k == 1 || k == 5 ? -6 : k == 3 ? -20 : 15);
}

// Stencil values around one point of (E_a, B_a) pairs or single fields, at offset k
// along x (immediate offsets from the point's address) or y (one 32-bit element
// offset per row; an array of these 2D grids has far fewer than 2^31 points).
// NC as for ldf.
template <bool NC, typename T>
struct Stencil2D {
  const F7<T>& u;
  uint32_t o, d0;
  __device__ __forceinline__ T x(int f, int k) const { return ldf<NC>(u.p[f] + o + k); }
  __device__ __forceinline__ T y(int f, int k) const {
    return ldf<NC>(u.p[f] + (uint32_t)(o + (uint32_t)k * d0));
  }
  __device__ __forceinline__ Pair<T> px(int a, int k) const { return pk(x(a, k), x(3 + a, k)); }
  __device__ __forceinline__ Pair<T> py(int a, int k) const { return pk(y(a, k), y(3 + a, k)); }
  // sum of w[k] times the pair a at the four points of diff1_4, or its own sum (before
  // its 1 / 12) in its order
  __device__ __forceinline__ Pair<T> dx(int a, const T w[4]) const {
    Pair<T> t = pmul(px(a, -2), both(w[0]));
    t = pfma(px(a, -1), both(w[1]), t);
    t = pfma(px(a, 1), both(w[2]), t);
    return pfma(px(a, 2), both(w[3]), t);
  }
  __device__ __forceinline__ Pair<T> dy(int a, const T w[4]) const {
    Pair<T> t = pmul(py(a, -2), both(w[0]));
    t = pfma(py(a, -1), both(w[1]), t);
    t = pfma(py(a, 1), both(w[2]), t);
    return pfma(py(a, 2), both(w[3]), t);
  }
  __device__ __forceinline__ Pair<T> dx(int a) const {
    return psub(pfma(px(a, 1), both(T(8)), pfma(px(a, -1), both(T(-8)), px(a, -2))), px(a, 2));
  }
  __device__ __forceinline__ Pair<T> dy(int a) const {
    return psub(pfma(py(a, 1), both(T(8)), pfma(py(a, -1), both(T(-8)), py(a, -2))), py(a, 2));
  }
  __device__ __forceinline__ T dx1(int f) const {
    return sfma(T(8), x(f, 1) - x(f, -1), x(f, -2) - x(f, 2));
  }
  __device__ __forceinline__ T dy1(int f) const {
    return sfma(T(8), y(f, 1) - y(f, -1), y(f, -2) - y(f, 2));
  }
};

// ---- log-spherical helpers ----------------------------------------------
// wpert_sph_angle (field_solver_EZ_spherical.cu:576-595)
template <typename T>
__device__ __noinline__ T sph_wpert_angle(T t, T th, T tp_start, T tp_end, T dw0, T nT, T thp1,
                                          T thp2) {
  if (thp1 > thp2) {
    const T tmp = thp1;
    thp1 = thp2;
    thp2 = tmp;
  }
  const T mu = (thp1 + thp2) * T(0.5);
  if (t >= tp_start && t <= tp_end && th >= thp1 && th <= thp2) {
    const double a = cos((double)(th - mu) * M_PI / (double)(thp2 - thp1));
    const double b = sin((double)(t - tp_start) * M_PI / (double)(tp_end - tp_start));
    const double c = sin((double)(t - tp_start) * 2.0 * M_PI * (double)nT /
                         (double)(tp_end - tp_start));
    return (T)((double)dw0 * (a * a) * (b * b) * c);
  }
  return T(0);
}

// Star surface and interior of the log-spherical run
// (kernel_boundary_pulsar_sph, field_solver_EZ_spherical.cu:617-688).
template <typename T>
__device__ __noinline__ V7<T> sph_pulsar(const SphConst<T>& c, V7<T> v, T r, T sn, T cs, T th,
                                         T t) {
  if (!(r < c.radius + c.dx)) return v;
  const T w = c.omega +
              sph_wpert_angle(t, th, c.tp_start, c.tp_end, c.dw0, c.nT, c.thp1, c.thp2) +
              sph_wpert_angle(t, th, c.tp_start1, c.tp_end1, c.dw1, c.nT1, c.thp11, c.thp21);
  const T r3 = r * r * r;
  const T bxn = c.b0 * (T(2) * cs / r3);
  const T byn = c.b0 * (sn / r3);
  const T v3n = w * r * sn;
  const T exn = v3n * byn;
  const T eyn = -v3n * bxn;
  const T g11s = r;  // sqrt(r^2)
  const T g22s = r;
  if (fabs(r - c.radius) < c.dx * T(0.5)) {
    v.v[3] = fdiv(bxn, g11s);
    v.v[1] = fdiv(eyn, g22s);
    v.v[2] = T(0);
  } else if (r < c.radius - Tiny<T>::v) {
    v.v[3] = fdiv(bxn, g11s);
    v.v[4] = fdiv(byn, g22s);
    v.v[5] = T(0);  // bzn / g33 with bzn = 0
    v.v[0] = fdiv(exn, g11s);
    v.v[1] = fdiv(eyn, g22s);
    v.v[2] = T(0);
  }
  return v;
}

// E.B = 0 and |E| <= |B| with the diagonal metric
// (kernel_Epar_sph / kernel_EgtB_sph, field_solver_EZ_spherical.cu:361-442).
template <typename T>
__device__ __forceinline__ void sph_clamps(const SphConst<T>& c, T* v, T g11, T g33) {
  if (c.clean_ep) {
    T B2 = g11 * v[3] * v[3] + g11 * v[4] * v[4] + g33 * v[5] * v[5];
    if (B2 < Tiny<T>::v) B2 = Tiny<T>::v;
    const T EB = g11 * v[0] * v[3] + g11 * v[1] * v[4] + g33 * v[2] * v[5];
    const T q = fdiv(EB, B2);
    v[0] -= q * v[3];
    v[1] -= q * v[4];
    v[2] -= q * v[5];
  }
  if (c.check_egb) {
    T B2 = g11 * v[3] * v[3] + g11 * v[4] * v[4] + g33 * v[5] * v[5];
    if (B2 < Tiny<T>::v) B2 = Tiny<T>::v;
    const T E2 = g11 * v[0] * v[0] + g11 * v[1] * v[1] + g33 * v[2] * v[2];
    if (E2 > B2) {
      const T s = sqrt(fdiv(B2, E2));
      v[0] *= s;
      v[1] *= s;
      v[2] *= s;
    }
  }
}

// Absorbing layer in r (kernel_boundary_absorbing_sph,
// field_solver_EZ_spherical.cu:758-802): blend towards the start-of-step
// values where x > xh.
template <typename T>
__device__ __noinline__ V7<T> sph_absorb(const SphConst<T>& c, V7<T> v, V7<T> n, T x, T r) {
  if (!(x > c.xh)) return v;
  T sig = T(0);
  if (r > c.rh) {
    const T q = (r - c.rh) / c.pmllen;
    sig = c.sigpml * q * q * q;
  }
  if (sig > Tiny<T>::v) {
    const T e = exp(-sig);
    const T f = (T(1) - e) / sig;
    for (int a = 0; a < 6; ++a) v.v[a] = e * n.v[a] + f * (v.v[a] - n.v[a]);
  }
  return v;
}

// Stores the new values w of point (i, j) together with the axis boundary
// that follows every pass (kernel_boundary_axis_sph,
// field_solver_EZ_spherical.cu:690-748): on the theta = 0 row E_r, B_r, P take
// the next row's values and the other components vanish, and the three rows
// beyond the axis mirror E and B of the rows inside with the parity of each
// component; the theta = pi row (the first guard row) likewise.  So the
// threads of the three rows next to an axis also write their mirror rows, the
// one next to it also the axis row, and a thread on a row that another one
// writes stores only what the axis boundary leaves alone: nothing on the axis,
// P beyond it (rows that are in the box with shift_ghost > 0 only).  As a
// launch of its own, one thread per column, the boundary cost 20 us after
// each 80 us stage at 2048 x 1024 (one chain of dependent accesses).
template <typename T>
__device__ __forceinline__ void sph_store(const SphConst<T>& c, const int j, const uint32_t o32,
                                          const V7<T>& w, const F7<T>& out) {
  const long long o = o32;
  // rows above theta = 0 and below theta = pi (far from an axis not on the grid)
  const int up = c.axis_lo >= 0 ? j - c.axis_lo : 1 << 20;
  const int down = c.axis_hi >= 0 ? c.axis_hi - j : 1 << 20;
  if (min(up, down) > 3) {
#pragma unroll
    for (int a = 0; a < 7; ++a) out.p[a][o] = w.v[a];
    return;
  }
  if (up == 0 || down == 0) return;
  out.p[6][o] = w.v[6];
  if ((up < 0 && up >= -3) || (down < 0 && down >= -3)) return;
#pragma unroll
  for (int a = 0; a < 6; ++a) out.p[a][o] = w.v[a];
#pragma unroll 1
  for (int side = 0; side < 2; ++side) {
    const int l = side == 0 ? up : down;
    if (l < 1 || l > 3) continue;
    const long long d = side == 0 ? -(long long)c.d0 : (long long)c.d0;  // towards the axis
    const long long m = o + 2 * l * d;
    out.p[0][m] = w.v[0];
    out.p[1][m] = -w.v[1];
    out.p[2][m] = -w.v[2];
    out.p[3][m] = w.v[3];
    out.p[4][m] = -w.v[4];
    out.p[5][m] = -w.v[5];
    if (l == 1) {
      const long long x = o + d;
      out.p[0][x] = w.v[0];
      out.p[1][x] = T(0);
      out.p[2][x] = T(0);
      out.p[3][x] = w.v[3];
      out.p[4][x] = T(0);
      out.p[5][x] = T(0);
      out.p[6][x] = w.v[6];
    }
  }
}

// One LSRK stage of the log-spherical solver at point (i, j):
// kernel_compute_ElBl + kernel_rk_step1_sph + kernel_rk_step2_sph, then
// kernel_Epar_sph, kernel_EgtB_sph, kernel_boundary_pulsar_sph and, in the
// last stage, kernel_boundary_absorbing_sph (field_solver_EZ_spherical.cu:
// 175-802, order of :967-990).  FIRST: As = 0, dU is not read.  NC: field
// loads through the read-only path (ldf).
template <typename T, bool FIRST, bool NC = true>
__device__ __forceinline__ void sph_stage_point(const SphConst<T>& c, const int i, const int j,
                                                const F7<T>& u, const F7<T>& out,
                                                const F7<T>& du, const F7<T>& un,
                                                const F5<T>& aux, const T As, const T Bs,
                                                const T tst, const int flags) {
  const uint32_t d0 = (uint32_t)c.d0;
  const uint32_t o = (uint32_t)i + (uint32_t)j * d0;
  const Stencil2D<NC, T> st{u, o, d0};
  const T rc = __ldg(c.rt + i), sc = __ldg(c.st + j), asc = fabs(sc);
  const T g11 = rc * rc;
  const T g33 = (rc * sc) * (rc * sc);
  T gms = rc * rc * rc * asc;
  if (gms < Tiny<T>::v) gms = Tiny<T>::v;
  const T igms = T(1) / gms;

  // The lowered fields (El_x = r^2 E_x, El_y = r^2 E_y, El_z = (r sin th)^2 E_z,
  // metric_sph.h:90-122) and sqrt(gamma) = r^3 |sin th| of div4_sph
  // (field_solver_EZ_spherical.cu:99-124) are products of a power of r and one of
  // sin th: a derivative along r is summed with the weights of diff1_4 times the
  // power of r, one along theta with those times the power of sin th, both formed
  // once for the E and B of a pair.  What the four points share scales the finished
  // sum, and what both derivatives of a curl or divergence share scales their sum:
  // these sums cancel, and a factor multiplied into a weight or into one of two
  // derivatives rounds it to a value that no longer matches the others, at a point the
  // same one in every stage (B_theta and P of a run 5% farther from 64 bits).
  T r2[4], r3[4], s1[4], s2[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int n = k < 2 ? k - 2 : k - 1;
    const T r = __ldg(c.rt + i + n), sn = __ldg(c.st + j + n);
    r2[k] = diff4<T>(k) * (r * r);
    r3[k] = diff4<T>(k) * (r * r * r);
    s1[k] = diff4<T>(k) * fabs(sn);
    s2[k] = diff4<T>(k) * (sn * sn);
  }
  // (rot E, rot B) and (div E, div B)
  Pair<T> rot[3] = {pmul(st.dy(2, s2), both(c.inv_dy * g11)),
                    pmul(st.dx(2, r2), both(-c.inv_dx * (sc * sc))),
                    pfma(st.dx(1, r2), both(c.inv_dx), pmul(st.dy(0), both(-c.inv_dy * g11)))};
  Pair<T> dvg = pfma(st.dx(0, r3), both(c.inv_dx * asc),
                     pmul(st.dy(1, s1), both(c.inv_dy * (g11 * rc))));
  const T igms12 = igms * T(1.0 / 12.0);
#pragma unroll
  for (int a = 0; a < 3; ++a) rot[a] = pmul(rot[a], both(igms12));
  dvg = pmul(dvg, both(igms12));
  const T divE = first(dvg), divB = second(dvg);

  Pair<T> eb[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) eb[a] = st.px(a, 0);
  const T P = st.x(6, 0);
  T J[3] = {T(0), T(0), T(0)};
  if (c.calc_current) {
    const Pair<T> low[3] = {pmul(eb[0], both(g11)), pmul(eb[1], both(g11)), pmul(eb[2], both(g33))};
    const Pair<T> sq = pdot3(eb, low), lr = pdot3(low, rot);  // (E2, B2), (E.rotE, B.rotB)
    T B2 = second(sq);
    if (B2 < Tiny<T>::v) B2 = Tiny<T>::v;
    T Jp = second(lr) - first(lr);
    const T el[3] = {first(low[0]), first(low[1]), first(low[2])};
    const T bl[3] = {second(low[0]), second(low[1]), second(low[2])};
    const T C[3] = {el[1] * bl[2] - el[2] * bl[1], el[2] * bl[0] - el[0] * bl[2],
                    el[0] * bl[1] - el[1] * bl[0]};
    if (c.edotb) {
      const T chi2 = B2 - first(sq);
      const T EdotB = first(eb[0]) * bl[0] + first(eb[1]) * bl[1] + first(eb[2]) * bl[2];
      const T E02 = T(0.5) * (sqrt(chi2 * chi2 + T(4) * EdotB * EdotB) - chi2);
      Jp += c.gam_dt * EdotB;
      const T a = fdiv(divE * igms, E02 + B2);
      const T q = fdiv(Jp, B2);
#pragma unroll
      for (int n = 0; n < 3; ++n) J[n] = a * C[n] + q * second(eb[n]);
    } else {
      const T iB2 = fdiv(T(1), B2);
#pragma unroll
      for (int n = 0; n < 3; ++n) J[n] = (divE * C[n] * igms + Jp * second(eb[n])) * iB2;
    }
  }
  T gP[3] = {T(0), T(0), T(0)};
  if (c.divB_clean) {
    gP[0] = fdiv(st.dx1(6) * (c.inv_dx * T(1.0 / 12.0)), g11);
    gP[1] = fdiv(st.dy1(6) * (c.inv_dy * T(1.0 / 12.0)), g11);
    // Pz = dfdz(P) / gamma_33 with dfdz = 0; the reference's 0/0 on the
    // theta = 0 row only reaches dB_z of that row, which the axis
    // boundary overwrites.
  }
  const T dt = c.dt;
  if (flags & AX_WRITE_UN) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      un.p[a][o] = first(eb[a]);
      un.p[3 + a][o] = second(eb[a]);
    }
  }
  T v[7];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    Pair<T> d = pmul(pk(second(rot[a]) - J[a], first(rot[a]) + gP[a]), pk(dt, -dt));
    if constexpr (!FIRST) d = pfma(pk(du.p[a][o], du.p[3 + a][o]), both(As), d);
    du.p[a][o] = first(d);
    du.p[3 + a][o] = second(d);
    const Pair<T> n = pfma(d, both(Bs), eb[a]);
    v[a] = first(n);
    v[3 + a] = second(n);
  }
  {
    T d = -dt * c.ch2 * divB - div_const(P, c.tau, c.inv_tau);
    if constexpr (!FIRST) d = sfma(du.p[6][o], As, d);
    du.p[6][o] = d;
    v[6] = sfma(d, Bs, P);
  }
  if (flags & AX_AUX) {
    aux.p[0][o] = J[0];
    aux.p[1][o] = J[1];
    aux.p[2][o] = J[2];
    aux.p[3][o] = divE;
    aux.p[4][o] = divB;
  }
  sph_clamps(c, v, g11, g33);
  V7<T> w;
#pragma unroll
  for (int a = 0; a < 7; ++a) w.v[a] = v[a];
  // the out-of-line boundary code is entered only where it can act
  if (rc < c.radius + c.dx) {
    const T th = c.y0 + c.dy * (T)(j - c.g1);
    w = sph_pulsar(c, w, rc, sc, __ldg(c.ct + j), th, tst);
  }
  const T xi = c.x0 + c.dx * (T)(i - c.g0);
  if ((flags & AX_LAST) && c.absorbing && xi > c.xh) {
    V7<T> n;
#pragma unroll
    for (int a = 0; a < 6; ++a) n.v[a] = un.p[a][o];
    n.v[6] = T(0);
    w = sph_absorb(c, w, n, xi, rc);
  }
  sph_store(c, j, o, w, out);
}

template <typename T, bool FIRST>
__global__ void __launch_bounds__(256, kSphMinBlocks<T>) sph_stage_kernel(const __grid_constant__ SphConst<T> c,
                                                        const F7<T> u, const F7<T> out,
                                                        const F7<T> du, const F7<T> un,
                                                        const F5<T> aux, const T As,
                                                        const T Bs, const T tst,
                                                        const int flags) {
  const int i = c.lo0 + blockIdx.x * blockDim.x + threadIdx.x;
  const int j = c.lo1 + blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= c.hi0 || j >= c.hi1) return;
  sph_stage_point<T, FIRST>(c, i, j, u, out, du, un, aux, As, Bs, tst, flags);
}

// Kreiss-Oliger pass of the log-spherical solver at point (i, j):
// kernel_KO_step1_sph + kernel_KO_step2_sph, then kernel_Epar_sph,
// kernel_EgtB_sph and kernel_boundary_pulsar_sph at t + dt
// (field_solver_EZ_spherical.cu:444-555, order of :996-1004).  KO_geometry
// weights the 6th differences by sqrt(gamma) (KO_2d6, :150-173), otherwise
// they are plain (KO_2d0, :142-148).  NC as for sph_stage_point.
template <typename T, bool NC = true>
__device__ __forceinline__ void sph_ko_point(const SphConst<T>& c, const int i, const int j,
                                             const F7<T>& u, const F7<T>& out, const T tend) {
  const uint32_t d0 = (uint32_t)c.d0;
  const uint32_t o = (uint32_t)i + (uint32_t)j * d0;
  const Stencil2D<NC, T> st{u, o, d0};
  const T rc = __ldg(c.rt + i), sc = __ldg(c.st + j);
  T wx[7], wy[7], scale = c.ko_c;
  if (c.ko_geometry) {  // sqrt(gamma) at the stencil points over that of the point
    T gms = rc * rc * rc * fabs(sc);
    if (gms < Tiny<T>::v) gms = Tiny<T>::v;
    scale = c.ko_c / gms;
#pragma unroll
    for (int k = 0; k < 7; ++k) {
      const T rk = __ldg(c.rt + i - 3 + k);
      wx[k] = diff6<T>(k) * (rk * rk * rk * fabs(sc));
      wy[k] = diff6<T>(k) * (rc * rc * rc * fabs(__ldg(c.st + j - 3 + k)));
    }
  } else {
#pragma unroll
    for (int k = 0; k < 7; ++k) wx[k] = wy[k] = diff6<T>(k);
  }
  // one chain per axis from one end to the other, where the running sum stays
  // below 10 fields (a sum that starts with the point's own -40 rounds at that size)
  T v[7];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    Pair<T> tx = pmul(st.px(a, -3), both(wx[0])), ty = pmul(st.py(a, -3), both(wy[0]));
#pragma unroll
    for (int k = 1; k < 7; ++k) {
      tx = pfma(st.px(a, k - 3), both(wx[k]), tx);
      ty = pfma(st.py(a, k - 3), both(wy[k]), ty);
    }
    const Pair<T> n = pfma(padd(tx, ty), both(scale), st.px(a, 0));
    v[a] = first(n);
    v[3 + a] = second(n);
  }
  {
    T tx = st.x(6, -3) * wx[0], ty = st.y(6, -3) * wy[0];
#pragma unroll
    for (int k = 1; k < 7; ++k) {
      tx = sfma(st.x(6, k - 3), wx[k], tx);
      ty = sfma(st.y(6, k - 3), wy[k], ty);
    }
    v[6] = sfma(tx + ty, scale, st.x(6, 0));
  }
  sph_clamps(c, v, rc * rc, (rc * sc) * (rc * sc));
  V7<T> w;
#pragma unroll
  for (int a = 0; a < 7; ++a) w.v[a] = v[a];
  if (rc < c.radius + c.dx)
    w = sph_pulsar(c, w, rc, sc, __ldg(c.ct + j), c.y0 + c.dy * (T)(j - c.g1), tend);
  sph_store(c, j, o, w, out);
}

template <typename T>
__global__ void __launch_bounds__(256, kSphMinBlocks<T>) sph_ko_kernel(const __grid_constant__ SphConst<T> c,
                                                     const F7<T> u, const F7<T> out,
                                                     const T tend) {
  const int i = c.lo0 + blockIdx.x * blockDim.x + threadIdx.x;
  const int j = c.lo1 + blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= c.hi0 || j >= c.hi1) return;
  sph_ko_point(c, i, j, u, out, tend);
}

// The axis boundary of sph_store at column i of fields as they are: once per
// call, before the first stage (the stages and KO passes apply it to what
// they write).
template <typename T>
__device__ __forceinline__ void sph_axis_column(const SphConst<T>& c, const int i,
                                                const F7<T>& u) {
  const long long d0 = c.d0;
  constexpr T par[6] = {T(1), T(-1), T(-1), T(1), T(-1), T(-1)};
  for (int side = 0; side < 2; ++side) {
    const int j = side == 0 ? c.axis_lo : c.axis_hi;
    if (j < 0) continue;
    const int in = side == 0 ? 1 : -1;  // direction of the rows inside
    const long long o = i + j * d0;
    T v[3][6];  // loads before stores
#pragma unroll
    for (int l = 1; l <= 3; ++l)
#pragma unroll
      for (int a = 0; a < 6; ++a) v[l - 1][a] = u.p[a][o + in * l * d0];
    const T P = u.p[6][o + in * d0];
    u.p[0][o] = v[0][0];
    u.p[1][o] = T(0);
    u.p[2][o] = T(0);
    u.p[3][o] = v[0][3];
    u.p[4][o] = T(0);
    u.p[5][o] = T(0);
    u.p[6][o] = P;
#pragma unroll
    for (int l = 1; l <= 3; ++l)
#pragma unroll
      for (int a = 0; a < 6; ++a) u.p[a][o - in * l * d0] = par[a] * v[l - 1][a];
  }
}

template <typename T>
__global__ void sph_axis_kernel(const __grid_constant__ SphConst<T> c, const F7<T> u) {
  const int i = c.lo0 + blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= c.hi0) return;
  sph_axis_column(c, i, u);
}

// ---- batches of independent log-spherical runs ---------------------------
// One launch per phase covers every run of a batch: block b belongs to the
// run whose first block index is the largest one <= b.  The run's table
// entry (parameters and array pointers) is copied to shared memory, then the
// threads proceed exactly as the single-run kernels do.
constexpr int kSphBatchMax = 128;

template <typename T>
struct SphBatchEntry {
  SphConst<T> c;
  F7<T> A, B, dU, Un;
  F5<T> aux;
  int tile0;    // first stage/KO block of this run
  int tiles_x;  // blocks along i
  int axis0;    // first axis block of this run
  int want_aux;
  int index;    // position in the batch
};

// Times of the runs of a batch live in device memory (the current step's
// start time t and the time step dt of each run), so that one captured step
// serves every step.  A stage at t + cs dt evaluates that time exactly as the
// host loop of a single run does, in field precision with one rounding per
// operation (no fused multiply-add).
__device__ __forceinline__ float batch_time(float t, float cs, float dt) {
  return __fadd_rn(t, __fmul_rn(cs, dt));
}
__device__ __forceinline__ double batch_time(double t, double cs, double dt) {
  return __dadd_rn(t, __dmul_rn(cs, dt));
}

template <typename T>
__device__ __forceinline__ const SphBatchEntry<T>& sph_batch_entry(
    const SphBatchEntry<T>* __restrict__ tab, int n, int b, bool axis, unsigned char* buf) {
  __shared__ int m_s;
  const int tid = threadIdx.x + threadIdx.y * blockDim.x;
  const int nt = blockDim.x * blockDim.y;
  if (tid == 0) {
    int lo = 0, hi = n - 1;  // largest m with start(m) <= b
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      const int st = axis ? tab[mid].axis0 : tab[mid].tile0;
      if (st <= b) lo = mid;
      else hi = mid - 1;
    }
    m_s = lo;
  }
  __syncthreads();
  const int* src = reinterpret_cast<const int*>(tab + m_s);
  int* dst = reinterpret_cast<int*>(buf);
  for (int q = tid; q < (int)(sizeof(SphBatchEntry<T>) / 4); q += nt) dst[q] = src[q];
  __syncthreads();
  return *reinterpret_cast<const SphBatchEntry<T>*>(buf);
}

template <typename T, bool FIRST>
__global__ void __launch_bounds__(256, kSphBatchMinBlocks<T>) sph_stage_batch_kernel(
    const SphBatchEntry<T>* __restrict__ tab, const int n, const int to_b,
    const T* __restrict__ tnow, const T* __restrict__ tdt, const T cs, const T As, const T Bs,
    const int last) {
  __shared__ __align__(16) unsigned char buf[sizeof(SphBatchEntry<T>)];
  const SphBatchEntry<T>& e = sph_batch_entry(tab, n, (int)blockIdx.x, false, buf);
  const int lt = (int)blockIdx.x - e.tile0;
  const int i = e.c.lo0 + (lt % e.tiles_x) * blockDim.x + threadIdx.x;
  const int j = e.c.lo1 + (lt / e.tiles_x) * blockDim.y + threadIdx.y;
  if (i >= e.c.hi0 || j >= e.c.hi1) return;
  int flags = 0;
  if (last) flags |= AX_LAST | (e.want_aux ? AX_AUX : 0);
  if (FIRST && e.c.absorbing) flags |= AX_WRITE_UN;
  const T tst = batch_time(tnow[e.index], cs, tdt[e.index]);
  sph_stage_point<T, FIRST>(e.c, i, j, to_b ? e.A : e.B, to_b ? e.B : e.A, e.dU, e.Un, e.aux,
                            As, Bs, tst, flags);
}

template <typename T>
__global__ void __launch_bounds__(256, kSphBatchMinBlocks<T>) sph_ko_batch_kernel(
    const SphBatchEntry<T>* __restrict__ tab, const int n, const T* __restrict__ tnow,
    const T* __restrict__ tdt) {
  __shared__ __align__(16) unsigned char buf[sizeof(SphBatchEntry<T>)];
  const SphBatchEntry<T>& e = sph_batch_entry(tab, n, (int)blockIdx.x, false, buf);
  const int lt = (int)blockIdx.x - e.tile0;
  const int i = e.c.lo0 + (lt % e.tiles_x) * blockDim.x + threadIdx.x;
  const int j = e.c.lo1 + (lt / e.tiles_x) * blockDim.y + threadIdx.y;
  if (i >= e.c.hi0 || j >= e.c.hi1) return;
  sph_ko_point(e.c, i, j, e.B, e.A, batch_time(tnow[e.index], T(1), tdt[e.index]));
}

// end of a step: t += dt for every run, in field precision
template <typename T>
__global__ void sph_batch_advance_kernel(T* __restrict__ tnow, const T* __restrict__ tdt,
                                         const int n) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m < n) tnow[m] = batch_time(tnow[m], T(1), tdt[m]);
}

// axis boundary of every run's fields, once per call
template <typename T>
__global__ void sph_axis_batch_kernel(const SphBatchEntry<T>* __restrict__ tab, const int n) {
  __shared__ __align__(16) unsigned char buf[sizeof(SphBatchEntry<T>)];
  const SphBatchEntry<T>& e = sph_batch_entry(tab, n, (int)blockIdx.x, true, buf);
  if (e.c.axis_lo < 0 && e.c.axis_hi < 0) return;
  const int i = e.c.lo0 + ((int)blockIdx.x - e.axis0) * blockDim.x + threadIdx.x;
  if (i >= e.c.hi0) return;
  sph_axis_column(e.c, i, e.A);
}

// ---- the whole batch step in one persistent launch ----------------------
// One cooperative launch (every CTA resident) runs nsteps steps of every run
// of a batch: the phases of the per-phase launches (5 stages, KO), each over
// all runs, separated by grid-wide barriers.  In a phase the CTAs take
// kTicketTiles tiles at a time from a ticket counter (the tiles differ in
// cost: star and absorbing-layer points), asking for the next ticket before
// working on the current one.  On each tile a CTA runs the single-run per-point code, so
// the results are bitwise those of the per-phase launches.  The run times alternate between two
// rows of `tbuf`: during step s the stages read row s & 1 and CTA 0 writes
// t + dt into the other row, which the next step reads after the
// barriers between.
//
// Every barrier wait is bounded, by `limit_ns` of %globaltimer and by an
// iteration cap: a CTA that gives up records COFFEE_E_TIMEOUT, the barrier
// and its block in GridSync and returns, and the CTAs still waiting see the
// status and return as well, so the launch always ends.
struct GridSync {
  unsigned int count;  // arrivals so far (barrier q completes at (q + 1) * gridDim.x)
  int status;          // 0, or COFFEE_E_TIMEOUT once a wait has run out
  int where;           // index of the barrier that ran out
  int block;           // the CTA whose wait ran out first
  unsigned int tickets[2];  // tile tickets of the stage / KO phases (alternating)
};
// Tiles a CTA takes per ticket in the stage and KO phases.
constexpr int kTicketTiles = 4;
// Phase coefficients of the LSRK stages.
template <typename T>
struct LsrkCoef {
  T As[5], Bs[5], Cs[5];
};

__device__ __forceinline__ long long globaltimer_ns() {
  long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Grid-wide barrier number q (0, 1, ...).  `arrive` = false leaves this
// CTA's arrival out (the stalled-CTA test of the wait limit).  Returns
// false when the barrier gave up.
__device__ __forceinline__ bool grid_barrier(GridSync* gs, unsigned q, long long limit_ns,
                                             bool arrive) {
  __shared__ int ok_s;
  __syncthreads();
  if (threadIdx.x == 0 && threadIdx.y == 0) {
    int ok = 1;
    if (arrive) {
      __threadfence();  // this CTA's writes, seen by thread 0 through the barrier above
      atomicAdd(&gs->count, 1u);
    }
    const unsigned target = (q + 1u) * gridDim.x;
    const long long t0 = globaltimer_ns();
    const long long cap = limit_ns / 32 + 4096;  // iterations, should the timer stall
    for (long long it = 0;; ++it) {
      unsigned c;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(c) : "l"(&gs->count) : "memory");
      if (c >= target) break;
      if (*(volatile int*)&gs->status != 0) {
        ok = 0;
        break;
      }
      if (it >= cap || globaltimer_ns() - t0 > limit_ns) {
        if (atomicCAS(&gs->status, 0, (int)COFFEE_E_TIMEOUT) == 0) {
          gs->where = (int)q;
          gs->block = (int)blockIdx.x;
        }
        ok = 0;
        break;
      }
      __nanosleep(64);
    }
    __threadfence();
    ok_s = ok;
  }
  __syncthreads();
  return ok_s != 0;
}

template <typename T>
__global__ void __launch_bounds__(256, kSphBatchMinBlocks<T>) sph_batch_persistent_kernel(
    const SphBatchEntry<T>* __restrict__ tab, const int n, const int nblocks,
    T* __restrict__ tbuf, const T* __restrict__ tdt, const LsrkCoef<T> k, const int nsteps,
    GridSync* __restrict__ gs, const long long limit_ns, const int stall_block) {
  __shared__ __align__(16) unsigned char buf[sizeof(SphBatchEntry<T>)];
  const int tid = threadIdx.x + threadIdx.y * blockDim.x;
  const int nt = blockDim.x * blockDim.y;
  unsigned q = 0;  // barriers passed
  auto barrier = [&]() {
    const bool arrive = !(q == 0 && (int)blockIdx.x == stall_block);
    return grid_barrier(gs, q++, limit_ns, arrive);
  };
  // one stage (s = 0..4) or, for s = 5, the KO pass, over every tile
  __shared__ unsigned base_s;
  unsigned tp = 0;  // tile phases begun
  auto tiles = [&](const int s, const T* tcur) {
    // tile phase tp takes its tickets from counter tp & 1; the other
    // counter, last used by the tile phase before (finished at a barrier
    // before this one began), is cleared for the next
    unsigned* ctr = &gs->tickets[tp & 1];
    if (blockIdx.x == 0 && tid == 0) gs->tickets[(tp + 1) & 1] = 0u;
    ++tp;
    if (tid == 0) base_s = atomicAdd(ctr, (unsigned)kTicketTiles);
    __syncthreads();
    unsigned base = base_s;
    while (base < (unsigned)nblocks) {
      unsigned pending = 0;
      if (tid == 0) pending = atomicAdd(ctr, (unsigned)kTicketTiles);  // used after the tiles
      const int bend = min((int)base + kTicketTiles, nblocks);
      for (int b = (int)base; b < bend; ++b) {
        const SphBatchEntry<T>& e = sph_batch_entry(tab, n, b, false, buf);
        const int lt = b - e.tile0;
        const int i = e.c.lo0 + (lt % e.tiles_x) * blockDim.x + threadIdx.x;
        const int j = e.c.lo1 + (lt / e.tiles_x) * blockDim.y + threadIdx.y;
        if (i < e.c.hi0 && j < e.c.hi1) {
          if (s == 5) {
            sph_ko_point<T, false>(e.c, i, j, e.B, e.A,
                                   batch_time(tcur[e.index], T(1), tdt[e.index]));
          } else {
            const int to_b = (s % 2 == 0) ? 1 : 0;
            int flags = 0;
            if (s == 4) flags |= AX_LAST | (e.want_aux ? AX_AUX : 0);
            if (s == 0 && e.c.absorbing) flags |= AX_WRITE_UN;
            const T tst = batch_time(tcur[e.index], k.Cs[s], tdt[e.index]);
            if (s == 0)
              sph_stage_point<T, true, false>(e.c, i, j, e.A, e.B, e.dU, e.Un, e.aux, k.As[0],
                                              k.Bs[0], tst, flags);
            else
              sph_stage_point<T, false, false>(e.c, i, j, to_b ? e.A : e.B, to_b ? e.B : e.A,
                                               e.dU, e.Un, e.aux, k.As[s], k.Bs[s], tst, flags);
          }
        }
        __syncthreads();  // buf is refilled for the next tile
      }
      if (tid == 0) base_s = pending;
      __syncthreads();
      base = base_s;
    }
  };
  for (int step = 0; step < nsteps; ++step) {
    const T* tcur = tbuf + (step & 1) * n;
    if (blockIdx.x == 0)
      for (int m = tid; m < n; m += nt)
        tbuf[((step + 1) & 1) * n + m] = batch_time(tcur[m], T(1), tdt[m]);
    for (int s = 0; s < 5; ++s) {
      tiles(s, tcur);
      if (!barrier()) return;
    }
    tiles(5, tcur);
    if (!barrier()) return;
  }
}

// ---- cylindrical helpers ------------------------------------------------
// shape (src/algorithms/pulsar_impl.hpp:52-55)
template <typename T>
__device__ __forceinline__ T cyl_shape(T r, T r0, T del) {
  return T(0.5) * (T(1) - tanh((r - r0) / del));
}

// wpert of the cylindrical run (field_solver_EZ_cylindrical.cu:413-443); the
// angular window [th1, th2] = acos(sqrt(1 - 1/rpert)) is precomputed.
template <typename T>
__device__ __noinline__ T cyl_wpert(const CylConst<T>& c, T t, T R, T z) {
  const T r = sqrt(R * R + z * z);
  const T th = acos(z / r);  // NaN at the origin: no perturbation there
  const T mu = (c.th1 + c.th2) * T(0.5);
  const T s = (mu - c.th1) / T(3);
  if (t >= c.tp_start && t <= c.tp_end && th >= c.th1 && th <= c.th2) {
    const T q = (th - mu) / s;
    return c.dw0 * exp(T(-0.5) * q * q) *
           (T)sin((double)(t - c.tp_start) * 2.0 * M_PI / (double)(c.tp_end - c.tp_start)) *
           T(0.5) * (T(1) + tanh((r - T(0.5) * c.radius) / (T(0.05) * c.radius)));
  }
  return T(0);
}

// Rotating dipole star blended in over r < 2 R (kernel_boundary_pulsar_thread,
// field_solver_EZ_cylindrical.cu:445-530).  Components: 0 E_R, 1 E_z,
// 2 E_phi, 3 B_R, 4 B_z, 5 B_phi.
template <typename T>
__device__ __noinline__ V7<T> cyl_pulsar(const CylConst<T>& c, V7<T> v, T R, T z, T t) {
  T r2 = R * R + z * z;
  if (r2 < Tiny<T>::v) r2 = Tiny<T>::v;
  const T r = sqrt(r2);
  if (!(r < T(2) * c.radius)) return v;
  const T ri = T(0.5) * c.radius;
  const T sEpar = T(0.5) * c.dR, sEperp = T(0.25) * c.dR;
  const T sB = sEpar;
  const T d1 = T(4) * c.dR;
  // dipole_x / dipole_z (pulsar_impl.hpp:10-50) with alpha = phase = 0
  T rr = sqrt(R * R + z * z);
  if (fabs(rr) < Tiny<T>::v) rr = Tiny<T>::v;
  const T xn = R / rr, zn = z / rr;
  const T rr3 = rr * rr * rr + Tiny<T>::v;
  const T m3 = c.b0 * c.radius * c.radius * c.radius;
  const T bRn = m3 * ((T(3) * xn * zn) / rr3);
  const T bzn = m3 * ((T(3) * zn * zn - T(1)) / rr3);
  const T bfn = T(0);
  const T BR = v.v[3], Bz = v.v[4], Bf = v.v[5];
  const T ER = v.v[0], Ez = v.v[1], Ef = v.v[2];
  const T bnp = bRn * R + bzn * z, bp = BR * R + Bz * z;
  T s = cyl_shape(r, c.radius - d1, sB);
  T BRn = bnp * R / r2 * s + bp * R / r2 * (T(1) - s);
  T Bzn = bnp * z / r2 * s + bp * z / r2 * (T(1) - s);
  BRn += (bRn - bnp * R / r2) * s + (BR - bp * R / r2) * (T(1) - s);
  Bzn += (bzn - bnp * z / r2) * s + (Bz - bp * z / r2) * (T(1) - s);
  const T Bfn = bfn * s + Bf * (T(1) - s);
  const T w = c.omega + cyl_wpert(c, t, R, z);
  const T eRn = -w * R * Bz;
  const T ezn = w * R * BR;
  const T efn = T(0);
  const T enp = eRn * R + ezn * z, ep = ER * R + Ez * z;
  s = cyl_shape(r, c.radius, sEperp);
  T ERn = enp * R / r2 * s + ep * R / r2 * (T(1) - s);
  T Ezn = enp * z / (r * r) * s + ep * z / r2 * (T(1) - s);
  s = cyl_shape(r, c.radius, sEpar);
  ERn += (eRn - enp * R / r2) * s + (ER - ep * R / r2) * (T(1) - s);
  Ezn += (ezn - enp * z / r2) * s + (Ez - ep * z / r2) * (T(1) - s);
  const T Efn = efn * s + Ef * (T(1) - s);
  if (r < ri) {
    v.v[3] = bRn; v.v[4] = bzn; v.v[5] = bfn;
    v.v[0] = eRn; v.v[1] = ezn; v.v[2] = efn;
  } else {
    v.v[3] = BRn; v.v[4] = Bzn; v.v[5] = Bfn;
    v.v[0] = ERn; v.v[1] = Ezn; v.v[2] = Efn;
  }
  return v;
}

// pmlsigma (src/algorithms/boundary.cu:7-15)
template <typename T>
__device__ __forceinline__ T cyl_pmlsigma(T x, T xl, T xh, T scale, T sig0) {
  if (x > xh) {
    const T q = (x - xh) / scale;
    return sig0 * q * q * q;
  }
  if (x < xl) {
    const T q = (xl - x) / scale;
    return sig0 * q * q * q;
  }
  return T(0);
}

// Absorbing layer at large R and both z ends
// (kernel_boundary_absorbing_cylindrical, field_solver_EZ_cylindrical.cu:532-591).
template <typename T>
__device__ __noinline__ V7<T> cyl_absorb(const CylConst<T>& c, V7<T> v, V7<T> n, T R, T z) {
  if (!(R > c.xh || z < c.yl || z > c.yh)) return v;
  const T sig = cyl_pmlsigma(R, c.xl, c.xh, c.pmlscale, c.sigpml) +
                cyl_pmlsigma(z, c.yl, c.yh, c.pmlscale, c.sigpml);
  if (sig > Tiny<T>::v) {
    const T e = exp(-sig);
    const T f = (T(1) - e) / sig;
    for (int a = 0; a < 6; ++a) v.v[a] = e * n.v[a] + f * (v.v[a] - n.v[a]);
  }
  return v;
}

// kernel_Epar_thread / kernel_EgtB_thread (field_solver_EZ_cylindrical.cu:236-294)
template <typename T>
__device__ __forceinline__ void cyl_clamps(const CylConst<T>& c, T* v) {
  if (c.clean_ep) {
    T B2 = v[3] * v[3] + v[4] * v[4] + v[5] * v[5];
    if (B2 < Tiny<T>::v) B2 = Tiny<T>::v;
    const T q = fdiv(v[0] * v[3] + v[1] * v[4] + v[2] * v[5], B2);
    v[0] -= q * v[3];
    v[1] -= q * v[4];
    v[2] -= q * v[5];
  }
  if (c.check_egb) {
    T B2 = v[3] * v[3] + v[4] * v[4] + v[5] * v[5];
    if (B2 < Tiny<T>::v) B2 = Tiny<T>::v;
    const T E2 = v[0] * v[0] + v[1] * v[1] + v[2] * v[2];
    if (E2 > B2) {
      const T s = sqrt(fdiv(B2, E2));
      v[0] *= s;
      v[1] *= s;
      v[2] *= s;
    }
  }
}

// The point boundaries that follow the clamps in a cylindrical stage, in the
// reference's order (field_solver_EZ_cylindrical.cu:688-700): the axis
// boundary (kernel_boundary_axis_thread, :371-411), the star at time t and,
// in the last stage, the absorbing layer.  v holds this point's values after
// the clamps.  The axis boundary copies values of the three columns next to
// the axis before the star is applied to them, so the threads of those
// columns write the mirror columns (and the one next to the axis also the
// axis column, which it then passes through the star and the layer); the
// thread of the axis column itself writes nothing.
template <typename T>
__device__ __forceinline__ void cyl_finish(const CylConst<T>& c, int i, int j, long long o,
                                          const T* v, const F7<T>& out, const F7<T>& un,
                                          T t, bool last) {
  const T z = c.z0 + c.dz * (T)(j - c.g1);
  auto bc = [&](V7<T> w, long long p, T R) {
    // the out-of-line boundary code is entered only where it can act
    if (R * R + z * z < T(4) * c.radius * c.radius + Tiny<T>::v) w = cyl_pulsar(c, w, R, z, t);
    if (last && c.absorbing && (R > c.xh || z < c.yl || z > c.yh)) {
      V7<T> n;
      for (int a = 0; a < 6; ++a) n.v[a] = un.p[a][p];
      n.v[6] = T(0);
      w = cyl_absorb(c, w, n, R, z);
    }
    for (int a = 0; a < 7; ++a) out.p[a][p] = w.v[a];
  };
  const int da = c.axis_col >= 0 ? i - c.axis_col : -1;
  if (da == 0) return;
  if (da >= 1 && da <= 3) {
    // mirror column axis - da: E_z, B_z, P even, the rest odd
    constexpr T par[7] = {T(-1), T(1), T(-1), T(-1), T(1), T(-1), T(1)};
    const long long m = o - 2 * da;
    for (int a = 0; a < 7; ++a) out.p[a][m] = par[a] * v[a];
    if (da == 1) {
      V7<T> w;
      w.v[0] = T(0); w.v[1] = v[1]; w.v[2] = T(0);
      w.v[3] = T(0); w.v[4] = v[4]; w.v[5] = T(0);
      w.v[6] = v[6];
      bc(w, o - 1, c.R0 + c.dR * (T)(c.axis_col - c.g0));
    }
  }
  V7<T> w;
  for (int a = 0; a < 7; ++a) w.v[a] = v[a];
  bc(w, o, c.R0 + c.dR * (T)(i - c.g0));
}

// One LSRK stage of the cylindrical solver: kernel_rk_step1_thread +
// kernel_rk_step2_thread, the clamps, then cyl_finish
// (field_solver_EZ_cylindrical.cu:143-234, 674-703).  The reference's
// cylindrical stage writes no J / divE / divB.
template <typename T, bool FIRST>
__global__ void __launch_bounds__(256, kCylStageMinBlocks) cyl_stage_kernel(const __grid_constant__ CylConst<T> c,
                                                        const F7<T> u, const F7<T> out,
                                                        const F7<T> du, const F7<T> un,
                                                        const T As, const T Bs, const T tst,
                                                        const int flags) {
  const int i = c.lo0 + blockIdx.x * blockDim.x + threadIdx.x;
  const int j = c.lo1 + blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= c.hi0 || j >= c.hi1) return;
  const uint32_t d0 = (uint32_t)c.d0;
  const uint32_t o = (uint32_t)i + (uint32_t)j * d0;
  const Stencil2D<true, T> st{u, o, d0};
  T R = c.R0 + c.dR * (T)(i - c.g0);
  if (fabs(R) < Tiny<T>::v) R = Tiny<T>::v;
  // dfRdRR (:110-113): (R f)_R / R, 2 f_R on the axis, as the weights of diff1_4 times
  // R at the four points.  The factors stay out of the weights, as in sph_stage_point (B_z
  // of a run was 5% farther from 64 bits), and each difference is rounded as diff1_4
  // rounds it, 1 / 12 before 1 / delta: beside the dipole's singularity two points decide
  // the error of E_phi, and with 1 / 12 taken out of the curls it was 1.9 times that.
  const bool on_axis = fabs(R) < c.dR * T(0.25);
  const T iRR = on_axis ? T(2) * c.inv_dR : c.inv_dR / R;
  T wRR[4];
#pragma unroll
  for (int k = 0; k < 4; ++k)
    wRR[k] = diff4<T>(k) * (on_axis ? T(1) : R + T(k < 2 ? k - 2 : k - 1) * c.dR);
  // (rot E, rot B) along R, z, phi and (div E, div B)
  auto r12 = [](Pair<T> t) { return pmul(t, both(T(1.0 / 12.0))); };
  const Pair<T> rot[3] = {
      pmul(r12(st.dy(2)), both(-c.inv_dz)), pmul(r12(st.dx(2, wRR)), both(iRR)),
      pfma(r12(st.dy(0)), both(c.inv_dz), pmul(r12(st.dx(1)), both(-c.inv_dR)))};
  const Pair<T> dvg =
      pfma(r12(st.dx(0, wRR)), both(iRR), pmul(r12(st.dy(1)), both(c.inv_dz)));
  const T divE = first(dvg), divB = second(dvg);
  Pair<T> eb[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) eb[a] = st.px(a, 0);
  const T P = st.x(6, 0);
  const T E[3] = {first(eb[0]), first(eb[1]), first(eb[2])};
  const T B[3] = {second(eb[0]), second(eb[1]), second(eb[2])};
  T B2 = B[0] * B[0] + B[1] * B[1] + B[2] * B[2];
  if (B2 < Tiny<T>::v) B2 = Tiny<T>::v;
  const Pair<T> lr = pdot3(eb, rot);
  const T Jp = second(lr) - first(lr);
  const T iB2 = fdiv(T(1), B2);
  const T J[3] = {(divE * (E[2] * B[1] - E[1] * B[2]) + Jp * B[0]) * iB2,
                  (divE * (E[0] * B[2] - E[2] * B[0]) + Jp * B[1]) * iB2,
                  (divE * (E[1] * B[0] - E[0] * B[1]) + Jp * B[2]) * iB2};
  const T gP[3] = {st.dx1(6) * (c.inv_dR * T(1.0 / 12.0)),
                   st.dy1(6) * (c.inv_dz * T(1.0 / 12.0)), T(0)};
  const T dt = c.dt;
  if (flags & AX_WRITE_UN) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      un.p[a][o] = E[a];
      un.p[3 + a][o] = B[a];
    }
  }
  T v[7];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    Pair<T> d = pmul(pk(second(rot[a]) - J[a], first(rot[a]) + gP[a]), pk(dt, -dt));
    if constexpr (!FIRST) d = pfma(pk(du.p[a][o], du.p[3 + a][o]), both(As), d);
    du.p[a][o] = first(d);
    du.p[3 + a][o] = second(d);
    const Pair<T> n = pfma(d, both(Bs), eb[a]);
    v[a] = first(n);
    v[3 + a] = second(n);
  }
  {
    T d = -dt * c.ch2 * divB - div_const(P, c.tau, c.inv_tau);
    if constexpr (!FIRST) d = sfma(du.p[6][o], As, d);
    du.p[6][o] = d;
    v[6] = sfma(d, Bs, P);
  }
  cyl_clamps(c, v);
  cyl_finish(c, i, j, o, v, out, un, tst, (flags & AX_LAST) != 0);
}

// Kreiss-Oliger pass of the cylindrical solver (kernel_KO_step1_thread +
// _step2_thread, field_solver_EZ_cylindrical.cu:297-369; order of :705-712):
// plain 6th differences in R and z, the clamps, then cyl_finish at t + dt.
template <typename T>
__global__ void __launch_bounds__(256, kCylKoMinBlocks) cyl_ko_kernel(const __grid_constant__ CylConst<T> c,
                                                     const F7<T> u, const F7<T> out,
                                                     const F7<T> un, const T tend) {
  const int i = c.lo0 + blockIdx.x * blockDim.x + threadIdx.x;
  const int j = c.lo1 + blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= c.hi0 || j >= c.hi1) return;
  const uint32_t d0 = (uint32_t)c.d0;
  const uint32_t o = (uint32_t)i + (uint32_t)j * d0;
  const Stencil2D<true, T> st{u, o, d0};
  // the 6th differences, one chain per axis as in sph_ko_point
  T v[7];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    Pair<T> tx = st.px(a, -3), ty = st.py(a, -3);
#pragma unroll
    for (int k = 1; k < 7; ++k) {
      tx = pfma(st.px(a, k - 3), both(diff6<T>(k)), tx);
      ty = pfma(st.py(a, k - 3), both(diff6<T>(k)), ty);
    }
    const Pair<T> n = pfma(padd(tx, ty), both(c.ko_c), st.px(a, 0));
    v[a] = first(n);
    v[3 + a] = second(n);
  }
  {
    T tx = st.x(6, -3), ty = st.y(6, -3);
#pragma unroll
    for (int k = 1; k < 7; ++k) {
      tx = sfma(st.x(6, k - 3), diff6<T>(k), tx);
      ty = sfma(st.y(6, k - 3), diff6<T>(k), ty);
    }
    v[6] = sfma(tx + ty, c.ko_c, st.x(6, 0));
  }
  cyl_clamps(c, v);
  cyl_finish(c, i, j, o, v, out, un, tend, false);
}

}  // namespace coffee
