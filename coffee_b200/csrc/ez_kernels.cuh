// Flat-Cartesian EZ kernels: one fused LSRK stage, and the Kreiss-Oliger
// pass that closes a step.
//
// Both kernels stream along z.  A CTA owns a TX x TY column of points and a
// chunk of z planes.  Each z plane of the 7 fields (E, B, P), with a halo of
// H points in x and y, is copied global -> shared memory by cp.async into a
// ring of planes, PF planes ahead of the plane being computed, so the HBM
// reads of the next planes overlap the arithmetic of this one.  The new
// E, B, P go to a second buffer (stencil reads of other points still need
// the old values), together with their periodic guard images, so no separate
// halo-exchange pass is needed.
//
// The kernels are bound by instruction issue more than by anything else, so
// the stencil loops are written to cost one instruction per operand: shared
// memory is addressed by 32-bit addresses with the field / neighbour offsets
// as compile-time immediates (lds<T, OFF>), loops over the 7 fields are
// unrolled at compile time (static_for), and the guard-image bookkeeping is
// skipped for points that have no image.  Global element offsets are 32-bit
// (an array has fewer than 2^31 points: flat_plan checks it), so that every
// global address is one wide multiply-add of an offset onto an array base.
#pragma once

#include "ez_pair.cuh"
#include "ez_physics.cuh"

namespace coffee {

// Flags of the stage kernel.
enum StageFlags { ST_LAST = 1, ST_AUX = 2, ST_WRITE_UN = 4 };

// Minimum resident CTAs for __launch_bounds__: two 256-thread CTAs (or the
// equivalent) per SM in FP32, which caps registers at 128 per thread.
#ifndef COFFEE_F32_THREADS_PER_SM
#define COFFEE_F32_THREADS_PER_SM 512
#endif
template <typename T, int NT>
constexpr int min_blocks() {
  return (sizeof(T) == 4)
             ? ((COFFEE_F32_THREADS_PER_SM / NT) > 0 ? COFFEE_F32_THREADS_PER_SM / NT : 1)
             : 1;
}

// 4th-order first derivative (reference diff1_4, finite_diff.h:13-18):
// ((f-2 - f+2) + 8 (f+1 - f-1)) * inv_delta / 12.
template <typename T>
__device__ __forceinline__ T d1_4(T m2, T m1, T p1, T p2, T s) {
  return ((m2 - p2) + (T)8 * (p1 - m1)) * s;
}

// The same of both fields of a pair.  XA: diff1_4 of the reference
// (finite_diff_simd.h:15-25) before its inv_delta factor, the division by 12
// as q = t (1/12), q + (t - 12 q) (1/12) with the exact residual, t noted in `g`.  This
// is the IEEE quotient of every float but 0 < |t| < 2^-124, whose quotient is subnormal
// and which the guard finds, and -0, of which it makes +0 (where results are called the
// same bit for bit, 0 and -0 are one value): tests/c/div12_check.c,
// tests/cuda/pair_check.cu.
template <bool XA, typename T>
__device__ __forceinline__ Pair<T> pd1_4(Pair<T> m2, Pair<T> m1, Pair<T> p1, Pair<T> p2,
                                         const T inv12, Guard<T>& g) {
  if constexpr (XA) {
    const Pair<T> r12 = both((T)(1.0 / 12.0));
    Pair<T> t = pfma(m1, both((T)-8), m2);
    t = pfma(p1, both((T)8), t);
    t = psub(t, p2);
    g.small(t);
    const Pair<T> q = pmul(t, r12);
    return pfma(pfma(q, both((T)-12), t), r12, q);
  } else {
    return pmul(pfma(psub(p1, m1), both((T)8), psub(m2, p2)), both(inv12));
  }
}
template <bool XA, typename T>
__device__ __forceinline__ T sd1_4(T m2, T m1, T p1, T p2, const T inv12, Guard<T>& g) {
  if constexpr (XA) {
    const T r12 = (T)(1.0 / 12.0);
    T t = sfma(m1, (T)-8, m2);
    t = sfma(p1, (T)8, t);
    t = xa::sub(t, p2);
    g.small(t);
    const T q = smul(t, r12);
    return sfma(sfma(q, (T)-12, t), r12, q);
  } else {
    return d1_4(m2, m1, p1, p2, inv12);
  }
}

// 6th-order, 2nd-difference KO operator along one axis (reference diff6_2,
// finite_diff.h:25-30): f-3 - 6 f-2 + 15 f-1 - 20 f0 + 15 f+1 - 6 f+2 + f+3.
template <typename T>
__device__ __forceinline__ T d6_2(T m3, T m2, T m1, T c, T p1, T p2, T p3) {
  return ((m3 + p3) - (T)6 * (m2 + p2)) + ((T)15 * (m1 + p1) - (T)20 * c);
}

// The same of both fields of a pair; XA: diff6_2 of the reference
// (finite_diff_simd.h:41-58), each weighted term fused into the running sum, f+3 added
// last.
template <bool XA, typename T>
__device__ __forceinline__ Pair<T> pd6_2(Pair<T> m3, Pair<T> m2, Pair<T> m1, Pair<T> c, Pair<T> p1,
                                         Pair<T> p2, Pair<T> p3) {
  if constexpr (XA) {
    Pair<T> t = pfma(m2, both((T)-6), m3);
    t = pfma(m1, both((T)15), t);
    t = pfma(c, both((T)-20), t);
    t = pfma(p1, both((T)15), t);
    t = pfma(p2, both((T)-6), t);
    return padd(p3, t);
  } else {
    Pair<T> t = pfma(padd(m2, p2), both((T)-6), padd(m3, p3));
    t = pfma(padd(m1, p1), both((T)15), t);
    return pfma(c, both((T)-20), t);
  }
}

// The CPU build's clamps (apply_clamps_xa) on v = (E, B, P) with the
// straight-line quotients; a point outside their range is done again with the
// IEEE operations.
template <typename T>
__device__ __forceinline__ void apply_clamps_mid(T v[7]) {
  Guard<T> g;
  const T N2 = xa::floor_tiny(xa::dot3(v[3], v[3], v[4], v[4], v[5], v[5]));
  const T EB = xa::dot3(v[3], v[0], v[4], v[1], v[5], v[2]);
  const T y = rcp_mid(N2);
  const Pair<T> q01 = pdiv_mid(pk(xa::mul(EB, v[3]), xa::mul(EB, v[4])), both(-N2), both(y), g);
  const Pair<T> q2 = pdiv_mid(both(xa::mul(EB, v[5])), both(-N2), both(y), g);
  T e[3] = {xa::sub(v[0], first(q01)), xa::sub(v[1], second(q01)), xa::sub(v[2], first(q2))};
  const T E2 = xa::dot3(e[0], e[0], e[1], e[1], e[2], e[2]);
  g.below(N2, MidRange<T>::den_max);
  g.below(E2, MidRange<T>::num_max);
  if (g.bad() || E2 > N2) {
    apply_clamps_xa(v[0], v[1], v[2], v[3], v[4], v[5]);
  } else {
#pragma unroll
    for (int a = 0; a < 3; ++a) v[a] = e[a];
  }
}

// Write the 7 new values of point (i, j, k) (linear index o) to `out` at the
// point and at its periodic guard images.
template <typename T>
__device__ __forceinline__ void store_with_images(const GridGeom& g, const ColumnCtx<T>& col,
                                                  const F7<T>& out, int k, uint32_t o,
                                                  const T u[7]) {
  if (col.xy_simple && only_self(g, 2, k)) {
#pragma unroll
    for (int f = 0; f < 7; ++f) out.p[f][o] = u[f];
    return;
  }
  int xs[2], ys[2], zs[2];
  const int nx = periodic_targets(g, 0, col.i, xs);
  const int ny = periodic_targets(g, 1, col.j, ys);
  const int nz = periodic_targets(g, 2, k, zs);
#pragma unroll
  for (int cz = 0; cz < 2; ++cz) {
    if (cz >= nz) break;
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      if (b >= ny) break;
#pragma unroll
      for (int a = 0; a < 2; ++a) {
        if (a >= nx) break;
        const uint32_t q = (uint32_t)zs[cz] * (uint32_t)g.sz + (uint32_t)ys[b] * (uint32_t)g.sy +
                           (uint32_t)xs[a];
#pragma unroll
        for (int f = 0; f < 7; ++f) out.p[f][q] = u[f];
      }
    }
  }
}

// The guard images of a box with a periodic axis of fewer than 2 guard points, where a
// point may have one beyond each face and store_with_images writes one of them: a pass
// of its own after each stage and KO pass of such a box, so that the others pay nothing
// (in store_with_images a third target cost a box of 128^3 4%).  Every guard point of a
// periodic axis takes the value at its wrapped coordinates if the kernels update
// that point; one thread per point, and no source is a target.
template <typename T>
__global__ void __launch_bounds__(256) ez_images_kernel(const GridGeom g, const F7<T> u) {
  const long long n = g.sz * g.dims[2];
  for (long long q = blockIdx.x * 256LL + threadIdx.x; q < n; q += gridDim.x * 256LL) {
    const int k = (int)(q / g.sz), r = (int)(q - k * g.sz), j = r / g.dims[0];
    int c[3] = {r - j * g.dims[0], j, k};
    bool image = false, updated = true;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      if (g.periodic[a]) {
        const int s = c[a] < g.guard[a] ? g.N[a] : c[a] >= g.dims[a] - g.guard[a] ? -g.N[a] : 0;
        image = image || s != 0;
        c[a] += s;
      } else {
        updated = updated && c[a] >= g.lo[a] && c[a] < g.hi[a];
      }
    }
    if (!image || !updated) continue;
    const long long o = c[2] * g.sz + c[1] * g.sy + c[0];
#pragma unroll
    for (int f = 0; f < 7; ++f) u.p[f][q] = u.p[f][o];
  }
}

// Curl, divergence and gradient of the fields at one point, as the stage
// needs them (all inv_delta-scaled 4th-order differences).
template <typename T>
struct Derivs {
  T rotE[3], rotB[3], divE, divB, gradP[3];
};

// What a stage computes at one point before the boundaries: the new
// accumulators and fields, the current and the divergences.
template <typename T>
struct StageValues {
  T d[7], nu[7], J[3], divE, divB;
};

// One stage at a point in the CPU build's own arithmetic, operation for
// operation (rk_step and clean_epar_check_eGTb, field_solver_EZ.cpp:143-259,
// 552-634; ez_refarith.cuh), with the IEEE divisions and roots.  With DG the
// clamps add to the energy-change diagnostics at point o.
template <bool FIRST, bool DG, typename T>
__device__ __forceinline__ void stage_values_ieee(const EzConst<T>& c, const T u[7],
                                                  const Derivs<T>& dv, const T dold[7],
                                                  const T As, const T Bs,
                                                  const ColumnCtx<T>& col, const int k,
                                                  const F6<T>& dg, const uint32_t o,
                                                  StageValues<T>& r) {
  const T ex = u[0], ey = u[1], ez = u[2], bx = u[3], by = u[4], bz = u[5], P = u[6];
  const T rotBx = dv.rotB[0], rotBy = dv.rotB[1], rotBz = dv.rotB[2];
  const T rotEx = dv.rotE[0], rotEy = dv.rotE[1], rotEz = dv.rotE[2];
  const T divE = dv.divE;
  const T divB = dv.divB;
  T* d = r.d;
  T Jx, Jy, Jz;
  const T B2 = xa::floor_tiny(xa::dot3(bx, bx, by, by, bz, bz));
  const T BrotB = xa::dot3(bx, rotBx, by, rotBy, bz, rotBz);
  const T ErotE = xa::dot3(ex, rotEx, ey, rotEy, ez, rotEz);
  const T cx = xa::fma(-by, ez, xa::mul(bz, ey));
  const T cy = xa::fma(-bz, ex, xa::mul(bx, ez));
  const T cz = xa::fma(-bx, ey, xa::mul(by, ex));
  if (c.use_edotb) {
    const T E2 = xa::dot3(ex, ex, ey, ey, ez, ez);
    const T chi2 = xa::sub(B2, E2);
    const T EdotB = xa::dot3(bx, ex, by, ey, bz, ez);
    const T E02 = xa::fma(
        xa::sub(xa::sqrt(xa::fma(xa::mul(EdotB, (T)4), EdotB, xa::mul(chi2, chi2))), chi2),
        (T)0.5, B2);
    const T Jp = xa::fma(EdotB, c.gam_dt, xa::sub(BrotB, ErotE));
    Jx = xa::add(xa::div(xa::mul(divE, cx), E02), xa::div(xa::mul(bx, Jp), B2));
    Jy = xa::add(xa::div(xa::mul(divE, cy), E02), xa::div(xa::mul(by, Jp), B2));
    Jz = xa::add(xa::div(xa::mul(divE, cz), E02), xa::div(xa::mul(bz, Jp), B2));
  } else {
    const T Jp = xa::sub(BrotB, ErotE);
    Jx = xa::div(xa::fma(bx, Jp, xa::mul(divE, cx)), B2);
    Jy = xa::div(xa::fma(by, Jp, xa::mul(divE, cy)), B2);
    Jz = xa::div(xa::fma(bz, Jp, xa::mul(divE, cz)), B2);
  }
  T Px = 0, Py = 0, Pz = 0;
  if (c.divB_clean) {
    Px = dv.gradP[0];
    Py = dv.gradP[1];
    Pz = dv.gradP[2];
  }
  const T s = p_taper_xa(c, col, k);
  const T dt = c.dt;
  // dU As (As = 0 on the first stage, where the old dU is not read)
  T da[7];
#pragma unroll
  for (int f = 0; f < 7; ++f) {
    if constexpr (FIRST) da[f] = (T)0;
    else da[f] = xa::mul(dold[f], As);
  }
  d[0] = xa::fma(dt, xa::sub(rotBx, Jx), da[0]);
  d[1] = xa::fma(dt, xa::sub(rotBy, Jy), da[1]);
  d[2] = xa::fma(dt, xa::sub(rotBz, Jz), da[2]);
  d[3] = xa::fma(-dt, xa::fma(Px, s, rotEx), da[3]);
  d[4] = xa::fma(-dt, xa::fma(Py, s, rotEy), da[4]);
  d[5] = xa::fma(-dt, xa::fma(Pz, s, rotEz), da[5]);
  // dP As - P / tau with the product fused, minus dt (divB ch2)
  if constexpr (FIRST)
    d[6] = xa::fma(-dt, xa::mul(divB, c.ch2), -xa::div(P, c.tau));
  else
    d[6] = xa::fma(-dt, xa::mul(divB, c.ch2), xa::fma(dold[6], As, -xa::div(P, c.tau)));
  // mul_add(dU, Bs, U), then clean_epar_check_eGTb
  T* nu = r.nu;
#pragma unroll
  for (int f = 0; f < 7; ++f) nu[f] = xa::fma(d[f], Bs, u[f]);
  if constexpr (DG)
    apply_clamps_xa_dg<FIRST>(nu[0], nu[1], nu[2], nu[3], nu[4], nu[5], dg, o);
  else
    apply_clamps_xa(nu[0], nu[1], nu[2], nu[3], nu[4], nu[5]);
  r.J[0] = Jx;
  r.J[1] = Jy;
  r.J[2] = Jz;
  r.divE = divE;
  r.divB = divB;
}

// The derivatives of one point from global memory with the IEEE division.
template <typename T>
__device__ __noinline__ Derivs<T> point_derivatives_ieee(const EzConst<T>& c,
                                                         const F7<const T> uin, const uint32_t o) {
  const uint32_t st[3] = {1u, (uint32_t)c.g.sy, (uint32_t)c.g.sz};
  T g[7][3];
  for (int f = 0; f < 7; ++f) {
    const T* p = uin.p[f] + o;
    for (int a = 0; a < 3; ++a) {
      const long long t = st[a];
      g[f][a] = xa::dq(p[-2 * t], p[-t], p[t], p[2 * t]);
    }
  }
  const T ix = c.inv_delta[0], iy = c.inv_delta[1], iz = c.inv_delta[2];
  Derivs<T> dv;
  auto curl_div = [&](int b, T* rot, T& dvg) {
    rot[0] = xa::fma(-iz, g[b + 1][2], xa::mul(iy, g[b + 2][1]));
    rot[1] = xa::fma(-ix, g[b + 2][0], xa::mul(iz, g[b][2]));
    rot[2] = xa::fma(-iy, g[b][1], xa::mul(ix, g[b + 1][0]));
    dvg = xa::fma(iz, g[b + 2][2], xa::fma(iy, g[b + 1][1], xa::mul(ix, g[b][0])));
  };
  curl_div(0, dv.rotE, dv.divE);
  curl_div(3, dv.rotB, dv.divB);
  dv.gradP[0] = xa::mul(ix, g[6][0]);
  dv.gradP[1] = xa::mul(iy, g[6][1]);
  dv.gradP[2] = xa::mul(iz, g[6][2]);
  return dv;
}

// The same stage of one point from global memory, out of line: for the rare
// points whose operands the straight-line arithmetic of stage_values_pair
// does not cover (Guard).  Were all points of that kind (fields below 2^-124 on a uniform
// B), a step of 512^3 would take 137 ms instead of 25, of 128^3 1.74 instead of 0.50.
template <bool FIRST, typename T>
__device__ __noinline__ StageValues<T> stage_point_ieee(const EzConst<T>& c, const F7<const T> uin,
                                                        const F7<T> du, const ColumnCtx<T> col,
                                                        const int k, const uint32_t o, const T As,
                                                        const T Bs) {
  T u[7], dold[7];
  for (int f = 0; f < 7; ++f) {
    u[f] = uin.p[f][o];
    dold[f] = FIRST ? (T)0 : du.p[f][o];
  }
  const Derivs<T> dv = point_derivatives_ieee(c, uin, o);
  StageValues<T> r;
  F6<T> none;
  stage_values_ieee<FIRST, false>(c, u, dv, dold, As, Bs, col, k, none, o, r);
  return r;
}

// One stage at a point from its pairs: eb[a] = (E_a, B_a), rot and dvg the
// pairs of their curls and divergences, dold the old accumulators of (E_a,
// B_a) and of P.  XA: the CPU build's arithmetic, with straight-line
// quotients and roots (ez_pair.cuh); `g` notes operands outside their range,
// and the caller then uses stage_point_ieee.  Otherwise the regrouped
// arithmetic: the same algorithm with shared divisions.
template <bool FIRST, bool XA, typename T>
__device__ __forceinline__ void stage_values_pair(const EzConst<T>& c, const Pair<T> eb[3],
                                                  const T P, const Pair<T> rot[3],
                                                  const Pair<T> dvg, const T gradP[3],
                                                  const Pair<T> dold[3], const T doldP, const T As,
                                                  const T Bs, const ColumnCtx<T>& col, const int k,
                                                  Pair<T> d[3], T& dP, Pair<T> nu[3], T& nuP,
                                                  T J[3], Guard<T>& g) {
  const T divE = first(dvg), divB = second(dvg);
  const T e[3] = {first(eb[0]), first(eb[1]), first(eb[2])};
  const T b[3] = {second(eb[0]), second(eb[1]), second(eb[2])};
  const Pair<T> sq = pdot3(eb, eb), br = pdot3(eb, rot);  // (E2, B2), (E.rotE, B.rotB)
  const T B2 = xa::floor_tiny(second(sq));
  const T dt = c.dt;
  const T C[3] = {xa::fma(-b[1], e[2], xa::mul(b[2], e[1])),
                  xa::fma(-b[2], e[0], xa::mul(b[0], e[2])),
                  xa::fma(-b[0], e[1], xa::mul(b[1], e[0]))};
  T Jp = xa::sub(second(br), first(br));
  T Ptau;  // P / tau
  T q[3];  // (E.B) B_a / B^2 of the clamps
  if constexpr (XA) {
    if (c.use_edotb) {
      const T chi2 = xa::sub(B2, first(sq));
      const T EdotB = xa::dot3(b[0], e[0], b[1], e[1], b[2], e[2]);
      const T s2 = xa::fma(xa::mul(EdotB, (T)4), EdotB, xa::mul(chi2, chi2));
      const T E02 = xa::fma(xa::sub(sqrt_floor(s2), chi2), (T)0.5, B2);
      Jp = xa::fma(EdotB, c.gam_dt, Jp);
      g.below(E02, MidRange<T>::den_max);
      const Pair<T> nden = pk(-E02, -B2);
      Pair<T> y = pk(rcp_seed(E02), rcp_seed(B2));
      y = pfma(pfma(nden, y, both((T)1)), y, y);
      const Pair<T> f = pk(divE, Jp);
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const Pair<T> t = pdiv_mid(pmul(f, pk(C[a], b[a])), nden, y, g);
        J[a] = xa::add(first(t), second(t));
      }
    } else {
      g.below(B2, MidRange<T>::den_max);
      const Pair<T> nden = both(-B2), y = both(rcp_mid(B2));
      T n[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) n[a] = xa::fma(b[a], Jp, xa::mul(divE, C[a]));
      const Pair<T> t01 = pdiv_mid(pk(n[0], n[1]), nden, y, g);
      J[0] = first(t01);
      J[1] = second(t01);
      J[2] = first(pdiv_mid(both(n[2]), nden, y, g));
    }
  } else if (c.use_edotb) {
    // J with E.B damping (field_solver_EZ.cpp:170-186, .cu:72-91)
    const T chi2 = B2 - first(sq);
    const T EdotB = e[0] * b[0] + e[1] * b[1] + e[2] * b[2];
    const T E02 = (T)0.5 * (sqrt(chi2 * chi2 + (T)4 * EdotB * EdotB) - chi2) + B2;
    const T x = fdiv(divE, E02), y = fdiv(Jp + EdotB * c.gam_dt, B2);
#pragma unroll
    for (int a = 0; a < 3; ++a) J[a] = x * C[a] + y * b[a];
  } else {
    const T rB2 = fdiv((T)1, B2);
#pragma unroll
    for (int a = 0; a < 3; ++a) J[a] = (divE * C[a] + Jp * b[a]) * rB2;
  }
  // the P gradient with its taper (CPU semantics), 0 without the cleaning
  T s = 0;
  if (c.divB_clean) {
    if constexpr (XA) s = p_taper_mid(c, col, k, g);
    else s = c.semantics == SEM_CPU_REF ? p_taper(c, col, k) : (T)1;
  }
  // new accumulators and fields
  const Pair<T> pdt = pk(dt, -dt);
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const Pair<T> da = FIRST ? both((T)0) : pmul(dold[a], both(As));
    // without the cleaning P may be anything (XA: a point of which w is not finite is
    // done again)
    const T gp = XA || c.divB_clean ? gradP[a] : (T)0;
    const Pair<T> w = pk(xa::sub(second(rot[a]), J[a]), xa::fma(gp, s, first(rot[a])));
    d[a] = pfma(pdt, w, da);
    nu[a] = pfma(d[a], both(Bs), eb[a]);
  }
  // E.B = 0 and |E| <= |B|
  T ne[3] = {first(nu[0]), first(nu[1]), first(nu[2])};
  const T nb[3] = {second(nu[0]), second(nu[1]), second(nu[2])};
  if constexpr (XA) {
    const T N2 = xa::floor_tiny(xa::dot3(nb[0], nb[0], nb[1], nb[1], nb[2], nb[2]));
    const T EB = xa::dot3(nb[0], ne[0], nb[1], ne[1], nb[2], ne[2]);
    const T y = rcp_mid(N2);
    const Pair<T> q01 =
        pdiv_mid(pk(xa::mul(EB, nb[0]), xa::mul(EB, nb[1])), both(-N2), both(y), g);
    const Pair<T> q2P = pdiv_mid(pk(xa::mul(EB, nb[2]), P), pk(-N2, -c.tau), pk(y, c.inv_tau), g);
    q[0] = first(q01);
    q[1] = second(q01);
    q[2] = first(q2P);
    Ptau = second(q2P);
    g.below(N2, MidRange<T>::den_max);
    g.below(xa::mul(P, P), MidRange<T>::num_max);
#pragma unroll
    for (int a = 0; a < 3; ++a) ne[a] = xa::sub(ne[a], q[a]);
    const T E2 = xa::dot3(ne[0], ne[0], ne[1], ne[1], ne[2], ne[2]);
    g.below(E2, MidRange<T>::num_max);
    if (E2 > N2) {
      const T m = xa::sqrt(xa::div(N2, E2));
#pragma unroll
      for (int a = 0; a < 3; ++a) ne[a] = xa::mul(ne[a], m);
    }
  } else {
    Ptau = P * c.inv_tau;
    apply_clamps(c, ne[0], ne[1], ne[2], nb[0], nb[1], nb[2]);
  }
#pragma unroll
  for (int a = 0; a < 3; ++a) nu[a] = pk(ne[a], nb[a]);
  // dP As - P / tau with the product fused, minus dt (divB ch2)
  dP = xa::fma(-dt, xa::mul(divB, c.ch2), FIRST ? -Ptau : xa::fma(doldP, As, -Ptau));
  nuP = xa::fma(dP, Bs, P);
}

// The rest of a stage at one point: the start-of-step copy, the stores of the
// accumulators and of J, div E and div B, the star boundary, the absorbing
// layer and the store of the fields with their guard images.
template <bool BC, typename T>
__device__ __forceinline__ void stage_finish(const EzConst<T>& c, const T u[7], const T d[7],
                                             T nu[7], const T J[3], const T divE, const T divB,
                                             const T tst, const int flags,
                                             const ColumnCtx<T>& col, const int k,
                                             const uint32_t o, const F7<T>& du, const F7<T>& un,
                                             const F5<T>& aux, const F7<T>& uout) {
  // the start-of-step copy is only read inside the absorbing layer
  T sig = (T)0;
  if constexpr (BC) sig = c.absorbing ? absorbing_sigma(c, col.i, col.j, k) : (T)0;
  if (BC && (flags & ST_WRITE_UN) != 0 && sig > (T)0) {
#pragma unroll
    for (int f = 0; f < 7; ++f) un.p[f][o] = u[f];
  }
#pragma unroll
  for (int f = 0; f < 7; ++f) du.p[f][o] = d[f];
  if ((flags & ST_AUX) != 0) {
    aux.p[0][o] = J[0];
    aux.p[1][o] = J[1];
    aux.p[2][o] = J[2];
    aux.p[3][o] = divE;
    aux.p[4][o] = divB;
  }
  if constexpr (BC) star_boundary(c, col.i, col.j, k, tst, nu);
  if (BC && (flags & ST_LAST) != 0 && sig > (T)0) {
    V7<T> uv, unv;
#pragma unroll
    for (int f = 0; f < 7; ++f) {
      uv.v[f] = nu[f];
      unv.v[f] = un.p[f][o];
    }
    uv = absorbing_apply(c, col.i, col.j, k, sig, uv, unv);
#pragma unroll
    for (int f = 0; f < 7; ++f) nu[f] = uv.v[f];
  }
  store_with_images(c.g, col, uout, k, o, nu);
}

// Per-thread table of the shared-memory slots and global offsets that a
// CTA's threads copy for one (TX + 2H) x (TY + 2H) tile of one field plane.
// V = 1 copies one element per cp.async; V = 2 copies aligned pairs (8 bytes
// in FP32), which needs an even row length d0: the copied row then starts at
// the even column at or left of the tile's first column, `xoff` (0 or 1)
// columns before it, and a row holds TX + 2H + 2 elements.
template <typename T, int TX, int TY, int H, int V = 1, int THREADS = TX * TY>
struct TileLoader {
  static_assert(V == 1 || V == 2, "one element or an aligned pair per copy");
  static constexpr int SX = TX + 2 * H + (V == 2 ? 2 : 0);  // shared row stride (elements)
  static constexpr int SY = TY + 2 * H, NT = THREADS;
  static constexpr int PER_ROW = SX / V;                    // copies per row
  static constexpr int NCOPY = PER_ROW * SY;
  static constexpr int NLOAD = (NCOPY + NT - 1) / NT;
  static constexpr int FB = SX * SY * (int)sizeof(T);       // bytes of one field plane
  uint32_t sadd[NLOAD];  // shared byte address within slot 0, field 0
  uint32_t eoff[NLOAD];  // element offset within a global plane
  bool lv[NLOAD];
  int xoff;               // shared column of the tile's first column

  __device__ __forceinline__ TileLoader(const GridGeom& g, uint32_t sbase, int tid, int gx0,
                                        int gy0) {
    xoff = (V == 2) ? (gx0 & 1) : 0;
    const int xs = gx0 - xoff;
#pragma unroll
    for (int m = 0; m < NLOAD; ++m) {
      const int e = tid + m * NT;
      const int r = e / PER_ROW, cl = (e - r * PER_ROW) * V;
      const int gx = xs + cl, gy = gy0 + r;
      lv[m] = (e < NCOPY) && gx + (V - 1) < g.dims[0] && gy < g.dims[1];
      sadd[m] = sbase + (uint32_t)((r * SX + cl) * (int)sizeof(T));
      eoff[m] = (uint32_t)gy * (uint32_t)g.sy + (uint32_t)gx;
    }
  }

  // Copy one plane (element offset pe into each field array) of the 7
  // fields into the ring slot at byte offset `slot`.
  __device__ __forceinline__ void copy(const F7<const T>& uin, uint32_t pe,
                                       uint32_t slot) const {
#pragma unroll
    for (int m = 0; m < NLOAD; ++m) {
      if (!lv[m]) continue;
      const uint32_t e = pe + eoff[m], d = sadd[m] + slot;
      static_for<7>([&](auto fc) {
        constexpr int f = decltype(fc)::value;
        cp_async_off<sizeof(T) * V, f * FB>(d, uin.p[f] + e);
      });
    }
  }
};

// Per-thread copies of one (TX + 2H) x (TY + 2H) tile of one plane of the 7
// fields into a ring slot, interleaved: element e of pair a (E_a, B_a) lies at a
// PB + 2 e elements, of P at 3 PB + e, so that one 64-bit shared load (FP32)
// reads both halves of a pair.  The copies are one element each: they need no
// alignment of a row.
template <typename T, int TX, int TY, int H>
struct PairLoader {
  static constexpr int SX = TX + 2 * H, SY = TY + 2 * H, NT = TX * TY;
  static constexpr int NCOPY = SX * SY, NLOAD = (NCOPY + NT - 1) / NT;
  static constexpr int ES = (int)sizeof(T);
  static constexpr int PB = 2 * NCOPY * ES;      // bytes of a pair's plane
  static constexpr int SB = 7 * NCOPY * ES;      // bytes of a ring slot
  static constexpr uint32_t kNone = 0xFFFFFFFFu;
  uint32_t pair0, p0;     // shared addresses of this thread's first element in slot 0
  uint32_t eoff[NLOAD];   // element offsets within a global plane, or kNone

  __device__ __forceinline__ PairLoader(const GridGeom& g, uint32_t sbase, int tid, int gx0,
                                        int gy0) {
    pair0 = sbase + (uint32_t)(2 * tid * ES);
    p0 = sbase + (uint32_t)(3 * PB + tid * ES);
#pragma unroll
    for (int m = 0; m < NLOAD; ++m) {
      const int e = tid + m * NT, r = e / SX, x = gx0 + e - r * SX, y = gy0 + r;
      eoff[m] = e < NCOPY && x < g.dims[0] && y < g.dims[1]
                    ? (uint32_t)y * (uint32_t)g.sy + (uint32_t)x
                    : kNone;
    }
  }
  __device__ __forceinline__ void copy(const F7<const T>& uin, uint32_t pe, uint32_t slot) const {
    static_for<NLOAD>([&](auto mc) {
      constexpr int m = decltype(mc)::value;
      if (eoff[m] == kNone) return;
      const uint32_t e = pe + eoff[m], d = pair0 + slot;
      static_for<3>([&](auto ac) {
        constexpr int a = decltype(ac)::value;
        cp_async_off<ES, a * PB + 2 * m * NT * ES>(d, uin.p[a] + e);
        cp_async_off<ES, a * PB + (2 * m * NT + 1) * ES>(d, uin.p[3 + a] + e);
      });
      cp_async_off<ES, m * NT * ES>(p0 + slot, uin.p[6] + e);
    });
  }
};

// ---------------------------------------------------------------------------
// One LSRK stage (reference rk_step + clamps + star boundary + absorbing
// layer + send_guard_cells, src/algorithms/field_solver_EZ.cpp:1024-1055,
// .cu:669-694).  BC = false compiles the kernel without the star and
// absorbing-layer code, for runs that have neither (their out-of-line calls
// cost registers even when not taken):
//   dU  <- As dU + dt RHS(U)        (FIRST: As = 0, so dU is not read)
//   U'  <- U + Bs dU
//   U'  <- clamps, star boundary at tst, absorbing layer (ST_LAST)
// reading U from `uin` and writing U' (with guard images) to `uout`.
//
// This is the FP64 kernel (and the FP32 one of runs with both the boundary code and the
// diagnostics: 256^3 with the star, 7345 us a step with the register window, 6230 here).
// The ring of 5 + PF planes (k-2 .. k+2, the prefetch) holds the whole stencil as pairs, read at
// compile-time offsets; with the z neighbours in the ring instead of a register
// window a thread's registers hold one point only, which in FP64 lets 12 warps of 168
// registers share an SM.  FP64 stage at 256^3: 2610 us with a register window, 4 warps
// a CTA and IEEE divisions, 1320 us here.  What bounds it is the latency between
// dependent FP64 operations.  The old dU of a point is loaded at the top of its plane
// and used after the derivatives.
// ---------------------------------------------------------------------------
template <typename T, int TX, int TY, int PF>
constexpr size_t stage_smem_bytes() {
  return (size_t)(5 + PF) * PairLoader<T, TX, TY, 2>::SB;
}

// DG (with XA only): also accumulate the CPU build's energy-change
// diagnostics of the clamps into dg.
template <typename T, int TX, int TY, int PF, int MINB, bool FIRST, bool BC, bool XA, bool DG>
__global__ void __launch_bounds__(TX * TY, MINB)
    ez_stage_kernel(const __grid_constant__ EzConst<T> c, const F7<const T> uin,
                    const F7<T> uout, const F7<T> du, const F7<T> un, const F5<T> aux,
                    const F6<T> dg, const T As, const T Bs, const T tst, const int kchunk,
                    const int flags) {
  static_assert(XA || !DG, "the energy diagnostics need the reference arithmetic");
  using L = PairLoader<T, TX, TY, 2>;
  constexpr int R = 5 + PF;  // ring slots
  constexpr int ES = (int)sizeof(T), SX = L::SX, PB = L::PB, SB = L::SB;
  constexpr int CEN = (2 * SX + 2) * 2 * ES;  // own pair, from the corner of its 5 x 5 patch
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const uint32_t sbase = smem_u32(smem_raw);

  const GridGeom& g = c.g;
  const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * TX + tx;
  const int i = g.lo[0] + blockIdx.x * TX + tx;
  const int j = g.lo[1] + blockIdx.y * TY + ty;
  const int k0 = g.lo[2] + blockIdx.z * kchunk;
  const int k1 = min(k0 + kchunk, g.hi[2]);
  const bool active = (i < g.hi[0]) && (j < g.hi[1]);
  // lanes of this warp that compute points: the fences between the field
  // groups below are executed by these lanes only (a tile that overhangs
  // the grid has idle lanes, which must not be named in the mask)
  const unsigned amask = __ballot_sync(0xffffffffu, active);
  const uint32_t sz = (uint32_t)g.sz;
  const uint32_t own = (uint32_t)j * (uint32_t)g.sy + (uint32_t)i;
  const ColumnCtx<T> col = make_column<XA>(c, i, j);
  const L loader(g, sbase, tid, g.lo[0] + (int)blockIdx.x * TX - 2,
                 g.lo[1] + (int)blockIdx.y * TY - 2);
  const int kend = k1 + 2;  // planes [k0-2, k1+2) are read
  auto issue = [&](int kp, uint32_t slot) {
    if (kp < kend) loader.copy(uin, (uint32_t)kp * sz, slot);
    cp_async_commit();
  };
  // plane k0 - 2 + q goes to slot q; the first wait needs planes up to k0 + 2
#pragma unroll 1
  for (int p = 0; p < 5 + PF; ++p) issue(k0 - 2 + p, (uint32_t)(p * SB));

  const T six = c.inv_delta[0] / (T)12, siy = c.inv_delta[1] / (T)12,
          siz = c.inv_delta[2] / (T)12;
  const T ix = c.inv_delta[0], iy = c.inv_delta[1], iz = c.inv_delta[2];
  const uint32_t pcorner = sbase + (uint32_t)((ty * SX + tx) * 2 * ES);
  const uint32_t scorner = sbase + (uint32_t)(3 * PB + (ty * SX + tx) * ES);
  uint32_t head = 0;  // slot of plane k - 2
#pragma unroll 1
  for (int k = k0; k < k1; ++k) {
    cp_async_wait<PF>();  // planes up to k+2 have landed
    __syncthreads();
    auto slot = [&](int q) -> uint32_t {  // of plane k - 2 + q
      const uint32_t s = head + (uint32_t)(q * SB);
      return s >= (uint32_t)(R * SB) ? s - (uint32_t)(R * SB) : s;
    };
    if (active) {
      const uint32_t o = (uint32_t)k * sz + own;
      Pair<T> dold[3];
      T doldP = 0;
      if constexpr (!FIRST) {
#pragma unroll
        for (int a = 0; a < 3; ++a) dold[a] = pk(du.p[a][o], du.p[3 + a][o]);
        doldP = du.p[6][o];
      }
      const uint32_t zs[5] = {slot(0), slot(1), slot(2), slot(3), slot(4)};
      const uint32_t a0 = pcorner + zs[2], s0 = scorner + zs[2];
      // The stencil is consumed component by component, then P; the
      // warp-level fence between groups keeps the shared loads of the next
      // group from being hoisted, which bounds the live registers.  d[a]: the
      // derivatives along axis a of (E_x, B_x), ..., unscaled (the quotients of
      // diff1_4) in the reference arithmetic, which scales and combines them
      // as rk_step does (field_solver_EZ.cpp:143-150: the first product of a
      // curl rounded, the second fused), inv_delta-scaled otherwise.
      Guard<T> gd;
      gd.large = !c.tau_mid;
      auto derivatives = [&](auto ac, Pair<T> d[3]) {
        constexpr int O = decltype(ac)::value * PB, P2 = 2 * ES;
        d[0] = pd1_4<XA>(ldsp<T, O + CEN - 2 * P2>(a0), ldsp<T, O + CEN - P2>(a0),
                         ldsp<T, O + CEN + P2>(a0), ldsp<T, O + CEN + 2 * P2>(a0), six, gd);
        d[1] = pd1_4<XA>(ldsp<T, O + 2 * P2>(a0), ldsp<T, O + (SX + 2) * P2>(a0),
                         ldsp<T, O + (3 * SX + 2) * P2>(a0), ldsp<T, O + (4 * SX + 2) * P2>(a0),
                         siy, gd);
        d[2] = pd1_4<XA>(ldsp<T, O + CEN>(pcorner + zs[0]), ldsp<T, O + CEN>(pcorner + zs[1]),
                         ldsp<T, O + CEN>(pcorner + zs[3]), ldsp<T, O + CEN>(pcorner + zs[4]),
                         siz, gd);
      };
      Pair<T> rot[3], dvg;
      T gradP[3];
      {
        Pair<T> xd[3], yd[3], zd[3];
        derivatives(std::integral_constant<int, 0>{}, xd);
        __syncwarp(amask);
        derivatives(std::integral_constant<int, 1>{}, yd);
        __syncwarp(amask);
        derivatives(std::integral_constant<int, 2>{}, zd);
        if constexpr (XA) {
          rot[0] = pfma(both(-iz), yd[2], pmul(both(iy), zd[1]));
          rot[1] = pfma(both(-ix), zd[0], pmul(both(iz), xd[2]));
          rot[2] = pfma(both(-iy), xd[1], pmul(both(ix), yd[0]));
          dvg = pfma(both(iz), zd[2], pfma(both(iy), yd[1], pmul(both(ix), xd[0])));
        } else {
          rot[0] = psub(zd[1], yd[2]);
          rot[1] = psub(xd[2], zd[0]);
          rot[2] = psub(yd[0], xd[1]);
          dvg = padd(padd(xd[0], yd[1]), zd[2]);
        }
      }
      __syncwarp(amask);
      constexpr int CE1 = CEN / 2;  // own P, from the corner of its patch
      gradP[0] = sd1_4<XA>(lds<T, CE1 - 2 * ES>(s0), lds<T, CE1 - ES>(s0), lds<T, CE1 + ES>(s0),
                           lds<T, CE1 + 2 * ES>(s0), six, gd);
      gradP[1] = sd1_4<XA>(lds<T, 2 * ES>(s0), lds<T, (SX + 2) * ES>(s0),
                           lds<T, (3 * SX + 2) * ES>(s0), lds<T, (4 * SX + 2) * ES>(s0), siy, gd);
      gradP[2] = sd1_4<XA>(lds<T, CE1>(scorner + zs[0]), lds<T, CE1>(scorner + zs[1]),
                           lds<T, CE1>(scorner + zs[3]), lds<T, CE1>(scorner + zs[4]), siz, gd);
      if constexpr (XA) {
        gradP[0] = xa::mul(ix, gradP[0]);
        gradP[1] = xa::mul(iy, gradP[1]);
        gradP[2] = xa::mul(iz, gradP[2]);
      }
      Pair<T> eb[3] = {ldsp<T, CEN>(a0), ldsp<T, PB + CEN>(a0), ldsp<T, 2 * PB + CEN>(a0)};
      const T P = lds<T, CE1>(s0);
      if constexpr (DG) {
        const T u[7] = {first(eb[0]),  first(eb[1]),  first(eb[2]), second(eb[0]),
                        second(eb[1]), second(eb[2]), P};
        Derivs<T> dv;
        T old[7];
        StageValues<T> r;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          dv.rotE[a] = first(rot[a]);
          dv.rotB[a] = second(rot[a]);
          dv.gradP[a] = gradP[a];
          old[a] = first(dold[a]);
          old[3 + a] = second(dold[a]);
        }
        dv.divE = first(dvg);
        dv.divB = second(dvg);
        old[6] = doldP;
        if (gd.bad()) dv = point_derivatives_ieee(c, uin, o);
        stage_values_ieee<FIRST, true>(c, u, dv, old, As, Bs, col, k, dg, o, r);
        stage_finish<BC>(c, u, r.d, r.nu, r.J, r.divE, r.divB, tst, flags, col, k, o, du, un, aux,
                         uout);
      } else {
        Pair<T> dn[3], nu[3];
        T dP, nuP, J[3];
        stage_values_pair<FIRST, XA>(c, eb, P, rot, dvg, gradP, dold, doldP, As, Bs, col, k, dn,
                                     dP, nu, nuP, J, gd);
        T divE = first(dvg), divB = second(dvg);
        if (XA && gd.bad()) {
          const StageValues<T> r = stage_point_ieee<FIRST>(c, uin, du, col, k, o, As, Bs);
#pragma unroll
          for (int a = 0; a < 3; ++a) {
            dn[a] = pk(r.d[a], r.d[3 + a]);
            nu[a] = pk(r.nu[a], r.nu[3 + a]);
            J[a] = r.J[a];
          }
          dP = r.d[6];
          nuP = r.nu[6];
          divE = r.divE;
          divB = r.divB;
        }
        const T u[7] = {first(eb[0]),  first(eb[1]),  first(eb[2]), second(eb[0]),
                        second(eb[1]), second(eb[2]), P};
        const T d7[7] = {first(dn[0]),  first(dn[1]),  first(dn[2]), second(dn[0]),
                         second(dn[1]), second(dn[2]), dP};
        T n7[7] = {first(nu[0]),  first(nu[1]),  first(nu[2]), second(nu[0]),
                   second(nu[1]), second(nu[2]), nuP};
        stage_finish<BC>(c, u, d7, n7, J, divE, divB, tst, flags, col, k, o, du, un, aux, uout);
      }
    }
    __syncthreads();
    issue(k + 3 + PF, head);  // into the slot of plane k-2
    head = slot(1);
  }
  cp_async_wait<0>();
}

// ---------------------------------------------------------------------------
// The same stage in FP32 with the z neighbours in a register window: planes k-2 ..
// k+2 of a thread's column travel through 35 registers (the z loop unrolled by ZU = 5,
// which renames instead of moving them; ZU = 1 with the boundary code, whose five
// copies would spill), each plane read from the ring once, as the leading one, so a field costs 9
// shared loads instead of 13; rows of even length are copied by aligned pairs.
// With 128 registers 16 warps share an SM.  Bound by dependency latency and the
// shared-memory queue (issue 52%, 613 instructions a point).  Stage at 512^3: 4526 us
// with one field per instruction and IEEE divisions, 4313 us here; with the ring
// kernel above instead (24 warps, but 13 shared loads per field and 4-byte copies)
// 5.0 ms, with two rows per thread (8 warps, 251 registers) 6.4 ms.
// ---------------------------------------------------------------------------
template <int PF>
__host__ __device__ constexpr int window_ring() {
  return 4 + PF;  // planes k .. k+2, the prefetch, a spare slot
}
template <typename T, int TX, int TY, int PF, int V>
constexpr size_t window_smem_bytes(bool first) {
  return (size_t)window_ring<PF>() * 7 * TileLoader<T, TX, TY, 2, V>::FB +
         (first ? 0 : (size_t)(PF + 2) * 7 * TX * TY * sizeof(T));
}

template <typename T, int TX, int TY, int PF, int ZU, bool FIRST, bool BC, int V, bool XA, bool DG>
__global__ void __launch_bounds__(TX * TY, min_blocks<T, TX * TY>())
    ez_stage_window_kernel(const __grid_constant__ EzConst<T> c, const F7<const T> uin,
                    const F7<T> uout, const F7<T> du, const F7<T> un, const F5<T> aux, const F6<T> dg,
                    const T As, const T Bs, const T tst, const int kchunk,
                    const int flags) {
  using L = TileLoader<T, TX, TY, 2, V>;
  constexpr int R = window_ring<PF>();    // field ring slots
  constexpr int DR = PF + 2;              // dU ring slots

  constexpr int ES = (int)sizeof(T);
  constexpr int SX = L::SX, FB = L::FB, SB = 7 * FB;
  constexpr int NT = TX * TY, DFB = NT * ES, DSB = 7 * DFB;
  constexpr int CEN = (2 * SX + 2) * ES;  // own point, from the corner of its 5x5 patch
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const uint32_t sbase = smem_u32(smem_raw);
  const uint32_t dbase = sbase + (uint32_t)(R * SB);

  const GridGeom& g = c.g;
  const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * TX + tx;
  const int i = g.lo[0] + blockIdx.x * TX + tx;
  const int j = g.lo[1] + blockIdx.y * TY + ty;
  const int k0 = g.lo[2] + blockIdx.z * kchunk;
  const int k1 = min(k0 + kchunk, g.hi[2]);
  const bool active = (i < g.hi[0]) && (j < g.hi[1]);
  // lanes of this warp that compute points: the fences between the field
  // groups below are executed by these lanes only (a tile that overhangs
  // the grid has idle lanes, which must not be named in the mask)
  const unsigned amask = __ballot_sync(0xffffffffu, active);
  const uint32_t sz = (uint32_t)g.sz;
  const uint32_t own = (uint32_t)j * (uint32_t)g.sy + (uint32_t)i;
  const ColumnCtx<T> col = make_column<XA>(c, i, j);
  const L loader(g, sbase, tid, g.lo[0] + (int)blockIdx.x * TX - 2,
                 g.lo[1] + (int)blockIdx.y * TY - 2);
  const uint32_t dme = dbase + (uint32_t)(tid * ES);
  const int kend = k1 + 2;  // planes [k0-2, k1+2) are read
  const int lo2 = g.lo[2];
  // byte offsets of the ring slots of plane k + OFF in window phase S:
  // compile-time constants in the unrolled loop
  auto fslot = [&](auto sc, auto oc, int k) -> uint32_t {
    constexpr int S = decltype(sc)::value, OFF = decltype(oc)::value;
    if constexpr (ZU == R) return (uint32_t)(((S + OFF) % R) * SB);
    else return (uint32_t)(((k + OFF - lo2) % R) * SB);
  };
  auto dslot = [&](auto sc, auto oc, int k) -> uint32_t {
    constexpr int S = decltype(sc)::value, OFF = decltype(oc)::value;
    if constexpr (ZU == DR) return (uint32_t)(((S + OFF) % DR) * DSB);
    else return (uint32_t)(((k + OFF - lo2) % DR) * DSB);
  };

  // copy plane kp into field slot fs and the dU of plane kp - 2 into dU
  // slot ds
  auto issue = [&](int kp, uint32_t fs, uint32_t dsl) {
    if (kp < kend) loader.copy(uin, (uint32_t)kp * sz, fs);
    if constexpr (!FIRST) {
      const int kd = kp - 2;
      if (kd >= k0 && kd < k1 && active) {
        const uint32_t ds = dme + dsl;
        const uint32_t e = (uint32_t)kd * sz + own;
        static_for<7>([&](auto fc) {
          constexpr int f = decltype(fc)::value;
          cp_async_off<sizeof(T), f * DFB>(ds, du.p[f] + e);
        });
      }
    }
    cp_async_commit();
  };
#pragma unroll 1
  for (int p = 0; p < 3 + PF; ++p)
    issue(k0 + p, (uint32_t)(((k0 + p - lo2) % R) * SB),
          (uint32_t)((((k0 + p - 2 - lo2) % DR + DR) % DR) * DSB));

  const T six = c.inv_delta[0] / (T)12, siy = c.inv_delta[1] / (T)12,
          siz = c.inv_delta[2] / (T)12;
  const T ix = c.inv_delta[0], iy = c.inv_delta[1], iz = c.inv_delta[2];
  const uint32_t corner = sbase + (uint32_t)((ty * SX + tx + loader.xoff) * ES);
  // Register window: in window phase S, w[(S + q) % 5][a] = (E_a, B_a) and
  // wp[(S + q) % 5] = P at (i, j, k - 2 + q).  Planes k-2 .. k+1 are carried
  // from the previous plane and k+2 is read from the ring into the slot of the
  // dead plane k-3, so advancing the window moves no registers when the z loop
  // is unrolled by the window length (ZU = 5).
  Pair<T> w[5][3];
  T wp[5];
  if (active) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint32_t e = (uint32_t)(k0 - 2 + q) * sz + own;
#pragma unroll
      for (int a = 0; a < 3; ++a) w[q][a] = pk(uin.p[a][e], uin.p[3 + a][e]);
      wp[q] = uin.p[6][e];
    }
  }

  auto plane = [&](auto sc, const int k) {
    constexpr int S = decltype(sc)::value;
    cp_async_wait<PF>();  // planes up to k+2 (and the dU of k) have landed
    __syncthreads();
    using Z = std::integral_constant<int, 0>;
    using P2 = std::integral_constant<int, 2>;
    using PN = std::integral_constant<int, 3 + PF>;   // the plane issued now
    using PD = std::integral_constant<int, 1 + PF>;   // and its dU plane
    issue(  // into the slot of plane k-1
        k + 3 + PF, fslot(sc, PN{}, k), dslot(sc, PD{}, k));
    if (active && k < k1) {
      const uint32_t a0 = corner + fslot(sc, Z{}, k);
      const uint32_t ap2 = corner + fslot(sc, P2{}, k);
      constexpr int W0 = S % 5, W1 = (S + 1) % 5, W2 = (S + 2) % 5, W3 = (S + 3) % 5,
                    W4 = (S + 4) % 5;
      // The stencil is consumed component by component, then P; the
      // warp-level fence between groups keeps the shared loads of the next
      // group from being hoisted, which bounds the live registers.  d[a]: the
      // derivatives along axis a of (E_x, B_x), ..., unscaled (the quotients of
      // diff1_4) in the reference arithmetic, which scales and combines them
      // as rk_step does (field_solver_EZ.cpp:143-150: the first product of a
      // curl rounded, the second fused), inv_delta-scaled otherwise.
      Guard<T> g;
      g.large = !c.tau_mid;
      auto derivatives = [&](auto ac, Pair<T> d[3]) {
        constexpr int a = decltype(ac)::value;
        auto at = [&](auto oc) {
          constexpr int off = decltype(oc)::value;
          return pk(lds<T, a * FB + off>(a0), lds<T, (3 + a) * FB + off>(a0));
        };
        using std::integral_constant;
        d[0] = pd1_4<XA>(at(integral_constant<int, CEN - 2 * ES>{}),
                         at(integral_constant<int, CEN - ES>{}),
                         at(integral_constant<int, CEN + ES>{}),
                         at(integral_constant<int, CEN + 2 * ES>{}), six, g);
        d[1] = pd1_4<XA>(at(integral_constant<int, 2 * ES>{}),
                         at(integral_constant<int, (SX + 2) * ES>{}),
                         at(integral_constant<int, (3 * SX + 2) * ES>{}),
                         at(integral_constant<int, (4 * SX + 2) * ES>{}), siy, g);
        w[W4][a] = pk(lds<T, a * FB + CEN>(ap2), lds<T, (3 + a) * FB + CEN>(ap2));
        d[2] = pd1_4<XA>(w[W0][a], w[W1][a], w[W3][a], w[W4][a], siz, g);
      };
      Pair<T> rot[3], dvg;
      T gradP[3];
      {
        Pair<T> xd[3], yd[3], zd[3];
        derivatives(std::integral_constant<int, 0>{}, xd);
        __syncwarp(amask);
        derivatives(std::integral_constant<int, 1>{}, yd);
        __syncwarp(amask);
        derivatives(std::integral_constant<int, 2>{}, zd);
        if constexpr (XA) {
          rot[0] = pfma(both(-iz), yd[2], pmul(both(iy), zd[1]));
          rot[1] = pfma(both(-ix), zd[0], pmul(both(iz), xd[2]));
          rot[2] = pfma(both(-iy), xd[1], pmul(both(ix), yd[0]));
          dvg = pfma(both(iz), zd[2], pfma(both(iy), yd[1], pmul(both(ix), xd[0])));
        } else {
          rot[0] = psub(zd[1], yd[2]);
          rot[1] = psub(xd[2], zd[0]);
          rot[2] = psub(yd[0], xd[1]);
          dvg = padd(padd(xd[0], yd[1]), zd[2]);
        }
      }
      __syncwarp(amask);
      {
        constexpr int o6 = 6 * FB;
        gradP[0] = sd1_4<XA>(lds<T, o6 + CEN - 2 * ES>(a0), lds<T, o6 + CEN - ES>(a0),
                             lds<T, o6 + CEN + ES>(a0), lds<T, o6 + CEN + 2 * ES>(a0), six, g);
        gradP[1] = sd1_4<XA>(lds<T, o6 + 2 * ES>(a0), lds<T, o6 + (SX + 2) * ES>(a0),
                             lds<T, o6 + (3 * SX + 2) * ES>(a0),
                             lds<T, o6 + (4 * SX + 2) * ES>(a0), siy, g);
        wp[W4] = lds<T, o6 + CEN>(ap2);
        gradP[2] = sd1_4<XA>(wp[W0], wp[W1], wp[W3], wp[W4], siz, g);
        if constexpr (XA) {
          gradP[0] = xa::mul(ix, gradP[0]);
          gradP[1] = xa::mul(iy, gradP[1]);
          gradP[2] = xa::mul(iz, gradP[2]);
        }
      }
      Pair<T> dold[3];
      T doldP = 0;
      if constexpr (!FIRST) {
        const uint32_t ad = dme + dslot(sc, Z{}, k);
        static_for<3>([&](auto ac) {
          constexpr int a = decltype(ac)::value;
          dold[a] = pk(lds<T, a * DFB>(ad), lds<T, (3 + a) * DFB>(ad));
        });
        doldP = lds<T, 6 * DFB>(ad);
      }
      const uint32_t o = (uint32_t)k * sz + own;
      const Pair<T>* eb = w[W2];
      const T u[7] = {first(eb[0]),  first(eb[1]),  first(eb[2]), second(eb[0]),
                      second(eb[1]), second(eb[2]), wp[W2]};
      if constexpr (DG) {
        Derivs<T> dv;
        T old[7];
        StageValues<T> r;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          dv.rotE[a] = first(rot[a]);
          dv.rotB[a] = second(rot[a]);
          dv.gradP[a] = gradP[a];
          old[a] = first(dold[a]);
          old[3 + a] = second(dold[a]);
        }
        dv.divE = first(dvg);
        dv.divB = second(dvg);
        old[6] = doldP;
        if (g.bad()) dv = point_derivatives_ieee(c, uin, o);
        stage_values_ieee<FIRST, true>(c, u, dv, old, As, Bs, col, k, dg, o, r);
        stage_finish<BC>(c, u, r.d, r.nu, r.J, r.divE, r.divB, tst, flags, col, k, o, du, un, aux,
                         uout);
      } else {
        Pair<T> dn[3], nu[3];
        T dP, nuP, J[3];
        stage_values_pair<FIRST, XA>(c, eb, u[6], rot, dvg, gradP, dold, doldP, As, Bs, col, k, dn,
                                     dP, nu, nuP, J, g);
        T d7[7], n7[7], divE = first(dvg), divB = second(dvg);
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          d7[a] = first(dn[a]);
          d7[3 + a] = second(dn[a]);
          n7[a] = first(nu[a]);
          n7[3 + a] = second(nu[a]);
        }
        d7[6] = dP;
        n7[6] = nuP;
        if (XA && g.bad()) {
          const StageValues<T> r = stage_point_ieee<FIRST>(c, uin, du, col, k, o, As, Bs);
#pragma unroll
          for (int f = 0; f < 7; ++f) {
            d7[f] = r.d[f];
            n7[f] = r.nu[f];
          }
#pragma unroll
          for (int a = 0; a < 3; ++a) J[a] = r.J[a];
          divE = r.divE;
          divB = r.divB;
        }
        stage_finish<BC>(c, u, d7, n7, J, divE, divB, tst, flags, col, k, o, du, un, aux, uout);
      }
      if constexpr (ZU == 1) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
#pragma unroll
          for (int a = 0; a < 3; ++a) w[q][a] = w[q + 1][a];
          wp[q] = wp[q + 1];
        }
      }
    }
  };
  if constexpr (ZU == 5) {
    // planes past k1 in the last group only wait, synchronise and commit
    // empty copy groups (issue() copies nothing past kend), so the ring's
    // group accounting stays the same as plane-by-plane
#pragma unroll 1
    for (int k = k0; k < k1; k += 5) {
      plane(std::integral_constant<int, 0>{}, k);
      plane(std::integral_constant<int, 1>{}, k + 1);
      plane(std::integral_constant<int, 2>{}, k + 2);
      plane(std::integral_constant<int, 3>{}, k + 3);
      plane(std::integral_constant<int, 4>{}, k + 4);
    }
  } else {
#pragma unroll 1
    for (int k = k0; k < k1; ++k) plane(std::integral_constant<int, 0>{}, k);
  }
  cp_async_wait<0>();
}

// ---------------------------------------------------------------------------
// Kreiss-Oliger dissipation + clamps + star boundary at t + dt + guard fill
// (reference Kreiss_Oliger and the tail of evolve_fields,
// field_solver_EZ.cpp:324-457, 1057-1072; .cu:272-392, 696-706):
//   f' = f + (-KOeps * KO_const) * sum_axes diff6_2(f)
// for E and B (CPU build) or E, B and P (GPU build).  The operator has 18
// neighbours per field, so the z direction is held in a register window of
// planes k-3..k+3 per thread; shared memory keeps plane k (x/y neighbours)
// and the arriving planes k+1..k+3+PF.
// ---------------------------------------------------------------------------
// Spare ring slots (0 or 1) of the KO kernel.  With a spare slot the copies of
// a new plane are issued right after the one barrier at the top of an
// iteration; without it they wait for a second barrier after the iteration's
// arithmetic.  Measured at 512^3: faster without (two CTAs per SM).
#ifndef COFFEE_KO_RING_SPARE
#define COFFEE_KO_RING_SPARE 0
#endif
constexpr int kKoRingSpare = COFFEE_KO_RING_SPARE;
static_assert(kKoRingSpare == 0 || kKoRingSpare == 1, "0 or 1 spare ring slot");

// z-loop unroll of the KO kernel: 7 (the window length, no register moves)
// or 1 (one plane per iteration, window shifted by moves), per instance
// (with and without the boundary code); both are faster unrolled.
#ifndef COFFEE_KO_ZUNROLL
#define COFFEE_KO_ZUNROLL 7
#endif
#ifndef COFFEE_KO_ZUNROLL_BC
#define COFFEE_KO_ZUNROLL_BC 7
#endif
template <bool BC>
__host__ __device__ constexpr int ko_zunroll() {
  return BC ? COFFEE_KO_ZUNROLL_BC : COFFEE_KO_ZUNROLL;
}
static_assert((ko_zunroll<false>() == 1 || ko_zunroll<false>() == 7) &&
                  (ko_zunroll<true>() == 1 || ko_zunroll<true>() == 7),
              "KO z unroll is 1 or 7");

// Ring slots of the KO kernel (plane k in slot (k - lo[2]) % R).  A 7-slot
// ring, matching the z unroll, would make the slots compile-time constants
// but measured far slower (its shared memory leaves the two resident CTAs
// little L1 cache).
template <bool BC, int PF>
__host__ __device__ constexpr int ko_ring() {
  return 4 + PF + kKoRingSpare;
}

template <typename T, int TX, int TY, int PF, int V, bool BC>
constexpr size_t ko_smem_bytes() {
  return (size_t)ko_ring<BC, PF>() * 7 * TileLoader<T, TX, TY, 3, V>::FB;
}

template <typename T, int TX, int TY, int PF, bool BC, int V, bool XA, bool DG>
__global__ void __launch_bounds__(TX * TY, min_blocks<T, TX * TY>())
    ez_ko_kernel(const __grid_constant__ EzConst<T> c, const F7<const T> uin,
                 const F7<T> uout, const F6<T> dg, const T tko, const int kchunk) {
  static_assert(XA || !DG, "the energy diagnostics need the reference arithmetic");
  using L = TileLoader<T, TX, TY, 3, V>;
  constexpr int R = ko_ring<BC, PF>();
  constexpr int ZU = ko_zunroll<BC>();

  constexpr int ES = (int)sizeof(T);
  constexpr int SX = L::SX, FB = L::FB, SB = 7 * FB;
  constexpr int CEN = (3 * SX + 3) * ES;  // own point, from the corner of its 7x7 patch
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const uint32_t sbase = smem_u32(smem_raw);

  const GridGeom& g = c.g;
  const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * TX + tx;
  const int i = g.lo[0] + blockIdx.x * TX + tx;
  const int j = g.lo[1] + blockIdx.y * TY + ty;
  const int k0 = g.lo[2] + blockIdx.z * kchunk;
  const int k1 = min(k0 + kchunk, g.hi[2]);
  const bool active = (i < g.hi[0]) && (j < g.hi[1]);
  const uint32_t sz = (uint32_t)g.sz;
  const uint32_t own = (uint32_t)j * (uint32_t)g.sy + (uint32_t)i;
  const ColumnCtx<T> col = make_column<XA>(c, i, j);
  const L loader(g, sbase, tid, g.lo[0] + (int)blockIdx.x * TX - 3,
                 g.lo[1] + (int)blockIdx.y * TY - 3);
  const int kend = k1 + 3;  // planes [k0, k1+3) pass through shared memory
  const int lo2 = g.lo[2];
  // byte offset of the ring slot of plane k + OFF in window phase S
  auto fslot = [&](auto sc, auto oc, int k) -> uint32_t {
    constexpr int S = decltype(sc)::value, OFF = decltype(oc)::value;
    if constexpr (ZU == R) return (uint32_t)(((S + OFF) % R) * SB);
    else return (uint32_t)(((k + OFF - lo2) % R) * SB);
  };
  auto issue = [&](int kp, uint32_t fs) {
    if (kp < kend) loader.copy(uin, (uint32_t)kp * sz, fs);
    cp_async_commit();
  };
#pragma unroll 1
  for (int p = 0; p < 4 + PF; ++p) issue(k0 + p, (uint32_t)(((k0 + p - lo2) % R) * SB));

  // Register window: in window phase S, w[(S + q) % 7][a] = (E_a, B_a) and
  // wp[(S + q) % 7] = P at (i, j, k - 3 + q); planes k-3 .. k+2 are carried,
  // k+3 is read from the ring into the slot of the dead plane k-4 (no register
  // moves when the z loop is unrolled by the window length, ZU = 7).
  Pair<T> w[7][3];
  T wp[7];
  if (active) {
#pragma unroll
    for (int q = 0; q < 6; ++q) {
      const uint32_t e = (uint32_t)(k0 - 3 + q) * sz + own;
#pragma unroll
      for (int a = 0; a < 3; ++a) w[q][a] = pk(uin.p[a][e], uin.p[3 + a][e]);
      wp[q] = uin.p[6][e];
    }
  }
  const bool ko_p = (c.semantics != SEM_CPU_REF);
  const uint32_t corner = sbase + (uint32_t)((ty * SX + tx + loader.xoff) * ES);
  auto plane = [&](auto sc, const int k) {
    constexpr int S = decltype(sc)::value;
    cp_async_wait<PF>();  // plane k+3 has landed
    __syncthreads();
    using PN = std::integral_constant<int, 4 + PF>;  // the plane issued now
    if constexpr (kKoRingSpare == 1) issue(k + 4 + PF, fslot(sc, PN{}, k));  // slot of plane k-1
    if (active && k < k1) {
      const uint32_t a0 = corner + fslot(sc, std::integral_constant<int, 0>{}, k);
      const uint32_t a3 = corner + fslot(sc, std::integral_constant<int, 3>{}, k);
      constexpr int C3 = (S + 3) % 7;  // the window slot of plane k
      Pair<T> nu[3];
      T nuP = wp[C3];
      static_for<3>([&](auto ac) {
        constexpr int a = decltype(ac)::value;
        using std::integral_constant;
        auto at = [&](auto oc) {
          constexpr int off = decltype(oc)::value;
          return pk(lds<T, a * FB + off>(a0), lds<T, (3 + a) * FB + off>(a0));
        };
        w[(S + 6) % 7][a] = pk(lds<T, a * FB + CEN>(a3), lds<T, (3 + a) * FB + CEN>(a3));
        const Pair<T> cv = w[C3][a];
        const Pair<T> kx = pd6_2<XA>(at(integral_constant<int, CEN - 3 * ES>{}),
                                     at(integral_constant<int, CEN - 2 * ES>{}),
                                     at(integral_constant<int, CEN - ES>{}), cv,
                                     at(integral_constant<int, CEN + ES>{}),
                                     at(integral_constant<int, CEN + 2 * ES>{}),
                                     at(integral_constant<int, CEN + 3 * ES>{}));
        const Pair<T> ky = pd6_2<XA>(at(integral_constant<int, 3 * ES>{}),
                                     at(integral_constant<int, (SX + 3) * ES>{}),
                                     at(integral_constant<int, (2 * SX + 3) * ES>{}), cv,
                                     at(integral_constant<int, (4 * SX + 3) * ES>{}),
                                     at(integral_constant<int, (5 * SX + 3) * ES>{}),
                                     at(integral_constant<int, (6 * SX + 3) * ES>{}));
        const Pair<T> kz = pd6_2<XA>(w[S % 7][a], w[(S + 1) % 7][a], w[(S + 2) % 7][a], cv,
                                     w[(S + 4) % 7][a], w[(S + 5) % 7][a], w[(S + 6) % 7][a]);
        // the reference arithmetic sums the axes x, y, z left to right and
        // fuses f + KO (-KOeps KO_const) (field_solver_EZ.cpp:350-420)
        nu[a] = pfma(both(c.ko_c), padd(padd(kx, ky), kz), cv);
      });
      wp[(S + 6) % 7] = lds<T, 6 * FB + CEN>(a3);
      if (ko_p) {
        constexpr int o6 = 6 * FB;
        const T kx = d6_2(lds<T, o6 + CEN - 3 * ES>(a0), lds<T, o6 + CEN - 2 * ES>(a0),
                          lds<T, o6 + CEN - ES>(a0), nuP, lds<T, o6 + CEN + ES>(a0),
                          lds<T, o6 + CEN + 2 * ES>(a0), lds<T, o6 + CEN + 3 * ES>(a0));
        const T ky = d6_2(lds<T, o6 + 3 * ES>(a0), lds<T, o6 + (SX + 3) * ES>(a0),
                          lds<T, o6 + (2 * SX + 3) * ES>(a0), nuP,
                          lds<T, o6 + (4 * SX + 3) * ES>(a0), lds<T, o6 + (5 * SX + 3) * ES>(a0),
                          lds<T, o6 + (6 * SX + 3) * ES>(a0));
        const T kz = d6_2(wp[S % 7], wp[(S + 1) % 7], wp[(S + 2) % 7], nuP, wp[(S + 4) % 7],
                          wp[(S + 5) % 7], wp[(S + 6) % 7]);
        nuP = sfma(kx + ky + kz, c.ko_c, nuP);
      }
      const uint32_t o = (uint32_t)k * sz + own;
      T n7[7] = {first(nu[0]),  first(nu[1]),  first(nu[2]), second(nu[0]),
                 second(nu[1]), second(nu[2]), nuP};
      if constexpr (DG) {
        // dU_KO = (|B|^2 + |E|^2) after the pass minus before it, and
        // dU_KO_cum += it (field_solver_EZ.cpp:398-455)
        const Pair<T> s0 = pdot3(w[C3], w[C3]), s1 = pdot3(nu, nu);
        const T dko = xa::sub(xa::add(second(s1), first(s1)), xa::add(second(s0), first(s0)));
        dg.p[5][o] = xa::add(dko, dg.p[5][o]);
        dg.p[2][o] = dko;
        apply_clamps_xa_dg<false>(n7[0], n7[1], n7[2], n7[3], n7[4], n7[5], dg, o);
      } else if constexpr (XA) {
        apply_clamps_mid(n7);
      } else {
        apply_clamps(c, n7[0], n7[1], n7[2], n7[3], n7[4], n7[5]);
      }
      if constexpr (BC) star_boundary(c, i, j, k, tko, n7);
      store_with_images(g, col, uout, k, o, n7);
      if constexpr (ZU == 1) {
#pragma unroll
        for (int q = 0; q < 6; ++q) {
#pragma unroll
          for (int a = 0; a < 3; ++a) w[q][a] = w[q + 1][a];
          wp[q] = wp[q + 1];
        }
      }
    }
    if constexpr (kKoRingSpare == 0) {
      __syncthreads();
      issue(k + 4 + PF, fslot(sc, PN{}, k));  // into the slot of plane k (or k-2 of 7)
    }
  };
  if constexpr (ZU == 7) {
    // planes past k1 in the last group only wait, synchronise and commit
    // empty copy groups (issue() copies nothing past kend)
#pragma unroll 1
    for (int k = k0; k < k1; k += 7) {
      plane(std::integral_constant<int, 0>{}, k);
      plane(std::integral_constant<int, 1>{}, k + 1);
      plane(std::integral_constant<int, 2>{}, k + 2);
      plane(std::integral_constant<int, 3>{}, k + 3);
      plane(std::integral_constant<int, 4>{}, k + 4);
      plane(std::integral_constant<int, 5>{}, k + 5);
      plane(std::integral_constant<int, 6>{}, k + 6);
    }
  } else {
#pragma unroll 1
    for (int k = k0; k < k1; ++k) plane(std::integral_constant<int, 0>{}, k);
  }
  cp_async_wait<0>();
}

// ---------------------------------------------------------------------------
// The stage and the KO pass with one point per thread, straight from global memory.
// A small grid fills the GPU with neither tiles nor planes (at 32^3 the streaming
// kernels run 14 CTAs, each waiting for one plane after the other), and up to some
// 200^3 points the stencil's 13 planes of 7 fields stay in L2 and L1, so that loads
// without tiles, barriers or a window cost less than they save: 80 registers, 24
// warps per SM, neighbours in z within a block (32 x 4 x 2 threads).  The arithmetic
// is the streaming kernels' (bit for bit in the reference arithmetic).  Stage of one
// point per thread against the streaming one, us: 32^3 13 / 19, 128^3 87 / 94, 192^3
// 258 / 283, 256^3 591 / 570, 512^3 5128 / 4313; with the star 192^3 298 / 426, 384^3
// 2264 / 2370.  What bounds it is the latency of the loads (FP32) and, from 256^3 on,
// L2 misses.
// ---------------------------------------------------------------------------
#ifndef COFFEE_DIRECT_Y
#define COFFEE_DIRECT_Y 4
#endif
#ifndef COFFEE_DIRECT_Z
#define COFFEE_DIRECT_Z 2
#endif
#ifndef COFFEE_DIRECT_MINB
#define COFFEE_DIRECT_MINB 3
#endif
constexpr int kDirectX = 32, kDirectY = COFFEE_DIRECT_Y;
template <typename T>
__host__ __device__ constexpr int direct_z() {
  return sizeof(T) == 4 ? COFFEE_DIRECT_Z : 1;
}

template <typename T, bool FIRST, bool BC, bool XA>
__global__ void __launch_bounds__(kDirectX * kDirectY * direct_z<T>(),
                                  sizeof(T) == 4 ? COFFEE_DIRECT_MINB : 2)
    ez_stage_direct_kernel(const __grid_constant__ EzConst<T> c, const F7<const T> uin,
                           const F7<T> uout, const F7<T> du, const F7<T> un, const F5<T> aux,
                           const T As, const T Bs, const T tst, const int flags, const int j0,
                           const int k0) {
  const GridGeom& g = c.g;
  const int i = g.lo[0] + blockIdx.x * kDirectX + threadIdx.x;
  const int j = j0 + blockIdx.y * kDirectY + threadIdx.y;
  const int k = k0 + blockIdx.z * direct_z<T>() + threadIdx.z;
  if (i >= g.hi[0] || j >= g.hi[1] || k >= g.hi[2]) return;
  const uint32_t sy = (uint32_t)g.sy, sz = (uint32_t)g.sz;
  const uint32_t o = (uint32_t)k * sz + (uint32_t)j * sy + (uint32_t)i;
  const ColumnCtx<T> col = make_column<XA>(c, i, j);
  Pair<T> dold[3];
  T doldP = 0;
  if constexpr (!FIRST) {
#pragma unroll
    for (int a = 0; a < 3; ++a) dold[a] = pk(du.p[a][o], du.p[3 + a][o]);
    doldP = du.p[6][o];
  }
  const T ix = c.inv_delta[0], iy = c.inv_delta[1], iz = c.inv_delta[2];
  const uint32_t st[3] = {1u, sy, sz};
  Guard<T> gd;
  gd.large = !c.tau_mid;
  Pair<T> d[3][3];  // d[a][x]: component a along axis x
  T dp[3];
#pragma unroll
  for (int x = 0; x < 3; ++x) {
    const T f12 = c.inv_delta[x] / (T)12;
    const uint32_t q[4] = {o - 2 * st[x], o - st[x], o + st[x], o + 2 * st[x]};
    T p[4];
#pragma unroll
    for (int n = 0; n < 4; ++n) p[n] = __ldg(uin.p[6] + q[n]);
    dp[x] = sd1_4<XA>(p[0], p[1], p[2], p[3], f12, gd);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      Pair<T> v[4];
#pragma unroll
      for (int n = 0; n < 4; ++n) v[n] = pk(__ldg(uin.p[a] + q[n]), __ldg(uin.p[3 + a] + q[n]));
      d[a][x] = pd1_4<XA>(v[0], v[1], v[2], v[3], f12, gd);
    }
  }
  Pair<T> rot[3], dvg;
  if constexpr (XA) {
    rot[0] = pfma(both(-iz), d[1][2], pmul(both(iy), d[2][1]));
    rot[1] = pfma(both(-ix), d[2][0], pmul(both(iz), d[0][2]));
    rot[2] = pfma(both(-iy), d[0][1], pmul(both(ix), d[1][0]));
    dvg = pfma(both(iz), d[2][2], pfma(both(iy), d[1][1], pmul(both(ix), d[0][0])));
    dp[0] = xa::mul(ix, dp[0]);
    dp[1] = xa::mul(iy, dp[1]);
    dp[2] = xa::mul(iz, dp[2]);
  } else {
    rot[0] = psub(d[2][1], d[1][2]);
    rot[1] = psub(d[0][2], d[2][0]);
    rot[2] = psub(d[1][0], d[0][1]);
    dvg = padd(padd(d[0][0], d[1][1]), d[2][2]);
  }
  Pair<T> eb[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) eb[a] = pk(__ldg(uin.p[a] + o), __ldg(uin.p[3 + a] + o));
  const T P = __ldg(uin.p[6] + o);
  StageValues<T> r;
  {
    Pair<T> dn[3], nu[3];
    stage_values_pair<FIRST, XA>(c, eb, P, rot, dvg, dp, dold, doldP, As, Bs, col, k, dn, r.d[6],
                                 nu, r.nu[6], r.J, gd);
    r.divE = first(dvg);
    r.divB = second(dvg);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      r.d[a] = first(dn[a]);
      r.d[3 + a] = second(dn[a]);
      r.nu[a] = first(nu[a]);
      r.nu[3 + a] = second(nu[a]);
    }
  }
  if (XA && gd.bad()) r = stage_point_ieee<FIRST>(c, uin, du, col, k, o, As, Bs);
  const T u[7] = {first(eb[0]),  first(eb[1]),  first(eb[2]), second(eb[0]),
                  second(eb[1]), second(eb[2]), P};
  stage_finish<BC>(c, u, r.d, r.nu, r.J, r.divE, r.divB, tst, flags, col, k, o, du, un, aux, uout);
}

template <typename T, bool BC, bool XA>
__global__ void __launch_bounds__(kDirectX * kDirectY * direct_z<T>(),
                                  sizeof(T) == 4 ? COFFEE_DIRECT_MINB : 2)
    ez_ko_direct_kernel(const __grid_constant__ EzConst<T> c, const F7<const T> uin,
                        const F7<T> uout, const T tko, const int j0, const int k0) {
  const GridGeom& g = c.g;
  const int i = g.lo[0] + blockIdx.x * kDirectX + threadIdx.x;
  const int j = j0 + blockIdx.y * kDirectY + threadIdx.y;
  const int k = k0 + blockIdx.z * direct_z<T>() + threadIdx.z;
  if (i >= g.hi[0] || j >= g.hi[1] || k >= g.hi[2]) return;
  const uint32_t st[3] = {1u, (uint32_t)g.sy, (uint32_t)g.sz};
  const uint32_t o = (uint32_t)k * st[2] + (uint32_t)j * st[1] + (uint32_t)i;
  const ColumnCtx<T> col = make_column<XA>(c, i, j);
  T n7[7];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    auto at = [&](uint32_t q) { return pk(__ldg(uin.p[a] + q), __ldg(uin.p[3 + a] + q)); };
    const Pair<T> cv = at(o);
    Pair<T> s[3];
#pragma unroll
    for (int x = 0; x < 3; ++x)
      s[x] = pd6_2<XA>(at(o - 3 * st[x]), at(o - 2 * st[x]), at(o - st[x]), cv, at(o + st[x]),
                       at(o + 2 * st[x]), at(o + 3 * st[x]));
    const Pair<T> v = pfma(both(c.ko_c), padd(padd(s[0], s[1]), s[2]), cv);
    n7[a] = first(v);
    n7[3 + a] = second(v);
  }
  n7[6] = __ldg(uin.p[6] + o);
  if (c.semantics != SEM_CPU_REF) {
    const T* p = uin.p[6];
    T s[3];
#pragma unroll
    for (int x = 0; x < 3; ++x)
      s[x] = d6_2(__ldg(p + (o - 3 * st[x])), __ldg(p + (o - 2 * st[x])), __ldg(p + (o - st[x])),
                  n7[6], __ldg(p + (o + st[x])), __ldg(p + (o + 2 * st[x])),
                  __ldg(p + (o + 3 * st[x])));
    n7[6] = sfma(s[0] + s[1] + s[2], c.ko_c, n7[6]);
  }
  if constexpr (XA) apply_clamps_mid(n7);
  else apply_clamps(c, n7[0], n7[1], n7[2], n7[3], n7[4], n7[5]);
  if constexpr (BC) star_boundary(c, i, j, k, tko, n7);
  store_with_images(g, col, uout, k, o, n7);
}

}  // namespace coffee
