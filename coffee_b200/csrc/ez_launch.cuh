// Host-side helpers shared by the translation units that launch the flat
// EZ kernels: the environment record, tile shapes and their shared-memory
// sizes, the LSRK coefficients, the z-chunk choice and the construction of
// the kernels' parameter block from the simulation parameters.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>

#include "coffee_b200.h"
#include "coffee_internal.h"
#include "ez_kernels.cuh"

// sim_environment of one rank on one GPU
struct coffee_env {
  coffee_params p;
  coffee_grid grid;
  int device;
  // fields and solvers created on this environment keep it alive: it is
  // deleted when it has been destroyed and the last of them is gone, in
  // whatever order the host releases them
  std::atomic<int> users{0};
  std::atomic<bool> released{false};
};

namespace coffee {


template <typename T> struct Shape;
// FP32 tile shapes; the defaults are the tuned values, the macros exist so
// that a build can be made with other shapes to measure them.
#ifndef COFFEE_F32_STY
#define COFFEE_F32_STY 12
#endif
#ifndef COFFEE_F32_SPF
#define COFFEE_F32_SPF 1
#endif
#ifndef COFFEE_F32_SMINB
#define COFFEE_F32_SMINB 2
#endif
#ifndef COFFEE_F32_KTY
#define COFFEE_F32_KTY 8
#endif
#ifndef COFFEE_F32_KPF
#define COFFEE_F32_KPF 1
#endif
template <> struct Shape<float> {
  // stage tile, planes of prefetch, resident CTAs per SM
  static constexpr int STX = 32, STY = COFFEE_F32_STY, SPF = COFFEE_F32_SPF;
  static constexpr int SMINB = COFFEE_F32_SMINB;
  static constexpr int KTX = 32, KTY = COFFEE_F32_KTY, KPF = COFFEE_F32_KPF;  // KO tile, prefetch
};
template <> struct Shape<double> {
  static constexpr int STX = 32, STY = 12, SPF = 1, SMINB = 1;
  static constexpr int KTX = 32, KTY = 4, KPF = 1;
};

template <typename T, int V, bool BC>
size_t ko_smem() {
  using S = Shape<T>;
  return ko_smem_bytes<T, S::KTX, S::KTY, S::KPF, V, BC>();
}

// LSRK(5,4) coefficients of the reference (field_solver_EZ.cpp:1009-1014)
constexpr double kAs[5] = {0, -0.4178904745, -1.192151694643, -1.697784692471, -1.514183444257};
constexpr double kBs[5] = {0.1496590219993, 0.3792103129999, 0.8229550293869, 0.6994504559488,
                       0.1530572479681};
constexpr double kCs[5] = {0, 0.1496590219993, 0.3704009573644, 0.6222557631345, 0.9582821306784};

// Choose the z chunk of a CTA: enough CTAs to fill the GPU in whole waves,
// while the 2H halo planes each chunk re-reads stay a small fraction.  The
// chunk is a multiple of `mult` (the kernel's z unroll, whose ring slots are
// then compile-time constants), except that it may be all nz planes.
inline int pick_kchunk(int nz, int nxy_tiles, int slots, int halo, int mult) {
  int best = nz;
  double best_cost = 1e300;
  const int step = mult > 1 ? mult : 4;
  for (int kc = step; kc <= nz + step - 1; kc += step) {
    const int kk = std::min(kc, nz);
    const long long ctas = (long long)nxy_tiles * ((nz + kk - 1) / kk);
    const double waves = std::ceil((double)ctas / (double)slots);
    const double cost = waves * (kk + 0.5 * halo);
    if (cost < best_cost - 1e-9) {
      best_cost = cost;
      best = kk;
    }
    if (kk == nz) break;
  }
  return best;
}

template <typename T>
void build_const(const coffee_env* env, int semantics, EzConst<T>* c) {
  const coffee_params& p = env->p;
  const coffee_grid& gr = env->grid;
  std::memset(c, 0, sizeof(*c));
  GridGeom& g = c->g;
  for (int a = 0; a < 3; ++a) {
    g.dims[a] = gr.dims[a];
    g.guard[a] = gr.guard[a];
    g.N[a] = gr.dims[a] - 2 * gr.guard[a];
    g.lo[a] = gr.guard[a] - p.shift_ghost;
    g.hi[a] = gr.dims[a] - gr.guard[a] + p.shift_ghost;
    g.periodic[a] = p.periodic_boundary[a] ? 1 : 0;
    c->delta[a] = (T)(T(p.size[a]) / (T)p.N[a]);
    c->inv_delta[a] = (T)(1.0 / (double)c->delta[a]);
    c->lower[a] = (T)p.lower[a];
  }
  g.sy = gr.dims[0];
  g.sz = (long long)gr.dims[0] * gr.dims[1];
  c->dt = (T)p.dt;
  c->ch2 = (T)p.ch2;
  c->tau = (T)p.tau;
  c->inv_tau = (T)1 / c->tau;  // correctly rounded: the quotients P / tau need it
  // -KOeps * KO_const with KO_const = -1/64 (FFE_DISSIPATION_ORDER 6)
  c->ko_c = -(T)p.KOeps * (T)(-1.0 / 64.0);
  c->gam_dt = (T)p.damp_gamma / (T)p.dt;
  c->use_edotb = p.use_edotb_damping;
  c->divB_clean = p.divB_clean;
  c->clean_ep = p.clean_ep;
  c->check_egb = p.check_egb;
  c->semantics = semantics;
  c->taper_lanes = (sizeof(T) == 4) ? 16 : 8;  // AVX-512 width of the reference CPU build
  // Quotients by tau stay in the range of the straight-line division: a point's |P| is
  // below 2^50 there, so that 2^64 P / tau, which it forms in FP32, stays below 2^127.
  // (A step with a smaller tau diverges: P's decay rate is 1 / tau per stage.)
  c->tau_mid = std::fabs((double)c->tau) >= 1.0 / 8192 && std::fabs((double)c->tau) < 1e6;
  c->problem = p.problem;
  bool abs_any = p.shift_ghost > 0;
  for (int a = 0; a < 3; ++a) {
    const T pm = (T)p.pml[a] * c->delta[a];
    c->pml_hi[a] = (T)p.lower[a] + (T)p.size[a] - pm;
    c->pml_lo[a] = (T)p.lower[a] + pm;
    c->pml_scale[a] = (T)p.pmllen * (semantics == SEM_CPU_REF ? c->delta[a] : c->delta[0]);
    if (p.pml[a] > 0) abs_any = true;
  }
  c->absorbing = abs_any ? 1 : 0;
  c->sigpml = (T)p.sigpml;
  c->radius = (T)p.radius;
  c->omega = (T)p.omega;
  c->b0 = (T)p.b0;
  c->p1 = (T)p.p1; c->p2 = (T)p.p2; c->p3 = (T)p.p3;
  c->q11 = (T)p.q11; c->q12 = (T)p.q12; c->q13 = (T)p.q13; c->q22 = (T)p.q22;
  c->q23 = (T)p.q23;
  c->qox = (T)p.q_offset_x; c->qoy = (T)p.q_offset_y; c->qoz = (T)p.q_offset_z;
  c->tp_start = (T)p.tp_start; c->tp_end = (T)p.tp_end; c->rpert1 = (T)p.rpert1;
  c->rpert2 = (T)p.rpert2; c->dw0 = (T)p.dw0; c->nT = (T)p.nT; c->ph1 = (T)p.ph1;
  c->ph2 = (T)p.ph2; c->dph = (T)p.dph; c->theta0 = (T)p.theta0; c->drpert = (T)p.drpert;
  c->tp_start1 = (T)p.tp_start1; c->tp_end1 = (T)p.tp_end1; c->rpert11 = (T)p.rpert11;
  c->rpert21 = (T)p.rpert21; c->dw1 = (T)p.dw1; c->nT1 = (T)p.nT1; c->ph11 = (T)p.ph11;
  c->ph21 = (T)p.ph21; c->dph1 = (T)p.dph1;
  c->pert_type = p.pert_type;
}

template <typename T>
inline F7<T> f7(void* const* a) {
  F7<T> r;
  for (int f = 0; f < 7; ++f) r.p[f] = static_cast<T*>(a[f]);
  return r;
}
template <typename T>
inline F7<const T> f7c(void* const* a) {
  F7<const T> r;
  for (int f = 0; f < 7; ++f) r.p[f] = static_cast<const T*>(a[f]);
  return r;
}

inline int num_sms(int device) {
  int n = 148;
  cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device);
  return n;
}

// Whether a run needs the star / absorbing-layer code in its kernels (the
// kernels are compiled with and without it, see ez_stage_kernel).
inline bool flat_needs_bc(const coffee_params& p, int semantics) {
  if (p.problem == 1 || (p.problem == 2 && semantics == SEM_CPU_REF)) return true;
  if (p.shift_ghost > 0) return true;
  for (int a = 0; a < 3; ++a)
    if (p.pml[a] > 0) return true;
  return false;
}

// Points up to which the one-point-per-thread kernels are the faster ones (us, one
// point per thread / streaming): FP32 stage 192^3 258 / 283, 256^3 591 / 570; FP32 KO
// 128^3 76 / 76, 192^3 226 / 202; regrouped arithmetic, stage and KO 96^3 38 + 37 / 43
// + 35, 128^3 85 + 87 / 79 + 76; FP64 stage 160^3 360 / 372, 256^3 1418 / 1320, KO
// 256^3 978 / 1044.  With the boundary code the stage in the reference arithmetic is
// faster up to 450^3 (192^3 298 / 421, 384^3 2264 / 2370) and within the runs' spread at
// 512^3 (5807 / 5732; whole steps 32.4 / 32.2 ms, +- 0.4): the only one.  Its KO pass is
// faster up to 384^3 (1762 / 1790; 512^3 4538 / 3793), the regrouped ones
// below 256^3 (192^3 300 + 271 / 334 + 317, 256^3 681 + 619 / 586 + 521).
struct DirectPoints {
  long long stage, ko;
};
template <typename T>
constexpr DirectPoints direct_points(bool bc, bool xa) {
  if (sizeof(T) == 8) return {8000000, 20000000};
  if (bc && xa) return {1LL << 31, 57000000};
  if (bc) return {10000000, 10000000};
  if (xa) return {12000000, 2200000};
  return {1200000, 1200000};
}

// Launch geometry of the flat kernels for one grid.
struct FlatLaunch {
  bool bc;   // star / absorbing-layer code compiled in
  bool vec;  // planes copied as aligned element pairs (even row length d0)
  bool xa;   // the CPU build's own arithmetic (CPU semantics, ez_refarith.cuh)
  bool dg;   // and its energy-change diagnostics (xa only)
  // one point per thread (not with the diagnostics)
  bool direct_stage, direct_ko;
  bool two_images;  // N < 2 guard on a periodic axis (ez_images_kernel)
  int kchunk_stage, kchunk_ko;
  dim3 grid_stage, grid_ko;
};

template <typename T, bool BC, int V, bool XA, bool DG = false>
struct FlatKernels {
  using S = Shape<T>;
  // the stage kernel: in FP32 the register window, but for the boundary code in the
  // reference arithmetic, which has one point per thread at every size and, with the
  // diagnostics, the plane ring; in FP64 the plane ring
  static constexpr bool kFloat = std::is_same<T, float>::value;
  static constexpr bool kDirectOnly = kFloat && BC && XA && !DG;  // the stage kernel
  static constexpr bool kWindow = kFloat && !(BC && XA);
  static constexpr int kTileX = 32, kTileY = kWindow ? 16 : S::STY;  // points of a stage CTA
  static constexpr int kZU = BC ? 1 : 5;                 // z unroll of the window kernel
  static constexpr int kChunkMult = kWindow ? kZU : 1;   // z chunks are multiples of it
  template <bool FIRST>
  static constexpr auto stage_fn() {
    if constexpr (kWindow)
      return ez_stage_window_kernel<T, kTileX, kTileY, S::SPF, kZU, FIRST, BC, V, XA, DG>;
    else
      return ez_stage_kernel<T, S::STX, S::STY, S::SPF, S::SMINB, FIRST, BC, XA, DG>;
  }
  static constexpr size_t stage_bytes(bool first) {
    if constexpr (kWindow) return window_smem_bytes<T, kTileX, kTileY, S::SPF, V>(first);
    else return stage_smem_bytes<T, S::STX, S::STY, S::SPF>();
  }
  static constexpr auto ko_fn() {
    return ez_ko_kernel<T, S::KTX, S::KTY, S::KPF, BC, V, XA, DG>;
  }


  static cudaError_t set_attributes() {
    cudaError_t e = cudaSuccess;
    if constexpr (!kDirectOnly) {
      e = cudaFuncSetAttribute(stage_fn<true>(), cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)stage_bytes(true));
      if (e == cudaSuccess)
        e = cudaFuncSetAttribute(stage_fn<false>(), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)stage_bytes(false));
    }
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(ko_fn(), cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)ko_smem<T, V, BC>());
    return e;
  }
  static cudaError_t occupancy(int* stage, int* kop) {
    cudaError_t e = cudaSuccess;
    if constexpr (!kDirectOnly)
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(stage, stage_fn<false>(), kTileX * kTileY,
                                                        stage_bytes(false));
    if (e == cudaSuccess)
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(kop, ko_fn(), S::KTX * S::KTY,
                                                        ko_smem<T, V, BC>());
    return e;
  }
  // launches of the one-point-per-thread kernels: fn(grid, first row, first plane),
  // more than one where an axis has more blocks than a grid dimension takes
  template <class Fn>
  static void direct_launches(const GridGeom& g, Fn&& fn) {
    constexpr int kMax = 65535, bz = direct_z<T>();
    const int n0 = g.hi[0] - g.lo[0];
    for (int k = g.lo[2]; k < g.hi[2]; k += kMax * bz)
      for (int j = g.lo[1]; j < g.hi[1]; j += kMax * kDirectY) {
        const int n1 = std::min(g.hi[1] - j, kMax * kDirectY), n2 = std::min(g.hi[2] - k, kMax * bz);
        fn(dim3((n0 + kDirectX - 1) / kDirectX, (n1 + kDirectY - 1) / kDirectY, (n2 + bz - 1) / bz),
           j, k);
      }
  }
  static void stage(bool is_first, const FlatLaunch& L, cudaStream_t st, const EzConst<T>& c,
                    const F7<const T>& src, const F7<T>& dst, const F7<T>& du, const F7<T>& un,
                    const F5<T>& aux, const F6<T>& dg, T As, T Bs, T tst, int flags) {
    auto launch = [&](auto fc) {
      constexpr bool FIRST = decltype(fc)::value;
      if constexpr (!DG) {
        if (kDirectOnly || L.direct_stage) {
          direct_launches(c.g, [&](dim3 grid, int j0, int k0) {
            ez_stage_direct_kernel<T, FIRST, BC, XA>
                <<<grid, dim3(kDirectX, kDirectY, direct_z<T>()), 0, st>>>(
                    c, src, dst, du, un, aux, As, Bs, tst, flags, j0, k0);
          });
          return;
        }
      }
      if constexpr (!kDirectOnly)
        stage_fn<FIRST>()<<<L.grid_stage, dim3(kTileX, kTileY), stage_bytes(FIRST), st>>>(
            c, src, dst, du, un, aux, dg, As, Bs, tst, L.kchunk_stage, flags);
    };
    if (is_first) launch(std::true_type{});
    else launch(std::false_type{});
  }
  static void ko_pass(const FlatLaunch& L, cudaStream_t st, const EzConst<T>& c,
                      const F7<const T>& src, const F7<T>& dst, const F6<T>& dg, T tko) {
    if constexpr (!DG) {
      if (L.direct_ko) {
        direct_launches(c.g, [&](dim3 grid, int j0, int k0) {
          ez_ko_direct_kernel<T, BC, XA><<<grid, dim3(kDirectX, kDirectY, direct_z<T>()), 0, st>>>(
              c, src, dst, tko, j0, k0);
        });
        return;
      }
    }
    ko_fn()<<<L.grid_ko, dim3(S::KTX, S::KTY), ko_smem<T, V, BC>(), st>>>(c, src, dst, dg, tko,
                                                                         L.kchunk_ko);
  }
};

// Calls fn(FlatKernels<T, BC, V, XA, DG>{}) for the kernel set L selects.
template <typename T, bool XA, bool DG, class Fn>
inline void with_flat_kernels_xa(const FlatLaunch& L, Fn&& fn) {
  if (L.bc) {
    if (L.vec) fn(FlatKernels<T, true, 2, XA, DG>{});
    else fn(FlatKernels<T, true, 1, XA, DG>{});
  } else {
    if (L.vec) fn(FlatKernels<T, false, 2, XA, DG>{});
    else fn(FlatKernels<T, false, 1, XA, DG>{});
  }
}
template <typename T, class Fn>
inline void with_flat_kernels(const FlatLaunch& L, Fn&& fn) {
  if (L.xa && L.dg) with_flat_kernels_xa<T, true, true>(L, fn);
  else if (L.xa) with_flat_kernels_xa<T, true, false>(L, fn);
  else with_flat_kernels_xa<T, false, false>(L, fn);
}

// Set the shared-memory limits of every flat kernel of precision T on the
// current device and plan the launch geometry of `env`'s grid.
// reference_arith: the CPU semantics run in the CPU build's own arithmetic
// (the default); false selects the regrouped, faster arithmetic.
// energy_diag: with the reference arithmetic, also accumulate the CPU
// build's energy-change diagnostics.  streaming: the plane-streaming kernels at every
// size (where there are any).
template <typename T>
inline int flat_plan(const coffee_env* env, int semantics, FlatLaunch* L,
                     bool reference_arith = true, bool energy_diag = false,
                     bool streaming = false) {
  using S = Shape<T>;
  L->bc = flat_needs_bc(env->p, semantics);
  L->vec = env->grid.dims[0] % 2 == 0;
  L->xa = reference_arith && semantics == SEM_CPU_REF;
  L->dg = L->xa && energy_diag;
  L->two_images = false;
  for (int a = 0; a < 3; ++a)
    if (env->p.periodic_boundary[a] && env->p.N[a] < 2 * env->p.guard[a]) L->two_images = true;
  // the shared-memory limits of the four kernel sets of this arithmetic (a
  // caller may still switch the pair copies off, as coffee_noalloc.cu does)
  if (L->dg) {
    COFFEE_CUDA_TRY((FlatKernels<T, true, 1, true, true>::set_attributes()));
    COFFEE_CUDA_TRY((FlatKernels<T, false, 1, true, true>::set_attributes()));
    COFFEE_CUDA_TRY((FlatKernels<T, true, 2, true, true>::set_attributes()));
    COFFEE_CUDA_TRY((FlatKernels<T, false, 2, true, true>::set_attributes()));
  } else if (L->xa) {
    COFFEE_CUDA_TRY((FlatKernels<T, true, 1, true>::set_attributes()));
    COFFEE_CUDA_TRY((FlatKernels<T, false, 1, true>::set_attributes()));
    COFFEE_CUDA_TRY((FlatKernels<T, true, 2, true>::set_attributes()));
    COFFEE_CUDA_TRY((FlatKernels<T, false, 2, true>::set_attributes()));
  } else {
    COFFEE_CUDA_TRY((FlatKernels<T, true, 1, false>::set_attributes()));
    COFFEE_CUDA_TRY((FlatKernels<T, false, 1, false>::set_attributes()));
    COFFEE_CUDA_TRY((FlatKernels<T, true, 2, false>::set_attributes()));
    COFFEE_CUDA_TRY((FlatKernels<T, false, 2, false>::set_attributes()));
  }
  // the flat kernels index an array with 32-bit element offsets (an FP32
  // array of 2^31 points alone would take a twentieth of the GPU's memory,
  // and a run holds at least 21 of them)
  const long long npts =
      (long long)env->grid.dims[0] * env->grid.dims[1] * (long long)env->grid.dims[2];
  if (npts >= (1LL << 31))
    return fail(COFFEE_E_CONFIG, "%lld points per array: the flat solver takes fewer than 2^31",
                npts);
  int per_sm_stage = 1, per_sm_ko = 1, tile_y = 1, stage_mult = 1;
  cudaError_t occ = cudaSuccess;
  with_flat_kernels<T>(*L, [&](auto K) {
    occ = decltype(K)::occupancy(&per_sm_stage, &per_sm_ko);
    tile_y = decltype(K)::kTileY;
    stage_mult = decltype(K)::kChunkMult;
  });
  COFFEE_CUDA_TRY(occ);
  if (per_sm_stage < 1 || per_sm_ko < 1)
    return fail(COFFEE_E_CUDA, "stage/KO kernels cannot be resident (occupancy 0)");
  const int sms = num_sms(env->device);
  const coffee_params& p = env->p;
  int box[3];
  for (int a = 0; a < 3; ++a) box[a] = p.N[a] + 2 * p.shift_ghost;
  const int sx = (box[0] + S::STX - 1) / S::STX, sy = (box[1] + tile_y - 1) / tile_y;
  // a kernel whose ring length equals its z unroll needs chunks of a
  // multiple of it (its ring slots are then compile-time constants)
  auto chunk_mult = [](int unroll, int ring) { return unroll == ring ? unroll : 1; };
  L->kchunk_stage = pick_kchunk(
      box[2], sx * sy, sms * per_sm_stage, 4, stage_mult);
  L->grid_stage = dim3(sx, sy, (box[2] + L->kchunk_stage - 1) / L->kchunk_stage);
  const int kx = (box[0] + S::KTX - 1) / S::KTX, ky = (box[1] + S::KTY - 1) / S::KTY;
  L->kchunk_ko = pick_kchunk(box[2], kx * ky, sms * per_sm_ko, 6,
                             L->bc ? chunk_mult(ko_zunroll<true>(), ko_ring<true, S::KPF>())
                                   : chunk_mult(ko_zunroll<false>(), ko_ring<false, S::KPF>()));
  L->grid_ko = dim3(kx, ky, (box[2] + L->kchunk_ko - 1) / L->kchunk_ko);
  const long long pts = (long long)box[0] * box[1] * box[2];
  const DirectPoints dp = direct_points<T>(L->bc, L->xa);
  L->direct_stage = !L->dg && !streaming && pts <= dp.stage;
  L->direct_ko = !L->dg && !streaming && pts <= dp.ko;
  return COFFEE_OK;
}

// Optional callbacks around every launch of flat_steps (timing).
struct LaunchHook {
  virtual int before(int kind) = 0;  // kind: COFFEE_KERNEL_*
  virtual int after(int kind) = 0;
  virtual ~LaunchHook() {}
};

template <typename T>
inline cudaError_t flat_images(const FlatLaunch& L, const GridGeom& g, const F7<T>& u,
                               cudaStream_t st) {
  if (!L.two_images) return cudaSuccess;
  const long long n = g.sz * g.dims[2];
  ez_images_kernel<T><<<(unsigned)std::min<long long>((n + 255) / 256, 148 * 8), 256, 0, st>>>(g, u);
  return cudaGetLastError();
}

// nsteps evolve_fields calls from `time` (reference field_solver_EZ.cpp:1007-1073):
// 5 stages A -> B -> A -> B -> A -> B, then the KO pass B -> A, advancing
// time by dt in field precision after each step (src/main-alfven3d.cpp:61,119).
template <typename T>
inline int flat_steps(const EzConst<T>& c, const FlatLaunch& L, const F7<T>& A, const F7<T>& Bb,
                      const F7<T>& dU, const F7<T>& Un, const F5<T>& aux, bool want_aux,
                      double time, int nsteps, cudaStream_t st, LaunchHook* hook,
                      const F6<T>* dg = nullptr) {
  F6<T> dgv;
  for (int a = 0; a < 6; ++a) dgv.p[a] = dg ? dg->p[a] : nullptr;
  if (L.dg && !dg) return fail(COFFEE_E_INVALID, "energy diagnostics planned without arrays");
  const T dt = c.dt;
  T t = (T)time;
  for (int step = 0; step < nsteps; ++step) {
    for (int i = 0; i < 5; ++i) {
      const F7<T>& src = (i % 2 == 0) ? A : Bb;
      const F7<T>& dst = (i % 2 == 0) ? Bb : A;
      F7<const T> srcc;
      for (int a = 0; a < 7; ++a) srcc.p[a] = src.p[a];
      int flags = 0;
      if (i == 4) flags |= ST_LAST;
      if (i == 4 && want_aux) flags |= ST_AUX;
      if (i == 0 && c.absorbing) flags |= ST_WRITE_UN;
      const T tst = t + (T)kCs[i] * dt;
      const int kind = (i == 0) ? COFFEE_KERNEL_STAGE_FIRST : COFFEE_KERNEL_STAGE;
      if (hook) {
        int rc = hook->before(kind);
        if (rc) return rc;
      }
      with_flat_kernels<T>(L, [&](auto K) {
        decltype(K)::stage(i == 0, L, st, c, srcc, dst, dU, Un, aux, dgv, (T)kAs[i], (T)kBs[i],
                           tst, flags);
      });
      COFFEE_CUDA_TRY(cudaGetLastError());
      COFFEE_CUDA_TRY(flat_images(L, c.g, dst, st));
      if (hook) {
        int rc = hook->after(kind);
        if (rc) return rc;
      }
    }
    F7<const T> srcc;
    for (int a = 0; a < 7; ++a) srcc.p[a] = Bb.p[a];
    if (hook) {
      int rc = hook->before(COFFEE_KERNEL_KO);
      if (rc) return rc;
    }
    with_flat_kernels<T>(L, [&](auto K) { decltype(K)::ko_pass(L, st, c, srcc, A, dgv, t + dt); });
    COFFEE_CUDA_TRY(cudaGetLastError());
    COFFEE_CUDA_TRY(flat_images(L, c.g, A, st));
    if (hook) {
      int rc = hook->after(COFFEE_KERNEL_KO);
      if (rc) return rc;
    }
    t = t + dt;
  }
  return COFFEE_OK;
}

}  // namespace coffee
