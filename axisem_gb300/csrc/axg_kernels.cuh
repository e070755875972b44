// axg_kernels.cuh -- sm_103a kernels of the AxiSEM time loop: shared types and
// helpers, the patch kernel of the no-allocation entry point, attenuation at
// every GLL point, the final drift, seismograms and wavefield dumps.  The
// steps' element and point passes are in axg_stream.cuh.
//
// These kernels hold an element in a warp, one lane per GLL point (i, j) =
// (lane % 5, lane / 5), lanes 25..31 idle.  The 5x5 tensor-product
// contractions of the reference (mxm_4 / vxm_4 of
// SOLVER/unrolled_loops.f90) are done with warp shuffles: lane (i, j) reads
// the five values of its column (k, j) or row (i, k) from the other lanes.
// Per-lane copies of the needed rows/columns of G1, G2 stay in registers.
//
// The patch kernel (stiffness + assembly, one CTA per patch of axg_plan.h)
// has three phases:
//   1. gather: the patch's global points are read once into shared memory;
//   2. elements, sub-round by sub-round: each warp computes its element's
//      stiffness and adds it into the shared point accumulators (elements
//      of one sub-round share no point, so there is no race);
//   3. write-back: the accumulators (which started from the partial sums of
//      earlier writers) are stored to the global force.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "axg_plan.h"
#include "axg_tma.cuh"

namespace axg {

// Debug variant (-DAXG_DEVICE_CHECKS): every global and shared index is
// checked against its bound; the first violation is recorded in
// g_axg_check = {flag, kernel id, source line, 0, index lo, index hi, bound lo,
// bound hi} and the access is skipped.  Nothing traps.  Normal builds compile
// the checks away.
#ifdef AXG_DEVICE_CHECKS
static __device__ int32_t g_axg_check[8];  // one per translation unit
static __device__ __noinline__ bool axg_record(int kern, int line, long long idx, long long bound) {
  if (atomicCAS(&g_axg_check[0], 0, 1) == 0) {
    g_axg_check[1] = kern;
    g_axg_check[2] = line;
    g_axg_check[4] = (int32_t)(idx & 0xffffffff);
    g_axg_check[5] = (int32_t)(idx >> 32);
    g_axg_check[6] = (int32_t)(bound & 0xffffffff);
    g_axg_check[7] = (int32_t)(bound >> 32);
  }
  return false;
}
#define AXG_BOUND(idx, bound, kern)                                                          \
  ((((long long)(idx)) >= 0 && ((long long)(idx)) < ((long long)(bound)))                    \
       ? true                                                                               \
       : axg_record((kern), __LINE__, (long long)(idx), (long long)(bound)))
#else
#define AXG_BOUND(idx, bound, kern) true
#endif

constexpr int kWarps = 8;
constexpr int kThreads = 32 * kWarps;
constexpr unsigned kFull = 0xffffffffu;

enum { POLE_MONO = 0, POLE_DI = 1, POLE_QUAD = 2 };
// FORCE: stiffness + assembly; NEWMARK: a Newmark step
// (SOLVER/time_evol_wave.F90:264-502); SYMPLECTIC: one stage of a symplectic
// step (SOLVER/time_evol_wave.F90:516-742): drift u + c_d v on the gather,
// kick v + c_v a by the last writer
enum { MODE_FORCE = 0, MODE_NEWMARK = 1, MODE_SYMPLECTIC = 2 };

// slot of each metric array inside an element's block (same order as the
// host packing, SOLID_TERMS_USED of the Python mirror)
enum : int {
  S_M1 = 0, S_M2, S_M3, S_M4, S_MW1, S_M11S, S_M21S, S_M41S, S_M12S, S_M22S, S_M32S, S_M42S,
  S_M11Z, S_M21Z, S_M41Z,
  S_M5 = 15, S_M6, S_M7, S_M8, S_MW2, S_MW3,
  // dipole
  S_M13S = 21, S_M33S, S_M43S,
  // quadrupole
  S_MW4 = 21, S_MW5, S_M1PHI, S_M2PHI, S_M4PHI
};
__host__ __device__ constexpr int n_terms(int pole) { return pole == POLE_MONO ? 15 : (pole == POLE_DI ? 24 : 26); }
__host__ __device__ constexpr int n_axial(int pole) { return pole == POLE_MONO ? 3 : (pole == POLE_DI ? 9 : 6); }
// solid element block: nt*25 metric floats, then 25 uint16 patch-local point
// indices (50 bytes), 2 bytes pad, the int32 element info word; 16-byte multiple
__host__ __device__ constexpr int solid_idx_off(int nt) { return nt * 25; }      // in floats
__host__ __device__ constexpr int solid_info_off(int nt) { return nt * 25 + 13; }  // in floats
__host__ __device__ constexpr int solid_block_stride(int nt) { return ((nt * 25 + 14 + 3) / 4) * 4; }

struct SpecDev {
  float g1[25], g2[25], g0[5];
};

struct SrcTable {           // solid source points (<= 200)
  const int32_t *gidx;      // global point
  const float *val;         // (n, 3)
  const double *val_dp;     // (n, 3) in FP64, applied in FP64 by the compensated mode; or null
  int32_t n;
};

struct DomainArgs {
  const PatchMeta *meta;
  const uint32_t *pts;
  const float *metric;      // per element solid_block_stride(nt) floats (launch order)
  const float *m0;          // per axial slot n_axial*5 floats
  int32_t patch_begin;
  int64_t n_patches, n_pts, n_elem, n_m0;   // buffer extents (checked builds)
};

// A solve's control words (device).  Each of a step's two passes reads what the
// other writes: the element pass CTL_ITER and CTL_STOP, which the end of the
// step sets; the point pass the copies that the element pass makes of them.
enum {
  CTL_ITER = 0,    // the step counter (1-based iteration of the next step)
  CTL_BLOWUP = 1,  // first iteration whose displacement blew up (0: none)
  CTL_ERR = 2,     // AXG_ERR_TIMEOUT when a bounded wait gave up
  CTL_ITER_P = 3,
  CTL_STOP = 4,    // CTL_BLOWUP of the steps completed: the solve has stopped
  CTL_STOP_P = 5,
  CTL_PARITY = 6,  // roles of the displacement buffers after the last step that was not skipped
  kCtlWords = 8
};

struct StateArgs {
  float *u[3];              // disp (solid, gvec layout) / chi (fluid: u[0]); plain Newmark: the
                            // buffer the step stores the next step's prediction into
  float *v[3];              // velo / dchi
  float *a[3];              // acc0 / ddchi0
  float *f[3];              // force partial sums
  float *cu[3], *cv[3];     // compensated mode: running compensation of disp / velo (chi / dchi), else null
  float *cup[3];            // compensated Newmark: the compensation after the step's prediction, else null
  float *up[3];             // Newmark: the step's predicted displacement (chi), which becomes its
                            // new displacement (the two buffers trade roles every step); else null
  const float *inv_mass;    // per global point
  // the FP64 inverse mass (compensated mode) or null: as FP32 pairs, or where
  // a mass is out of their range in FP64
  const float2 *inv_mass_pair;
  const double *inv_mass_dp;
  const float *gamma;       // absorbing gamma per global point or null
  const float *stf;         // (niter)
  const int32_t *iter;      // device iteration counter (1-based iter of this step)
  int32_t *blowup;          // first iteration that blew up (0 = none)
  const int32_t *stop;      // set in the steps after it: they do nothing
  int32_t *err;             // device error word (AXG_ERR_TIMEOUT when a bounded wait gave up)
  float thresh;             // 10 |magnitude|
  // Newmark: deltat, deltat/2, deltat^2/2; symplectic stage: dt = coefd(i) deltat,
  // kick = coefv(i) deltat; each an FP32 pair (value + _lo = the FP64 value)
  float dt, hdt, hdt2, dt_lo, hdt_lo, hdt2_lo;
  float kick, kick_lo;
  SrcTable src;
  int64_t nglob;            // extent of the state arrays (checked builds)
  int32_t niter;            // extent of stf
};

// ------------------------------------------------------------ work descriptors

// A launch's per-solve arguments, passed in its parameter space
// (__grid_constant__).  One<W>: one solve owns all of the launch's work items
// (its points, its receivers).  Many<W>: up to kMaxBatch
// solves advanced together by one launch; solve s owns the items
// [start[s], start[s + 1]), and a CTA or thread finds its solve from them.
constexpr int kMaxBatch = 32;

template <class W>
struct One {
  static constexpr bool kMany = false;
  W w;
  int32_t n_items;
  __device__ __forceinline__ int32_t items() const { return n_items; }
  __device__ __forceinline__ int locate(int32_t) const { return 0; }
  __device__ __forceinline__ int32_t first(int) const { return 0; }
  __device__ __forceinline__ const W &at(int) const { return w; }
};

template <class W>
struct Many {
  static constexpr bool kMany = true;
  int32_t n;                       // solves, 1..kMaxBatch
  int32_t start[kMaxBatch + 1];    // item prefix over the solves
  W w[kMaxBatch];
  __device__ __forceinline__ int32_t items() const { return start[n]; }
  __device__ __forceinline__ int locate(int32_t it) const {
    int s = 0;
    while (s + 1 < n && start[s + 1] <= it) ++s;
    return s;
  }
  __device__ __forceinline__ int32_t first(int s) const { return start[s]; }
  __device__ __forceinline__ const W &at(int s) const { return w[s]; }
};

// Attenuation: the fields of the cg4 constants, in groups of four points
// (A_* + 4 k' is field k' of the element's cg points (1,1), (1,3), (3,1),
// (3,3), the order of the reference's (1:4) arrays; packing in axg_stream.cuh).
constexpr int kMaxSls = 8;

// attenuation at every GLL point (anel_full_kernel)
struct AnelArgs {
  const float *consts;      // per element kFullConst floats (slot order)
  float *state;             // per element state_stride floats (slot order)
  const float *qtab;        // per distinct Q: ts_fac_t(j) a_j(Q) at [0, kMaxSls), ts_fac_tm1(j) a_j(Q) after
  float ex[kMaxSls];        // exp_w_j_deltat
  int32_t nsls, state_stride, n_q;
};

// ------------------------------------------------------------ small helpers

// Time-step coefficients as FP32 pairs.  The reference multiplies its FP32
// fields by FP64 coefficients (deltat, half_dt, half_dt_sq, coefd(i) and
// coefv(i) times deltat) and rounds each update once.  A coefficient rounded
// to FP32 is off by up to 3e-8 relative, the same in every step: over 1e5
// steps a steady drift of the solution's time scale, which the compensated
// summation cannot remove.  With the low part the increments carry only the
// FP32 rounding of the product.
// c x for the coefficient c + c_lo
__device__ __forceinline__ float mul2(float c, float c_lo, float x) { return fmaf(c, x, c_lo * x); }
// the predictor's increment deltat*velo + half_dt_sq*acc0
__device__ __forceinline__ float pred_inc(float v, float a, const StateArgs &st) {
  return fmaf(st.hdt2, a, fmaf(st.dt, v, fmaf(st.hdt2_lo, a, st.dt_lo * v)));
}
// disp + deltat*velo + half_dt_sq*acc0 (SOLVER/time_evol_wave.F90:357-364);
// a symplectic stage's drift disp + coefd(i) velo (hdt2 = 0)
__device__ __forceinline__ float predict(float d, float v, float a, const StateArgs &st) {
  return d + pred_inc(v, a, st);
}

// Compensated mode (no counterpart in the reference): x + inc by Kahan's
// compensated summation.  c carries the low-order part the previous additions
// lost; it is taken off the increment before the addition and replaced by
// what this addition loses, so that rounding does not accumulate over many
// steps.  (No fast-math: the compiler keeps (t - x) - y as written.)
__device__ __forceinline__ float kahan_add(float x, float inc, float &c) {
  const float y = inc - c;
  const float t = x + y;
  c = (t - x) - y;
  return t;
}
// components apply_axis_mask_{onecomp,twocomp,threecomp} zero on the axis
// (SOLVER/apply_masks.f90): s (monopole), phi and z (dipole), all (quadrupole)
template <int POLE>
__device__ __forceinline__ bool axis_masked(int comp) {
  return POLE == POLE_QUAD || (POLE == POLE_MONO ? comp == 0 : comp != 0);
}

// The predictor of the compensated mode: the increment's FP32 part, added by
// compensated summation.  Its low-coefficient part was taken off the stored
// compensation by the previous step's last writer (comp_after_step), so
// that the gathers, which hold many points' values at once, need no more
// registers than the increment takes.
__device__ __forceinline__ float predict_comp(float d, float v, float a, const StateArgs &st, float &c) {
  return kahan_add(d, fmaf(st.hdt2, a, st.dt * v), c);
}
// the compensation a last writer stores with the new state: c less the low
// part of the next predictor's increment deltat*velo + half_dt_sq*acc0
__device__ __forceinline__ float comp_after_step(float c, float v, float a, const StateArgs &st) {
  return c - fmaf(st.hdt2_lo, a, st.dt_lo * v);
}
// a symplectic stage's compensated drift disp + coefd(i) velo
__device__ __forceinline__ float drift_comp(float d, float v, const StateArgs &st, float &c) {
  return kahan_add(d, mul2(st.dt, st.dt_lo, v), c);
}

// (float)(m x) for an FP64 factor m held as an FP32 pair m.x + m.y: the product
// of the high part and its exact rounding error, with the low part's product.
// Equal to the FP64 product rounded once but for values within about 2^-20
// of an ulp from a tie.  FP64 runs at 1/64 of the FP32 rate here: on 305 000
// points of three components a compensated step took 27.6 us with FP64
// products and took 25.1 with pairs; errors against FP64 are alike (2.5e-7).
// The product's error term is 2^-24 of it and flushed to zero below 2^-126:
// small products are formed 2^60 times larger (|x| is below 2^30 then, unless
// the mass is zero).  One that is infinite or no number stays what it is.  (No
// measurable cost: 4.02 ms for 200 steps of 18 944 elements with and without.)
__device__ __forceinline__ float mul_pair(float2 m, float x) {
  float p = __fmul_rn(m.x, x);
  const bool small = fabsf(p) < 0x1p-60f && fabsf(x) < 0x1p60f;
  if (small) x = x * 0x1p60f;
  if (small) p = __fmul_rn(m.x, x);
  const float r = __fadd_rn(p, fmaf(m.y, x, fmaf(m.x, x, -p)));
  return !(fabsf(p) <= 3.402823466e38f) ? p : small ? r * 0x1p-60f : r;
}

// X(i,j) = sum_k c[k] * v(k,j)   (v(k,j) held by lane k + 5 j)
__device__ __forceinline__ float dxi(float v, const float (&c)[5], int j5) {
  float s = c[0] * __shfl_sync(kFull, v, j5);
  s = fmaf(c[1], __shfl_sync(kFull, v, j5 + 1), s);
  s = fmaf(c[2], __shfl_sync(kFull, v, j5 + 2), s);
  s = fmaf(c[3], __shfl_sync(kFull, v, j5 + 3), s);
  s = fmaf(c[4], __shfl_sync(kFull, v, j5 + 4), s);
  return s;
}
// X(i,j) = sum_k v(i,k) * c[k]   (v(i,k) held by lane i + 5 k)
__device__ __forceinline__ float deta(float v, const float (&c)[5], int i) {
  float s = __shfl_sync(kFull, v, i) * c[0];
  s = fmaf(__shfl_sync(kFull, v, i + 5), c[1], s);
  s = fmaf(__shfl_sync(kFull, v, i + 10), c[2], s);
  s = fmaf(__shfl_sync(kFull, v, i + 15), c[3], s);
  s = fmaf(__shfl_sync(kFull, v, i + 20), c[4], s);
  return s;
}

// per-lane rows/columns of the derivative matrices (column-major G(a,b) = g[a+5b])
struct LaneCoef {
  float xi2[5], xi1[5];    // G2(k,i), G1(k,i): first stage d/dxi  (mxm_4(G2T,u))
  float eta[5];            // G2(k,j): first stage d/deta          (mxm_4(u,G2))
  float sxi2[5], sxi1[5];  // G2(i,k), G1(i,k): second stage       (mxm_4(G2,S))
  float seta[5];           // G2(j,k): second stage                (mxm_4(S,G2T))
  float g0i;               // G0(i)
  float g0[5];             // G0(k)
};

__device__ __forceinline__ void load_coef(const SpecDev &sp, int i, int j, LaneCoef &c) {
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    c.xi2[k] = sp.g2[k + 5 * i];
    c.xi1[k] = sp.g1[k + 5 * i];
    c.eta[k] = sp.g2[k + 5 * j];
    c.sxi2[k] = sp.g2[i + 5 * k];
    c.sxi1[k] = sp.g1[i + 5 * k];
    c.seta[k] = sp.g2[j + 5 * k];
    c.g0[k] = sp.g0[k];
  }
  c.g0i = sp.g0[i];
}

template <bool AX>
__device__ __forceinline__ const float (&cxi(const LaneCoef &c))[5] { return AX ? c.xi1 : c.xi2; }
template <bool AX>
__device__ __forceinline__ const float (&csxi(const LaneCoef &c))[5] { return AX ? c.sxi1 : c.sxi2; }

// element-local value of metric array `slot` at point `lane` (< 25); `blk` is
// the element's block staged in shared memory
__device__ __forceinline__ float ldm(const float *blk, int slot, int lane) { return blk[slot * 25 + lane]; }

// ------------------------------------------------------------ element stiffness

// glob_stiffness_mono_4 (SOLVER/stiffness_mono.f90:60-157) for lane (i, j)
template <bool AX>
__device__ __forceinline__ void stiff_mono(const LaneCoef &c, const float *blk, const float *m0, int lane,
                                           int i, int j, float us, float uz, float &fs, float &fz) {
  const int j5 = 5 * j;
  float X1 = dxi(us, cxi<AX>(c), j5);
  float X2 = dxi(uz, cxi<AX>(c), j5);
  float X3 = deta(us, c.eta, i);
  float X4 = deta(uz, c.eta, i);
  const float m1 = ldm(blk, S_M1, lane), m2 = ldm(blk, S_M2, lane), m3 = ldm(blk, S_M3, lane),
              m4 = ldm(blk, S_M4, lane), mw1 = ldm(blk, S_MW1, lane);
  const float m11s = ldm(blk, S_M11S, lane), m21s = ldm(blk, S_M21S, lane), m41s = ldm(blk, S_M41S, lane),
              m12s = ldm(blk, S_M12S, lane), m22s = ldm(blk, S_M22S, lane), m32s = ldm(blk, S_M32S, lane),
              m42s = ldm(blk, S_M42S, lane), m11z = ldm(blk, S_M11Z, lane), m21z = ldm(blk, S_M21Z, lane),
              m41z = ldm(blk, S_M41Z, lane);
  float ls = m4 * X4 + m2 * X3 + m1 * X1 + m3 * X2 + us * mw1;
  const float S1s = m11s * X3 + m21s * X1 + m12s * X4 + m22s * X2 + m1 * us;
  const float S2s = m11s * X1 + m41s * X3 + m32s * X2 + m42s * X4 + m2 * us;
  const float S1z = m11z * X4 + m21z * X2 + m32s * X3 + m22s * X1 + m3 * us;
  const float S2z = m11z * X2 + m41z * X4 + m12s * X1 + m42s * X3 + m4 * us;
  X2 = deta(S2s, c.seta, i);
  X4 = deta(S2z, c.seta, i);
  X1 = dxi(S1s, csxi<AX>(c), j5);
  X3 = dxi(S1z, csxi<AX>(c), j5);
  ls = ls + X1 + X2;
  float lz = X3 + X4;
  if (AX) {
    const float w1 = m0[0 * 5 + j], w2 = m0[1 * 5 + j], w3 = m0[2 * 5 + j];
    float V1 = dxi(us, c.g0, j5);   // vxm_4(G0, us)
    float V2 = deta(uz, c.eta, 0);  // vxm_4(uz(0,:), G2)
    float V4 = w1 * V1 + w3 * V2;
    const float V3 = dxi(uz, c.g0, j5);
    V4 = V4 + w2 * V3;
    float Xa = c.g0i * (w2 * V1);
    const float V2b = w3 * V1;
    const float V1b = deta(V2b, c.seta, 0);  // vxm_4(V2, G2T)
    if (i == 0) Xa = Xa + V1b;
    ls = ls + c.g0i * V4;
    lz = Xa + lz;
  }
  fs = ls;
  fz = lz;
}

// glob_stiffness_di_4 (SOLVER/stiffness_di.f90:60-256)
template <bool AX>
__device__ __forceinline__ void stiff_di(const LaneCoef &c, const float *blk, const float *m0, int lane, int i,
                                         int j, float u1, float u2, float u3, float &f1, float &f2, float &f3) {
  const int j5 = 5 * j;
  float X4 = deta(u1, c.eta, i), X5 = deta(u2, c.eta, i), X6 = deta(u3, c.eta, i);
  float X1 = dxi(u1, cxi<AX>(c), j5), X2 = dxi(u2, cxi<AX>(c), j5), X3 = dxi(u3, cxi<AX>(c), j5);
  const float X7 = X1 + X2, X8 = X4 + X5;
  const float m1 = ldm(blk, S_M1, lane), m2 = ldm(blk, S_M2, lane), m3 = ldm(blk, S_M3, lane),
              m4 = ldm(blk, S_M4, lane), m5 = ldm(blk, S_M5, lane), m6 = ldm(blk, S_M6, lane),
              m7 = ldm(blk, S_M7, lane), m8 = ldm(blk, S_M8, lane);
  const float mw1 = ldm(blk, S_MW1, lane), mw2 = ldm(blk, S_MW2, lane), mw3 = ldm(blk, S_MW3, lane);
  const float m11s = ldm(blk, S_M11S, lane), m21s = ldm(blk, S_M21S, lane), m41s = ldm(blk, S_M41S, lane),
              m12s = ldm(blk, S_M12S, lane), m22s = ldm(blk, S_M22S, lane), m42s = ldm(blk, S_M42S, lane),
              m13s = ldm(blk, S_M13S, lane), m23s = ldm(blk, S_M32S, lane), m33s = ldm(blk, S_M33S, lane),
              m43s = ldm(blk, S_M43S, lane), m11z = ldm(blk, S_M11Z, lane), m21z = ldm(blk, S_M21Z, lane),
              m41z = ldm(blk, S_M41Z, lane);
  const float ls2 = m8 * X6 + m7 * X3 + m1 * X1 + m5 * X2 + m2 * X4 + m6 * X5 + mw1 * u2 + mw2 * u3;
  const float ls3 = m4 * X4 - m4 * X5 + m3 * X1 - m3 * X2 + mw2 * u2 + mw3 * u3;
  float c1 = m13s * X6, c2 = m23s * X3, c3 = m3 * u3;
  float s1p = c1 + c2 + c3 + m11s * X4 + m21s * X1 + m12s * X5 + m22s * X2 + m1 * u2;
  float s1m = c1 + c2 - c3 + m11s * X5 + m21s * X2 + m12s * X4 + m22s * X1 + m5 * u2;
  c1 = m33s * X3;
  c2 = m43s * X6;
  c3 = m4 * u3;
  const float s2p = c1 + c2 + c3 + m11s * X1 + m41s * X4 + m12s * X2 + m42s * X5 + m2 * u2;
  const float s2m = c1 + c2 - c3 + m11s * X2 + m41s * X5 + m12s * X1 + m42s * X4 + m6 * u2;
  float S1z = m33s * X8 + m23s * X7 + m11z * X6 + m21z * X3 + m7 * u2;
  const float S2z = m13s * X7 + m43s * X8 + m11z * X3 + m41z * X6 + m8 * u2;
  X1 = dxi(s1p, csxi<AX>(c), j5);
  X3 = dxi(s1m, csxi<AX>(c), j5);
  X5 = dxi(S1z, csxi<AX>(c), j5);
  X2 = deta(s2p, c.seta, i);
  X4 = deta(s2m, c.seta, i);
  X6 = deta(S2z, c.seta, i);
  float l1 = X1 + X2;
  float l2 = X3 + X4 + ls2;
  float l3 = X5 + X6 + ls3;
  if (AX) {
    // M0_w slots: 0:w1 1:w2 2:w3 3:w4 4:w6 5:w7 6:w8 7:w9 8:w10
    const float w1 = m0[0 * 5 + j], w2 = m0[1 * 5 + j], w3 = m0[2 * 5 + j], w4 = m0[3 * 5 + j],
                w6 = m0[4 * 5 + j], w7 = m0[5 * 5 + j], w8 = m0[6 * 5 + j], w9 = m0[7 * 5 + j],
                w10 = m0[8 * 5 + j];
    const float V1 = dxi(u1, c.g0, j5), V2 = dxi(u2, c.g0, j5), V3 = dxi(u3, c.g0, j5);
    const float V4 = deta(u1, c.eta, 0), V5 = deta(u2, c.eta, 0);
    (void)V5;
    const float a_p = w1 * V2 + w3 * V3;
    const float a_m = w1 * V1 + (w2 + w6) * V4 + w9 * V2 + w10 * V3;
    const float a_z = w3 * V1 + (w4 + w8) * V4 + w7 * V3 + w10 * V2;
    float S1p = c.g0i * a_p;
    const float S1m = c.g0i * a_m;
    S1z = c.g0i * a_z;
    const float V4b = (w2 + w6) * V2 + (w4 + w8) * V3;
    const float V1b = deta(V4b, c.seta, 0);
    if (i == 0) S1p = S1p + V1b;
    l1 = l1 + S1p;
    l2 = l2 + S1m;
    l3 = l3 + S1z;
  }
  f1 = l1;
  f2 = l2;
  f3 = l3;
}

// glob_stiffness_quad_4 (SOLVER/stiffness_quad.f90:238-414)
template <bool AX>
__device__ __forceinline__ void stiff_quad(const LaneCoef &c, const float *blk, const float *m0, int lane,
                                           int i, int j, float us, float up, float uz, float &f1, float &f2,
                                           float &f3) {
  const int j5 = 5 * j;
  float X1 = dxi(us, cxi<AX>(c), j5), X2 = dxi(up, cxi<AX>(c), j5), X3 = dxi(uz, cxi<AX>(c), j5);
  float X4 = deta(us, c.eta, i), X5 = deta(up, c.eta, i), X6 = deta(uz, c.eta, i);
  const float m1 = ldm(blk, S_M1, lane), m2 = ldm(blk, S_M2, lane), m3 = ldm(blk, S_M3, lane),
              m4 = ldm(blk, S_M4, lane), m5 = ldm(blk, S_M5, lane), m6 = ldm(blk, S_M6, lane),
              m7 = ldm(blk, S_M7, lane), m8 = ldm(blk, S_M8, lane);
  const float mw1 = ldm(blk, S_MW1, lane), mw2 = ldm(blk, S_MW2, lane), mw3 = ldm(blk, S_MW3, lane),
              mw4 = ldm(blk, S_MW4, lane), mw5 = ldm(blk, S_MW5, lane);
  const float m11s = ldm(blk, S_M11S, lane), m21s = ldm(blk, S_M21S, lane), m41s = ldm(blk, S_M41S, lane),
              m12s = ldm(blk, S_M12S, lane), m22s = ldm(blk, S_M22S, lane), m32s = ldm(blk, S_M32S, lane),
              m42s = ldm(blk, S_M42S, lane), m11z = ldm(blk, S_M11Z, lane), m21z = ldm(blk, S_M21Z, lane),
              m41z = ldm(blk, S_M41Z, lane), m1p = ldm(blk, S_M1PHI, lane), m2p = ldm(blk, S_M2PHI, lane),
              m4p = ldm(blk, S_M4PHI, lane);
  const float c1 = m2 * X4, c2 = m1 * X1, c3 = m6 * X5, c4 = m5 * X2, c5 = m4 * X6, c6 = m3 * X3;
  float ls = c1 + c2 + 2.f * (c3 + c4) + c5 + c6 + mw1 * us + mw2 * up + 2.f * mw3 * uz;
  float lp = -2.f * (c1 + c2 + c5 + c6) - (c3 + c4) + mw2 * us + mw4 * up - mw3 * uz;
  float lz = 2.f * (m8 * X5 + m7 * X2) + mw3 * (2.f * us - up) + mw5 * uz;
  const float usm = us - 2.f * up, ups = 2.f * us - up;
  const float S1s = m11s * X4 + m21s * X1 + m12s * X6 + m22s * X3 + m1 * usm;
  const float S2s = m11s * X1 + m41s * X4 + m32s * X3 + m42s * X6 + m2 * usm;
  const float S1z = m11z * X6 + m21z * X3 + m32s * X4 + m22s * X1 + m3 * usm;
  const float S2z = m11z * X3 + m41z * X6 + m12s * X1 + m42s * X4 + m4 * usm;
  const float S1p = m1p * X5 + m2p * X2 + m5 * ups + 2.f * m7 * uz;
  const float S2p = m1p * X2 + m4p * X5 + m6 * ups + 2.f * m8 * uz;
  X2 = deta(S2s, c.seta, i);
  X4 = deta(S2p, c.seta, i);
  X6 = deta(S2z, c.seta, i);
  X1 = dxi(S1s, csxi<AX>(c), j5);
  X3 = dxi(S1p, csxi<AX>(c), j5);
  X5 = dxi(S1z, csxi<AX>(c), j5);
  ls = ls + X1 + X2;
  lp = lp + X3 + X4;
  lz = lz + X5 + X6;
  if (AX) {
    const float w1 = m0[0 * 5 + j], w2 = m0[1 * 5 + j], w3 = m0[2 * 5 + j], w4 = m0[3 * 5 + j],
                w5 = m0[4 * 5 + j], w6 = m0[5 * 5 + j];
    const float V1 = dxi(us, c.g0, j5), V2 = dxi(up, c.g0, j5), V3 = dxi(uz, c.g0, j5);
    ls = ls + c.g0i * (w1 * V1 + w2 * V2 + w3 * V3);
    lp = lp + c.g0i * (w2 * V1 + w4 * V2 + w5 * V3);
    lz = lz + c.g0i * (w3 * V1 + w5 * V2 + w6 * V3);
  }
  f1 = ls;
  f2 = lp;
  f3 = lz;
}

// ------------------------------------------------------------ solid patch kernel

constexpr int kStages = 2;  // element blocks in flight per warp (TMA ring depth)

// shared-memory layout (bytes); NB buffers of the patch state (u, f, point
// words), STG ring stages per warp
template <int NC, int BS, int STG, int NB, int ROW>
struct SolidSmem {
  static constexpr int u_bytes = NC * ROW * 4, w_bytes = kMaxPatchPoints * 4;
  static constexpr int u_off = 0;
  static constexpr int f_off = u_off + NB * u_bytes;
  static constexpr int w_off = f_off + NB * u_bytes;
  static constexpr int ring_off = ((w_off + NB * w_bytes + 127) / 128) * 128;
  static constexpr int bar_off = ring_off + kWarps * STG * BS * 4;
  static constexpr int bytes = bar_off + kWarps * STG * 8;
};
// Bank swizzle of the shared point arrays: patch point t lives at
// t + kPad * (t / 32).  An element's 25 points sit in five runs of five
// consecutive patch points, one run per element row; on structured blocks
// the runs lie a patch width (33 for 8 x 8 patches) apart, so unpadded they
// share only 9 of the 32 banks (5-way conflicts), padded by 4 words per 32
// they fall on 25 distinct banks.
constexpr int kPad = 4;
__host__ __device__ constexpr int solid_row() { return kMaxPatchPoints + kPad * ((kMaxPatchPoints + 31) / 32); }

// the sub-round ends of a patch held in registers (8 bits per round), so
// that no per-patch array is indexed at run time: a PatchMeta indexed that
// way lives in local memory, and each lookup is a local load
struct PatchRounds {
  uint64_t lo;  // round_end[0..7]
  uint32_t hi;  // round_end[8..11]
  int n;
  __device__ __forceinline__ explicit PatchRounds(const PatchMeta &m) : lo(0), hi(0), n(m.n_rounds) {
    static_assert(kMaxSubrounds <= 12, "PatchRounds holds 12 rounds");
#pragma unroll
    for (int r = 0; r < 8; ++r) lo |= (uint64_t)m.round_end[r] << (8 * r);
#pragma unroll
    for (int r = 0; r < 4; ++r) hi |= (uint32_t)m.round_end[8 + r] << (8 * r);
  }
  __device__ __forceinline__ int end(int r) const {
    return r < 8 ? (int)((lo >> (8 * r)) & 0xFFu) : (int)((hi >> (8 * (r - 8))) & 0xFFu);
  }
};

// the elements warp `w` processes in a patch, in order: sub-round by
// sub-round, elements w, w + kWarps, ... of each round
struct WarpIter {
  int r, s;
  __device__ __forceinline__ void norm(const PatchRounds &m, int w) {
    while (r < m.n && s >= m.end(r)) {
      ++r;
      s = m.end(r - 1) + w;
    }
  }
  __device__ __forceinline__ bool valid(const PatchRounds &m) const { return r < m.n; }
};

// Stiffness + assembly of one colour's patches by persistent CTAs (two per
// SM: 128 registers, no spills, two patch buffers).  The gather is
// asynchronous (cp.async into shared memory, the next patch's during the
// current one's element rounds).
template <int POLE>
__global__ void __launch_bounds__(kThreads, 2)
    solid_patch_kernel(DomainArgs d, StateArgs st, SpecDev sp, int32_t n_colour_patches) {
  constexpr int NC = POLE == POLE_MONO ? 2 : 3;           // stored components
  constexpr int NT = n_terms(POLE), NA = n_axial(POLE);
  constexpr int BS = solid_block_stride(NT);
  constexpr uint32_t BSB = BS * 4;
  constexpr int STG = kStages, NB = 2;
  constexpr int ROW = solid_row();
  using L = SolidSmem<NC, BS, STG, NB, ROW>;
  extern __shared__ __align__(128) unsigned char smem[];
  auto su_of = [&](int b) { return reinterpret_cast<float(*)[ROW]>(smem + L::u_off + b * L::u_bytes); };
  auto sf_of = [&](int b) { return reinterpret_cast<float(*)[ROW]>(smem + L::f_off + b * L::u_bytes); };
  auto spos = [](int t) { return t + kPad * (t >> 5); };  // swizzled position of patch point t
  auto sw_of = [&](int b) { return reinterpret_cast<uint32_t *>(smem + L::w_off + b * L::w_bytes); };
  float *ring = reinterpret_cast<float *>(smem + L::ring_off);
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + L::bar_off);
  __shared__ int s_timeout;  // a bounded wait of this CTA gave up
  // sub-round r of a patch is complete when all threads have arrived on
  // s_round[r] after their accumulations of round r
  __shared__ __align__(8) uint64_t s_round[kMaxSubrounds];
  __shared__ __align__(8) uint64_t s_wbar[2];  // a patch's point words have landed in buffer b
  // component c of the shared arrays -> global component (mono: s, z)
  auto gc = [](int c) { return (POLE == POLE_MONO && c == 1) ? 2 : c; };

  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x < kWarps * STG) mbar_init(&bars[threadIdx.x], 1);
  if (threadIdx.x < kMaxSubrounds) mbar_init(&s_round[threadIdx.x], kThreads);
  if (threadIdx.x < 2) mbar_init(&s_wbar[threadIdx.x], 1);
  if (threadIdx.x == 0) s_timeout = 0;
  fence_mbar_init();
  __syncthreads();

  const bool active = lane < 25;
  const int i = lane % 5, j = active ? lane / 5 : 0;
  // idle lanes 25..31 take part in the shuffles; their reads of an element's
  // data go to point 24 so that no lane reads past the element's block
  const int ml = active ? lane : 24;
  LaneCoef coef;
  load_coef(sp, i, j, coef);
  const uint64_t pol = policy_evict_first();
  float *my_ring = ring + warp * STG * BS;
  uint64_t *my_bars = bars + warp * STG;
  uint32_t kcount = 0;  // elements this warp has consumed (slot = kcount % STG)
  uint32_t round_par = 0;  // bit r: parity of the next completion of s_round[r]
  uint32_t pcount = 0;     // patches this CTA has started: buffer pcount % NB, s_wbar parity (pcount / NB) & 1
  // one thread: start the copy of element `el` into ring slot `slot`
  auto issue = [&](uint32_t slot, int64_t el) {
    bulk_g2s(my_ring + slot * BS, d.metric + el * BS, BSB, &my_bars[slot], pol);
  };
  // one thread: bulk copy of a patch's point words into buffer b (each
  // patch's words start 16-byte aligned, padded to a multiple of four)
  auto issue_words = [&](int b, int32_t pt_start, int n_pts) {
    const uint32_t nw = ((uint32_t)n_pts + 3u) & ~3u;
    if (nw > 0 && AXG_BOUND((int64_t)pt_start + nw - 1, d.n_pts, 1)) {
      fence_proxy_async();  // earlier generic reads of the buffer precede the async-proxy write
      bulk_g2s(sw_of(b), d.pts + pt_start, nw * 4u, &s_wbar[b], pol);
    } else {
      mbar_arrive(&s_wbar[b]);
    }
  };
  // every thread: 4-byte copies of its points' u, and of the partial sums of
  // points an earlier colour holds, straight into buffer b.  A point's
  // accumulator starts from that partial sum, so that the write-back is a
  // plain store.
  auto issue_gather = [&](int b, int n_pts) {
    float(*gu)[ROW] = su_of(b);
    float(*gf)[ROW] = sf_of(b);
    const uint32_t *gw = sw_of(b);
    for (int t = threadIdx.x; t < n_pts; t += kThreads) {
      const uint32_t w = gw[t];
      const uint32_t g = w & kPtIndexMask;
      const int pt = spos(t);
      if (!AXG_BOUND(g, st.nglob, 1)) {
#pragma unroll
        for (int c = 0; c < NC; ++c) gu[c][pt] = gf[c][pt] = 0.f;
        continue;
      }
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        cp_async4(&gu[c][pt], st.u[gc(c)] + g);
        if (w & kPtFirst) gf[c][pt] = 0.f;
        else cp_async4(&gf[c][pt], st.f[gc(c)] + g);
      }
    }
    cp_async_commit();
  };
  // the CTA's first patch is gathered here, each later one while the CTA
  // computes the patch before it
  if ((int32_t)blockIdx.x < n_colour_patches && AXG_BOUND(d.patch_begin + blockIdx.x, d.n_patches, 1)) {
    const PatchMeta m0 = d.meta[d.patch_begin + blockIdx.x];
    if (threadIdx.x == 0) issue_words(0, m0.pt_start, m0.n_pts);
    if (!mbar_wait_bounded(&s_wbar[0], 0u, st.err)) s_timeout = 1;
    issue_gather(0, m0.n_pts);
  }

  for (int32_t pp = blockIdx.x; pp < n_colour_patches; pp += gridDim.x) {
    if (!AXG_BOUND(d.patch_begin + pp, d.n_patches, 1)) break;
    const PatchMeta m = d.meta[d.patch_begin + pp];
    const PatchRounds pr(m);
    const int buf = pcount % NB;
    float(*s_u)[ROW] = su_of(buf);
    float(*s_f)[ROW] = sf_of(buf);
    const uint32_t *s_w = sw_of(buf);
    // the next patch's point words go to the other buffer now
    int next_npts = 0;
    const int32_t ppn = pp + gridDim.x;
    if (ppn < n_colour_patches && AXG_BOUND(d.patch_begin + ppn, d.n_patches, 1)) {
      const PatchMeta mn = d.meta[d.patch_begin + ppn];
      next_npts = mn.n_pts;
      if (threadIdx.x == 0) issue_words(buf ^ 1, mn.pt_start, mn.n_pts);
    }
    // this warp's first STG element blocks
    WarpIter pf{0, warp};
    pf.norm(pr, warp);
    for (int q = 0; q < STG && pf.valid(pr); ++q) {
      if (lane == 0) {
        const int64_t el = (int64_t)m.elem_start + pf.s;
        if (AXG_BOUND(el, d.n_elem, 2)) issue((kcount + q) % STG, el);
      }
      pf.s += kWarps;
      pf.norm(pr, warp);
    }
    cp_async_wait_all();  // this thread's copies of the patch (issued during the previous one)
    __syncthreads();

    // elements, sub-round by sub-round
    int r0 = 0;
    for (int r = 0; r < pr.n; ++r) {
      const int r1 = pr.end(r);
      bool ready = r == 0;  // round r-1 complete (waited for)
      for (int s = r0 + warp; s < r1; s += kWarps) {
        const uint32_t slot = kcount % STG;
        if (!mbar_wait_bounded(&my_bars[slot], (kcount / STG) & 1u, st.err)) s_timeout = 1;
        const float *blk = my_ring + slot * BS;
        const int32_t info = *reinterpret_cast<const int32_t *>(blk + solid_info_off(NT));
        int axslot = (info & 0xFFFFFF) - 1;
        if (axslot >= 0 && !AXG_BOUND((int64_t)(axslot + 1) * NA * 5 - 1, d.n_m0, 2)) axslot = -1;
        int idx = active ? reinterpret_cast<const uint16_t *>(blk + solid_idx_off(NT))[lane] : 0;
        if (!AXG_BOUND(idx, m.n_pts, 2)) idx = 0;
        idx = spos(idx);
        float u[3] = {0.f, 0.f, 0.f};
        if (active) {
          u[0] = s_u[0][idx];
          if (POLE == POLE_MONO) {
            u[2] = s_u[1][idx];
          } else {
            u[1] = s_u[1][idx];
            u[2] = s_u[2][idx];
          }
        }
        const bool ax = axslot >= 0;
        if (ax && i == 0) {  // apply_axis_mask_{one,two,three}comp on disp
          if (POLE == POLE_MONO) u[0] = 0.f;
          if (POLE == POLE_DI) { u[1] = 0.f; u[2] = 0.f; }
          if (POLE == POLE_QUAD) { u[0] = 0.f; u[1] = 0.f; u[2] = 0.f; }
        }
        float f0, f1 = 0.f, f2;
        const float *m0 = ax ? d.m0 + (int64_t)axslot * (NA * 5) : nullptr;
        if (POLE == POLE_MONO) {
          if (ax) stiff_mono<true>(coef, blk, m0, ml, i, j, u[0], u[2], f0, f2);
          else stiff_mono<false>(coef, blk, m0, ml, i, j, u[0], u[2], f0, f2);
        } else if (POLE == POLE_DI) {
          if (ax) stiff_di<true>(coef, blk, m0, ml, i, j, u[0], u[1], u[2], f0, f1, f2);
          else stiff_di<false>(coef, blk, m0, ml, i, j, u[0], u[1], u[2], f0, f1, f2);
        } else {
          if (ax) stiff_quad<true>(coef, blk, m0, ml, i, j, u[0], u[1], u[2], f0, f1, f2);
          else stiff_quad<false>(coef, blk, m0, ml, i, j, u[0], u[1], u[2], f0, f1, f2);
        }
        if (ax && i == 0) {  // axis mask of acc1
          if (POLE == POLE_MONO) f0 = 0.f;
          if (POLE == POLE_DI) { f1 = 0.f; f2 = 0.f; }
          if (POLE == POLE_QUAD) { f0 = 0.f; f1 = 0.f; f2 = 0.f; }
        }
        // the previous sub-round's accumulations must be complete; the wait
        // comes after this element's stiffness, which hides it
        if (!ready) {
          if (!mbar_wait_bounded(&s_round[r - 1], (round_par >> (r - 1)) & 1u, st.err)) s_timeout = 1;
          ready = true;
        }
        if (active) {
          s_f[0][idx] += f0;
          if (POLE == POLE_MONO) {
            s_f[1][idx] += f2;
          } else {
            s_f[1][idx] += f1;
            s_f[2][idx] += f2;
          }
        }
        // the slot is free again: start the copy of the element STG ahead
        __syncwarp();
        if (pf.valid(pr)) {
          if (lane == 0) {
            const int64_t pel = (int64_t)m.elem_start + pf.s;
            fence_proxy_async();  // the warp's reads of the slot precede the async-proxy write
            if (AXG_BOUND(pel, d.n_elem, 2)) issue(slot, pel);
          }
          pf.s += kWarps;
          pf.norm(pr, warp);
        }
        ++kcount;
      }
      mbar_arrive(&s_round[r]);  // this thread's accumulations of round r are done
      r0 = r1;
      if (r == 0 && next_npts > 0) {
        // the next patch's words have landed in the other buffer: start its gather
        if (!mbar_wait_bounded(&s_wbar[buf ^ 1], ((pcount + 1) / NB) & 1u, st.err)) s_timeout = 1;
        issue_gather(buf ^ 1, next_npts);
      }
    }
    round_par ^= (1u << pr.n) - 1u;  // each used s_round completed once in this patch
    __syncthreads();

    // write-back
    for (int t = threadIdx.x; t < m.n_pts; t += kThreads) {
      const uint32_t g = s_w[t] & kPtIndexMask;
      if (!AXG_BOUND(g, st.nglob, 3)) continue;
#pragma unroll
      for (int c = 0; c < NC; ++c) st.f[gc(c)][g] = s_f[c][spos(t)];
    }
    __syncthreads();
    ++pcount;
  }
  // After a timeout, bulk copies of this CTA may still be in flight into its
  // shared memory: wait (bounded) for the last phase of each ring slot and of
  // the point-word buffer before the CTA exits.
  __syncthreads();
  if (s_timeout) {
    if (lane == 0)
      for (uint32_t q = 0; q < (uint32_t)STG && q < kcount; ++q) {
        const uint32_t k = kcount - 1 - q;  // the last element consumed from slot k % STG
        mbar_drain(&my_bars[k % STG], (k / STG) & 1u);
      }
    if (threadIdx.x == 0 && pcount > 0) mbar_drain(&s_wbar[(pcount - 1) % NB], ((pcount - 1) / NB) & 1u);
  }
}

// ------------------------------------------------------------ attenuation at every GLL point
//
// att_coarse_grained = .false.: memory variables at all 25 GLL points of
// every solid element.  Per launch slot the host packs kFullConst constants:
// [field][GLL point] of delta_mu, delta_kappa, Y, V_s_eta, V_s_xi, V_z_eta,
// V_z_xi, DsDeta_over_J_sol, DzDeta_over_J_sol, DsDxi_over_J_sol,
// DzDxi_over_J_sol, inv_s_solid; then [field][jpol] of Y0, V0_s_eta,
// V0_s_xi, V0_z_eta, V0_z_xi (zero off the axis); then the two Q-table rows.
// The state of a slot is memory_var(0:4,0:4,6,n_sls), src_tr_tm1(0:4,0:4),
// src_dev_tm1(0:4,0:4,6), the reference's layouts.
enum : int {
  F_DMU = 0, F_DKA = 25, F_Y = 50, F_VSE = 75, F_VSX = 100, F_VZE = 125, F_VZX = 150, F_DSDETA = 175,
  F_DZDETA = 200, F_DSDXI = 225, F_DZDXI = 250, F_INVS = 275, F_Y0 = 300, F_V0SE = 305, F_V0SX = 310,
  F_V0ZE = 315, F_V0ZX = 320, F_QMU = 325, F_QKA = 326
};
constexpr int kFullConst = 328;  // floats, a 16-byte multiple
__host__ __device__ constexpr int full_state_stride(int nsls) { return ((150 * nsls + 175 + 3) / 4) * 4; }

struct FullAnelArgs {
  AnelArgs an;            // consts (kFullConst per slot), state, qtab, ex, nsls, state_stride, n_q
  float *fx;              // per slot 3 x 25: minus the anelastic stiffness the next Newmark step adds
  const int32_t *gidx;    // per slot the element's 25 global points
  const uint8_t *axial;   // per slot 1 for an axial element
  int64_t nel;
};

// One warp per element (launch order), lane = GLL point.  UPDATE: the memory
// variables of the step from the displacement the step stored
// (time_step_memvars_4 with compute_strain_att_el_4, SOLVER/attenuation.f90:
// 210-334, 542-606: the gradients of axisym_gradient_solid_el_4, f / s of
// f_over_s_solid_el_4 with L'Hospital's df/ds on the axis).  Then, from the
// memory variables, the anelastic stiffness of glob_anel_stiffness_*_4
// (SOLVER/stiffness_mono.f90:409-507, SOLVER/stiffness_di.f90:604-723,
// SOLVER/stiffness_quad.f90:555-669), stored negated in fx for the next
// step's patch kernel.  Without UPDATE (before a run) only the latter.
template <int POLE, bool UPDATE>
__global__ void __launch_bounds__(kThreads) anel_full_kernel(const __grid_constant__ FullAnelArgs fa, StateArgs st,
                                                             SpecDev sp) {
  pdl_wait();
  pdl_trigger();
  if (*st.stop) return;
  const AnelArgs &an = fa.an;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool active = lane < 25;
  const int ml = active ? lane : 24;
  const int i = ml % 5, j = ml / 5, j5 = 5 * j;
  LaneCoef coef;
  load_coef(sp, i, j, coef);
  const int nsls = an.nsls;
  for (int64_t el = (int64_t)blockIdx.x * kWarps + warp; el < fa.nel; el += (int64_t)gridDim.x * kWarps) {
    const float *cs = an.consts + el * kFullConst;
    float *R = an.state + el * an.state_stride;
    float *trm1 = R + 150 * nsls, *devm1 = trm1 + 25;
    const bool ax = fa.axial[el] != 0;
    if (UPDATE) {
      int32_t g = fa.gidx[25 * el + ml];
      if (!AXG_BOUND(g, st.nglob, 52)) g = 0;
      float u[3] = {st.u[0][g], POLE == POLE_MONO ? 0.f : st.u[1][g], st.u[2][g]};
      if (ax && i == 0) {  // apply_axis_mask_* on disp
        if (POLE == POLE_MONO) u[0] = 0.f;
        if (POLE == POLE_DI) { u[1] = 0.f; u[2] = 0.f; }
        if (POLE == POLE_QUAD) { u[0] = 0.f; u[1] = 0.f; u[2] = 0.f; }
      }
      const float dsdeta = cs[F_DSDETA + ml], dzdeta = cs[F_DZDETA + ml];
      const float dsdxi = cs[F_DSDXI + ml], dzdxi = cs[F_DZDXI + ml], invs = cs[F_INVS + ml];
      // axisym_gradient_solid_el_4 of the field f held lane-wise: (d/ds, d/dz)
      auto grad = [&](float f, float &gs, float &gz) {
        const float m1 = ax ? dxi(f, coef.xi1, j5) : dxi(f, coef.xi2, j5);
        const float m2 = deta(f, coef.eta, i);
        gs = dzdeta * m1 + dzdxi * m2;
        gz = dsdeta * m1 + dsdxi * m2;
      };
      // f_over_s_solid_el_4: f / s; on the axis (ipol = 0 of an axial
      // element) df/ds (dsdf_elem_solid, G1T); the contractions run on every
      // lane of the warp (ax is uniform across it)
      auto fos = [&](float f) {
        float o = invs * f;
        if (ax) {
          float gs, gz;
          grad(f, gs, gz);
          if (i == 0) o = gs;
        }
        return o;
      };
      float gu[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};  // Voigt 1..6
      float b1s, b1z, b2s, b2z;
      grad(POLE == POLE_DI ? u[0] + u[1] : u[0], b1s, b1z);
      grad(u[2], b2s, b2z);
      gu[0] = b1s;
      gu[2] = b2z;
      gu[4] = b1z + b2s;
      if (POLE == POLE_MONO) {
        gu[1] = fos(u[0]);
      } else if (POLE == POLE_DI) {
        gu[1] = 2.f * fos(u[1]);
        grad(u[0] - u[1], b1s, b1z);
        const float t = fos(u[2]);
        gu[3] = -t - b1z;
        gu[5] = -gu[1] - b1s;
      } else {
        gu[1] = fos(u[0] - 2.f * u[1]);
        grad(u[1], b1s, b1z);
        const float t = fos(u[2]);
        const float t2 = fos(u[1] - 2.f * u[0]);
        gu[3] = -2.f * t - b1z;
        gu[5] = t2 - b1s;
      }
      if (active) {
        const float tr = gu[0] + gu[1] + gu[2];
        const float dm = cs[F_DMU + lane], dk = cs[F_DKA + lane];
        float src_dev[6];
#pragma unroll
        for (int v = 0; v < 3; ++v) src_dev[v] = (dm * 2.f) * (gu[v] - tr * (1.f / 3.f));
        src_dev[3] = POLE == POLE_MONO ? 0.f : dm * gu[3];
        src_dev[4] = dm * gu[4];
        src_dev[5] = POLE == POLE_MONO ? 0.f : dm * gu[5];
        const float src_tr = dk * tr;
        int qmu = __float_as_int(cs[F_QMU]), qka = __float_as_int(cs[F_QKA]);
        if (!AXG_BOUND(qmu, an.n_q, 52)) qmu = 0;
        if (!AXG_BOUND(qka, an.n_q, 52)) qka = 0;
        const float *tmu = an.qtab + qmu * 2 * kMaxSls, *tka = an.qtab + qka * 2 * kMaxSls;
        const float trp = trm1[lane];
        for (int q = 0; q < nsls; ++q) {
          const float trb = __ldg(tka + q) * src_tr + __ldg(tka + kMaxSls + q) * trp;
#pragma unroll
          for (int v = 0; v < 6; ++v) {
            if (POLE == POLE_MONO && (v == 3 || v == 5)) continue;  // never written for the monopole
            float *r = R + lane + 25 * (v + 6 * q);
            const float db = __ldg(tmu + q) * src_dev[v] + __ldg(tmu + kMaxSls + q) * devm1[lane + 25 * v];
            float nv = an.ex[q] * *r + db;
            if (v < 3) nv = nv + trb;
            *r = nv;
          }
        }
        trm1[lane] = src_tr;
#pragma unroll
        for (int v = 0; v < 6; ++v) devm1[lane + 25 * v] = src_dev[v];
      }
      __syncwarp();
    }
    // the summed memory variables at the lane's point
    float r[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (active)
      for (int q = 0; q < nsls; ++q)
#pragma unroll
        for (int v = 0; v < 6; ++v) r[v] = r[v] + R[lane + 25 * (v + 6 * q)];
    const float yl = cs[F_Y + ml], vse = cs[F_VSE + ml], vsx = cs[F_VSX + ml];
    const float vze = cs[F_VZE + ml], vzx = cs[F_VZX + ml];
    // X = mxm(G, S) (G1 on axial elements) and mxm(S, G2T)
    auto gx = [&](float S) { return ax ? dxi(S, coef.sxi1, j5) : dxi(S, coef.sxi2, j5); };
    auto ge = [&](float S) { return deta(S, coef.seta, i); };
    // axial vectors at jpol = j (lanes with ipol = 0 use them)
    const float y0 = cs[F_Y0 + j], v0se = cs[F_V0SE + j], v0sx = cs[F_V0SX + j];
    const float v0ze = cs[F_V0ZE + j], v0zx = cs[F_V0ZX + j];
    // outerprod(G0, V)(i, j) = G0(i) V(j), V held by lane (0, j)
    auto outer = [&](float V) { return coef.g0i * __shfl_sync(kFull, V, j5); };
    float l0, l1 = 0.f, l2;
    if (POLE == POLE_MONO) {
      const float S1s = vze * r[0] + vse * r[4], S2s = vzx * r[0] + vsx * r[4];
      const float S1z = vze * r[4] + vse * r[2], S2z = vzx * r[4] + vsx * r[2];
      l0 = gx(S1s) + ge(S2s) + yl * r[1];
      l2 = gx(S1z) + ge(S2z);
      if (ax) {
        const float V1 = v0ze * r[0] + v0se * r[4] + y0 * r[1];
        const float V2 = v0ze * r[4] + v0se * r[2];
        const float V3 = v0zx * r[4] + v0sx * r[2];
        const float V4 = deta(V3, coef.seta, 0);  // vxm(V3, G2T) on the lanes with ipol = 0
        l0 = l0 + outer(V1);
        l2 = l2 + outer(V2);
        if (i == 0) l2 = l2 + V4;
      }
    } else if (POLE == POLE_DI) {
      const float r16m = r[0] - r[5], r54m = r[4] - r[3], r16p = r[0] + r[5], r54p = r[4] + r[3];
      const float S1p = vze * r16m + vse * r54m, S2p = vzx * r16m + vsx * r54m;
      const float S1m = vze * r16p + vse * r54p, S2m = vzx * r16p + vsx * r54p;
      const float S1z = vze * r[4] + vse * r[2], S2z = vzx * r[4] + vsx * r[2];
      l0 = gx(S1p) + ge(S2p);
      l1 = gx(S1m) + ge(S2m) + 2.f * yl * (r[1] - r[5]);
      l2 = gx(S1z) + ge(S2z) - yl * r[3];
      if (ax) {
        const float V1 = v0ze * r16m + v0se * r54m;
        const float V2 = v0zx * r16m + v0sx * r54m;
        const float V3 = deta(V2, coef.seta, 0);
        l0 = l0 + outer(V1);
        if (i == 0) l0 = l0 + V3;
        const float V1m = v0ze * r16p + v0se * r54p + y0 * 2.f * (r[1] - r[5]);
        l1 = l1 + outer(V1m);
        l2 = l2 + outer(V2);  // the reference adds V2 here, as it writes it
      }
    } else {
      const float S1s = vze * r[0] + vse * r[4], S2s = vzx * r[0] + vsx * r[4];
      const float S1p = vze * r[5] + vse * r[3], S2p = vzx * r[5] + vsx * r[3];
      const float S1z = vze * r[4] + vse * r[2], S2z = vzx * r[4] + vsx * r[2];
      l0 = gx(S1s) + ge(S2s) + yl * (r[1] - 2.f * r[5]);
      l1 = -gx(S1p) - ge(S2p) + yl * (r[5] - 2.f * r[1]);
      l2 = gx(S1z) + ge(S2z) - 2.f * yl * r[3];
      if (ax) {
        l0 = l0 + outer(v0ze * r[0] + y0 * (r[1] - 2.f * r[5]));
        l1 = l1 + outer(-v0ze * r[5] + y0 * (r[5] - 2.f * r[1]));
        l2 = l2 + outer(v0se * r[2]);
      }
    }
    if (active) {
      float *x = fa.fx + el * 75;
      x[lane] = -l0;
      x[25 + lane] = -l1;
      x[50 + lane] = -l2;
    }
    __syncwarp();
  }
}

// The final drift of a symplectic step (SOLVER/time_evol_wave.F90:722-727):
// chi += dchi * coefd(nstages+1), disp += velo * coefd(nstages+1), on every
// global point.
struct DriftWork {
  StateArgs solid, fluid;
  float cd, cd_lo;  // coefd(nstages + 1) deltat, an FP32 pair
};
template <class P = One<DriftWork>>
__global__ void drift_kernel(const __grid_constant__ P p) {
  pdl_wait();
  pdl_trigger();
  const int32_t it = blockIdx.x * blockDim.x + threadIdx.x;  // a point of one of the solves
  if (it >= p.items()) return;
  const int sv = p.locate(it);
  const StateArgs &solid = p.at(sv).solid;
  const StateArgs &fluid = p.at(sv).fluid;
  const float cd = p.at(sv).cd, cd_lo = p.at(sv).cd_lo;
  if (*solid.stop) return;
  const int64_t q = it - p.first(sv);
  // u + coefd(nstages+1) v; compensated where the handle keeps compensation
  auto drift = [&](float *u, const float *v, float *cu) {
    if (cu) {
      float k = cu[q];
      u[q] = kahan_add(u[q], mul2(cd, cd_lo, v[q]), k);
      cu[q] = k;
    } else {
      u[q] = u[q] + mul2(cd, cd_lo, v[q]);
    }
  };
  if (q < solid.nglob)
    for (int c = 0; c < 3; ++c)
      if (solid.u[c]) drift(solid.u[c], solid.v[c], solid.cu[c]);
  if (fluid.u[0] && q < fluid.nglob) drift(fluid.u[0], fluid.v[0], fluid.cu[0]);
}

// The Newmark step's predicted displacement up = disp + deltat*velo +
// half_dt_sq*acc0 (SOLVER/time_evol_wave.F90:357-364) of the current state,
// before a run: the point pass keeps it from there on (compensated: with the
// compensation the prediction leaves).  axmask (or null): per point, bit c
// set where the axis mask zeroes component c; those are stored as zero, as
// the step leaves them in its state.
static __global__ void predict_kernel(StateArgs st, const uint8_t *axmask) {
  const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= st.nglob || *st.stop) return;
  const uint32_t m = axmask ? axmask[q] : 0u;
  for (int c = 0; c < 3; ++c) {
    if (!st.up[c]) continue;
    const bool zero = (m >> c) & 1u;
    if (st.cup[c]) {
      float k = st.cu[c][q];
      const float p = predict_comp(st.u[c][q], st.v[c][q], st.a[c][q], st, k);
      st.up[c][q] = zero ? 0.f : p;
      st.cup[c][q] = zero ? 0.f : k;
    } else {
      st.up[c][q] = zero ? 0.f : predict(st.u[c][q], st.v[c][q], st.a[c][q], st);
    }
  }
}

// ------------------------------------------------------------ solid-fluid coupling

struct Coupling {
  // per boundary point (of the receiving domain): CSR of contributions
  const int32_t *pt_gidx;   // receiving global point
  const int32_t *start;     // n+1
  const int32_t *src_gidx;  // sending global point per contribution
  const float *b1, *b2;     // bdry_matr(ipol, b, 1/2) per contribution
  const float *mask;        // per contribution: 0 where the receiving copy is masked, else 1 (or fs mask)
  int32_t n;
  int64_t n_contrib, nglob_recv, nglob_send;  // extents (checked builds)
};

// ------------------------------------------------------------ receivers, step counter

// nc_compute_recfile_seis_bare (SOLVER/seismograms.f90:783-820) every seis_it
// steps into rec(nseismo, 3, num_rec); advances the step counter afterwards.
// One CTA per solve.
struct RecWork {
  StateArgs solid;
  const int32_t *rec_gidx;
  int32_t num_rec, seis_it, pole, nseismo;
  float *rec;
  int32_t *ctl;
};
template <class P = One<RecWork>>
__global__ void receivers_kernel(const __grid_constant__ P p) {
  pdl_wait();
  pdl_trigger();
  if ((int32_t)blockIdx.x >= p.items()) return;
  const RecWork &rw = p.at(p.locate(blockIdx.x));
  const StateArgs &solid = rw.solid;
  const int32_t *rec_gidx = rw.rec_gidx;
  const int32_t num_rec = rw.num_rec, seis_it = rw.seis_it, pole = rw.pole, nseismo = rw.nseismo;
  float *rec = rw.rec;
  const int32_t iter = rw.ctl[CTL_ITER];
  __syncthreads();
  if (!*solid.blowup && seis_it > 0 && iter % seis_it == 0) {
    const int32_t is = iter / seis_it;
    if (is < nseismo) {
      for (int r = threadIdx.x; r < num_rec; r += blockDim.x) {
        const int g = rec_gidx[r];
        if (!AXG_BOUND(g, solid.nglob, 31)) continue;
        const float us = solid.u[0][g], uz = solid.u[2][g];
        const float up = pole == POLE_MONO ? 0.f : solid.u[1][g];
        float v1 = us, v2 = up, v3 = uz;
        if (pole == POLE_MONO) v2 = 0.f;
        if (pole == POLE_DI) { v1 = us + up; v2 = us - up; }
        const int64_t n = nseismo;
        rec[is + n * (0 + 3 * (int64_t)r)] = v1;
        rec[is + n * (1 + 3 * (int64_t)r)] = v2;
        rec[is + n * (2 + 3 * (int64_t)r)] = v3;
      }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    rw.ctl[CTL_STOP] = *solid.blowup;
    rw.ctl[CTL_ITER] = iter + 1;
  }
}

// ------------------------------------------------------------ kernel wavefield dumps

// dump_stuff (SOLVER/time_evol_wave.F90:1201-1249): the fields of one
// snapshot from the state at the end of a step.  One warp per element in the
// reference's element order, lane = GLL point (i, j); the gradients are the
// reference's axisym_gradient_* (SOLVER/pointwise_derivatives.f90:329-545)
// as shuffle contractions: mxm1 = G1T f (axial element) or G2T f, mxm2 = f G2,
// d/ds = dzdeta mxm1 + dzdxi mxm2, d/dz = dsdeta mxm1 + dsdxi mxm2.
enum { DUMP_DISPL_ONLY = 1, DUMP_STRAIN_ONLY = 2, DUMP_DISPL_VELO = 3, DUMP_FULLFIELDS = 4 };

struct DumpArgs {
  const int32_t *gidx;     // (25, nel): the element's points (0-based, internal numbering)
  const uint8_t *axial;    // per element: 1 on the axis
  const float *pw[5];      // DsDeta, DzDeta, DsDxi, DzDxi over J, 1/s: (25, nel)
  const float *inv_rho;    // fluid: 1/rho (25, nel)
  const float *u[3];       // solid disp (u[1] null for the monopole) / fluid chi (u[0])
  const float *v[3];       // solid velo / fluid dchi (v[0])
  float *out;              // the domain's first field
  int64_t nel, nglob;
  int32_t type, ibeg, iend, jbeg, jend;
  const int32_t *kwf;      // kernel wavefield layout: position of each element point (25, nel), -1: none; or null
  int64_t npt;             // points per field in that layout
  int32_t nsrcel;          // solid: elements whose values are dumped as zero (src_dump_type = 'mask')
  int32_t srcel[8];        // ... their 0-based indices
};

struct DumpLane {
  float dsdeta, dzdeta, dsdxi, dzdxi, inv_s;
};

// (d/ds f, d/dz f) at this lane; warp-uniform `ax`
__device__ __forceinline__ void dump_grad(const LaneCoef &c, const DumpLane &w, bool ax, int i, int j5, float f,
                                          float &gs, float &gz) {
  const float m1 = ax ? dxi(f, c.xi1, j5) : dxi(f, c.xi2, j5);
  const float m2 = deta(f, c.eta, i);
  gs = fmaf(w.dzdeta, m1, w.dzdxi * m2);
  gz = fmaf(w.dsdeta, m1, w.dsdxi * m2);
}

// f_over_s_*: f / s, and at the axis (i = 0 of an axial element) L'Hospital's
// df/ds (dsdf_*_allaxis, with G1T)
__device__ __forceinline__ float dump_fos(const LaneCoef &c, const DumpLane &w, bool ax, int i, int j5, float f) {
  float r = w.inv_s * f;
  if (ax) {
    const float m1 = dxi(f, c.xi1, j5), m2 = deta(f, c.eta, i);
    if (i == 0) r = fmaf(w.dzdeta, m1, w.dzdxi * m2);
  }
  return r;
}

template <int POLE, bool FLUID>
__global__ void __launch_bounds__(kThreads) wavefield_dump_kernel(DumpArgs a, SpecDev sp) {
  const int lane = threadIdx.x & 31;
  const bool active = lane < 25;
  const int ml = active ? lane : 24;  // idle lanes take part in the shuffles on point 24's data
  const int i = ml % 5, j = ml / 5, j5 = 5 * j;
  LaneCoef coef;
  load_coef(sp, i, j, coef);
  const int ni = a.iend - a.ibeg + 1, nj = a.jend - a.jbeg + 1;
  const int64_t np = (int64_t)ni * nj;
  const bool mine = active && i >= a.ibeg && i <= a.iend && j >= a.jbeg && j <= a.jend;
  const int64_t pidx = (i - a.ibeg) + (int64_t)ni * (j - a.jbeg);
  const int64_t nwarps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t e = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); e < a.nel; e += nwarps) {
    const int64_t q = 25 * e + ml;
    int32_t g = a.gidx[q];
    if (!AXG_BOUND(g, a.nglob, 41)) g = 0;
    const bool ax = a.axial[e] != 0;
    const DumpLane w{a.pw[0][q], a.pw[1][q], a.pw[2][q], a.pw[3][q], a.pw[4][q]};
    int fld = 0;
    const int32_t kpos = a.kwf && active ? a.kwf[q] : -1;
    // src_dump_type = 'mask': the source elements' solid values are zero
    // (eradicate_src_elem_values, SOLVER/wavefields_io.f90:1123-1153)
    bool masked = false;
    if (!FLUID)
      for (int k = 0; k < a.nsrcel && k < 8; ++k) masked = masked || a.srcel[k] == e;
    auto put = [&](float val) {
      if (masked) val = 0.f;
      if (a.kwf) {
        if (kpos >= 0 && AXG_BOUND(kpos, a.npt, 42)) a.out[fld * a.npt + kpos] = val;
      } else if (mine) {
        a.out[(fld * a.nel + e) * np + pidx] = val;
      }
      ++fld;
    };
    constexpr bool nonmono = POLE != POLE_MONO;
    if (!FLUID) {
      const float x1 = a.u[0][g], x2 = nonmono ? a.u[1][g] : 0.f, x3 = a.u[2][g];
      if (a.type == DUMP_STRAIN_ONLY || a.type == DUMP_FULLFIELDS) {
        // compute_strain, SOLVER/time_evol_wave.F90:1286-1345
        float g1, g2, h1, h2;
        dump_grad(coef, w, ax, i, j5, POLE == POLE_DI ? x1 + x2 : x1, g1, g2);  // dsus, dzus
        put(g1);
        dump_grad(coef, w, ax, i, j5, x3, h1, h2);                              // dsuz, dzuz
        const float n1 = (g2 + h1) / 2.f, n2 = g1 + h2;
        put(n1);                                                                // E31
        float buff;
        if (POLE == POLE_MONO) buff = dump_fos(coef, w, ax, i, j5, x1);
        else if (POLE == POLE_DI) buff = 2.f * dump_fos(coef, w, ax, i, j5, x2);
        else buff = dump_fos(coef, w, ax, i, j5, x1 - 2.f * x2);
        put(buff);                                                              // E22
        put(buff + n2);                                                         // Ekk
        if (POLE == POLE_DI) {
          float p1, p2;
          dump_grad(coef, w, ax, i, j5, x1 - x2, p1, p2);                       // dsup, dzup
          put(-dump_fos(coef, w, ax, i, j5, x2) - p1 / 2.f);                    // E12
          put(-(dump_fos(coef, w, ax, i, j5, x3) + p2) / 2.f);                  // E23
        } else if (POLE == POLE_QUAD) {
          float p1, p2;
          dump_grad(coef, w, ax, i, j5, x2, p1, p2);
          put(-dump_fos(coef, w, ax, i, j5, x1 + x2 / 2.f) - p1 / 2.f);
          put(-dump_fos(coef, w, ax, i, j5, x3) - p2 / 2.f);
        }
      }
      // dump_disp_global / dump_velo_global transform the dipole to (s, phi);
      // dump_disp / dump_velo_dchi write the state as it is
      const bool global = a.type != DUMP_DISPL_VELO;
      auto vec = [&](float y1, float y2, float y3) {
        put(global && POLE == POLE_DI ? y1 + y2 : y1);
        if (nonmono) put(global && POLE == POLE_DI ? y1 - y2 : y2);
        put(y3);
      };
      if (a.type == DUMP_DISPL_ONLY || a.type == DUMP_DISPL_VELO) vec(x1, x2, x3);
      if (a.type == DUMP_DISPL_VELO || a.type == DUMP_FULLFIELDS)
        vec(a.v[0][g], nonmono ? a.v[1][g] : 0.f, a.v[2][g]);
    } else {
      const float chi = a.u[0][g];
      const float irho = a.inv_rho[q];
      if (a.type == DUMP_DISPL_VELO) {
        put(chi);
        put(a.v[0][g]);
        continue;
      }
      if (a.type == DUMP_STRAIN_ONLY || a.type == DUMP_FULLFIELDS) {
        // SOLVER/time_evol_wave.F90:1347-1408: usz = grad(chi) / rho
        float c1, c2, g1, g2, h1, h2;
        dump_grad(coef, w, ax, i, j5, chi, c1, c2);
        const float us = c1 * irho, uz = c2 * irho;
        dump_grad(coef, w, ax, i, j5, us, g1, g2);
        put(g1);
        dump_grad(coef, w, ax, i, j5, uz, h1, h2);
        const float n1 = (g2 + h1) / 2.f, n2 = g1 + h2;
        put(n1);
        const float fs = dump_fos(coef, w, ax, i, j5, us);
        put(fs);
        put(fs + n2);
        if (POLE == POLE_DI) {
          put((-fs) / 2.f);
          put(dump_fos(coef, w, ax, i, j5, uz) / 2.f);
        } else if (POLE == POLE_QUAD) {
          put(-fs);
          put(-dump_fos(coef, w, ax, i, j5, uz));
        }
      }
      auto flu_vec = [&](float f) {  // inv_rho grad(f): s, phi (zero), z
        float c1, c2;
        dump_grad(coef, w, ax, i, j5, f, c1, c2);
        put(irho * c1);
        if (nonmono) put(0.f);
        put(irho * c2);
      };
      if (a.type == DUMP_DISPL_ONLY) flu_vec(chi);
      if (a.type == DUMP_FULLFIELDS) flu_vec(a.v[0][g]);
    }
  }
}

}  // namespace axg
