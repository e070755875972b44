// axg_stream.cuh -- the step in two launches: an element pass and a point pass.
//
// The element pass computes the element contributions, the point pass sums
// each remaining point's in a fixed order, adds the solid-fluid coupling and
// applies the source and the corrector.  There are no colours and no atomics;
// the summation order is fixed, so results are bit-reproducible.  The solid's
// element pass has two forms:
//   scattered (meshes whose contributions stay in L2): every element writes
//     its 25 contributions to a buffer (fel), the point pass sums the copies
//     of every point (CSR over ent).  Any number of warps work at once, so a
//     small mesh's step is two short launches;
//   patched (large meshes): a CTA holds a patch of elements, accumulates them
//     in shared memory in a fixed order, and finishes the points that only the
//     patch holds; a deferred point (shared with another patch, or coupled to
//     the fluid) gets a partial sum per patch, and the point pass finishes it.
//     The contributions never leave the SM, so that the step moves little more
//     than the bytes it cannot do without.
//
// An element is held in five lanes, one per GLL column j (i = 0..4 in
// registers), six elements per warp (30 of 32 lanes).  With a column per lane
// the xi contractions are in-lane FMAs with constant-bank matrices, and the
// eta contractions read the other columns from a per-warp shared buffer as
// broadcast 16-byte loads: 4 stores and 20 loads per warp and stage for six
// elements, where a lane per point takes 30 shuffles per element.  Warp
// instructions counted per solid element (with a fifth to a third as many fluid
// elements): 193 scattered quadrupole, 320 dipole with cg4 attenuation, 337 patched
// quadrupole and 248 monopole, which finish points as well; a lane per point took
// 380 without those.  Issue slots are 24 to 40 % used: what bounds the pass from
// HBM is the loads in flight of 11 to 16 resident warps per SM.
//
// Element arrays are packed per group of up to six consecutive element slots,
// in rows of eight floats per lane (one 256-bit load each): a lane's values
// are its five points (scattered: five global indices; patched: five 11-bit
// patch-local indices in two words), then the points' metric terms, point by
// point.
#pragma once

#include "axg_kernels.cuh"

namespace axg {

constexpr int kGrp = 6;             // elements per warp
constexpr int kGrpLanes = 5 * kGrp;
constexpr int kGrpWarps = 4;        // warps per CTA of the element pass
constexpr int kGrpThreads = 32 * kGrpWarps;

// a lane's values: kOff index words, then 5 NT metric terms; kRows rows of
// eight floats, and (patched, where it saves padding) kTail floats in an
// array of their own
template <int POLE, bool PATCH>
struct SolidGrp {
  static constexpr int NT = n_terms(POLE), NC = POLE == POLE_MONO ? 2 : 3, NA = n_axial(POLE);
  static constexpr int kOff = PATCH ? 2 : 5;
  static constexpr int kValues = kOff + 5 * NT;
  static constexpr int kRest = kValues % 8;
  static constexpr int kTail = PATCH && (kRest == 2 || kRest == 4) ? kRest : 0;
  static constexpr int kRows = (kValues - kTail + 7) / 8;
};
constexpr int solid_fs(int pole) { return pole == POLE_MONO ? 12 : 16; }  // contribution floats per (element, j)
constexpr int kFluidFs = 8;
__host__ __device__ constexpr int64_t grp_count(int64_t nel) { return (nel + kGrp - 1) / kGrp; }
// bit 31 of a lane's first index word: axial element
constexpr uint32_t kGrpAxial = 1u << 31, kGrpIdx = 0x0FFFFFFFu;
static_assert(kGrpIdx == kPtIndexMask, "the planner refuses meshes of more points");

// A group: its first element slot, its element count and (patched) how many
// groups of its patch must have accumulated before it may.
struct GroupMeta {
  int32_t slot0;
  uint16_t n, wait;
};
// Group `grp` of a scattered solid: the elements off the axis, then the axial
// ones from slot n_off on, each kind in groups of its own.  A group of both is
// computed twice, and on a small mesh, whose groups all run at once, that was
// the step's length: 3.40 against 3.14 ms for 400 steps of the PREM 50 s mesh,
// 2.33 against 1.95 ms for 250 steps of 45 elements, before and after.
__host__ __device__ inline GroupMeta scatter_meta(int32_t grp, int64_t n_off, int64_t nel) {
  const int64_t g1 = grp_count(n_off);
  const int64_t s = grp < g1 ? (int64_t)grp * kGrp : n_off + (grp - g1) * kGrp, end = grp < g1 ? n_off : nel;
  return GroupMeta{(int32_t)s, (uint16_t)(end - s < kGrp ? end - s : kGrp), 0};
}
__host__ __device__ inline int64_t scatter_groups(int64_t n_off, int64_t nel) {
  return grp_count(n_off) + grp_count(nel - n_off);
}
// place of lane value v of element e (column j) of a group, in rows of `row`
// floats per lane and `rows` rows
__host__ __device__ constexpr int64_t grp_at(const GroupMeta &g, int e, int j, int v, int rows, int row) {
  return ((int64_t)g.slot0 * 5 * rows + (int64_t)(v / row) * 5 * g.n + 5 * e + j) * row + v % row;
}

// A patch: its own points are int_start .. int_start + n_int, its deferred
// points the slots def_start .. def_start + n_def of the deferred lists; a
// local point index below n_int is an own point, others count the deferred.
struct PatchInfo {
  int32_t group0;
  int32_t int_start, def_start;
  uint16_t n_groups, n_int, n_def, axis;  // axis: the patch has own points on the axis
  int32_t pad[3];
};
static_assert(sizeof(PatchInfo) == 32, "PatchInfo must be 32 bytes");
constexpr int kMaxDef = kMaxPatchPoints;  // deferred points of a patch (shared memory)

// flags of a point's CSR start word: the first entry of the point is a
// coupling row (not a copy); on the axis; carries a solid source term
constexpr uint32_t kStCoupled = 1u << 31, kStAxis = 1u << 30, kStSource = 1u << 29, kStMask = kStSource - 1u;

// Attenuation (cg4) in group layout: the four cg points of the group's
// elements side by side (lane 4 e + k): constants as three float4 rows
// (delta_mu, delta_kappa, Y, V_s_eta | V_s_xi, V_z_eta, V_z_xi, DsDeta |
// DzDeta, DsDxi, DzDxi, 1/s); state per SLS three float2 rows (components
// 0..5), then three float2 rows of src_dev_tm1 and one float row of
// src_tr_tm1.
constexpr int kCgLanes = 4 * kGrp;
__host__ __device__ constexpr int cg_state_floats(int nsls) { return 6 * nsls + 7; }  // per cg point
// place of component v of solid q (q = nsls: src_dev_tm1; v = 6: src_tr_tm1)
// at cg point k of element e of a group
__host__ __device__ constexpr int64_t cg_state_at(const GroupMeta &g, int e, int k, int q, int v, int nsls) {
  const int64_t b = (int64_t)g.slot0 * 4 * cg_state_floats(nsls);
  if (v == 6) return b + (int64_t)6 * (nsls + 1) * 4 * g.n + 4 * e + k;
  return b + ((int64_t)(3 * q + v / 2) * 4 * g.n + 4 * e + k) * 2 + v % 2;
}
__host__ __device__ constexpr int64_t cg_const_at(const GroupMeta &g, int e, int k, int f) {
  return (int64_t)g.slot0 * 48 + ((int64_t)(f / 4) * 4 * g.n + 4 * e + k) * 4 + f % 4;
}

struct CgArgs {
  const float *consts;      // 48 floats per element slot
  const int2 *q;            // per element slot: Q rows of Q_mu, Q_kappa
  float *state;             // 4 cg_state_floats(nsls) floats per element slot
  const float *qtab;        // per distinct Q: ts_fac_t(j) a_j(Q) at [0, kMaxSls), ts_fac_tm1(j) a_j(Q) after
  float ex[kMaxSls];        // exp_w_j_deltat
  int32_t nsls, n_q;
};

struct StreamDomain {
  const float *blocks;      // the groups' rows
  const float *tails;       // patched: the groups' tail values, or null
  const int32_t *elinfo;    // per slot: bits 0..23 axial slot + 1, bits 24..27 source slot + 1
  const float *m0;          // axial vectors
  const float *aux;         // solid: fx (3 x 25 per slot) or null; fluid: free-surface mask (25 per slot) or null
  const float *srcfl;       // fluid source terms (8, 25) or null
  float *fel;               // contributions; patched: the deferred points' partial sums (4 floats per slot)
  const int32_t *start;     // CSR start words (kSt* flags) of the point pass's points
  const int32_t *ent;       // per point: [coupling row,] the fel index of each copy or partial sum
  // patched
  const PatchInfo *patches;
  const GroupMeta *groups;
  const int32_t *def;       // the deferred points' global indices, patch by patch
  int32_t src_patch[8];     // patches whose own points (scattered: element slots whose inner points) carry source terms
  int32_t n_src_patch, n_patches;
  int64_t n_off;            // scattered solid: elements off the axis
  int64_t nel, nglob, n_m0, n_ent, n_fel, n_def;
};

// One launch of a solve's step.  Its CTAs are, in order: element-pass CTAs of
// the solid (one per patch, or kGrpWarps groups each), of the fluid groups,
// the rows of the coupling into the fluid; or point-pass CTAs of a scattered
// solid's inner points [0, p0), of the solid points [p0, nglob), of the fluid
// points, and the receivers' CTA.
struct StreamWork {
  StreamDomain ds, df;
  StateArgs solid, fluid;
  Coupling to_fluid, to_solid;
  float *ffl;               // the fluid force partial sums (coupling into the fluid)
  const uint8_t *axmask;    // the solid's per-point axis mask bits or null
  CgArgs cg;
  int32_t p0;               // first solid point of the point pass
  int32_t nb_se, nb_fe, nb_cp, nb_si, nb_sp, nb_fp, nb_rec;  // CTAs per role
  int32_t prefetch;         // element pass: CTAs ahead whose blocks are prefetched into L2 (0: none)
  int32_t *ctl;             // the solve's control words (CTL_*)
  int32_t parity;           // CTL_PARITY after a Newmark step
  const int32_t *memvar_gidx;  // memvar_kernel: each element slot's 25 points
  RecWork rec;
};

// up to kMaxStream solves advanced by one launch (parameter space)
constexpr int kMaxStream = 12;
struct StreamOne {
  static constexpr bool kMany = false;
  StreamWork w;
  __device__ __forceinline__ const StreamWork &find(int &) const { return w; }
};
struct StreamMany {
  static constexpr bool kMany = true;
  int32_t n;
  int32_t start[kMaxStream + 1];  // CTA prefix over the solves
  StreamWork w[kMaxStream];
  __device__ __forceinline__ const StreamWork &find(int &b) const {
    int s = 0;
    while (s + 1 < n && start[s + 1] <= b) ++s;
    b -= start[s];
    return w[s];
  }
};

// ------------------------------------------------------------ loads and stores

__device__ __forceinline__ void ldg8(const float *p, float (&v)[8], uint64_t pol) {
  asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8], %9;"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
               : "l"(p), "l"(pol));
}
__device__ __forceinline__ void stg8(float *p, const float (&v)[8]) {
  asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]),
               "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
               : "memory");
}
__device__ __forceinline__ uint64_t policy_evict_normal() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ void prefetch_l2(const void *p, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// A flag of a solve that has stopped, read before the wait for the step before.
// It is set once and stays, so a set one is true whenever it is read, and a CTA
// that reads it before it is set finds it after the wait.  Loaded with a warp's
// first rows it costs nothing; a return that waits for a load after the wait
// cost 4 to 12 % of every step (24.4 for 21.8 ms on 786 432 elements).
__device__ __forceinline__ bool stopped_before(const int32_t *flag) {
  int32_t f;
  asm volatile("ld.relaxed.cta.global.s32 %0, [%1];" : "=r"(f) : "l"(flag));
  return f != 0;
}

// ------------------------------------------------------------ column helpers

// exchange buffer: NV values per lane, 16-byte rows; strides of 20 (15 values)
// and 12 (10 or 5) floats put the 16-byte accesses of eight lanes on
// distinct banks
template <int NV>
struct Xch {
  static constexpr int kRows = (NV + 3) / 4;
  static constexpr int kStride = NV > 12 ? 20 : 12;
};
constexpr int kXchFloats = 32 * 20;  // per warp

template <int NC>
__device__ __forceinline__ void xch_put(float *xw, int lane, const float (&v)[NC][5]) {
  float4 *p = reinterpret_cast<float4 *>(xw + lane * Xch<5 * NC>::kStride);
#pragma unroll
  for (int q = 0; q < Xch<5 * NC>::kRows; ++q) {
    float4 t;
    auto at = [&](int x) { return x < 5 * NC ? v[x / 5][x % 5] : 0.f; };
    t.x = at(4 * q);
    t.y = at(4 * q + 1);
    t.z = at(4 * q + 2);
    t.w = at(4 * q + 3);
    p[q] = t;
  }
}
// out[c][i] = sum_k v_k[c][i] coef[k], v_k the values lane e5 + k put
template <int NC>
__device__ __forceinline__ void xch_eta(const float *xw, int e5, const float (&coef)[5], float (&out)[NC][5]) {
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    const float4 *p = reinterpret_cast<const float4 *>(xw + (e5 + k) * Xch<5 * NC>::kStride);
#pragma unroll
    for (int q = 0; q < Xch<5 * NC>::kRows; ++q) {
      const float4 t = p[q];
      const float tv[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int x = 4 * q + r;
        if (x < 5 * NC) out[x / 5][x % 5] = k == 0 ? tv[r] * coef[k] : fmaf(tv[r], coef[k], out[x / 5][x % 5]);
      }
    }
  }
}
// out[c][i] = sum_k v[c][k] M(k, i) with M(k, i) = g[k + 5 i] (first stage)
// or g[i + 5 k] (second stage)
template <int NC, bool SECOND>
__device__ __forceinline__ void col_xi(const float *g, const float (&v)[NC][5], float (&out)[NC][5]) {
#pragma unroll
  for (int c = 0; c < NC; ++c)
#pragma unroll
    for (int i = 0; i < 5; ++i) {
      float s = g[SECOND ? i : 5 * i] * v[c][0];
#pragma unroll
      for (int k = 1; k < 5; ++k) s = fmaf(SECOND ? g[i + 5 * k] : g[k + 5 * i], v[c][k], s);
      out[c][i] = s;
    }
}

// out[c][i] += sum_k g[i + 5 k] v[c][k], term by term
template <int NC>
__device__ __forceinline__ void col_xi_add(const float *g, const float (&v)[NC][5], float (&out)[NC][5]) {
#pragma unroll
  for (int c = 0; c < NC; ++c)
#pragma unroll
    for (int i = 0; i < 5; ++i)
#pragma unroll
      for (int k = 0; k < 5; ++k) out[c][i] = fmaf(g[i + 5 * k], v[c][k], out[c][i]);
}

// component c of a group array is the axis-masked one of the pole (group
// arrays hold s, z for the monopole)
template <int POLE>
__device__ __forceinline__ constexpr bool col_masked(int c) {
  return POLE == POLE_QUAD || (POLE == POLE_MONO ? c == 0 : c != 0);
}

// ------------------------------------------------------------ attenuation in the element pass

// The memory-variable work of the group's cg points, lane 4 e + k: returns in
// `sc` (shared, 9 floats per cg lane) the anelastic stress terms the
// stiffness subtracts at that point -- S1 (three components), S2 (three), y
// (three), in the order of the displacement components -- and, with UPDATE,
// advances the memory variables (time_step_memvars_cg4,
// SOLVER/attenuation.f90:81-202) from the derivatives the columns left in xw
// (per lane 5 e + j, j in {1, 3}: two points of gx[NC], ge[NC], u[NC]).  The
// sums are those of glob_anel_stiffness_*_cg4; subtracting the terms from S1,
// S2 and the local part before the second stage makes their contraction part
// of the elastic one.
constexpr int kCgBatch = 5;  // solids whose memory variables are in flight together

// What cg_point reads, copied to shared memory by the cg lane itself while its
// warp gathers the displacements: the constants before the step's wait, the
// state of the first kCgBatch solids and the last source terms after it.
// In a warp's scratch `sc`, after the 9 results per cg lane.  Dipole steps with
// 5 solids took 133.3 us on 99 450 elements and 371.6 on 278 297 with these
// read where they are used, and take 131.9 and 369.2.  (Held in registers from
// the gather on they spill: 157.)
constexpr int kScConst = 9 * kCgLanes, kScState = kScConst + 12 * kCgLanes,
              kScTr = kScState + 6 * (kCgBatch + 1) * kCgLanes;
constexpr int kScFloats = kScTr + kCgLanes;  // per warp
static_assert(kScConst % 4 == 0 && kScState % 2 == 0 && kScFloats % 4 == 0, "aligned copies");
__device__ __forceinline__ void cg_stage_consts(const CgArgs &cg, float *sc, const GroupMeta &g, int lane) {
  const int nl = 4 * g.n;
  if (lane >= nl) return;
  const float *cs = cg.consts + (int64_t)g.slot0 * 48 + 4 * lane;
#pragma unroll
  for (int r = 0; r < 3; ++r) cp_async16(sc + kScConst + 4 * (r * kCgLanes + lane), cs + (int64_t)4 * r * nl);
}
__device__ __forceinline__ void cg_stage_state(const CgArgs &cg, float *sc, const GroupMeta &g, int lane) {
  const int nl = 4 * g.n, nsls = cg.nsls;
  if (lane >= nl) return;
  const float *b = cg.state + (int64_t)g.slot0 * 4 * cg_state_floats(nsls);
  float *s = sc + kScState + 2 * lane;
#pragma unroll
  for (int w = 0; w < 3; ++w)
    cp_async8(s + 2 * (3 * kCgBatch + w) * kCgLanes, b + 2 * ((int64_t)(3 * nsls + w) * nl + lane));
  cp_async4(sc + kScTr + lane, b + 6 * (nsls + 1) * nl + lane);
#pragma unroll
  for (int q = 0; q < kCgBatch; ++q)
    if (q < nsls)
#pragma unroll
      for (int w = 0; w < 3; ++w)
        cp_async8(s + 2 * (3 * q + w) * kCgLanes, b + 2 * ((int64_t)(3 * q + w) * nl + lane));
}

// STAGED: what the two functions above copied is read from there.
template <int POLE, bool UPDATE, bool STAGED>
__device__ __forceinline__ void cg_point(const CgArgs &cg, const float *xw, float *sc, const GroupMeta &g, int lane,
                                         bool mine) {
  constexpr int NC = POLE == POLE_MONO ? 2 : 3;
  const int nl = 4 * g.n;  // cg lanes of the group
  const int cl = lane < nl ? lane : 0;
  const int e = cl >> 2, k = cl & 3, jj = (k & 1) ? 3 : 1, ip = k >> 1;
  const int nsls = cg.nsls;
  const float4 *cs = reinterpret_cast<const float4 *>(cg.consts + (int64_t)g.slot0 * 48) + cl;
  const float4 *cst = STAGED ? reinterpret_cast<const float4 *>(sc + kScConst) + cl : cs;
  const int crow = STAGED ? kCgLanes : nl;
  if (STAGED) cp_async_wait_all();
  const float4 c0 = cst[0], c1 = cst[crow], c2 = cst[2 * crow];
  const float2 *ss = reinterpret_cast<const float2 *>(sc + kScState) + cl;
  const float dmu = c0.x, dka = c0.y, yl = c0.z, vse = c0.w, vsx = c1.x, vze = c1.y, vzx = c1.z;
  float *sbase = cg.state + (int64_t)g.slot0 * 4 * cg_state_floats(nsls);
  float2 *st = reinterpret_cast<float2 *>(sbase) + cl;
  float *trp = sbase + 6 * (nsls + 1) * nl + cl;
  float src[6], tr = 0.f, sk = 0.f;
  if (UPDATE) {
    const float *x = xw + (5 * e + jj) * 20 + ip * 3 * NC;
    const float dsdeta = c1.w, dzdeta = c2.x, dsdxi = c2.y, dzdxi = c2.z, invs = c2.w;
    auto grad_s = [&](float m1, float m2) { return dzdeta * m1 + dzdxi * m2; };
    auto grad_z = [&](float m1, float m2) { return dsdeta * m1 + dsdxi * m2; };
    float gx[NC], ge[NC], u[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      gx[c] = x[c];
      ge[c] = x[NC + c];
      u[c] = x[2 * NC + c];
    }
    float g[6];
    const float b1x = POLE == POLE_DI ? gx[0] + gx[1] : gx[0], b1e = POLE == POLE_DI ? ge[0] + ge[1] : ge[0];
    const float b1s = grad_s(b1x, b1e), b1z = grad_z(b1x, b1e);
    const float b2s = grad_s(gx[NC - 1], ge[NC - 1]), b2z = grad_z(gx[NC - 1], ge[NC - 1]);
    g[0] = b1s;
    g[2] = b2z;
    g[4] = b1z + b2s;
    if (POLE == POLE_MONO) {
      g[1] = invs * u[0];
      g[3] = g[5] = 0.f;
    } else if (POLE == POLE_DI) {
      g[1] = 2.f * (invs * u[1]);
      const float cx = gx[0] - gx[1], ce = ge[0] - ge[1];
      g[3] = -(invs * u[NC - 1]) - grad_z(cx, ce);
      g[5] = -g[1] - grad_s(cx, ce);
    } else {
      g[1] = invs * (u[0] - 2.f * u[1]);
      g[3] = -2.f * (invs * u[NC - 1]) - grad_z(gx[1], ge[1]);
      g[5] = invs * (u[1] - 2.f * u[0]) - grad_s(gx[1], ge[1]);
    }
    tr = g[0] + g[1] + g[2];
#pragma unroll
    for (int v = 0; v < 3; ++v) src[v] = (dmu * 2.f) * (g[v] - tr * (1.f / 3.f));
    src[3] = POLE == POLE_MONO ? 0.f : dmu * g[3];
    src[4] = dmu * g[4];
    src[5] = POLE == POLE_MONO ? 0.f : dmu * g[5];
    sk = dka * tr;
  }
  float r[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (UPDATE) {
    int2 qr = __ldg(cg.q + g.slot0 + e);
    if (!AXG_BOUND(qr.x, cg.n_q, 61)) qr.x = 0;
    if (!AXG_BOUND(qr.y, cg.n_q, 61)) qr.y = 0;
    const float *tmu = cg.qtab + qr.x * 2 * kMaxSls, *tka = cg.qtab + qr.y * 2 * kMaxSls;
    float dv[6];
#pragma unroll
    for (int w = 0; w < 3; ++w) {
      const float2 t = STAGED ? ss[(3 * kCgBatch + w) * kCgLanes] : st[(3 * nsls + w) * nl];
      dv[2 * w] = t.x;
      dv[2 * w + 1] = t.y;
    }
    const float tk = STAGED ? sc[kScTr + cl] : *trp;
    const bool store = mine && lane < nl;
    constexpr int kB = STAGED ? 1 : kCgBatch;
    for (int q0 = 0; q0 < nsls; q0 += kB) {
      // the batch's loads are issued together, before its stores
      float2 R[kB][3];
#pragma unroll
      for (int b = 0; b < kB; ++b)
        if (q0 + b < nsls)
#pragma unroll
          for (int w = 0; w < 3; ++w)
            R[b][w] = STAGED && q0 < kCgBatch ? ss[(3 * q0 + w) * kCgLanes] : st[(3 * (q0 + b) + w) * nl];
#pragma unroll
      for (int b = 0; b < kB; ++b) {
        const int q = q0 + b;
        if (q >= nsls) break;
        const float tm = __ldg(tmu + q), tm1 = __ldg(tmu + kMaxSls + q);
        const float trb = __ldg(tka + q) * sk + __ldg(tka + kMaxSls + q) * tk;
        const float ex = cg.ex[q];
        auto next = [&](int v, float o) {
          r[v] = r[v] + o;
          if (POLE == POLE_MONO && (v == 3 || v == 5)) return o;  // never written for the monopole
          float nv = ex * o + (tm * src[v] + tm1 * dv[v]);
          if (v < 3) nv = nv + trb;
          return nv;
        };
#pragma unroll
        for (int w = 0; w < 3; ++w) {
          const float2 nw = make_float2(next(2 * w, R[b][w].x), next(2 * w + 1, R[b][w].y));
          if (store) st[(3 * q + w) * nl] = nw;
        }
      }
    }
    if (store) {
#pragma unroll
      for (int w = 0; w < 3; ++w) st[(3 * nsls + w) * nl] = make_float2(src[2 * w], src[2 * w + 1]);
      *trp = sk;
    }
  } else {
    for (int q = 0; q < nsls; ++q)
#pragma unroll
      for (int w = 0; w < 3; ++w) {
        const float2 old = st[(3 * q + w) * nl];
        r[2 * w] = r[2 * w] + old.x;
        r[2 * w + 1] = r[2 * w + 1] + old.y;
      }
  }
  float S1[3] = {0.f, 0.f, 0.f}, S2[3] = {0.f, 0.f, 0.f}, y[3] = {0.f, 0.f, 0.f};
  if (POLE == POLE_DI) {
    S1[0] = vze * (r[0] - r[5]) + vse * (r[4] - r[3]);
    S2[0] = vzx * (r[0] - r[5]) + vsx * (r[4] - r[3]);
    S1[1] = vze * (r[0] + r[5]) + vse * (r[4] + r[3]);
    S2[1] = vzx * (r[0] + r[5]) + vsx * (r[4] + r[3]);
  } else {
    S1[0] = vze * r[0] + vse * r[4];
    S2[0] = vzx * r[0] + vsx * r[4];
    if (POLE == POLE_QUAD) {
      S1[1] = -(vze * r[5] + vse * r[3]);
      S2[1] = -(vzx * r[5] + vsx * r[3]);
    }
  }
  S1[NC - 1] = vze * r[4] + vse * r[2];
  S2[NC - 1] = vzx * r[4] + vsx * r[2];
  if (POLE == POLE_MONO) {
    y[0] = yl * r[1];
  } else if (POLE == POLE_DI) {
    y[1] = 2.f * yl * (r[1] - r[5]);
    y[2] = -(yl * r[3]);
  } else {
    y[0] = yl * (r[1] - 2.f * r[5]);
    y[1] = yl * (r[5] - 2.f * r[1]);
    y[2] = -(2.f * yl * r[3]);
  }
  if (sc && lane < nl) {
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      sc[9 * cl + c] = S1[c];
      sc[9 * cl + 3 + c] = S2[c];
      sc[9 * cl + 6 + c] = y[c];
    }
  }
}

// the columns j = 1, 3 leave the derivatives and displacements of their two
// cg points for cg_point (18 of the lane's 20 exchange floats)
template <int POLE, int NC>
__device__ __forceinline__ void cg_put(float *xw, int lane, int j, const float (&gx)[NC][5], const float (&ge)[NC][5],
                                       const float (&u)[NC][5]) {
  if (lane < kGrpLanes && (j == 1 || j == 3)) {
    float *x = xw + lane * 20;
#pragma unroll
    for (int p = 0; p < 2; ++p)
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        x[p * 3 * NC + c] = gx[c][2 * p + 1];
        x[p * 3 * NC + NC + c] = ge[c][2 * p + 1];
        x[p * 3 * NC + 2 * NC + c] = u[c][2 * p + 1];
      }
  }
}

// ------------------------------------------------------------ solid element pass

// The stiffness of a group's elements, a column per lane
// (glob_stiffness_{mono,di,quad}_4 as in stiff_mono / stiff_di / stiff_quad,
// the same products per point).  mv holds the first point's rows on entry
// (with attenuation row 0 alone: the others follow the memory variables,
// whose registers they then take); each point's other rows are loaded one
// point ahead of their use.  u: the displacement column, masked on the axis;
// f: the column's contributions.
template <int POLE, bool PATCH, bool AX, int MODE, bool ANEL>
__device__ __forceinline__ void col_stiffness(const SpecDev &sp, const float (&eta)[5], const float (&seta)[5],
                                              const float *blk, const float *tail, int nl, uint64_t pol,
                                              float (&mv)[SolidGrp<POLE, PATCH>::kRows + 1][8], float *xw, float *sc,
                                              int lane, int e5, int j, float (&u)[SolidGrp<POLE, PATCH>::NC][5],
                                              const float *m0, const CgArgs &cg, const GroupMeta &g, bool mine_cg,
                                              float (&f)[SolidGrp<POLE, PATCH>::NC][5]) {
  using G = SolidGrp<POLE, PATCH>;
  constexpr int NC = G::NC, NT = G::NT, OFF = G::kOff;
  const float *gxi = AX ? sp.g1 : sp.g2;
  // rows [a, b] of the group (row kRows: the tail)
  auto rows = [&](int a, int b) {
#pragma unroll
    for (int r = a; r <= b; ++r) {
      if (r < G::kRows) {
        ldg8(blk + (int64_t)r * 8 * nl, mv[r], pol);
      } else if (G::kTail == 4) {
        const float4 t = __ldg(reinterpret_cast<const float4 *>(tail));
        mv[r][0] = t.x;
        mv[r][1] = t.y;
        mv[r][2] = t.z;
        mv[r][3] = t.w;
      } else if (G::kTail == 2) {
        const float2 t = __ldg(reinterpret_cast<const float2 *>(tail));
        mv[r][0] = t.x;
        mv[r][1] = t.y;
      }
    }
  };
  float X[NC][5], E[NC][5];
  xch_put<NC>(xw, lane, u);
  __syncwarp();
  col_xi<NC, false>(gxi, u, X);
  xch_eta<NC>(xw, e5, eta, E);
  __syncwarp();
  if (ANEL) {
    if (MODE == MODE_NEWMARK) cg_put<POLE, NC>(xw, lane, j, X, E, u);
    __syncwarp();
    cg_point<POLE, MODE == MODE_NEWMARK, MODE == MODE_NEWMARK>(cg, xw, sc, g, lane, mine_cg);
    rows(1, (OFF + NT - 1) / 8);
    __syncwarp();
  }
  float V[NC], W0 = 0.f;
  if (AX) {
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      V[c] = 0.f;
#pragma unroll
      for (int k = 0; k < 5; ++k) V[c] = fmaf(sp.g0[k], u[c][k], V[c]);  // vxm_4(G0, u)
    }
    W0 = POLE == POLE_MONO ? E[NC - 1][0] : E[0][0];  // vxm_4(u(0,:), G2)
  }
  float S2[NC][5];
#pragma unroll
  for (int i = 0; i < 5; ++i) {
    if (i < 4) rows((OFF + (i + 1) * NT - 1) / 8 + 1, (OFF + (i + 2) * NT - 1) / 8);  // the next point's
    auto m = [&](int t) { return mv[(OFF + i * NT + t) / 8][(OFF + i * NT + t) % 8]; };
    if constexpr (POLE == POLE_MONO) {
      const float us = u[0][i], X1 = X[0][i], X2 = X[1][i], X3 = E[0][i], X4 = E[1][i];
      const float m1 = m(S_M1), m2 = m(S_M2), m3 = m(S_M3), m4 = m(S_M4);
      f[0][i] = m4 * X4 + m2 * X3 + m1 * X1 + m3 * X2 + us * m(S_MW1);
      f[1][i] = 0.f;
      const float m11s = m(S_M11S), m12s = m(S_M12S), m22s = m(S_M22S), m32s = m(S_M32S), m42s = m(S_M42S),
                  m11z = m(S_M11Z);
      X[0][i] = m11s * X3 + m(S_M21S) * X1 + m12s * X4 + m22s * X2 + m1 * us;
      S2[0][i] = m11s * X1 + m(S_M41S) * X3 + m32s * X2 + m42s * X4 + m2 * us;
      X[1][i] = m11z * X4 + m(S_M21Z) * X2 + m32s * X3 + m22s * X1 + m3 * us;
      S2[1][i] = m11z * X2 + m(S_M41Z) * X4 + m12s * X1 + m42s * X3 + m4 * us;
    } else if constexpr (POLE == POLE_DI) {
      const float u2 = u[1][i], u3 = u[2][i];
      const float X1 = X[0][i], X2 = X[1][i], X3 = X[2][i], X4 = E[0][i], X5 = E[1][i], X6 = E[2][i];
      const float X7 = X1 + X2, X8 = X4 + X5;
      const float m1 = m(S_M1), m2 = m(S_M2), m3 = m(S_M3), m4 = m(S_M4), m5 = m(S_M5), m6 = m(S_M6), m7 = m(S_M7),
                  m8 = m(S_M8), mw2 = m(S_MW2);
      f[0][i] = 0.f;
      f[1][i] = m8 * X6 + m7 * X3 + m1 * X1 + m5 * X2 + m2 * X4 + m6 * X5 + m(S_MW1) * u2 + mw2 * u3;
      f[2][i] = m4 * X4 - m4 * X5 + m3 * X1 - m3 * X2 + mw2 * u2 + m(S_MW3) * u3;
      const float m11s = m(S_M11S), m21s = m(S_M21S), m41s = m(S_M41S), m12s = m(S_M12S), m22s = m(S_M22S),
                  m42s = m(S_M42S), m13s = m(S_M13S), m23s = m(S_M32S), m33s = m(S_M33S), m43s = m(S_M43S),
                  m11z = m(S_M11Z);
      float c1 = m13s * X6, c2 = m23s * X3, c3 = m3 * u3;
      X[0][i] = c1 + c2 + c3 + m11s * X4 + m21s * X1 + m12s * X5 + m22s * X2 + m1 * u2;
      X[1][i] = c1 + c2 - c3 + m11s * X5 + m21s * X2 + m12s * X4 + m22s * X1 + m5 * u2;
      c1 = m33s * X3;
      c2 = m43s * X6;
      c3 = m4 * u3;
      S2[0][i] = c1 + c2 + c3 + m11s * X1 + m41s * X4 + m12s * X2 + m42s * X5 + m2 * u2;
      S2[1][i] = c1 + c2 - c3 + m11s * X2 + m41s * X5 + m12s * X1 + m42s * X4 + m6 * u2;
      X[2][i] = m33s * X8 + m23s * X7 + m11z * X6 + m(S_M21Z) * X3 + m7 * u2;
      S2[2][i] = m13s * X7 + m43s * X8 + m11z * X3 + m(S_M41Z) * X6 + m8 * u2;
    } else {
      const float us = u[0][i], up = u[1][i], uz = u[2][i];
      const float X1 = X[0][i], X2 = X[1][i], X3 = X[2][i], X4 = E[0][i], X5 = E[1][i], X6 = E[2][i];
      const float m1 = m(S_M1), m2 = m(S_M2), m3 = m(S_M3), m4 = m(S_M4), m5 = m(S_M5), m6 = m(S_M6), m7 = m(S_M7),
                  m8 = m(S_M8), mw2 = m(S_MW2), mw3 = m(S_MW3);
      const float a = m2 * X4 + m1 * X1 + m4 * X6 + m3 * X3, b = m6 * X5 + m5 * X2;
      const float usm = us - 2.f * up, ups = 2.f * us - up;
      f[0][i] = a + 2.f * b + m(S_MW1) * us + mw2 * up + 2.f * mw3 * uz;
      f[1][i] = -2.f * a - b + mw2 * us + m(S_MW4) * up - mw3 * uz;
      f[2][i] = 2.f * (m8 * X5 + m7 * X2) + mw3 * ups + m(S_MW5) * uz;
      const float m11s = m(S_M11S), m12s = m(S_M12S), m22s = m(S_M22S), m32s = m(S_M32S), m42s = m(S_M42S),
                  m11z = m(S_M11Z), m1p = m(S_M1PHI);
      X[0][i] = m11s * X4 + m(S_M21S) * X1 + m12s * X6 + m22s * X3 + m1 * usm;
      S2[0][i] = m11s * X1 + m(S_M41S) * X4 + m32s * X3 + m42s * X6 + m2 * usm;
      X[2][i] = m11z * X6 + m(S_M21Z) * X3 + m32s * X4 + m22s * X1 + m3 * usm;
      S2[2][i] = m11z * X3 + m(S_M41Z) * X6 + m12s * X1 + m42s * X4 + m4 * usm;
      X[1][i] = m1p * X5 + m(S_M2PHI) * X2 + m5 * ups + 2.f * m7 * uz;
      S2[1][i] = m1p * X2 + m(S_M4PHI) * X5 + m6 * ups + 2.f * m8 * uz;
    }
    if (ANEL && (i == 1 || i == 3)) {
      // minus the anelastic terms at the cg points (cg lane 4 e + 2 (i >> 1) + (j >> 1))
      if (j == 1 || j == 3) {
        const float *s = sc + 9 * (4 * (e5 / 5) + 2 * (i >> 1) + (j >> 1));
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          X[c][i] = X[c][i] - s[c];
          S2[c][i] = S2[c][i] - s[3 + c];
          f[c][i] = f[c][i] - s[6 + c];
        }
      }
    }
  }
  // second stage: f and mxm(G, S1) and mxm(S2, G2T), S1 in X.  All ten terms in a
  // chain on top of f round at f's magnitude; the second sum at least is formed
  // apart.  Stiffness errors against FP64, 1e-8, quadrupole, random metric terms /
  // PREM mesh: chain 8.58 / 7.43, both sums apart as the reference adds them 8.23 /
  // 6.90, the second one apart 8.16 / 6.61.  The last is the faster one for a
  // scattered quadrupole's or monopole's pass (200 compensated steps of 18 944
  // elements: 3.97, 4.05 and 3.83 ms); patched, attenuated and dipole passes are as
  // fast or faster with both apart (32 steps of 786 432 elements 21.7 ms, 72 of
  // 99 450 attenuated 9.4, where the last takes 9.8).  A stiffness call of 2^20
  // quadrupoles took 0.629 ms with the chain and takes 0.641.
  xch_put<NC>(xw, lane, S2);
  __syncwarp();
  float Y[NC][5];
  auto local = [](int c) { return POLE == POLE_DI ? c != 0 : POLE == POLE_QUAD || c == 0; };  // f[c] has a local part
  if (PATCH || ANEL || POLE == POLE_DI) {
    col_xi<NC, true>(gxi, X, Y);
    xch_eta<NC>(xw, e5, seta, E);
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
      for (int i = 0; i < 5; ++i) {
        if (!local(c)) f[c][i] = Y[c][i] + E[c][i];
        else if (POLE == POLE_DI) f[c][i] = Y[c][i] + E[c][i] + f[c][i];
        else f[c][i] = f[c][i] + Y[c][i] + E[c][i];
      }
  } else {
    col_xi_add<NC>(gxi, X, f);
    xch_eta<NC>(xw, e5, seta, E);
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
      for (int i = 0; i < 5; ++i) f[c][i] = f[c][i] + E[c][i];
  }
  __syncwarp();
  if (AX) {
    auto w = [&](int q) { return m0[5 * q + j]; };
    auto outer = [&](int c, float v) {
#pragma unroll
      for (int i = 0; i < 5; ++i) f[c][i] = fmaf(sp.g0[i], v, f[c][i]);
    };
    auto along = [&](float v) {  // vxm_4(v, G2T) over the element's columns
      float s = 0.f;
#pragma unroll
      for (int k = 0; k < 5; ++k) s = fmaf(__shfl_sync(kFull, v, e5 + k), seta[k], s);
      return s;
    };
    if constexpr (POLE == POLE_MONO) {
      const float w1 = w(0), w2 = w(1), w3 = w(2);
      outer(0, w1 * V[0] + w3 * W0 + w2 * V[1]);
      outer(1, w2 * V[0]);
      f[1][0] = f[1][0] + along(w3 * V[0]);
    } else if constexpr (POLE == POLE_DI) {
      // M0_w slots: 0:w1 1:w2 2:w3 3:w4 4:w6 5:w7 6:w8 7:w9 8:w10
      const float w26 = w(1) + w(4), w48 = w(3) + w(6), w10 = w(8);
      outer(0, w(0) * V[1] + w(2) * V[2]);
      outer(1, w(0) * V[0] + w26 * W0 + w(7) * V[1] + w10 * V[2]);
      outer(2, w(2) * V[0] + w48 * W0 + w(5) * V[2] + w10 * V[1]);
      f[0][0] = f[0][0] + along(w26 * V[1] + w48 * V[2]);
    } else {
      const float w1 = w(0), w2 = w(1), w3 = w(2), w4 = w(3), w5 = w(4), w6 = w(5);
      outer(0, w1 * V[0] + w2 * V[1] + w3 * V[2]);
      outer(1, w2 * V[0] + w4 * V[1] + w5 * V[2]);
      outer(2, w3 * V[0] + w5 * V[1] + w6 * V[2]);
    }
  }
}

// The gather point's displacement component: a Newmark step's stored
// prediction, a symplectic stage's drift, the stiffness operation's u
template <int MODE, bool KAHAN>
__device__ __forceinline__ float gather_u(const StateArgs &st, int c, int32_t g) {
  if (MODE == MODE_NEWMARK) return st.up[c][g];
  if (MODE == MODE_SYMPLECTIC) {
    if (KAHAN) {
      float k = st.cu[c][g];
      return drift_comp(st.u[c][g], st.v[c][g], st, k);
    }
    return st.u[c][g] + mul2(st.dt, st.dt_lo, st.v[c][g]);
  }
  return st.u[c][g];
}

// Element pass of one group of solid elements by one warp.  PATCH: int_start,
// n_int and the deferred list s_def turn local point indices into global ones,
// and out(f, idx, mine) accumulates the columns of the lanes with `mine`;
// otherwise idx are global and out stores the columns.
// What the step before does not write (the group's rows) is loaded before
// `wait`, which waits for that step's kernels and returns whether the solve
// has stopped: nothing of the state is written then.  gone: that it had, as read
// before the wait.
template <int POLE, bool PATCH, int MODE, bool ANEL, bool KAHAN, class Wait, class Out>
__device__ __forceinline__ void solid_group(const StreamWork &w, const SpecDev &sp, const GroupMeta &g, float *xw,
                                            float *sc, int32_t int_start, int n_int, const int32_t *s_def, bool gone,
                                            Wait wait, Out out) {
  using G = SolidGrp<POLE, PATCH>;
  constexpr int NC = G::NC;
  const StreamDomain &d = w.ds;
  const StateArgs &st = w.solid;
  const int lane = threadIdx.x & 31;
  const int nl = 5 * g.n;
  const int ll = lane < nl ? lane : nl - 1;  // idle lanes follow the last column
  const int e = ll / 5, j = ll % 5, e5 = 5 * e;
  auto gc = [](int c) { return (POLE == POLE_MONO && c == 1) ? 2 : c; };
  const int64_t slot = (int64_t)g.slot0 + e;
  const float *blk = d.blocks + (int64_t)g.slot0 * (5 * 8 * G::kRows) + ll * 8;
  const float *tail = G::kTail ? d.tails + ((int64_t)g.slot0 * 5 + ll) * G::kTail : nullptr;
  // metric terms are read once per step: with a mesh beyond L2 they leave it first
  const uint64_t pol = w.prefetch > 0 ? policy_evict_first() : policy_evict_normal();
  float mv[G::kRows + 1][8];
  ldg8(blk, mv[0], pol);
  float eta[5], seta[5];
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    eta[k] = sp.g2[k + 5 * j];   // G2(k, j)
    seta[k] = sp.g2[j + 5 * k];  // G2(j, k)
  }
  const uint32_t w0 = __float_as_uint(mv[0][0]), w1 = __float_as_uint(mv[0][1]);
  const bool ax = (w0 & kGrpAxial) != 0;
  int32_t idx[5];  // PATCH: local, else global
  if (PATCH) {
    idx[0] = w0 & 0x7FF;
    idx[1] = (w0 >> 11) & 0x7FF;
    idx[2] = w1 & 0x7FF;
    idx[3] = (w1 >> 11) & 0x7FF;
    idx[4] = ((w0 >> 22) & 0x3F) | ((w1 >> 22) << 6);
  } else {
#pragma unroll
    for (int i = 0; i < 5; ++i) idx[i] = (int32_t)(__float_as_uint(mv[0][i]) & kGrpIdx);
  }
  const unsigned axm = __ballot_sync(kFull, ax);
  if (!PATCH && __any_sync(kFull, gone)) return;
  const int cge = (lane < 4 * g.n ? lane : 0) >> 2;  // the cg lane's element
#pragma unroll 1
  for (int pass = 0; pass < 2; ++pass) {
    // elements off the axis, then (if any) the axial ones; both by the whole warp
    if (pass == 0 ? axm == kFull : axm == 0u) continue;
    if (!ANEL)
#pragma unroll
      for (int r = 1; r <= (G::kOff + G::NT - 1) / 8; ++r) ldg8(blk + (int64_t)r * 8 * nl, mv[r], pol);
    constexpr bool staged = ANEL && MODE == MODE_NEWMARK;
    if (staged) cg_stage_consts(w.cg, sc, g, lane);
    const bool stopped = wait();
    if (staged) cg_stage_state(w.cg, sc, g, lane);
    float u[NC][5], f[NC][5];
#pragma unroll
    for (int i = 0; i < 5; ++i) {
      int32_t p = idx[i];
      if (PATCH) p = p < n_int ? int_start + p : AXG_BOUND(p - n_int, kMaxDef, 62) ? s_def[p - n_int] : 0;
      if (!AXG_BOUND(p, st.nglob, 62)) p = 0;
#pragma unroll
      for (int c = 0; c < NC; ++c) u[c][i] = gather_u<MODE, KAHAN>(st, gc(c), p);
    }
    if (MODE != MODE_FORCE && j == 1) {
      // runtime_info guard on disp(1,1,:,:) (SOLVER/time_evol_wave.F90:1042)
      const float mx = fmaxf(fabsf(u[0][1]), fmaxf(NC == 3 ? fabsf(u[1][1]) : 0.f, fabsf(u[NC - 1][1])));
      if (!(mx <= st.thresh)) atomicCAS(st.blowup, 0, *st.iter);
    }
    const bool mine_cg = !stopped && ((axm >> (5 * cge)) & 1u) == (unsigned)pass;
    if (pass == 0) {
      col_stiffness<POLE, PATCH, false, MODE, ANEL>(sp, eta, seta, blk, tail, nl, pol, mv, xw, sc, lane, e5, j, u,
                                                    nullptr, w.cg, g, mine_cg, f);
    } else {
      int axslot = (__ldg(d.elinfo + slot) & 0xFFFFFF) - 1;
      if (axslot < 0 || !AXG_BOUND((int64_t)(axslot + 1) * G::NA * 5 - 1, d.n_m0, 62)) axslot = 0;
#pragma unroll
      for (int c = 0; c < NC; ++c)
        if (col_masked<POLE>(c)) u[c][0] = 0.f;  // apply_axis_mask_{one,two,three}comp on disp
      col_stiffness<POLE, PATCH, true, MODE, ANEL>(sp, eta, seta, blk, tail, nl, pol, mv, xw, sc, lane, e5, j, u,
                                                   d.m0 + (int64_t)axslot * (G::NA * 5), w.cg, g, mine_cg, f);
    }
    if (MODE == MODE_NEWMARK && !ANEL && d.aux) {
      // attenuation at every GLL point: minus the anelastic stiffness
      // (glob_anel_stiffness_*_4), formed by anel_full_kernel
      const float *x = d.aux + slot * 75 + 5 * j;
#pragma unroll
      for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int i = 0; i < 5; ++i) f[c][i] = f[c][i] + x[25 * gc(c) + i];
    }
    if (pass == 1) {
#pragma unroll
      for (int c = 0; c < NC; ++c)
        if (col_masked<POLE>(c)) f[c][0] = 0.f;  // axis mask of acc1
    }
    out(f, idx, lane < nl && ax == (pass == 1), e, j);
  }
}

// Scattered element pass: the group's columns to its place in fel.
template <int POLE, int MODE, bool ANEL, bool KAHAN>
__device__ __forceinline__ void scatter_group(const StreamWork &w, const SpecDev &sp, int32_t grp, float *xw, float *sc) {
  constexpr int NC = SolidGrp<POLE, false>::NC, FS = solid_fs(POLE);
  const StreamDomain &d = w.ds;
  const GroupMeta g = scatter_meta(grp, d.n_off, d.nel);
  const bool gone = MODE != MODE_FORCE && stopped_before(w.solid.stop);
  auto prefetch = [&]() {
    if (w.prefetch <= 0 || (threadIdx.x & 31) != 0) return;
    // the blocks of the group that runs about one round of resident warps later
    const int64_t h = (int64_t)grp + w.prefetch * kGrpWarps;
    if (h < scatter_groups(d.n_off, d.nel)) {
      constexpr int row = 5 * 8 * SolidGrp<POLE, false>::kRows;
      const GroupMeta m = scatter_meta((int32_t)h, d.n_off, d.nel);
      const int64_t s = m.slot0;
      prefetch_l2(d.blocks + s * row, m.n * row * 4);
      if (ANEL) {
        prefetch_l2(w.cg.consts + s * 48, m.n * 48 * 4);
        prefetch_l2(w.cg.state + s * 4 * cg_state_floats(w.cg.nsls), m.n * 16 * cg_state_floats(w.cg.nsls));
      }
    }
  };
  if (ANEL) prefetch();  // (others: once the group's first rows are here, 4.04 against 4.11 ms for 200 steps of 18 944 elements)
  solid_group<POLE, false, MODE, ANEL, KAHAN>(
      w, sp, g, xw, sc, 0, 0, nullptr, gone,
      [&]() {
        if (!ANEL) prefetch();
        pdl_wait();
        return MODE != MODE_FORCE && *w.solid.stop != 0;
      },
      [&](const float (&f)[NC][5], const int32_t (&)[5], bool mine, int e, int j) {
        const int64_t o = (((int64_t)g.slot0 + e) * 5 + j) * FS;
        if (!mine || !AXG_BOUND(o + FS - 1, d.n_fel, 62)) return;
        float v[16];
#pragma unroll
        for (int q = 0; q < 16; ++q) v[q] = q < 5 * NC ? f[q < 5 * NC ? q / 5 : 0][q % 5] : 0.f;
        if (NC == 3) {
          stg8(d.fel + o, reinterpret_cast<const float(&)[8]>(v[0]));
          stg8(d.fel + o + 8, reinterpret_cast<const float(&)[8]>(v[8]));
        } else {
          float4 *p = reinterpret_cast<float4 *>(d.fel + o);
#pragma unroll
          for (int q = 0; q < 3; ++q) p[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
        }
      });
}

// ------------------------------------------------------------ fluid element pass

// The fluid's groups: rows of four floats per lane (a fluid column is too
// short for rows of eight): five point indices, then the points' 3 or 4 terms
__host__ __device__ constexpr int fgrp_rows(int nt) { return (5 + 5 * nt + 3) / 4; }
// chi at the step's gather point: a Newmark step's stored prediction, or a
// symplectic stage's drift (compensated or not)
template <int MODE, bool KAHAN>
__device__ __forceinline__ float stream_chi(const StateArgs &st, int64_t g, float &k) {
  if (MODE == MODE_NEWMARK) return st.up[0][g];
  if (KAHAN) {
    k = st.cu[0][g];
    return drift_comp(st.u[0][g], st.v[0][g], st, k);
  }
  return st.u[0][g] + mul2(st.dt, st.dt_lo, st.v[0][g]);
}

// glob_fluid_stiffness_4 (SOLVER/stiffness_fluid.f90:139-216) of a group, with
// the source, axis mask and free-surface mask
template <bool NONMONO, int MODE, bool KAHAN>
__device__ __forceinline__ void fluid_group(const StreamWork &w, const SpecDev &sp, int32_t grp, float *xw) {
  constexpr int NT = NONMONO ? 4 : 3, NR = fgrp_rows(NT);
  const StreamDomain &d = w.df;
  const StateArgs &st = w.fluid;
  const int lane = threadIdx.x & 31;
  const int64_t left = d.nel - (int64_t)grp * kGrp;
  const int nl = 5 * (int)(left < kGrp ? left : kGrp);
  const int ll = lane < nl ? lane : nl - 1;
  const int e = ll / 5, j = ll % 5, e5 = 5 * e;
  const int64_t slot = (int64_t)grp * kGrp + e;
  const float4 *blk = reinterpret_cast<const float4 *>(d.blocks) + (int64_t)grp * kGrp * 5 * NR + ll;
  float mv[NR * 4];
#pragma unroll
  for (int r = 0; r < NR; ++r) {
    const float4 t = __ldg(blk + r * nl);
    mv[4 * r] = t.x;
    mv[4 * r + 1] = t.y;
    mv[4 * r + 2] = t.z;
    mv[4 * r + 3] = t.w;
  }
  float eta[5], seta[5];
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    eta[k] = sp.g2[k + 5 * j];
    seta[k] = sp.g2[j + 5 * k];
  }
  const bool ax = (__float_as_uint(mv[0]) & kGrpAxial) != 0;
  const unsigned axm = __ballot_sync(kFull, ax);
  pdl_wait();  // (what comes before is the mesh's)
  const bool stopped = *st.stop != 0;
  float chi[1][5];
#pragma unroll
  for (int i = 0; i < 5; ++i) {
    int64_t g = __float_as_uint(mv[i]) & kGrpIdx;
    if (!AXG_BOUND(g, st.nglob, 63)) g = 0;
    float k = 0.f;
    chi[0][i] = stream_chi<MODE, KAHAN>(st, g, k);
  }
  if (__any_sync(kFull, stopped)) return;
  if (NONMONO && ax) chi[0][0] = 0.f;  // apply_axis_mask_scal
  float X[1][5], E[1][5], f[1][5];
  xch_put<1>(xw, lane, chi);
  __syncwarp();
  xch_eta<1>(xw, e5, eta, E);
  col_xi<1, false>(sp.g2, chi, X);
  if (axm) {
    float Y[1][5];
    col_xi<1, false>(sp.g1, chi, Y);
#pragma unroll
    for (int i = 0; i < 5; ++i)
      if (ax) X[0][i] = Y[0][i];
  }
  __syncwarp();
  float S2[1][5];
#pragma unroll
  for (int i = 0; i < 5; ++i) {
    const float *m = mv + 5 + i * NT;
    const float x1 = X[0][i], x2 = E[0][i];
    X[0][i] = m[0] * x2 + m[1] * x1;
    S2[0][i] = m[0] * x1 + m[2] * x2;
  }
  xch_put<1>(xw, lane, S2);
  __syncwarp();
  col_xi<1, true>(sp.g2, X, f);
  if (axm) {
    float Y[1][5];
    col_xi<1, true>(sp.g1, X, Y);
#pragma unroll
    for (int i = 0; i < 5; ++i)
      if (ax) f[0][i] = Y[0][i];
  }
  xch_eta<1>(xw, e5, seta, E);
#pragma unroll
  for (int i = 0; i < 5; ++i) {
    f[0][i] = f[0][i] + E[0][i];
    if (NONMONO) f[0][i] = fmaf(mv[5 + i * NT + NT - 1], chi[0][i], f[0][i]);
  }
  if (ax || d.srcfl) {
    const int32_t info = __ldg(d.elinfo + slot);
    int axslot = (info & 0xFFFFFF) - 1;
    if (axslot >= 0 && !AXG_BOUND((int64_t)axslot * 5 + 4, d.n_m0, 63)) axslot = -1;
    if (NONMONO && ax && axslot >= 0) {
      float v = 0.f;
#pragma unroll
      for (int k = 0; k < 5; ++k) v = fmaf(sp.g0[k], chi[0][k], v);
      v = d.m0[(int64_t)axslot * 5 + j] * v;
#pragma unroll
      for (int i = 0; i < 5; ++i) f[0][i] = fmaf(sp.g0[i], v, f[0][i]);
    }
    const int srcslot = ((info >> 24) & 0xF) - 1;
    if (srcslot >= 0 && d.srcfl) {
      const float stf1 = AXG_BOUND(*st.iter - 1, st.niter, 63) ? st.stf[*st.iter - 1] : 0.f;
      if (stf1 != 0.f)
#pragma unroll
        for (int i = 0; i < 5; ++i) f[0][i] = f[0][i] - d.srcfl[srcslot * 25 + 5 * j + i] * stf1;
    }
  }
  if (NONMONO && ax) f[0][0] = 0.f;
  if (d.aux)
#pragma unroll
    for (int i = 0; i < 5; ++i) f[0][i] = f[0][i] * __ldg(d.aux + slot * 25 + 5 * j + i);
  const int64_t o = (slot * 5 + j) * kFluidFs;
  if (lane < nl && AXG_BOUND(o + kFluidFs - 1, d.n_fel, 63)) {
    const float v[8] = {f[0][0], f[0][1], f[0][2], f[0][3], f[0][4], 0.f, 0.f, 0.f};
    stg8(d.fel + o, v);
  }
}

// one row of the coupling into the fluid (bdry_copy2fluid,
// SOLVER/time_evol_wave.F90:1532-1571): the fluid force starts with
// -(b1 u_s [+ u_phi] + b2 u_z) of the predicted solid displacement
template <int POLE, int MODE, bool KAHAN>
__device__ __forceinline__ void couple_row(const StreamWork &w, int q) {
  const Coupling &cp = w.to_fluid;
  const StateArgs &solid = w.solid;
  pdl_wait();
  float acc = 0.f;
  for (int k = cp.start[q]; k < cp.start[q + 1]; ++k) {
    if (!AXG_BOUND(k, cp.n_contrib, 64)) break;
    const int gs = cp.src_gidx[k];
    if (!AXG_BOUND(gs, cp.nglob_send, 64)) continue;
    auto pred = [&](int c) {
      if (MODE == MODE_SYMPLECTIC) {
        if (KAHAN) {
          float kk = solid.cu[c][gs];
          return drift_comp(solid.u[c][gs], solid.v[c][gs], solid, kk);
        }
        return predict(solid.u[c][gs], solid.v[c][gs], solid.a[c][gs], solid);
      }
      // the stored prediction has the axis-masked components zeroed; the
      // reference couples before its axis mask, with the prediction of the
      // displacement as it is (zero there, unless a caller set it)
      if (w.axmask && ((w.axmask[gs] >> c) & 1u)) {
        if (KAHAN) {
          float kk = solid.cu[c][gs];
          return predict_comp(solid.u[c][gs], solid.v[c][gs], solid.a[c][gs], solid, kk);
        }
        return predict(solid.u[c][gs], solid.v[c][gs], solid.a[c][gs], solid);
      }
      return solid.up[c][gs];
    };
    const float us = pred(0);
    const float uz = pred(2);
    const float x = POLE == POLE_DI ? us + pred(1) : us;
    acc = acc + cp.mask[k] * (-cp.b1[k] * x - cp.b2[k] * uz);
  }
  if (AXG_BOUND(cp.pt_gidx[q], cp.nglob_recv, 64)) w.ffl[cp.pt_gidx[q]] = acc;
}

// ------------------------------------------------------------ point pass

// The copies [k, s1) of a point, NC components FSTEP floats apart: the first
// four copies' indices (which no step writes) are loaded by the constructor,
// their contributions together by sum().
template <int NC, int FSTEP>
struct Copies {
  int32_t e[4];
  uint32_t k, s1;
  __device__ __forceinline__ Copies(const StreamDomain &d, uint32_t k0, uint32_t end) : k(k0), s1(end) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      e[q] = k + q < s1 && AXG_BOUND(k + q, d.n_ent, 65) ? __ldg(d.ent + k + q) : -1;
      if (e[q] >= 0 && !AXG_BOUND(e[q] + FSTEP * (NC - 1), d.n_fel, 65)) e[q] = -1;
    }
  }
  __device__ __forceinline__ void sum(const StreamDomain &d, float (&s)[NC]) const {
    float x[4][NC];
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int c = 0; c < NC; ++c) x[q][c] = e[q] >= 0 ? d.fel[e[q] + FSTEP * c] : 0.f;
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (e[q] >= 0)
#pragma unroll
        for (int c = 0; c < NC; ++c) s[c] = s[c] + x[q][c];
    for (uint32_t q = k + 4; q < s1; ++q) {
      if (!AXG_BOUND(q, d.n_ent, 65)) break;
      const int32_t f = __ldg(d.ent + q);
      if (!AXG_BOUND(f + FSTEP * (NC - 1), d.n_fel, 65)) break;
#pragma unroll
      for (int c = 0; c < NC; ++c) s[c] = s[c] + d.fel[f + FSTEP * c];
    }
  }
};

// -inv_mass_fluid * force at fluid point g, without absorbing terms; the
// force is the coupling partial sum, then the copies
struct FluidForce {
  uint32_t s0;
  Copies<1, 1> cp;
  __device__ __forceinline__ FluidForce(const StreamDomain &d, int64_t g)
      : s0((uint32_t)d.start[g]), cp(d, s0 & kStMask, (uint32_t)d.start[g + 1] & kStMask) {}
  template <bool KAHAN>
  __device__ __forceinline__ float accel(const StreamWork &w, int64_t g) const {
    float sum[1] = {(s0 & kStCoupled) ? w.ffl[g] : 0.f};
    cp.sum(w.df, sum);
    if (KAHAN && w.fluid.inv_mass_pair) return -mul_pair(w.fluid.inv_mass_pair[g], sum[0]);
    if (KAHAN && w.fluid.inv_mass_dp) return (float)(-w.fluid.inv_mass_dp[g] * (double)sum[0]);  // FP64, one rounding
    return -w.fluid.inv_mass[g] * sum[0];
  }
};

// One fluid point: ddchi = -inv_mass_fluid * force [- absorbing terms], dchi by
// the Newmark corrector or a symplectic kick, chi (zero on the axis for the
// non-monopole sources); a Newmark step stores the next prediction (the compensated one with the compensation it
// leaves, cup).
template <bool NONMONO, int MODE, bool KAHAN>
__device__ __forceinline__ void fluid_point(const StreamWork &w, int64_t g) {
  const StateArgs &st = w.fluid;
  const FluidForce ff(w.df, g);
  pdl_wait();
  if (w.ctl[CTL_STOP_P]) return;
  float a = ff.template accel<KAHAN>(w, g);
  float kc = 0.f;
  const float chi = stream_chi<MODE, KAHAN>(st, g, kc);
  if (KAHAN && MODE == MODE_NEWMARK) kc = st.cup[0][g];
  const float vel = st.v[0][g];
  if (st.gamma) {
    const float gam = st.gamma[g];
    a = a - 2.f * gam * vel - gam * gam * chi;
  }
  const float inc = MODE == MODE_SYMPLECTIC ? mul2(st.kick, st.kick_lo, a) : mul2(st.hdt, st.hdt_lo, st.a[0][g] + a);
  float vn;
  if (KAHAN) {
    float k = st.cv[0][g];
    vn = kahan_add(vel, inc, k);
    st.cv[0][g] = k;
  } else {
    vn = vel + inc;
  }
  st.v[0][g] = vn;
  st.a[0][g] = a;
  // apply_axis_mask_scal zeroes chi on the axis (non-monopole)
  const bool zero = NONMONO && (ff.s0 & kStAxis);
  const float un = zero ? 0.f : chi;
  if (MODE == MODE_SYMPLECTIC) {
    st.u[0][g] = un;
    if (KAHAN) st.cu[0][g] = zero ? 0.f : kc;
  } else if (KAHAN) {
    float k = zero ? 0.f : comp_after_step(kc, vn, a, st);
    st.cu[0][g] = k;
    const float p = predict_comp(un, vn, a, st, k);
    st.u[0][g] = zero ? 0.f : p;
    st.cup[0][g] = zero ? 0.f : k;
  } else {
    st.u[0][g] = zero ? 0.f : predict(un, vn, a, st);
  }
}

// One solid point: its state, loaded ahead of the force's sum, and the
// source and corrector (SOLVER/time_evol_wave.F90:466-494; a symplectic
// stage's kick, :688-717).
template <int POLE, int MODE, bool KAHAN>
struct SolidPoint {
  static constexpr int NC = POLE == POLE_MONO ? 2 : 3;
  static __device__ __forceinline__ int gc(int c) { return (POLE == POLE_MONO && c == 1) ? 2 : c; }
  float dsp[NC], vel[NC], acc[NC], kc[KAHAN ? NC : 1], kv[KAHAN ? NC : 1], gam;
  float2 im;  // (y: the low part of an FP64 inverse mass, else 0)

  __device__ __forceinline__ void load(const StateArgs &st, int64_t g) {
    if (KAHAN && st.inv_mass_pair) im = st.inv_mass_pair[g];
    else im = make_float2(st.inv_mass[g], 0.f);
    gam = st.gamma ? st.gamma[g] : 0.f;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      vel[c] = st.v[gc(c)][g];
      if (MODE == MODE_NEWMARK) {
        dsp[c] = st.up[gc(c)][g];
        acc[c] = st.a[gc(c)][g];
        if (KAHAN) kc[KAHAN ? c : 0] = st.cup[gc(c)][g];
      } else {
        dsp[c] = st.u[gc(c)][g];
        if (KAHAN) kc[KAHAN ? c : 0] = st.cu[gc(c)][g];
      }
      if (KAHAN) kv[KAHAN ? c : 0] = st.cv[gc(c)][g];
    }
  }

  // the source term of point g, if it has one, in step `iter` (the element
  // pass reads the step counter, the point pass the copy the element pass
  // makes of it: each pass writes the other's)
  static __device__ __forceinline__ void source(const StateArgs &st, int32_t iter, int64_t g, float (&sum)[NC]) {
    const float stf1 = AXG_BOUND(iter - 1, st.niter, 66) ? st.stf[iter - 1] : 0.f;
    if (stf1 == 0.f) return;
    for (int q = 0; q < st.src.n; ++q)
      if (st.src.gidx[q] == (int32_t)g) {
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          if (KAHAN && st.src.val_dp)  // the source projection in FP64, one rounding
            sum[c] = (float)((double)sum[c] - st.src.val_dp[3 * q + gc(c)] * (double)stf1);
          else
            sum[c] = sum[c] - st.src.val[3 * q + gc(c)] * stf1;
        }
      }
  }

  // the corrector of point g with the summed force
  __device__ __forceinline__ void finish(const StateArgs &st, int64_t g, bool axis, const float (&sum)[NC]) {
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const int cg = gc(c), q = KAHAN ? c : 0;
      const bool two = POLE == POLE_DI && cg == 2;  // the dipole's z component takes twice the acceleration
      if (MODE == MODE_SYMPLECTIC) {
        if (KAHAN) dsp[c] = drift_comp(dsp[c], vel[c], st, kc[q]);
        else dsp[c] = dsp[c] + mul2(st.dt, st.dt_lo, vel[c]);
      }
      // (a symplectic kick doubles the dipole's z component's increment, below)
      const float f = two && MODE != MODE_SYMPLECTIC ? 2.f * sum[c] : sum[c];
      float a;
      if (KAHAN && st.inv_mass_pair) a = -mul_pair(im, f);
      else if (KAHAN && st.inv_mass_dp) a = (float)(-st.inv_mass_dp[g] * (double)f);  // FP64, one rounding
      else a = -im.x * f;
      if (st.gamma) a = a - 2.f * gam * vel[c] - gam * gam * dsp[c];
      const float inc = MODE == MODE_SYMPLECTIC
                            ? mul2(two ? 2.f * st.kick : st.kick, two ? 2.f * st.kick_lo : st.kick_lo, a)
                            : mul2(st.hdt, st.hdt_lo, acc[c] + a);
      float vn;
      if (KAHAN) {
        vn = kahan_add(vel[c], inc, kv[q]);
        st.cv[cg][g] = kv[q];
      } else {
        vn = vel[c] + inc;
      }
      st.v[cg][g] = vn;
      st.a[cg][g] = a;
      // the axis masks of the reference zero these components of its state
      const bool zero = axis && axis_masked<POLE>(cg);
      const float un = zero ? 0.f : dsp[c];
      if (MODE == MODE_SYMPLECTIC) {
        st.u[cg][g] = un;
        if (KAHAN) st.cu[cg][g] = zero ? 0.f : kc[q];
      } else if (KAHAN) {
        // The new displacement is the gathered prediction, which stays in the
        // buffer it came from (up); st.u is the other buffer and receives the
        // next step's prediction, cup the compensation it leaves.
        float kk = zero ? 0.f : comp_after_step(kc[q], vn, a, st);
        st.cu[cg][g] = kk;
        const float p = predict_comp(un, vn, a, st, kk);
        st.u[cg][g] = zero ? 0.f : p;
        st.cup[cg][g] = zero ? 0.f : kk;
      } else {
        st.u[cg][g] = zero ? 0.f : predict(un, vn, a, st);
      }
    }
  }
};

// An inner GLL point of an element of a scattered solid (nine per element, 9/16
// of the points): one copy, whose place follows from the point's number
// 9 slot + 3 (j - 1) + i - 1, so no index is read: steps of 305 000 points took
// 25.1 us with all points through the lists below and take 24.9 (quadrupole,
// compensated), 24.0 / 21.6 (dipole); with cg4 on 99 450 elements 137.4 /
// 132.1.  (Finished by the element pass itself they cost more: its chain is the
// longer one.)
template <int POLE, int MODE, bool KAHAN>
__device__ __forceinline__ void inner_point(const StreamWork &w, int32_t g) {
  using S = SolidPoint<POLE, MODE, KAHAN>;
  constexpr int NC = S::NC;
  const StreamDomain &d = w.ds;
  const StateArgs &st = w.solid;
  const int32_t slot = g / 9, q = g - 9 * slot;
  const int64_t e = ((int64_t)slot * 5 + q / 3 + 1) * solid_fs(POLE) + q % 3 + 1;
  pdl_wait();
  const bool stopped = MODE != MODE_FORCE && w.ctl[CTL_STOP_P] != 0;
  S pt;
  if (MODE != MODE_FORCE) pt.load(st, g);
  if (!AXG_BOUND(e + 5 * (NC - 1), d.n_fel, 70)) return;
  float sum[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) sum[c] = 0.f + d.fel[e + 5 * c];
  if (MODE == MODE_FORCE) {
#pragma unroll
    for (int c = 0; c < NC; ++c) st.f[S::gc(c)][g] = sum[c];
    return;
  }
  if (stopped) return;
  for (int k = 0; k < d.n_src_patch; ++k)
    if (d.src_patch[k] == slot) S::source(st, w.ctl[CTL_ITER_P], g, sum);
  pt.finish(st, g, false, sum);
}

// A solid point of the point pass: the coupling, then the copies' (the
// patches') sums in order.
template <int POLE, int MODE, bool PATCH, bool KAHAN>
__device__ __forceinline__ void solid_point(const StreamWork &w, int64_t g) {
  using S = SolidPoint<POLE, MODE, KAHAN>;
  constexpr int NC = S::NC;
  const StreamDomain &d = w.ds;
  const StateArgs &st = w.solid;
  const int64_t r = g - w.p0;
  const uint32_t s0 = (uint32_t)d.start[r], s1 = (uint32_t)d.start[r + 1] & kStMask;
  const bool coupled = (s0 & kStCoupled) != 0;
  const Copies<NC, PATCH ? 1 : 5> cps(d, (s0 & kStMask) + (coupled ? 1 : 0), s1);
  pdl_wait();  // (what comes before no step writes)
  const bool stopped = MODE != MODE_FORCE && w.ctl[CTL_STOP_P] != 0;
  S pt;
  if (MODE != MODE_FORCE) pt.load(st, g);
  float sum[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) sum[c] = 0.f;
  if (coupled) {
    const int32_t q = AXG_BOUND(s0 & kStMask, d.n_ent, 66) ? __ldg(d.ent + (s0 & kStMask)) : 0;
    if (MODE != MODE_FORCE && AXG_BOUND(q, w.to_solid.n, 66)) {
      // bdry_copy2solid (SOLVER/time_evol_wave.F90:1577-1611): b1 ddchi (s [and
      // phi]) and b2 ddchi (z) of the new fluid acceleration, formed here from
      // the fluid's contributions (with absorbing terms, stored by the launch before)
      const Coupling &cp = w.to_solid;
      for (int x = cp.start[q]; x < cp.start[q + 1]; ++x) {
        if (!AXG_BOUND(x, cp.n_contrib, 66) || !AXG_BOUND(cp.src_gidx[x], cp.nglob_send, 66)) break;
        const int gf = cp.src_gidx[x];
        const float a = w.fluid.gamma ? w.fluid.a[0][gf] : FluidForce(w.df, gf).template accel<KAHAN>(w, gf);
        const bool masked = cp.mask[x] == 0.f;  // solid copy sits at ipol=0 of an axial element
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          const float b = S::gc(c) == 2 ? cp.b2[x] : (c == 0 || POLE == POLE_DI) ? cp.b1[x] : 0.f;
          sum[c] = sum[c] + (masked && axis_masked<POLE>(S::gc(c)) ? 0.f : b * a);
        }
      }
    }
  }
  cps.sum(d, sum);
  if (MODE == MODE_FORCE) {
#pragma unroll
    for (int c = 0; c < NC; ++c) st.f[S::gc(c)][g] = sum[c];
    return;
  }
  if (stopped) return;  // a stopped solve does nothing more
  if (s0 & kStSource) S::source(st, w.ctl[CTL_ITER_P], g, sum);
  pt.finish(st, g, (s0 & kStAxis) != 0, sum);
}

// ------------------------------------------------------------ patched element pass

constexpr uint64_t kTurnNs = 1000000000ull;  // a warp's wait for its turn gives up after 1 s

// Waits (bounded) until `need` groups of the patch have accumulated.
__device__ __forceinline__ void wait_turn(const volatile int32_t *done, int need, int lane, int32_t *err) {
  if (lane == 0 && *done < need) {
    const uint64_t t0 = globaltimer_ns();
    for (int k = 0; *done < need; ++k)
      if ((k & 63) == 63 && globaltimer_ns() - t0 > kTurnNs) {
        if (err) atomicCAS(err, 0, 5 /* AXG_ERR_TIMEOUT */);
        break;
      }
  }
  __threadfence_block();
  __syncwarp();
}

// shared memory of a patched CTA
template <int POLE>
struct PatchSmem {
  static constexpr int NC = POLE == POLE_MONO ? 2 : 3;
  float f[NC][kMaxPatchPoints];
  int32_t def[kMaxDef];
  int32_t done;
};

// One patch by one CTA.  Its groups go to the warps in turn; groups whose
// elements share points accumulate in the order of their rounds (a group
// waits until the groups of earlier rounds have accumulated; its stiffness,
// most of the work, comes before the wait), those of one round share none.
template <int POLE, int MODE, bool KAHAN>
__device__ __forceinline__ void patch_cta(const StreamWork &w, const SpecDev &sp, int32_t p, float *xw,
                                          PatchSmem<POLE> &s) {
  using S = SolidPoint<POLE, MODE, KAHAN>;
  constexpr int NC = S::NC;
  constexpr int row = 5 * 8 * SolidGrp<POLE, true>::kRows;
  const StreamDomain &d = w.ds;
  const StateArgs &st = w.solid;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool gone = MODE != MODE_FORCE && stopped_before(st.stop);
  const PatchInfo pi = d.patches[p];
  const int n_pts = pi.n_int + pi.n_def;
  GroupMeta g = warp < pi.n_groups ? d.groups[pi.group0 + warp] : GroupMeta{0, 0, 0};
  for (int t = threadIdx.x; t < n_pts; t += kGrpThreads)
#pragma unroll
    for (int c = 0; c < NC; ++c) s.f[c][t] = 0.f;
  for (int t = threadIdx.x; t < pi.n_def; t += kGrpThreads)
    s.def[t] = AXG_BOUND(pi.def_start + t, d.n_def, 69) ? __ldg(d.def + pi.def_start + t) : 0;
  if (threadIdx.x == 0) s.done = 0;
  if (MODE == MODE_FORCE) __syncthreads();
  else if (__syncthreads_or(gone)) return;
  // the own points' state, which the last phase reads, into L2 meanwhile
  if (w.prefetch > 0 && MODE != MODE_FORCE && warp == kGrpWarps - 1 && pi.n_int > 0) {
    auto range = [&](const float *a) {
      const uintptr_t x = (reinterpret_cast<uintptr_t>(a + pi.int_start)) & ~(uintptr_t)15;
      const uintptr_t y = (reinterpret_cast<uintptr_t>(a + pi.int_start + pi.n_int) + 15) & ~(uintptr_t)15;
      prefetch_l2(reinterpret_cast<const void *>(x), (uint32_t)(y - x));
    };
    const int c = lane % 3;
    // (mass pairs, 8 bytes per point, take longer with theirs: 338.2 us against
    // 335.1 for a compensated step of 327 680 elements)
    if (lane == 0 && !(KAHAN && st.inv_mass_pair)) range(st.inv_mass);
    if (lane >= 3 && lane < 6 && st.v[c]) range(st.v[c]);
    if (MODE == MODE_NEWMARK && lane >= 6 && lane < 9 && st.a[c]) range(st.a[c]);
    if (KAHAN && lane >= 9 && lane < 12 && st.cv[c]) range(st.cv[c]);
    if (KAHAN && MODE == MODE_NEWMARK && lane >= 12 && lane < 15 && st.cup[c]) range(st.cup[c]);
  }
  bool waited = false, stopped = false;
  for (int q = warp; q < pi.n_groups; q += kGrpWarps) {
    const bool more = q + kGrpWarps < pi.n_groups;
    GroupMeta next = more ? d.groups[pi.group0 + q + kGrpWarps] : GroupMeta{0, 0, 0};
    if (w.prefetch > 0) {
      // into L2: the warp's next group, or its first of the patch that runs
      // about one round of resident CTAs later
      GroupMeta h = next;
      if (!more && p + w.prefetch < d.n_patches) {
        const PatchInfo pn = d.patches[p + w.prefetch];
        if (warp < pn.n_groups) h = d.groups[pn.group0 + warp];
      }
      if (h.n > 0 && lane == 0) prefetch_l2(d.blocks + (int64_t)h.slot0 * row, h.n * row * 4);
    }
    bool turn = false;
    solid_group<POLE, true, MODE, false, KAHAN>(
        w, sp, g, xw, nullptr, pi.int_start, pi.n_int, s.def, false,
        [&]() {
          if (!waited) {
            pdl_wait();
            stopped = MODE != MODE_FORCE && *st.stop != 0;
          }
          waited = true;
          return stopped;
        },
        [&](const float (&f)[NC][5], const int32_t (&idx)[5], bool mine, int, int) {
          if (!turn) wait_turn(&s.done, g.wait, lane, st.err);
          turn = true;
          if (!mine) return;
#pragma unroll
          for (int i = 0; i < 5; ++i) {
            const int t = idx[i];
            if (!AXG_BOUND(t, n_pts, 69)) continue;
#pragma unroll
            for (int c = 0; c < NC; ++c) s.f[c][t] += f[c][i];
          }
        });
    __syncwarp();
    __threadfence_block();
    if (lane == 0) atomicAdd(&s.done, 1);
    g = next;
  }
  if (!waited) {
    pdl_wait();
    stopped = MODE != MODE_FORCE && *st.stop != 0;
  }
  __syncthreads();
  if (stopped) return;  // (the whole CTA: no flag changes between the wait and the end of the step)
  // the deferred points' partial sums
  for (int t = threadIdx.x; t < pi.n_def; t += kGrpThreads) {
    float4 v;
    v.x = s.f[0][pi.n_int + t];
    v.y = s.f[1][pi.n_int + t];
    v.z = NC == 3 ? s.f[NC - 1][pi.n_int + t] : 0.f;
    v.w = 0.f;
    if (AXG_BOUND(4 * (pi.def_start + t) + 3, d.n_fel, 69)) reinterpret_cast<float4 *>(d.fel)[pi.def_start + t] = v;
  }
  // the patch's own points; kB at a time, their loads together
  bool src = false;
  if (MODE != MODE_FORCE)
    for (int q = 0; q < d.n_src_patch; ++q) src = src || d.src_patch[q] == p;
  constexpr int kB = KAHAN ? 2 : 3;
  for (int t0 = threadIdx.x; t0 < pi.n_int; t0 += kB * kGrpThreads) {
    S pt[kB];
    uint8_t ax[kB];
    if (MODE != MODE_FORCE)
#pragma unroll
      for (int b = 0; b < kB; ++b) {
        const int t = t0 + b * kGrpThreads;
        if (t >= pi.n_int) continue;
        pt[b].load(st, (int64_t)pi.int_start + t);
        ax[b] = pi.axis && w.axmask ? w.axmask[pi.int_start + t] : 0;
      }
#pragma unroll
    for (int b = 0; b < kB; ++b) {
      const int t = t0 + b * kGrpThreads;
      if (t >= pi.n_int) continue;
      const int64_t g = (int64_t)pi.int_start + t;
      if (!AXG_BOUND(g, st.nglob, 69)) continue;
      float sum[NC];
#pragma unroll
      for (int c = 0; c < NC; ++c) sum[c] = s.f[c][t];
      if (MODE == MODE_FORCE) {
#pragma unroll
        for (int c = 0; c < NC; ++c) st.f[S::gc(c)][g] = sum[c];
      } else {
        if (src) S::source(st, *st.iter, g, sum);
        pt[b].finish(st, g, ax[b] != 0, sum);
      }
    }
  }
}

// The seismogram sample of the step (nc_compute_recfile_seis_bare,
// SOLVER/seismograms.f90:783-820) from the step's new displacement, which is
// the prediction it gathered, and the step counter.  One CTA.
template <int POLE>
__device__ __forceinline__ void stream_receivers(const StreamWork &w) {
  const RecWork &rw = w.rec;
  const StateArgs &s = w.solid;
  const int32_t iter = w.ctl[CTL_ITER_P];
  if (rw.seis_it > 0 && iter % rw.seis_it == 0 && !*s.blowup) {
    const int32_t is = iter / rw.seis_it;
    if (is < rw.nseismo)
      for (int r = threadIdx.x; r < rw.num_rec; r += blockDim.x) {
        const int g = rw.rec_gidx[r];
        if (!AXG_BOUND(g, s.nglob, 67)) continue;
        const float us = s.up[0][g], uz = s.up[2][g], up = POLE == POLE_MONO ? 0.f : s.up[1][g];
        const int64_t n = rw.nseismo;
        rw.rec[is + n * (0 + 3 * (int64_t)r)] = POLE == POLE_DI ? us + up : us;
        rw.rec[is + n * (1 + 3 * (int64_t)r)] = POLE == POLE_DI ? us - up : up;
        rw.rec[is + n * (2 + 3 * (int64_t)r)] = uz;
      }
  }
  if (threadIdx.x == 0) {
    if (!w.ctl[CTL_STOP_P]) w.ctl[CTL_PARITY] = w.parity;
    w.ctl[CTL_STOP] = *s.blowup;
    w.ctl[CTL_ITER] = iter + 1;
  }
}

// ------------------------------------------------------------ kernels

// The roles wait for the step before themselves, once they have loaded what
// it does not write.  The solid's first CTA hands the step number on to the
// point pass, and whether the solve has stopped.  A step whose displacement
// blows up is completed, as the reference completes it, by every CTA alike; those
// of the steps after it return at once or, where they have come too early to see
// it, write nothing of the state.
template <int POLE, bool PATCH, int MODE, bool ANEL, bool KAHAN, class P>
__device__ __forceinline__ void elem_cta(const P &p, const SpecDev &sp, float *xch, float *scr, PatchSmem<POLE> *ps) {
  pdl_trigger();
  int b = blockIdx.x;
  const StreamWork &w = p.find(b);
  const int warp = threadIdx.x >> 5;
  float *xw = xch + warp * kXchFloats, *sc = ANEL ? scr + warp * kScFloats : nullptr;
  if (b < w.nb_se) {
    if (MODE != MODE_FORCE && b == 0 && threadIdx.x == kGrpThreads - 1) {
      pdl_wait();
      w.ctl[CTL_ITER_P] = w.ctl[CTL_ITER];
      w.ctl[CTL_STOP_P] = w.ctl[CTL_STOP];
    }
    if constexpr (PATCH) {
      patch_cta<POLE, MODE, KAHAN>(w, sp, b, xw, *ps);
    } else {
      const int32_t grp = b * kGrpWarps + warp;
      if (grp < scatter_groups(w.ds.n_off, w.ds.nel)) scatter_group<POLE, MODE, ANEL, KAHAN>(w, sp, grp, xw, sc);
    }
    return;
  }
  if (MODE == MODE_FORCE) return;
  b -= w.nb_se;
  if (b < w.nb_fe) {
    const int32_t grp = b * kGrpWarps + warp;
    if (grp < grp_count(w.df.nel)) fluid_group<POLE != POLE_MONO, MODE, KAHAN>(w, sp, grp, xw);
    return;
  }
  const int q = (b - w.nb_fe) * kGrpThreads + threadIdx.x;
  if (q < w.to_fluid.n) couple_row<POLE, MODE, KAHAN>(w, q);
}

// The element pass of meshes whose contributions stay in L2.  CTAs: per SM; 4
// (up to 128 registers) where the blocks come from L2, 3 (up to 168) where a
// dipole's or quadrupole's come from HBM: more of a column's rows in flight per
// warp then weigh more than warps.  With attenuation the memory variables need
// the registers: 3.
template <int POLE, int MODE, bool ANEL, bool KAHAN, int CTAS, class P>
__global__ void __launch_bounds__(kGrpThreads, CTAS)
    scatter_kernel(const __grid_constant__ P p, const __grid_constant__ SpecDev sp) {
  __shared__ __align__(16) float xch[kGrpWarps * kXchFloats];
  __shared__ __align__(16) float scr[ANEL ? kGrpWarps * kScFloats : 1];
  elem_cta<POLE, false, MODE, ANEL, KAHAN>(p, sp, xch, scr, nullptr);
}
// The element pass of larger meshes (without coarse-grained attenuation): 3
// CTAs per SM took 21.7 ms where 4 took 23.1 (32 steps, quadrupole, 786 432
// solid elements); a monopole keeps 4 (18.1 ms against 20.3).
template <int POLE, int MODE, bool KAHAN, class P>
__global__ void __launch_bounds__(kGrpThreads, POLE != POLE_MONO ? 3 : 4)
    patch_kernel(const __grid_constant__ P p, const __grid_constant__ SpecDev sp) {
  __shared__ __align__(16) float xch[kGrpWarps * kXchFloats];
  __shared__ PatchSmem<POLE> ps;
  elem_cta<POLE, true, MODE, false, KAHAN>(p, sp, xch, nullptr, &ps);
}

template <int POLE, int MODE, bool PATCH, bool KAHAN, class P>
__global__ void __launch_bounds__(kGrpThreads) point_kernel(const __grid_constant__ P p) {
  pdl_trigger();
  int b = blockIdx.x;
  const StreamWork &w = p.find(b);
  if (MODE == MODE_NEWMARK && b == w.nb_si + w.nb_sp + w.nb_fp) {
    pdl_wait();
    if (w.nb_rec > 0) stream_receivers<POLE>(w);
    return;
  }
  if (!PATCH && b < w.nb_si) {
    const int32_t g = b * kGrpThreads + threadIdx.x;
    if (g < w.p0) inner_point<POLE, MODE, KAHAN>(w, g);
    return;
  }
  b -= w.nb_si;
  if (b < w.nb_sp) {
    const int64_t g = (int64_t)w.p0 + (int64_t)b * kGrpThreads + threadIdx.x;
    if (g < w.ds.nglob) solid_point<POLE, MODE, PATCH, KAHAN>(w, g);
  } else if (MODE != MODE_FORCE) {
    const int64_t g = (int64_t)(b - w.nb_sp) * kGrpThreads + threadIdx.x;
    if (b < w.nb_sp + w.nb_fp && g < w.df.nglob) fluid_point<POLE != POLE_MONO, MODE, KAHAN>(w, g);
  }
}

// time_step_memvars (SOLVER/attenuation.f90:81-202) once per step of the
// symplectic loop, from the drifted displacement: the element pass's first
// stage and memory-variable update alone, a warp per group.
template <int POLE>
__global__ void __launch_bounds__(kGrpThreads, 4)
    memvar_kernel(const __grid_constant__ StreamOne p, const __grid_constant__ SpecDev sp, int32_t n_groups) {
  __shared__ __align__(16) float xch[kGrpWarps * kXchFloats];
  using G = SolidGrp<POLE, false>;
  constexpr int NC = G::NC;
  const StreamWork &w = p.w;
  if (*w.solid.stop) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int32_t grp = blockIdx.x * kGrpWarps + warp;
  if (grp >= n_groups) return;
  const int32_t *ids = w.memvar_gidx;
  float *xw = xch + warp * kXchFloats;
  const GroupMeta g = scatter_meta(grp, w.ds.n_off, w.ds.nel);
  const int nl = 5 * g.n;
  const int ll = lane < nl ? lane : nl - 1;
  const int e = ll / 5, j = ll % 5, e5 = ll - j;
  auto gc = [](int c) { return (POLE == POLE_MONO && c == 1) ? 2 : c; };
  float row[8];
  ldg8(w.ds.blocks + (int64_t)g.slot0 * (5 * 8 * G::kRows) + ll * 8, row, policy_evict_normal());
  const bool ax = (__float_as_uint(row[0]) & kGrpAxial) != 0;
  float eta[5];
#pragma unroll
  for (int k = 0; k < 5; ++k) eta[k] = sp.g2[k + 5 * j];
  float u[NC][5], X[NC][5], Y[NC][5], E[NC][5];
#pragma unroll
  for (int i = 0; i < 5; ++i) {
    int32_t q = __ldg(ids + ((int64_t)g.slot0 + e) * 25 + 5 * j + i);
    if (!AXG_BOUND(q, w.solid.nglob, 68)) q = 0;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      u[c][i] = w.solid.u[gc(c)][q];
      if (i == 0 && ax && col_masked<POLE>(c)) u[c][i] = 0.f;
    }
  }
  xch_put<NC>(xw, lane, u);
  __syncwarp();
  col_xi<NC, false>(sp.g2, u, X);
  col_xi<NC, false>(sp.g1, u, Y);
  xch_eta<NC>(xw, e5, eta, E);
#pragma unroll
  for (int c = 0; c < NC; ++c)
#pragma unroll
    for (int i = 0; i < 5; ++i)
      if (ax) X[c][i] = Y[c][i];
  __syncwarp();
  cg_put<POLE, NC>(xw, lane, j, X, E, u);
  __syncwarp();
  cg_point<POLE, true, false>(w.cg, xw, nullptr, g, lane, true);
}

}  // namespace axg
