// walk_mixed.cu -- warp-group Barnes-Hut walk in mixed precision.
//
// The mixed path walks ONE combined tree of both species (net-charge moments
// about each cell's particle centroid, net.cu).  One warp (in small clouds a
// team of warps) owns a target group -- a contiguous sorted range of at most 32
// particles of either species inside one cell, built by k_groups -- and
// builds ONE interaction list for it:
//   * group MAC: a cell is accepted when rcrit = s/theta + dx (the reference
//     criterion, tree.f90:736-743) is below the distance from the cell's charge
//     centre to the group's bounding box, so every target of the group would
//     also accept it on its own;
//   * accepted cells go to a shared-memory ring of far-field (M2P) entries,
//     the particles of leaves and of twigs with at most `bucket` go to a list
//     of pair (P2P) sources, other twigs push their children on a per-warp
//     stack;
//   * every 32 entries the warp stages them in shared memory and each lane
//     evaluates them for its own target in FP32, two cells or two sources at a
//     time on the packed f32x2 pipeline.
// Precision: positions, the group centre and the MAC stay FP64.  Cells are
// evaluated in FP32 relative to the group centre; particle pairs use a
// two-float (hi + lo) split of the FP64 offsets, so a pair separation keeps
// ~1e-7 relative accuracy even for the closest e-i pairs.  Chunk sums of 32
// terms are added into Kahan-compensated per-lane accumulators.
// Far field: net monopole, dipole and trace-free quadrupole (octupole at order
// 3, hexadecapole at order 4) about the centroid -- the Coulomb expansion of
// tree.f90:744-779 carried to full subtree moments and further, for cells
// whose net charge nearly cancels; accepted cells far from the group go into
// the group's fourth-order local expansion (local.cuh), evaluated once per
// target.  Near field: erf-Kelbg (or the reference laws) for every particle
// pair.  With a trained model, cells the fixed test opens may be accepted by
// the learned criterion (mac.cuh, mac_batch below).
#include <atomic>
#include <cstdio>
#include "local.cuh"
#include "mac.cuh"
#include "walk_mixed.h"

namespace tg {

constexpr int kStackCap = 8192;   // node indices per warp
constexpr int kM2pRing = 64;      // power of two, > 31 + 32
constexpr int kLocRing = 64;      // power of two, > 31 + 32
constexpr int kLocStride = kLocCoef | 1;  // odd row stride of the coefficient rows
constexpr int kMaxBucket = 8;
constexpr int kP2pBuf = 31 + 32 * kMaxBucket + 1;  // what a batch of nodes can leave
constexpr int kMaxBlocksPerSm = 4;
// One block per SM.  The fixed test without RDF counts runs 20 warps of 96
// registers: N = 1M takes 11.0 ms, against 11.6 ms for 16 warps (of 96 too) and
// 11.6 ms for 24 of 80.  The learned criterion's build runs 16 warps of 128:
// 70.3 ms at N = 4M and 50.5 ms on the ensemble of 64 clouds.  The line was
// drawn with a far field of fewer operations and more live registers, where
// 20 of 96 were 1.4 % slower and 0.6 % faster; with this one they take 68.4 and
// 49.1 ms, 24 of 80 71.6 and 50.1.  The builds with RDF counts run 16 warps:
// their histograms (2 x 10001 u32, added to the global bins once, when the
// block ends) leave no room for more.
constexpr int kWarpStep = 8;      // warps per unit of the blocks_per_sm tunable
constexpr int kStackWarps = 32;   // per SM: stacks of the walk's and the sampler's warps
template <bool RDF, bool LEARNED>
constexpr int walk_warps() { return RDF || LEARNED ? 16 : 20; }

// Warps that share a group.  Below about 30,000 particles there are fewer
// groups (of about 25 targets) than half the warps of the GPU, and a group is a
// serial walk; a team's leader walks, and its warps evaluate the same batches
// that one warp would, in rounds, so the forces are the same to the last bit.
// Walk ms for 1, 2, 4, 8, 16 warps (hexadecapole, theta 0.42, fixed | with RDF):
//   N = 1,000   0.092 0.076 0.061 0.054 0.050 | 0.131 0.094 0.074 0.064 0.059
//   N = 4,096   0.273 0.213 0.165 0.143 0.173 | 0.362 0.250 0.185 0.161 0.189
//   N = 8,192   0.387 0.317 0.252 0.268 0.339 | 0.483 0.358 0.275 0.292 0.364
//   N = 12,000  0.454 0.365 0.300 0.375 0.522 | 0.518 0.398 0.326 0.407 0.551
//   N = 16,384  0.540 0.443 0.439 0.514 0.723 | 0.598 0.479 0.474 0.557 0.764
//   N = 20,000  0.657 0.517 0.555 0.662 0.965 | 0.720 0.562 0.595 0.718 1.018
//   N = 28,000  1.133 0.956 1.132 1.457 2.173 | 1.320 1.056 1.220 1.568 2.292
//   N = 32,768  1.336 1.266 1.380 1.789 2.714 | 1.472 1.376 1.484 1.932 2.847
// A cloud's longest groups count: on another one of 32,768 two warps took 0.832
// against 0.803 of one, which is why the line lies below that size.
int walk_team(int n) {
  return n < 3000 ? 16 : (n < 6000 ? 8 : (n < 16000 ? 4 : (n < 30000 ? 2 : 1)));
}

constexpr int kCandRing = 64;     // power of two, > 31 + 32
constexpr int kCellF4 = 9;        // float4 per staged far-field cell (order 4)
constexpr int kPartF4 = 5;        // float4 per staged source pair (4 used + pad)

struct WarpSmem {
  int m2p[kM2pRing];
  int loc[kLocRing];       // far cells summed into the group's local expansion
  int p2p[kP2pBuf];        // particle entries; at most 31 between batches
  int cq_node[kCandRing];  // learned-MAC candidates waiting for a full batch
  // The far-field and pair staging areas (and the learned MAC's feature
  // rows, in `cell`) are used one at a time by the warp: one buffer.
  union {
    // staged cells, kCellF4 float4 each: (dx, dy, dz, Q), (Dx, Dy, Dz, q_ion),
    // (Sxx, Syy, Szz, Sxy), (Syz, Szx, Txxx, Tyyy), (Tzzz, Txxy, Txxz, Txyy),
    // (Tyyz, Txzz, Tyzz, Txyz), then for order 4 (Hxxxx, Hxxxy, Hxxxz, Hxxyy),
    // (Hxxyz, Hxyyy, Hxyyz, Hyyyy), (Hyyyz, Hxxzz, Hxyzz, Hyyzz) -- S, T and
    // H trace-free
    float4 cell[32 * kCellF4];
    // staged sources in pairs, kPartF4 float4 per pair: sources 2b and 2b+1
    // side by side, (nhx nhx' nhy nhy') (nhz nhz' q q') (nlx nlx' nly nly')
    // (nlz nlz' idx idx'): negated hi / lo offsets from the group centre,
    // charge, sorted index bits
    float4 part[16 * kPartF4];
    // local-expansion coefficients of up to 32 cells, one row per lane
    // (odd stride: conflict-free rows and columns)
    float loc_rows[32 * kLocStride];
  };
  // pair constants of the group's cloud: 1/lambda^2 (ee, ei, ii), 1/rs,
  // 1/lambda (ee, ei, ii)
  float pk[8];
  // the group's box: centre and half extents (read where used, so that they
  // hold no registers across the walk loop)
  double gx, gy, gz, bx, by, bz;
  double hl2;  // the group's squared half-diagonal (local-expansion test)
  // learned criterion, per group: log10 of the error budget (-inf: none),
  // and the cells sent to the network / kept on the fixed decision.  Kept
  // here rather than in registers, which the walk loop needs for its
  // evaluations.
  float lbud;
  unsigned n_mlp, n_fallback;
  double2 phi[32];  // per lane: unscaled potential (all sources, ion part)
};

__device__ __forceinline__ void phi_add(WarpSmem& sm, int lane, double all, double ion) {
  double2 p = sm.phi[lane];
  p.x += all;
  p.y += ion;
  sm.phi[lane] = p;
}

// A team of warps and its queue of batches: the leader walks and fills it, every
// warp evaluates one batch a round, the leader adds the results in order.
constexpr int kTeamMin = 2;
constexpr int kTeamQueue = 15 + 13;  // one short of the largest team, and what a walk's end adds
struct TeamSmem {
  int item, take;            // the team's group; batches of this round (0: group done)
  int info[kTeamQueue];      // 4 * entries + kind: 1 far field, 2 particles, 3 local
  int idx[kTeamQueue][32];
};

struct MixedArgs {
  const double4* __restrict__ node_c;
  const float4* __restrict__ mom;
  const int32_t* __restrict__ kids;
  const int32_t* __restrict__ first;
  const int32_t* __restrict__ count;
  const double4* __restrict__ xs;
  const uint32_t* __restrict__ order;
  const int32_t* __restrict__ bounds;
  const int2* __restrict__ groups;
  const int32_t* __restrict__ n_groups;
  int32_t* control;
  int32_t* stack;
  int team;  // warps that share a group (TEAM builds; a power of two)
  int bucket;
  int p2p_max;  // accepted cells with at most this many particles go to P2P
  // accepted cells far from the group go to its local expansion: h / d <=
  // loc_eps, h the group's half-diagonal, d the distance from its centre to
  // the cell's centroid; loc_eps = 0: never
  double loc_eps2;
  float inv_lam2_ee, inv_lam2_ei, inv_lam2_ii;
  float inv_lam_ee, inv_lam_ei, inv_lam_ii;
  float rs_inv;
  float dx_ei_inv_f, dx_ii_inv_f;  // 1 / RDF bin widths
  double* f;
  double2* epot_part;
  uint32_t* rdf;
  unsigned long long* counters;
  int32_t* err;
  // learned acceptance
  const MlpPacked* packed;
  const float* fmin;
  const float* fmax;
  const float4* geom;
  const float4* mom3;
  const float4* mom4;
  // per cell: its part K of the pre-filter (mac.cuh) and the distance
  // s / rho_hi + dx below which its acceptance ratio s / (d - dx) exceeds
  // rho_hi (the learned criterion's band)
  const float2* mac_k;
  const float* margins;  // m_lo, m_hi, pre-filter coefficients c0..c4
  const double* f_prev;
  float eta_over_eps;
  // ensemble of clouds (nseg > 0): cloud ranges, roots, pair constants
  int nseg;
  const int32_t* ens_start;
  const int32_t* roots;
  const float4* cloud_pk;  // 2 per cloud, the layout of WarpSmem::pk
};

struct Acc {
  float sx, sy, sz, cx, cy, cz;  // Kahan sums of the unscaled force
  // The unscaled potential (all sources, ion part) is summed in FP64 in the
  // warp's shared memory, one slot per lane (WarpSmem::phi): it is touched
  // once per batch of 32 entries and need not hold registers in between.
};

// What one batch of 32 entries gives this lane: unscaled force and potential
// (all sources, ion part) of its target, or one local-expansion coefficient.
struct alignas(16) Batch {
  float fx, fy, fz, loc;
  double pa, pi;
};

__device__ __forceinline__ void kahan_add(float& s, float& c, float v) {
  float y = v - c;
  float t = s + y;
  c = (t - s) - y;
  s = t;
}

__device__ __forceinline__ void batch_add(WarpSmem& sm, int lane, Acc& acc, const Batch& b) {
  kahan_add(acc.sx, acc.cx, b.fx);
  kahan_add(acc.sy, acc.cy, b.fy);
  kahan_add(acc.sz, acc.cz, b.fz);
  phi_add(sm, lane, b.pa, b.pi);
}

// Inclusive scan over the warp; the shuffle's own predicate says which lanes add.
__device__ __forceinline__ int warp_incl_scan(int v) {
#define TG_SCAN(o)                                                     \
  asm volatile("{ .reg .s32 t; .reg .pred p;\n"                       \
               "  shfl.sync.up.b32 t|p, %0, " #o ", 0, 0xffffffff;\n" \
               "  @p add.s32 %0, %0, t; }\n"                          \
               : "+r"(v))
  TG_SCAN(1);
  TG_SCAN(2);
  TG_SCAN(4);
  TG_SCAN(8);
  TG_SCAN(16);
#undef TG_SCAN
  return v;
}

__device__ __forceinline__ double warp_min_d(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ double warp_max_d(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// ---------------------------------------------------------------- M2P ----
// Net monopole Q, dipole D, trace-free second moment S (from 1/2 sum q a a^T),
// third moment T (from sum q a a a) and fourth moment H about the cell
// centroid.  With d = target - centroid, r = |d|, s = 1/r, n = d / r:
//   r phi = Q + s D.n + 3 s^2 S(n,n) + 5/2 s^3 T(n,n,n) + 35/8 s^4 H(n,n,n,n),
//   r^2 (-grad phi) = g n - s D - 6 s^2 S n - 15/2 s^3 T(.,n,n) - 35/2 s^4 H(.,n,n,n),
//   g = Q + 3 s D.n + 15 s^2 S(n,n) + 35/2 s^3 T(n,n,n) + 315/8 s^4 H(n,n,n,n).
// Normalised form: every intermediate is bounded by n (a/r)^k -- escaped
// electrons millions of um away would otherwise overflow T(d,d,d) ~ |T| r^3
// while 1/r^7 underflows.
// T is trace-free (T_iik = 0), so T_kzz = -T_kxx - T_kyy and each component
// of T(., n, n) takes five terms with a2 = nx^2 - nz^2, b2 = ny^2 - nz^2; each
// component of H(., n, n, n) is a combination of seven cubic harmonics P1..P7
// of n, its z component reading the dependent components xxzz, xyzz, yyzz
// staged with the others.  About 120 multiply-adds at order 4.  The ion part
// of phi for the Epot_e/Epot_i split is taken at monopole order (q_ion / r).
//
// The order of the operations below is part of the results: a loop of steps
// amplifies a last-bit difference by the close passages of the electrons (ten
// steps at N = 32,768: 1.2e-5 of the electron positions, 9e-4 of a single one).
// The walk without RDF counts adds the cells up one after the other, the one with
// counts in two sums, and the two form P1, P5 and P6 in different orders, as
// their first versions did.

// 1/sqrt(x) of a normal number, without rsqrtf's rescaling of subnormal ones.
__device__ __forceinline__ float rsqrt_normal(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// The rows of a staged cell (WarpSmem::cell).
template <int ORDER, int ROWS>
__device__ __forceinline__ void m2p_rows(const MixedArgs& a, int node, double Gx, double Gy,
                                         double Gz, float4 (&r)[ROWS]) {
  const double4 c = ldg_d4(&a.node_c[node]);
  const float4* mp = a.mom + 3 * (int64_t)node;
  const float4 m0 = __ldg(mp), m2 = __ldg(mp + 2);
  r[0] = make_float4((float)(Gx - c.x), (float)(Gy - c.y), (float)(Gz - c.z), m0.x);
  r[1] = make_float4(m0.y, m0.z, m0.w, m2.w);
  r[2] = __ldg(mp + 1);
  r[3] = make_float4(m2.x, m2.y, 0.f, 0.f);
  if constexpr (ORDER >= 3) {
    const float4* tp = a.mom3 + 3 * (int64_t)node;
    const float4 t0 = __ldg(tp), t1 = __ldg(tp + 1), t2 = __ldg(tp + 2);
    r[3].z = t0.x;
    r[3].w = t0.y;
    r[4] = make_float4(t0.z, t0.w, t1.x, t1.y);
    r[5] = make_float4(t1.z, t1.w, t2.x, t2.y);
  }
  if constexpr (ORDER >= 4) {
    const float4* hp = a.mom4 + 3 * (int64_t)node;
#pragma unroll
    for (int k = 0; k < 3; ++k) r[6 + k] = __ldg(hp + k);
  }
}

// The far field runs two cells at a time on the packed FP32 (f32x2) pipeline:
// cells 2b and 2b+1 are staged side by side, so one 16-byte shared load gives
// two float2 operands and every multiply-add serves both cells.
__device__ __forceinline__ float2 f2(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
// a + b that is not merged into a multiply-add with a product a or b, which
// __fadd2_rn is.
__device__ __forceinline__ float2 add2_apart(float2 a, float2 b) {
  return make_float2(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y));
}

// sum += a b for the two cells of a pair: side by side, or one after the other
// in sum.x (sum.y stays 0).
template <bool SIDE>
__device__ __forceinline__ void m2p_sum(float2& sum, float2 a, float2 b) {
  if (SIDE) {
    sum = fma2(a, b, sum);
  } else {
    sum.x = fmaf(a.x, b.x, sum.x);
    sum.x = fmaf(a.y, b.y, sum.x);
  }
}

template <int ORDER, bool RDF>
__device__ __forceinline__ void eval_m2p(WarpSmem& sm, const int* list, int mask, int head, int cnt,
                                            const MixedArgs& a, double Gx, double Gy,
                                            double Gz, float tx, float ty, float tz,
                                            int lane, Batch& out) {
  constexpr int kRows = ORDER >= 4 ? 9 : (ORDER == 3 ? 6 : 4);
  {
    // this lane's cell as kRows float4 rows (see WarpSmem::cell), or past cnt a
    // chargeless dummy whose r^2 overflows to infinity: its powers of 1/r are 0
    // (at a distance that a target can lie at, they could overflow instead)
    float4 r[kRows];
    if (lane < cnt) {
      m2p_rows<ORDER>(a, list[(head + lane) & mask], Gx, Gy, Gz, r);
    } else {
      r[0] = make_float4(1.0e20f, 1.0e20f, 1.0e20f, 0.f);
#pragma unroll
      for (int j = 1; j < kRows; ++j) r[j] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    // pair block b = lane / 2: row j of both cells as (x x' y y') (z z' w w');
    // the even lane writes the first float4, the odd lane the second
    const bool odd = lane & 1;
    float4* blk = sm.cell + 2 * kCellF4 * (lane >> 1);
#pragma unroll
    for (int j = 0; j < kRows; ++j) {
      const float s0 = odd ? r[j].x : r[j].z, s1 = odd ? r[j].y : r[j].w;
      const float p0 = __shfl_xor_sync(0xffffffffu, s0, 1);
      const float p1 = __shfl_xor_sync(0xffffffffu, s1, 1);
      blk[2 * j + (odd ? 1 : 0)] = odd ? make_float4(p0, r[j].z, p1, r[j].w)
                                       : make_float4(r[j].x, p0, r[j].y, p1);
    }
  }
  __syncwarp();
  const float2 tx2 = f2(tx), ty2 = f2(ty), tz2 = f2(tz);
  float2 fx = f2(0.f), fy = fx, fz = fx, pa = fx, pi = fx;
  const int npair = (cnt + 1) >> 1;
#pragma unroll 1
  for (int b = 0; b < npair; ++b) {
    const float4* bl = sm.cell + 2 * kCellF4 * b;
    float4 q = bl[0];
    const float2 Ax = make_float2(q.x, q.y), Ay = make_float2(q.z, q.w);
    q = bl[1];
    const float2 Az = make_float2(q.x, q.y), Q = make_float2(q.z, q.w);
    const float2 dx = add2(tx2, Ax), dy = add2(ty2, Ay), dz = add2(tz2, Az);
    const float2 r2 = fma2(dx, dx, fma2(dy, dy, fma2(dz, dz, f2(1e-30f))));
    const float2 s = make_float2(rsqrt_normal(r2.x), rsqrt_normal(r2.y));
    const float2 s2 = mul2(s, s);
    const float2 nx = mul2(dx, s), ny = mul2(dy, s), nz = mul2(dz, s);
    q = bl[4];
    const float2 Sxx = make_float2(q.x, q.y), Syy = make_float2(q.z, q.w);
    q = bl[5];
    const float2 Szz = make_float2(q.x, q.y), Sxy = make_float2(q.z, q.w);
    q = bl[6];
    const float2 Syz = make_float2(q.x, q.y), Szx = make_float2(q.z, q.w);
    const float2 Sx = fma2(Sxx, nx, fma2(Sxy, ny, mul2(Szx, nz)));
    const float2 Sy = fma2(Sxy, nx, fma2(Syy, ny, mul2(Syz, nz)));
    const float2 Sz = fma2(Szx, nx, fma2(Syz, ny, mul2(Szz, nz)));
    const float2 u = fma2(nx, Sx, fma2(ny, Sy, mul2(nz, Sz)));
    q = bl[2];
    const float2 Dx = make_float2(q.x, q.y), Dy = make_float2(q.z, q.w);
    q = bl[3];
    const float2 Dz = make_float2(q.x, q.y), Qi = make_float2(q.z, q.w);
    const float2 Dn = fma2(Dx, nx, fma2(Dy, ny, mul2(Dz, nz)));
    const float2 su = mul2(s, u);
    float2 gp = fma2(s, fma2(f2(15.f), su, mul2(f2(3.f), Dn)), Q);
    float2 ph = fma2(s, fma2(f2(3.f), su, Dn), Q);
    const float2 c5 = mul2(f2(-6.f), s2), ms = mul2(f2(-1.f), s);
    float2 gx = fma2(c5, Sx, mul2(ms, Dx));
    float2 gy = fma2(c5, Sy, mul2(ms, Dy));
    float2 gz = fma2(c5, Sz, mul2(ms, Dz));
    const float2 mnz = mul2(f2(-1.f), nz);
    if (ORDER >= 3) {
      // (Syz Szx Txxx Tyyy) (Tzzz Txxy Txxz Txyy) (Tyyz Txzz Tyzz Txyz)
      q = bl[7];
      const float2 Txxx = make_float2(q.x, q.y), Tyyy = make_float2(q.z, q.w);
      q = bl[8];
      const float2 Txxy = make_float2(q.z, q.w);
      q = bl[9];
      const float2 Txxz = make_float2(q.x, q.y), Txyy = make_float2(q.z, q.w);
      q = bl[10];
      const float2 Tyyz = make_float2(q.x, q.y), Txzz = make_float2(q.z, q.w);
      q = bl[11];
      const float2 Tyzz = make_float2(q.x, q.y), Txyz = make_float2(q.z, q.w);
      const float2 mzz = mul2(nz, mnz);
      const float2 a2 = fma2(nx, nx, mzz), b2 = fma2(ny, ny, mzz);
      const float2 x2 = mul2(f2(2.f), nx);
      const float2 xy2 = mul2(x2, ny), xz2 = mul2(x2, nz), yz2 = mul2(mul2(f2(2.f), ny), nz);
      const float2 Tx = fma2(Txxx, a2, fma2(Txyy, b2, fma2(Txxy, xy2, fma2(Txxz, xz2, mul2(Txyz, yz2)))));
      const float2 Ty = fma2(Txxy, a2, fma2(Tyyy, b2, fma2(Txyy, xy2, fma2(Txyz, xz2, mul2(Tyyz, yz2)))));
      const float2 Tz = fma2(Txxz, a2, fma2(Tyyz, b2, fma2(Txyz, xy2, fma2(Txzz, xz2, mul2(Tyzz, yz2)))));
      const float2 T3 = fma2(nx, Tx, fma2(ny, Ty, mul2(nz, Tz)));
      const float2 s3 = mul2(s2, s);
      const float2 s3T3 = mul2(s3, T3);
      gp = fma2(f2(17.5f), s3T3, gp);
      ph = fma2(f2(2.5f), s3T3, ph);
      const float2 c7 = mul2(f2(-7.5f), s3);
      gx = fma2(c7, Tx, gx);
      gy = fma2(c7, Ty, gy);
      gz = fma2(c7, Tz, gz);
    }
    if (ORDER >= 4) {
      // (xxxx xxxy xxxz xxyy) (xxyz xyyy xyyz yyyy) (yyyz xxzz xyzz yyzz)
      q = bl[12];
      const float2 H0 = make_float2(q.x, q.y), H1 = make_float2(q.z, q.w);
      q = bl[13];
      const float2 H2 = make_float2(q.x, q.y), H3 = make_float2(q.z, q.w);
      q = bl[14];
      const float2 H4 = make_float2(q.x, q.y), H5 = make_float2(q.z, q.w);
      q = bl[15];
      const float2 H6 = make_float2(q.x, q.y), H7 = make_float2(q.z, q.w);
      q = bl[16];
      const float2 H8 = make_float2(q.x, q.y), H9 = make_float2(q.z, q.w);
      q = bl[17];
      const float2 H10 = make_float2(q.x, q.y), H11 = make_float2(q.z, q.w);
      const float2 xx = mul2(nx, nx), yy = mul2(ny, ny);
      float2 P1, P5, P6;
      if (RDF) {
        const float2 mzz3 = mul2(f2(-3.f), mul2(nz, nz));
        P1 = mul2(nx, add2_apart(xx, mzz3));
        P6 = mul2(ny, add2_apart(yy, mzz3));
        P5 = mul2(mul2(f2(6.f), nx), mul2(ny, nz));
      } else {
        const float2 m3nz = mul2(f2(-3.f), nz);
        P1 = mul2(nx, fma2(m3nz, nz, xx));
        P6 = mul2(ny, fma2(m3nz, nz, yy));
        P5 = mul2(mul2(mul2(f2(6.f), nx), ny), nz);
      }
      const float2 P2 = mul2(mul2(f2(3.f), ny), fma2(nz, mnz, xx));
      const float2 P4 = mul2(mul2(f2(3.f), nx), fma2(nz, mnz, yy));
      const float2 mzz = mul2(mnz, nz);
      const float2 P3 = mul2(nz, fma2(f2(3.f), xx, mzz));
      const float2 P7 = mul2(nz, fma2(f2(3.f), yy, mzz));
      const float2 Vx = fma2(H0, P1, fma2(H1, P2, fma2(H2, P3, fma2(H3, P4,
                        fma2(H4, P5, fma2(H5, P6, mul2(H6, P7)))))));
      const float2 Vy = fma2(H1, P1, fma2(H3, P2, fma2(H4, P3, fma2(H5, P4,
                        fma2(H6, P5, fma2(H7, P6, mul2(H8, P7)))))));
      const float2 Vz = fma2(H2, P1, fma2(H4, P2, fma2(H9, P3, fma2(H6, P4,
                        fma2(H10, P5, fma2(H8, P6, mul2(H11, P7)))))));
      const float2 H4n = fma2(nx, Vx, fma2(ny, Vy, mul2(nz, Vz)));
      const float2 s4 = mul2(s2, s2);
      const float2 s4H = mul2(s4, H4n);
      gp = fma2(f2(39.375f), s4H, gp);
      ph = fma2(f2(4.375f), s4H, ph);
      const float2 c9 = mul2(f2(-17.5f), s4);
      gx = fma2(c9, Vx, gx);
      gy = fma2(c9, Vy, gy);
      gz = fma2(c9, Vz, gz);
    }
    m2p_sum<RDF>(fx, s2, fma2(gp, nx, gx));
    m2p_sum<RDF>(fy, s2, fma2(gp, ny, gy));
    m2p_sum<RDF>(fz, s2, fma2(gp, nz, gz));
    m2p_sum<RDF>(pa, s, ph);
    m2p_sum<RDF>(pi, Qi, s);
  }
  __syncwarp();
  out.fx = fx.x + fx.y;
  out.fy = fy.x + fy.y;
  out.fz = fz.x + fz.y;
  out.pa = (double)pa.x + (double)pa.y;
  out.pi = (double)pi.x + (double)pi.y;
}

// -------------------------------------------------------------- local ----
// Up to 32 far cells, one per lane: each lane expands its cell's field about
// the group centre G (local.cuh) into its row of `loc_rows`; lanes 0..28 then
// add up one coefficient each over the rows.  The
// group's targets evaluate the summed expansion once, after the walk.
template <int ORDER>
__device__ __forceinline__ void eval_local(WarpSmem& sm, const int* list, int mask, int head, int cnt,
                                           const MixedArgs& a, double Gx, double Gy,
                                           double Gz, int lane, Batch& out) {
  constexpr int kStride = kLocStride;
  if (lane < cnt) {
    const int node = list[(head + lane) & mask];
    const double4 c = ldg_d4(&a.node_c[node]);
    CellMoments m;
    const float4* mp = a.mom + 3 * (int64_t)node;
    const float4 m0 = __ldg(mp), m1 = __ldg(mp + 1), m2 = __ldg(mp + 2);
    m.q = m0.x;
    m.d[0] = m0.y; m.d[1] = m0.z; m.d[2] = m0.w;
    m.s[0] = m1.x; m.s[1] = m1.y; m.s[2] = m1.z; m.s[3] = m1.w;
    m.s[4] = m2.x; m.s[5] = m2.y;
    m.q_ion = m2.w;
    if (ORDER >= 3) {
      const float4* tp = a.mom3 + 3 * (int64_t)node;
      const float4 t0 = __ldg(tp), t1 = __ldg(tp + 1), t2 = __ldg(tp + 2);
      m.t[0] = t0.x; m.t[1] = t0.y; m.t[2] = t0.z; m.t[3] = t0.w;
      m.t[4] = t1.x; m.t[5] = t1.y; m.t[6] = t1.z; m.t[7] = t1.w;
      m.t[8] = t2.x; m.t[9] = t2.y;
    }
    if (ORDER >= 4) {
      const float4* hp = a.mom4 + 3 * (int64_t)node;
      const float4 h0 = __ldg(hp), h1 = __ldg(hp + 1), h2 = __ldg(hp + 2);
      m.h[0] = h0.x; m.h[1] = h0.y; m.h[2] = h0.z; m.h[3] = h0.w;
      m.h[4] = h1.x; m.h[5] = h1.y; m.h[6] = h1.z; m.h[7] = h1.w;
      m.h[8] = h2.x; m.h[9] = h2.y; m.h[10] = h2.z; m.h[11] = h2.w;
    }
    local_coefs<ORDER>((float)(Gx - c.x), (float)(Gy - c.y), (float)(Gz - c.z), m,
                       sm.loc_rows + kStride * lane);
  }
  __syncwarp();
  float t = 0.f;
  if (lane < kLocCoef)
    for (int k = 0; k < cnt; ++k) t += sm.loc_rows[kStride * k + lane];
  out.loc = t;
  __syncwarp();
}

// ---------------------------------------------------------------- P2P ----
// Staged pair block (kPartF4 float4, sources 2b and 2b+1 side by side):
//   q0 (nhx nhx' nhy nhy')  q1 (nhz nhz' q q')  q2 (nlx nlx' nly nly')
//   q3 (nlz nlz' idx idx')
// negated hi / lo FP32 parts of each source's FP64 offset from the group
// centre, its charge (-1 electron, +1 ion; 0 for padding) and its sorted index.
//
// A pair's separation is formed from the hi parts alone.  Each hi part is
// within 2^-24 of its offset, so the separation r is within 2^-24 (2h + r)
// of the exact one (h the group's half-diagonal, which bounds the target's
// offset); for r^2 > h^2/32 that is below 7.3e-7 r.  Closer pairs -- a few in
// a thousand, among them every pair of the Kelbg core, the target itself and
// particles on one point -- are redone with hi + lo, whose FP32 roundings are
// relative to their own results, and only they need the source index.

// RDF counts of two pairs (e-i for every target, i-i for ion targets, as
// Search_Tree_ie/ei/ii bin them).  The bin is the FP32 distance r = r2 /
// sqrt(r2) (rsqrt within 2 ulp) over the bin width: within about 1e-6
// relative of the FP64 distance (see above), so a pair within that of a bin
// edge can land in the neighbouring bin; the FP64 path bins in FP64.
// s0 / s1: the source indices, or -1 when a pair was not close (it is then
// not the target).
template <int PHYS>
__device__ __forceinline__ void rdf_count2(const MixedArgs& a, uint32_t* hist, float2 r2,
                                           float2 rinv, float2 q, int s0, int s1,
                                           int p_self, int tsp) {
  const float tq = tsp ? 1.f : -1.f;
  const bool same0 = q.x == tq, same1 = q.y == tq;
  const float2 inv = make_float2(same0 ? a.dx_ii_inv_f : a.dx_ei_inv_f,
                                 same1 ? a.dx_ii_inv_f : a.dx_ei_inv_f);
  const float2 t = __fmul2_rn(__fmul2_rn(r2, rinv), inv);
  // counted pairs: a source (q != 0) of the other species, or an ion for an
  // ion target; never the target itself (Kelbg) or inside the same-species
  // cutoff (reference laws)
  const bool ok0 = q.x != 0.f && (!same0 || tsp == 1) &&
                   (PHYS == 1 ? s0 != p_self : (same0 ? r2.x > 0.01f : true));
  const bool ok1 = q.y != 0.f && (!same1 || tsp == 1) &&
                   (PHYS == 1 ? s1 != p_self : (same1 ? r2.y > 0.01f : true));
  // r2 = 0 (distinct particles on one point): bin 0
  const float t0 = r2.x > 0.f ? t.x : 0.f, t1 = r2.y > 0.f ? t.y : 0.f;
  if (ok0 && t0 < (float)kRdfBins) atomicAdd(&hist[(same0 ? kRdfBins : 0) + (int)t0], 1u);
  if (ok1 && t1 < (float)kRdfBins) atomicAdd(&hist[(same1 ? kRdfBins : 0) + (int)t1], 1u);
}

// hist[...] += 1 at a shared-memory address.
__device__ __forceinline__ void rdf_inc(uint32_t at) {
  asm volatile("red.shared.add.u32 [%0], 1;" ::"r"(at) : "memory");
}

// One source against this lane's target with every case of the pair laws:
// "special" pairs leave the plain Coulomb law -- the target itself (r = 0),
// pairs inside the Kelbg core (exp(-x^2) still visible in FP32), and for the
// reference laws same-species pairs inside the r^2 <= 0.01 cutoff and e-i
// pairs where exp(-r/rs) is visible.
template <int PHYS>
__device__ __noinline__ float2 p2p_special(float r2, float ssign, float il, float rs_inv) {
  // (force over separation, potential) of a special pair that interacts
  float fs = 0.f, ve;
  if (PHYS == 1) {
    const float sqrtpi = 1.77245385f;
    if (r2 > 0.f) {
      const float r = sqrtf(r2);
      const float ri = 1.f / r;
      const float x2 = r2 * il * il;
      const float g = -expm1f(-x2);
      fs = ssign * g * ri * ri * ri;
      ve = g * ri + sqrtpi * erfcf(r * il) * il;
    } else {
      ve = sqrtpi * il;  // distinct particles on one point: V(0)
    }
  } else if (r2 > 0.f) {
    const float r = sqrtf(r2);
    const float ri = 1.f / r;
    const float e = expf(-r * rs_inv);
    const float g = ri - e * (ri + rs_inv);
    fs = ssign * g * ri * ri;
    ve = (1.f - e) * ri;
  } else {
    ve = rs_inv;  // r -> 0 limit of (1 - exp(-r/rs))/r
  }
  return make_float2(fs, ssign * ve);
}

template <int PHYS>
__device__ __forceinline__ void p2p_one(const WarpSmem& sm, float r2, float dx, float dy,
                                        float dz, float ssign, int s, int p_self, int tsp,
                                        float& fx, float& fy, float& fz, float& pa,
                                        float& pq) {
  const bool same = ssign == (tsp ? 1.f : -1.f);
  const float il2 = PHYS == 1 ? (same ? (tsp ? sm.pk[2] : sm.pk[0]) : sm.pk[1]) : 0.f;
  const float rs_inv = sm.pk[3];
  bool special;
  if (PHYS == 1) special = r2 * il2 < 40.f;
  else special = same ? !(r2 > 0.01f) : r2 * (rs_inv * rs_inv) < 400.f;
  float fs = 0.f, ph = 0.f;
  if (!special) {
    const float rinv = rsqrtf(r2);
    fs = ssign * rinv * rinv * rinv;
    ph = ssign * rinv;
  } else if (PHYS == 1 ? s != p_self : !same) {
    // the target itself, and same species inside the cutoff: nothing
    const float il = PHYS == 1 ? (same ? (tsp ? sm.pk[6] : sm.pk[4]) : sm.pk[5]) : 0.f;
    const float2 v = p2p_special<PHYS>(r2, ssign, il, rs_inv);
    fs = v.x;
    ph = v.y;
  }
  fx = fmaf(fs, dx, fx);
  fy = fmaf(fs, dy, fy);
  fz = fmaf(fs, dz, fz);
  pa += ph;
  pq = fmaf(ssign, ph, pq);
}

// Pair interactions of up to 32 staged sources with this lane's target, two
// sources per packed FP32 (f32x2) instruction.  The common pair is plain
// Coulomb from the hi parts; a close pair (r^2 <= close2) is redone with the
// exact offsets, and a pair with a special member goes through p2p_one.
template <int PHYS, bool RDF>
__device__ __forceinline__ void eval_p2p(WarpSmem& sm, const int* list, int cnt,
                                         const MixedArgs& a, double Gx,
                                         double Gy, double Gz, float thx,
                                         float thy, float thz, float tlx,
                                         float tly, float tlz, float close2,
                                         int p_self, int tsp, bool act, int lane,
                                         uint32_t* hist, Batch& out) {
  {
    // this lane's source (or, past cnt, a chargeless dummy: its r^2 overflows to
    // infinity, whose inverse root is 0 and whose bin, 0 times infinity, is none)
    float v[8];
    if (lane < cnt) {
      const int s = list[lane];
      const double4 xs = a.xs[s];
      const double rx = Gx - xs.x, ry = Gy - xs.y, rz = Gz - xs.z;
      const float hx = (float)rx, hy = (float)ry, hz = (float)rz;
      v[0] = hx; v[1] = hy; v[2] = hz; v[3] = xs.w > 0.5 ? 1.f : -1.f;
      v[4] = (float)(rx - (double)hx); v[5] = (float)(ry - (double)hy);
      v[6] = (float)(rz - (double)hz); v[7] = __int_as_float(s);
    } else {
      v[0] = v[1] = v[2] = 1.0e20f;
      v[3] = 0.f;
      v[4] = v[5] = v[6] = 0.f;
      v[7] = __int_as_float(-1);
    }
    const bool odd = lane & 1;
    float2* pb = reinterpret_cast<float2*>(sm.part + kPartF4 * (lane >> 1)) + (odd ? 1 : 0);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float lo = v[2 * j], hi = v[2 * j + 1];
      const float o_lo = __shfl_xor_sync(0xffffffffu, lo, 1);
      const float o_hi = __shfl_xor_sync(0xffffffffu, hi, 1);
      pb[2 * j] = odd ? make_float2(o_hi, hi) : make_float2(lo, o_lo);
    }
  }
  __syncwarp();
  // the source charge that makes a pair "same species" for this target, and
  // the FP32 screening constants of the special-pair test
  const float tq = tsp ? 1.f : -1.f;
  const float il2_to_e = PHYS == 1 ? (tsp ? sm.pk[1] : sm.pk[0]) : 0.f;  // electron source
  const float il2_to_i = PHYS == 1 ? (tsp ? sm.pk[2] : sm.pk[1]) : 0.f;  // ion source
  const float rs2 = sm.pk[3] * sm.pk[3];
  // one test sends a pair to the exact offsets or a special law: the largest
  // squared distance at which any of them could apply (1.01: its rounding)
  const float near2 =
      fmaxf(close2, 1.01f * (PHYS == 1 ? 40.f / fminf(il2_to_e, il2_to_i)
                                       : fmaxf(0.01f, 400.f / rs2)));
  // RDF counts of the other pairs: bin = trunc(r * rdf_inv), read off the low
  // bits of r * rdf_inv + 2^23 (rounded towards zero; + the ii histogram's
  // offset); a scale of 1e30 puts pairs that are not counted (electrons for an
  // electron target, every pair of an idle lane) beyond the last bin
  float inv_i = 1e30f, inv_e = 1e30f, bin_i = 8388608.f;
  uint32_t hist_at = 0;
  if (RDF) {
    if (act) inv_i = tsp ? a.dx_ii_inv_f : a.dx_ei_inv_f;
    if (act && tsp) inv_e = a.dx_ei_inv_f;
    if (tsp) bin_i += (float)kRdfBins;
    // (0x4B000000 + bin) * 4 + hist_at = address of the bin, modulo 2^32
    hist_at = (uint32_t)__cvta_generic_to_shared(hist) - (0x4B000000u << 2);
  }
  const float2 thx2 = make_float2(thx, thx), thy2 = make_float2(thy, thy), thz2 = make_float2(thz, thz);
  float2 fx = make_float2(0.f, 0.f), fy = fx, fz = fx, pa = fx, pq = fx;
  const int npair = (cnt + 1) >> 1;
#pragma unroll 1
  for (int b = 0; b < npair; ++b) {
    const float4* blk = sm.part + kPartF4 * b;
    const float4 q0 = blk[0], q1 = blk[1];
    const float2 q = make_float2(q1.z, q1.w);  // source charges: -1 e, +1 ion
    float2 dx = __fadd2_rn(thx2, make_float2(q0.x, q0.y));
    float2 dy = __fadd2_rn(thy2, make_float2(q0.z, q0.w));
    float2 dz = __fadd2_rn(thz2, make_float2(q1.x, q1.y));
    float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
    if (fminf(r2.x, r2.y) > near2) {
      const float2 rinv = make_float2(rsqrt_normal(r2.x), rsqrt_normal(r2.y));
      const float2 ph = __fmul2_rn(q, rinv);
      const float2 fs = __fmul2_rn(ph, __fmul2_rn(rinv, rinv));
      fx = __ffma2_rn(fs, dx, fx);
      fy = __ffma2_rn(fs, dy, fy);
      fz = __ffma2_rn(fs, dz, fz);
      pa = __fadd2_rn(pa, ph);
      pq = __ffma2_rn(q, ph, pq);
      if (RDF) {
        const bool i0 = q.x > 0.f, i1 = q.y > 0.f;
        const float2 t = __fmul2_rn(__fmul2_rn(r2, rinv),
                                    make_float2(i0 ? inv_i : inv_e, i1 ? inv_i : inv_e));
        const float b0 = __fadd_rz(t.x, i0 ? bin_i : 8388608.f);
        const float b1 = __fadd_rz(t.y, i1 ? bin_i : 8388608.f);
        if (t.x < (float)kRdfBins) rdf_inc(hist_at + 4u * __float_as_uint(b0));
        if (t.y < (float)kRdfBins) rdf_inc(hist_at + 4u * __float_as_uint(b1));
      }
      continue;
    }
    int s0 = -1, s1 = -1;
    if (r2.x <= close2 || r2.y <= close2) {
      // close pair: the exact offsets (hi + lo) and the source indices
      const float4 q2 = blk[2], q3 = blk[3];
      dx = __fadd2_rn(__fadd2_rn(thx2, make_float2(q0.x, q0.y)),
                      __fadd2_rn(make_float2(tlx, tlx), make_float2(q2.x, q2.y)));
      dy = __fadd2_rn(__fadd2_rn(thy2, make_float2(q0.z, q0.w)),
                      __fadd2_rn(make_float2(tly, tly), make_float2(q2.z, q2.w)));
      dz = __fadd2_rn(__fadd2_rn(thz2, make_float2(q1.x, q1.y)),
                      __fadd2_rn(make_float2(tlz, tlz), make_float2(q3.x, q3.y)));
      r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
      s0 = __float_as_int(q3.z);
      s1 = __float_as_int(q3.w);
    }
    bool sp0, sp1;
    if (PHYS == 1) {
      sp0 = r2.x * (q.x < 0.f ? il2_to_e : il2_to_i) < 40.f;
      sp1 = r2.y * (q.y < 0.f ? il2_to_e : il2_to_i) < 40.f;
    } else {
      sp0 = q.x == tq ? !(r2.x > 0.01f) : r2.x * rs2 < 400.f;
      sp1 = q.y == tq ? !(r2.y > 0.01f) : r2.y * rs2 < 400.f;
    }
    const float2 rinv = make_float2(rsqrtf(r2.x), rsqrtf(r2.y));
    if (!(sp0 || sp1)) {
      const float2 ph = __fmul2_rn(q, rinv);
      const float2 fs = __fmul2_rn(ph, __fmul2_rn(rinv, rinv));
      fx = __ffma2_rn(fs, dx, fx);
      fy = __ffma2_rn(fs, dy, fy);
      fz = __ffma2_rn(fs, dz, fz);
      pa = __fadd2_rn(pa, ph);
      pq = __ffma2_rn(q, ph, pq);
    } else {
      p2p_one<PHYS>(sm, r2.x, dx.x, dy.x, dz.x, q.x, s0, p_self, tsp,
                    fx.x, fy.x, fz.x, pa.x, pq.x);
      p2p_one<PHYS>(sm, r2.y, dx.y, dy.y, dz.y, q.y, s1, p_self, tsp,
                    fx.y, fy.y, fz.y, pa.y, pq.y);
    }
    if (RDF && act) rdf_count2<PHYS>(a, hist, r2, rinv, q, s0, s1, p_self, tsp);
  }
  __syncwarp();
  out.fx = fx.x + fx.y;
  out.fy = fy.x + fy.y;
  out.fz = fz.x + fz.y;
  const double pad = (double)pa.x + (double)pa.y, pqd = (double)pq.x + (double)pq.y;
  out.pa = pad;
  out.pi = 0.5 * (pad + pqd);  // ion sources: (all + charge-weighted) / 2
}

// max(v, 0) of a finite number: three instructions instead of fmax's five.
__device__ __forceinline__ double clamp0(double v) { return __double2hiint(v) < 0 ? 0.0 : v; }

// Squared distance from a cell's centroid to the group's box, in an
// operation order pinned against contraction: the network batch recomputes
// it for its candidates and must see the value the walk's test saw.
__device__ __forceinline__ double box_dist2(const double4& c, const WarpSmem& sm) {
  const double ex = clamp0(fabs(c.x - sm.gx) - sm.bx);
  const double ey = clamp0(fabs(c.y - sm.gy) - sm.by);
  const double ez = clamp0(fabs(c.z - sm.gz) - sm.bz);
  return __dadd_rn(__dadd_rn(__dmul_rn(ex, ex), __dmul_rn(ey, ey)), __dmul_rn(ez, ez));
}

// ------------------------------------------------------ learned MAC ----
// One batch of queued candidates (lane < nb holds one) through the network.
// Returns 1 (accept) or 3 (open) for a candidate, 0 otherwise, plus 4 when
// its features fell outside the training range (the fixed decision, open,
// stands).  Out of line: it runs once per 32 candidates, and the network's
// fragments then take no registers from the walk loop around the call.
// A candidate's distance d and budget B = log10(budget d^2 / n) (the label's
// units) are recomputed here as the walk's test formed them.
__device__ __noinline__ int mac_batch(const double4* __restrict__ node_c,
                                      const float4* __restrict__ geom,
                                      const float4* __restrict__ mom,
                                      const float4* __restrict__ mom3, WarpSmem& sm,
                                      const MlpPacked* mlp, const float* frange, int node,
                                      bool cand, float n_act, int lane) {
  float* feat = reinterpret_cast<float*>(sm.cell) + lane * kMacFeatures;
  float cand_B = 0.f;
  if (cand) {
    const double4 c = ldg_d4(&node_c[node]);
    const float4 g4 = __ldg(&geom[node]);
    const float ddf = sqrtf((float)box_dist2(c, sm));
    cand_B = sm.lbud + 2.f * __log10f(ddf) - log10f(g4.z);
    const float4* mp = mom + 3 * (int64_t)node;
    const float4* tp = mom3 + 3 * (int64_t)node;
    mac_features(c.x, c.y, c.z, g4, __ldg(mp), __ldg(mp + 1), __ldg(mp + 2), __ldg(tp),
                 __ldg(tp + 1), __ldg(tp + 2), sm.gx, sm.gy, sm.gz, (float)sqrt(sm.hl2), ddf,
                 n_act, feat);
  } else {
#pragma unroll
    for (int k = 0; k < kMacFeatures; ++k) feat[k] = 0.f;
  }
  // range check on the raw features before the network normalises them
  bool in_range = true;
#pragma unroll
  for (int k = 0; k < kMacFeatures; ++k)
    in_range = in_range && feat[k] >= frange[k] && feat[k] <= frange[kMacFeatures + k];
  __syncwarp();
  const float y = mlp_forward_warp(reinterpret_cast<float*>(sm.cell), *mlp, lane);
  if (!cand) return 0;
  // predicted |dF| = 10^y * n / d^2 against the group's budget; out of the
  // training range the fixed-theta decision (open) stands
  return ((in_range && y <= cand_B) ? 1 : 3) | (in_range ? 0 : 4);
}

// Per cell, for the nodes [0, bounds[2]) of this build: its part K of the
// learned pre-filter (mac_node_term) and the distance s / rho_hi + dx inside
// which it lies outside the criterion's band.  Leaves are never tested; their
// records are not read.
__global__ void k_mac_node_terms(const float4* __restrict__ geom,
                                 const float4* __restrict__ mom3,
                                 const int32_t* __restrict__ bounds,
                                 const float* __restrict__ margins, float inv_rho_hi,
                                 float2* __restrict__ mac_k) {
  const int end = bounds[2];
  float c[kEstCoef];
#pragma unroll
  for (int k = 0; k < kEstCoef; ++k) c[k] = __ldg(&margins[2 + k]);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < end; i += gridDim.x * blockDim.x) {
    const float4 g4 = __ldg(&geom[i]);
    mac_k[i] = make_float2(mac_node_term(g4, __ldg(&mom3[3 * (int64_t)i + 2]).z, c),
                           fmaf(g4.x, inv_rho_hi, g4.y));
  }
}

// --------------------------------------------------------------- walk ----
// Dynamic shared memory: WarpSmem per warp, then (learned MAC only) the
// features' training range and, without RDF counts, the packed network, then
// (RDF only) the two block histograms.  With RDF counts the network stays in
// global memory: it is read once per 32 candidates, and its 11 KB bring the
// block under the step at which the SM keeps 60 KB of L1 instead of 28 KB.
constexpr size_t kFrangeBytes = sizeof(float) * (2 * kMacFeatures + 8);
template <bool LEARNED, bool RDF>
constexpr size_t walk_learned_bytes() {
  return LEARNED ? (kFrangeBytes + (RDF ? 0 : sizeof(MlpPacked)) + 15) / 16 * 16 : 0;
}
template <bool LEARNED, bool RDF>
constexpr size_t walk_smem_bytes(int warps) {
  return sizeof(WarpSmem) * warps + walk_learned_bytes<LEARNED, RDF>() +
         (RDF ? sizeof(uint32_t) * 2 * kRdfBins : 0);
}
constexpr size_t kTeamBytes = sizeof(TeamSmem) * (16 / kTeamMin);  // the most a launch takes
static_assert(walk_smem_bytes<true, true>(16) + kTeamBytes <= 227 * 1024, "team walk over 227 KB");
static_assert(walk_smem_bytes<true, true>(16) <= 195 * 1024, "RDF walk over the 196 KB step");
static_assert(walk_smem_bytes<false, false>(20) <= 163 * 1024, "walk over the 164 KB step");

__device__ __forceinline__ void team_sync(int team, int warps) {
  asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "r"(32 * warps) : "memory");
}

template <int PHYS, bool RDF, bool LEARNED, int ORDER, bool TEAM>
__global__ void __launch_bounds__(32 * (TEAM ? 16 : walk_warps<RDF, LEARNED>()), 1)
    k_walk_mixed(MixedArgs a) {
  extern __shared__ float4 dyn_smem[];
  WarpSmem* smem = reinterpret_cast<WarpSmem*>(dyn_smem);
  const int nwarps = blockDim.x >> 5;
  unsigned char* tail = reinterpret_cast<unsigned char*>(smem + nwarps);
  // training range of the features (fmin | fmax), then m_lo, m_hi and the
  // pre-filter coefficients, shared by the block
  float* frange = reinterpret_cast<float*>(tail);
  const float* fmodel = frange + 2 * kMacFeatures;
  MlpPacked* mlp_s = reinterpret_cast<MlpPacked*>(tail + kFrangeBytes);
  const MlpPacked* mlp = RDF ? a.packed : mlp_s;
  uint32_t* hist = reinterpret_cast<uint32_t*>(tail + walk_learned_bytes<LEARNED, RDF>());
  const int lane = threadIdx.x & 31;
  const int wib = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);  // known to be warp-uniform
  WarpSmem& sm = smem[wib];
  // this warp's team, and its rank in it (0: the leader)
  const int team = TEAM ? wib / a.team : wib, rank = TEAM ? wib & (a.team - 1) : 0;
  const int nteams = TEAM ? nwarps / a.team : nwarps;
  TeamSmem& ts = reinterpret_cast<TeamSmem*>(
      tail + walk_learned_bytes<LEARNED, RDF>() + (RDF ? sizeof(uint32_t) * 2 * kRdfBins : 0))[team];
  if (RDF) {
    for (int i = threadIdx.x; i < 2 * kRdfBins; i += blockDim.x) hist[i] = 0u;
    __syncthreads();
  }
  if (LEARNED) {
    if (!RDF) {
      const uint32_t* src = reinterpret_cast<const uint32_t*>(a.packed);
      uint32_t* dst = reinterpret_cast<uint32_t*>(mlp_s);
      for (int i = threadIdx.x; i < (int)(sizeof(MlpPacked) / 4); i += blockDim.x) dst[i] = src[i];
    }
    if (threadIdx.x < kMacFeatures) {
      frange[threadIdx.x] = __ldg(&a.fmin[threadIdx.x]);
      frange[kMacFeatures + threadIdx.x] = __ldg(&a.fmax[threadIdx.x]);
    }
    if (threadIdx.x < 2 + kEstCoef)
      frange[2 * kMacFeatures + threadIdx.x] = __ldg(&a.margins[threadIdx.x]);
    __syncthreads();
  }
  const int gwarp = blockIdx.x * nwarps + wib;
  int32_t* stack = a.stack + (int64_t)gwarp * kStackCap;
  const unsigned lt = (1u << lane) - 1u;
  if (*((volatile int32_t*)a.err) & (kErrCapacity | kErrDepth | kErrNonFinite)) return;
  const int root_end = a.bounds[2];  // combined tree: nodes [0, root_end)
  const int ngroups = *a.n_groups;
  int max_stack = 0;
  // The first group of each warp is fixed, spread over the SMs before the warps
  // of an SM: with fewer groups than warps, a cursor alone gives them all to
  // the blocks that start first (N = 32,768 kept 55 of the 148 SMs busy).
  int g = team * gridDim.x + blockIdx.x;
  for (bool own = true; root_end > 0; own = false) {
    if (!own) {
      if (lane == 0 && rank == 0) g = gridDim.x * nteams + atomicAdd(&a.control[0], 1);
      if (TEAM) {
        if (lane == 0 && rank == 0) ts.item = g;
        __syncwarp();
        team_sync(team, a.team);
        g = ts.item;
      } else {
        g = __shfl_sync(0xffffffffu, g, 0);
      }
    }
    if (g >= ngroups) break;
    const int2 grp = a.groups[g];
    const int p0 = grp.x, n_act = grp.y;
    const bool act = lane < n_act;
    const int pt = p0 + (act ? lane : n_act - 1);
    const double4 xt = a.xs[pt];
    const int tsp = xt.w > 0.5 ? 1 : 0;  // this lane's target species
    const double mnx = warp_min_d(xt.x), mny = warp_min_d(xt.y), mnz = warp_min_d(xt.z);
    const double mxx = warp_max_d(xt.x), mxy = warp_max_d(xt.y), mxz = warp_max_d(xt.z);
    const double Gx = 0.5 * (mnx + mxx), Gy = 0.5 * (mny + mxy), Gz = 0.5 * (mnz + mxz);
    const double hx = 0.5 * (mxx - mnx), hy = 0.5 * (mxy - mny), hz = 0.5 * (mxz - mnz);
    const double rtx = xt.x - Gx, rty = xt.y - Gy, rtz = xt.z - Gz;
    const float thx = (float)rtx, thy = (float)rty, thz = (float)rtz;
    const float tlx = (float)(rtx - (double)thx), tly = (float)(rty - (double)thy),
                tlz = (float)(rtz - (double)thz);
    // pairs closer than h / sqrt(32) (h the group's half-diagonal) take the
    // exact offsets (eval_p2p)
    const double hl2 = hx * hx + hy * hy + hz * hz;
    const float close2 = (float)(hl2 * (1.0 / 32.0));
    if (lane == 0) {
      sm.hl2 = hl2;
      sm.gx = Gx;
      sm.gy = Gy;
      sm.gz = Gz;
      sm.bx = hx;
      sm.by = hy;
      sm.bz = hz;
    }
    Acc acc{0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    sm.phi[lane] = make_double2(0.0, 0.0);
    // error budget of the learned MAC: eta * min |F_prev| / eps over the group
    if (LEARNED) {
      const int64_t o = a.order[pt];
      const double fx = a.f_prev[3 * o], fy = a.f_prev[3 * o + 1], fz = a.f_prev[3 * o + 2];
      float fm = act ? (float)sqrt(fx * fx + fy * fy + fz * fz) : 3.0e38f;
      for (int o2 = 16; o2 > 0; o2 >>= 1) fm = fminf(fm, __shfl_xor_sync(0xffffffffu, fm, o2));
      const float budget = a.eta_over_eps * fm;
      if (lane == 0) {
        sm.lbud = budget > 0.f ? log10f(budget) : -INFINITY;
        sm.n_mlp = 0u;
        sm.n_fallback = 0u;
      }
    }
    int ssize = 1;
    // the group's tree: its cloud's root and pair constants
    int root = 0;
    if (a.nseg > 0) {
      int c = 0;
      if (lane == 0) {
        int lo = 0, hi = a.nseg - 1;  // largest c with start[c] <= p0
        while (lo < hi) {
          const int mid = (lo + hi + 1) >> 1;
          if (__ldg(&a.ens_start[mid]) <= p0) lo = mid;
          else hi = mid - 1;
        }
        c = lo;
      }
      c = __shfl_sync(0xffffffffu, c, 0);
      root = __ldg(&a.roots[c]);
      if (lane < 8) sm.pk[lane] = __ldg(reinterpret_cast<const float*>(a.cloud_pk + 2 * c) + lane);
    } else if (lane == 0) {
      sm.pk[0] = a.inv_lam2_ee;
      sm.pk[1] = a.inv_lam2_ei;
      sm.pk[2] = a.inv_lam2_ii;
      sm.pk[3] = a.rs_inv;
      sm.pk[4] = a.inv_lam_ee;
      sm.pk[5] = a.inv_lam_ei;
      sm.pk[6] = a.inv_lam_ii;
      sm.pk[7] = 0.f;
    }
    if (lane == 0) stack[0] = root;
    __syncwarp();
    int m2h = 0, m2t = 0;  // ring head/tail (warp-uniform)
    int p2n = 0, p2tot = 0;  // particle entries waiting, evaluated
    int lch = 0, lct = 0;                    // local-expansion ring
    float lsum = 0.f;  // lanes below kLocCoef: one summed coefficient of the expansion
    bool overflow = false;
    int cqh = 0, cqt = 0;  // learned-MAC candidate ring (warp-uniform)
    bool fin = false;  // the walk has ended: what is left of the lists is next
    int qn = 0;  // TEAM: batches in the queue
    while (TEAM || !fin) {
      // ---- a batch of nodes (TEAM: until a round's worth of work waits) ----
      while (rank == 0 && !fin && (!TEAM || qn < a.team)) {
        int node = -1;
        int action = 0, pfirst = 0, pcnt = 0;  // 1 far field, 2 particles, 3 open
        if (LEARNED && (cqt - cqh >= 32 || (ssize == 0 && cqt > cqh))) {
          // ---- a batch of queued candidates goes through the network ----
          const int nb = min(32, cqt - cqh);
          const bool cand = lane < nb;
          if (cand) node = sm.cq_node[(cqh + lane) & (kCandRing - 1)];
          cqh += nb;
          __syncwarp();
          const int r = mac_batch(a.node_c, a.geom, a.mom, a.mom3, sm, mlp, frange, node, cand,
                                  (float)n_act, lane);
          if (cand) action = r & 3;  // candidates exceed a bucket: accept or open
          const unsigned fbm = __ballot_sync(0xffffffffu, (r & 4) != 0);
          if (lane == 0) {
            sm.n_mlp += (unsigned)nb;
            sm.n_fallback += (unsigned)__popc(fbm);
          }
        } else {
          // ---- a batch of nodes from the stack ----
          const int nb = min(32, ssize);
          node = lane < nb ? stack[ssize - 1 - lane] : -1;
          ssize -= nb;
          __syncwarp();
          bool cand = false;  // queued for the learned MAC
          if (node >= 0) {
            // the particle range and (learned criterion) the cell's pre-filter
            // record depend on the node index alone: issued with node_c, so a
            // batch waits for one round of loads instead of two or three
            const double4 c = ldg_d4(&a.node_c[node]);
            const int cnt = __ldg(&a.count[node]);
            const int fst = __ldg(&a.first[node]);
            const float2 kr = LEARNED ? __ldg(&a.mac_k[node]) : make_float2(0.f, 0.f);
            if (c.w < 0.0) {
              action = 2;
              pfirst = fst;
              pcnt = 1;
            } else {
              // group MAC: rcrit below the distance from the centroid to the box
              const double d2 = box_dist2(c, sm);
              bool accept = c.w * c.w < d2;  // the fixed-theta test
              if (LEARNED && !accept) {
                // learned criterion, on top of the fixed test: a cell the fixed
                // test opens is accepted anyway when its predicted acceptance
                // error is within the group's budget.  rho = s / (d - dx) places
                // it against the training band; est is the fitted log-linear
                // estimate of the label (mac.cuh) and B the budget in the same
                // units.  Cells whose estimate is clearly on one side of B
                // (training quantiles m_lo, m_hi of label - est) are decided at
                // once; the rest are queued for the network.  Only cells that
                // would otherwise open into more than a bucket of particle
                // pairs are worth a far-field evaluation.
                // rho = s / (d - dx) <= rho_hi  <=>  d >= s / rho_hi + dx
                const float d2f = (float)d2;
                if (d2f >= kr.y * kr.y && cnt > a.bucket) {
                  const float ddf = sqrtf(d2f);
                  // est - B = K - log10(budget) - (2 + c0) log10(d); no
                  // budget: log10(budget) = -inf, never accepted or queued
                  const float lb = sm.lbud, l10d = __log10f(ddf);
                  const float eb = fmaf(-(2.f + fmodel[2]), l10d, kr.x - lb);
                  if (eb + fmodel[1] <= 0.f) {
                    accept = true;
                  } else if (eb + fmodel[0] <= 0.f) {
                    cand = true;
                  }
                }
              }
              // a small accepted cell is cheaper and exact as particle pairs: an
              // M2P costs about as much as p2p_max pair interactions
              if (accept && cnt <= a.p2p_max) {
                action = 2;
                pfirst = fst;
                pcnt = cnt;
              } else if (accept) {
                action = 1;
                if (a.loc_eps2 > 0.0) {
                  // far from the group: summed into its local expansion
                  const double ux = c.x - sm.gx, uy = c.y - sm.gy, uz = c.z - sm.gz;
                  const double dc2 = ux * ux + uy * uy + uz * uz;
                  if (sm.hl2 <= a.loc_eps2 * dc2) action = 4;
                }
              } else if (!cand) {
                if (cnt <= a.bucket) {
                  action = 2;
                  pfirst = fst;
                  pcnt = cnt;
                } else {
                  action = 3;
                }
              }
            }
          }
          if (LEARNED) {
            const unsigned cm = __ballot_sync(0xffffffffu, cand);
            if (cand) {
              const int q = (cqt + __popc(cm & lt)) & (kCandRing - 1);
              sm.cq_node[q] = node;
            }
            cqt += __popc(cm);
          }
        }
        // far-field entries
        const unsigned bm = __ballot_sync(0xffffffffu, action == 1);
        if (action == 1) sm.m2p[(m2t + __popc(bm & lt)) & (kM2pRing - 1)] = node;
        m2t += __popc(bm);
        // local-expansion entries
        const unsigned lm = __ballot_sync(0xffffffffu, action == 4);
        if (action == 4) sm.loc[(lct + __popc(lm & lt)) & (kLocRing - 1)] = node;
        lct += __popc(lm);
        // opened twigs push their children (octant order)
        int4 k0 = make_int4(-1, -1, -1, -1), k1 = k0;
        if (action == 3) {
          const int4* kk = reinterpret_cast<const int4*>(a.kids + 8 * (int64_t)node);
          k0 = __ldg(kk);
          k1 = __ldg(kk + 1);
        }
        const int kv[8] = {k0.x, k0.y, k0.z, k0.w, k1.x, k1.y, k1.z, k1.w};
        int kc = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) kc += kv[j] >= 0 ? 1 : 0;
        // particle entries (at most 8 a lane) and children in one scan; the
        // traversal is bound by its instructions, a quarter of the walk's time
        // (L1 prefetches of the next nodes made it 2 % slower)
        const int mine = (kc << 16) | (action == 2 ? pcnt : 0);
        const int upto = warp_incl_scan(mine);
        const int tot = __shfl_sync(0xffffffffu, upto, 31);
        const int ptot = tot & 0xffff, ktot = tot >> 16;
        const int pex = (upto - mine) & 0xffff, kex = (upto - mine) >> 16;
        const int pmine = mine & 0xffff;
#pragma unroll
        for (int k = 0; k < kMaxBucket; ++k)
          if (k < pmine) sm.p2p[p2n + pex + k] = pfirst + k;
        p2n += ptot;
        if (ssize + ktot > kStackCap) {
          overflow = fin = true;
          qn = 0;
          break;
        }
        {
          int pos = ssize + kex;
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (kv[j] >= 0) stack[pos++] = kv[j];
        }
        ssize += ktot;
        max_stack = max(max_stack, ssize);
        __syncwarp();
        // remainders come after every full batch, in the order of the sums: a
        // walk that ends on a full far-field batch takes an empty turn more
        fin = ssize == 0 && cqt == cqh && m2t - m2h < 32;
        if (!TEAM) break;
        // full batches, and what is left once the walk has ended, to the queue
        int p2h = 0;
        while (p2n - p2h >= 32 || (fin && p2n > p2h)) {
          const int cnt = min(32, p2n - p2h);
          if (lane < cnt) ts.idx[qn][lane] = sm.p2p[p2h + lane];
          if (lane == 0) ts.info[qn] = 4 * cnt + 2;
          ++qn;
          p2h += cnt;
        }
        p2tot += p2h;
        p2n -= p2h;
        if (p2h > 0) {  // the remainder moves to the front
          const int e = lane < p2n ? sm.p2p[p2h + lane] : 0;
          __syncwarp();
          if (lane < p2n) sm.p2p[lane] = e;
        }
        while (m2t - m2h >= 32 || (fin && m2t > m2h)) {
          const int cnt = min(32, m2t - m2h);
          if (lane < cnt) ts.idx[qn][lane] = sm.m2p[(m2h + lane) & (kM2pRing - 1)];
          if (lane == 0) ts.info[qn] = 4 * cnt + 1;
          ++qn;
          m2h += cnt;
        }
        while (lct - lch >= 32 || (fin && lct > lch)) {
          const int cnt = min(32, lct - lch);
          if (lane < cnt) ts.idx[qn][lane] = sm.loc[(lch + lane) & (kLocRing - 1)];
          if (lane == 0) ts.info[qn] = 4 * cnt + 3;
          ++qn;
          lch += cnt;
        }
        __syncwarp();
      }
      // ---- evaluation: full batches of 32, and what is left once the walk has
      // ended.  One call site each: this is long straight-line code, and the
      // warps of an SM are in different parts of it. ----
      if (!TEAM && overflow) break;
      int take = 0, kind = 0, cnt = 0;
      Batch out;
      if (TEAM) out = {0.f, 0.f, 0.f, 0.f, 0.0, 0.0};
      int p2h = 0;
      if (TEAM) {
        if (rank == 0) {
          take = min(qn, a.team);
          if (lane == 0) ts.take = take;
        }
        __syncwarp();
        team_sync(team, a.team);
        take = ts.take;
        if (take == 0) break;
        if (rank < take) {
          kind = ts.info[rank] & 3;
          cnt = ts.info[rank] >> 2;
        }
      }
      while (TEAM ? kind == 2 : p2n - p2h >= 32 || (fin && p2n > p2h)) {
        if (!TEAM) cnt = min(32, p2n - p2h);
        eval_p2p<PHYS, RDF>(sm, TEAM ? ts.idx[rank] : sm.p2p + p2h, cnt, a, sm.gx, sm.gy, sm.gz,
                            thx, thy, thz, tlx, tly, tlz, close2, pt, tsp, act, lane, hist, out);
        if (TEAM) break;
        batch_add(sm, lane, acc, out);
        p2h += cnt;
      }
      if (!TEAM && p2h > 0) {  // the remainder moves to the front
        p2tot += p2h;
        p2n -= p2h;
        const int e = lane < p2n ? sm.p2p[p2h + lane] : 0;
        __syncwarp();
        if (lane < p2n) sm.p2p[lane] = e;
        __syncwarp();
      }
      while (TEAM ? kind == 1 : m2t - m2h >= 32 || (fin && m2t > m2h)) {
        if (!TEAM) cnt = min(32, m2t - m2h);
        eval_m2p<ORDER, RDF>(sm, TEAM ? ts.idx[rank] : sm.m2p, TEAM ? 31 : kM2pRing - 1, TEAM ? 0 : m2h,
                        cnt, a, sm.gx, sm.gy, sm.gz, thx, thy, thz, lane, out);
        if (TEAM) break;
        batch_add(sm, lane, acc, out);
        m2h += cnt;
      }
      while (TEAM ? kind == 3 : lct - lch >= 32 || (fin && lct > lch)) {
        if (!TEAM) cnt = min(32, lct - lch);
        eval_local<ORDER>(sm, TEAM ? ts.idx[rank] : sm.loc, TEAM ? 31 : kLocRing - 1,
                          TEAM ? 0 : lch, cnt, a, sm.gx, sm.gy, sm.gz, lane, out);
        if (TEAM) break;
        lsum += out.loc;
        lch += cnt;
      }
      if (TEAM) {
        // results stay in each warp's staging buffer until the leader has them
        if (rank < take) reinterpret_cast<Batch*>(sm.cell)[lane] = out;
        __syncwarp();
        team_sync(team, a.team);
        if (rank == 0) {
          for (int j = 0; j < take; ++j) {
            const Batch b = reinterpret_cast<const Batch*>(smem[wib + j].cell)[lane];
            if ((ts.info[j] & 3) == 3) lsum += b.loc;
            else batch_add(sm, lane, acc, b);
          }
          qn -= take;
          for (int j = 0; j < qn; ++j) {  // what is left of the queue moves up
            const int e = ts.idx[j + take][lane], f = ts.info[j + take];
            __syncwarp();
            ts.idx[j][lane] = e;
            if (lane == 0) ts.info[j] = f;
            __syncwarp();
          }
        }
      }
    }
    if (TEAM && rank != 0) continue;
    if (overflow) {
      if (lane == 0) set_error(a.err, kErrWalk);
      continue;
    }
    if (lct > 0) {
      // every target evaluates the group's summed local expansion
      if (lane < kLocCoef) sm.loc_rows[lane] = lsum;
      __syncwarp();
      float lfx, lfy, lfz, lph, lpi;
      local_eval(sm.loc_rows, thx, thy, thz, lfx, lfy, lfz, lph, lpi);
      __syncwarp();
      kahan_add(acc.sx, acc.cx, lfx);
      kahan_add(acc.sy, acc.cy, lfy);
      kahan_add(acc.sz, acc.cz, lfz);
      phi_add(sm, lane, (double)lph, (double)lpi);
    }
    if (act) {
      const double sc = tsp ? kEps : -kEps;  // eps * target charge
      const int64_t o = a.order[pt];
      a.f[3 * o] = sc * ((double)acc.sx - (double)acc.cx);
      a.f[3 * o + 1] = sc * ((double)acc.sy - (double)acc.cy);
      a.f[3 * o + 2] = sc * ((double)acc.sz - (double)acc.cz);
      const double2 phi = sm.phi[lane];
      const double all = 0.5 * sc * phi.x;
      const double from_i = 0.5 * sc * phi.y;
      // Epot_e = ee + ie + ei, Epot_i = ii (tree.f90:674-715)
      a.epot_part[o] = tsp ? make_double2(all - from_i, from_i)
                           : make_double2(all, 0.0);
    }
    if (lane == 0) {
      // every queued entry was evaluated: the ring tails are the counts
      atomicAdd(&a.counters[0], (unsigned long long)m2t * n_act);
      atomicAdd(&a.counters[1], (unsigned long long)p2tot * n_act);
      if (lct > 0) atomicAdd(&a.counters[8], (unsigned long long)lct);
    }
    if (LEARNED) {
      if (lane == 0) {
        atomicAdd(&a.counters[2], (unsigned long long)sm.n_mlp);
        atomicAdd(&a.counters[3], (unsigned long long)sm.n_fallback);
      }
    }
  }
  if (lane == 0) atomicMax(&a.control[1], max_stack);
  if (RDF) {
    // every warp of the block has left the group loop: add the block's bins
    __syncthreads();
    for (int i = threadIdx.x; i < 2 * kRdfBins; i += blockDim.x) {
      const uint32_t v = hist[i];
      if (v) atomicAdd(&a.rdf[i], v);
    }
  }
}

// ------------------------------------------------------------- memory ----
template <class T>
static int realloc_dev(T** p, size_t count) {
  if (*p) cudaFree(*p);
  *p = nullptr;
  if (count == 0) count = 1;
  return cudaMalloc((void**)p, count * sizeof(T)) == cudaSuccess ? 0 : 1;
}

int mixed_alloc_nodes(MixedBuffers& mb, int cap) {
  mb.cap = cap;
  int rc = 0;
  rc |= realloc_dev(&mb.kids, 8 * (size_t)cap);
  rc |= realloc_dev(&mb.first, (size_t)cap);
  rc |= realloc_dev(&mb.count, (size_t)cap);
  rc |= realloc_dev(&mb.digit, (size_t)cap);
  rc |= realloc_dev(&mb.m64, (size_t)kM64 * cap);
  rc |= realloc_dev(&mb.mom3, 3 * (size_t)cap);
  rc |= realloc_dev(&mb.mom4, 3 * (size_t)cap);
  rc |= realloc_dev(&mb.mom, 3 * (size_t)cap);
  rc |= realloc_dev(&mb.geom, (size_t)cap);
  rc |= realloc_dev(&mb.mac_k, (size_t)cap);
  rc |= realloc_dev(&mb.lvl_list, (size_t)cap);
  rc |= realloc_dev(&mb.cls, (size_t)net_cls_entries(cap));
  return rc;
}

int mixed_alloc_particles(MixedBuffers& mb, int n) {
  mb.n = n;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  mb.sms = sms;
  mb.grid_warps = sms * kStackWarps;
  int rc = 0;
  rc |= realloc_dev(&mb.xs, (size_t)n);
  rc |= realloc_dev(&mb.groups, (size_t)n);
  rc |= realloc_dev(&mb.stack, (size_t)mb.grid_warps * kStackCap);
  rc |= realloc_dev(&mb.control, 4);
  rc |= realloc_dev(&mb.lvl, 3 * (size_t)kLevelSlots);
  return rc;
}

void mixed_free(MixedBuffers& mb) {
  void* ptrs[] = {mb.kids, mb.first, mb.count, mb.digit, mb.m64, mb.mom,
                  mb.mom3, mb.mom4, mb.geom, mb.mac_k, mb.xs, mb.groups, mb.stack, mb.control,
                  mb.lvl_list, mb.lvl, mb.cls};
  for (void* p : ptrs)
    if (p) cudaFree(p);
  mb = MixedBuffers();
}

MixedNodes mixed_nodes(const MixedBuffers& mb) {
  MixedNodes m;
  m.kids = mb.kids;
  m.first = mb.first;
  m.count = mb.count;
  m.digit = mb.digit;
  m.m64 = mb.m64;
  m.mom = mb.mom;
  m.mom3 = mb.mom3;
  m.mom4 = mb.mom4;
  m.geom = mb.geom;
  m.xs = mb.xs;
  m.groups = mb.groups;
  m.n_groups = mb.control + 2;
  m.lvl_list = mb.lvl_list;
  m.lvl = mb.lvl;
  m.cls = mb.cls;
  return m;
}

int walk_mixed(MixedBuffers& mb, const BuildBuffers& b, int n,
               const TreeView& tv, const WalkParams& wp,
               const MixedTuning& tune, const LearnedMac* learned,
               const Ensemble& ens, const float4* cloud_pk,
               double* f, double2* epot_part,
               uint32_t* rdf, unsigned long long* counters, int32_t* err,
               cudaStream_t st) {
  if (n == 0) return 0;
  MixedArgs a;
  a.node_c = tv.node_c;
  a.mom = mb.mom;
  a.kids = mb.kids;
  a.first = mb.first;
  a.count = mb.count;
  a.xs = mb.xs;
  a.order = b.vals;
  a.bounds = tv.tree_bounds;
  a.groups = mb.groups;
  a.n_groups = mb.control + 2;
  a.control = mb.control;
  a.stack = mb.stack;
  a.bucket = tune.bucket < 1 ? 1 : (tune.bucket > kMaxBucket ? kMaxBucket : tune.bucket);
  // an accepted cell of at most p2p_max particles is summed as pairs: with
  // the hexadecapole far field (measured at N = 1M, learned criterion) one
  // far-field evaluation costs about two pair interactions, at order 3 about
  // four
  a.p2p_max = tune.order >= 4 ? 2 : (tune.order == 3 ? 4 : 2);
  if (a.p2p_max > a.bucket) a.p2p_max = a.bucket;
  a.loc_eps2 = (double)tune.loc_eps * tune.loc_eps;
  a.inv_lam2_ee = (float)(1.0 / (wp.lam_ee * wp.lam_ee));
  a.inv_lam2_ei = (float)(1.0 / (wp.lam_ei * wp.lam_ei));
  a.inv_lam2_ii = (float)(1.0 / (wp.lam_ii * wp.lam_ii));
  a.inv_lam_ee = (float)(1.0 / wp.lam_ee);
  a.inv_lam_ei = (float)(1.0 / wp.lam_ei);
  a.inv_lam_ii = (float)(1.0 / wp.lam_ii);
  a.rs_inv = (float)(1.0 / wp.rs);
  a.dx_ei_inv_f = (float)(1.0 / wp.dx_ei);
  a.dx_ii_inv_f = (float)(1.0 / wp.dx_ii);
  a.f = f;
  a.epot_part = epot_part;
  a.rdf = rdf;
  a.counters = counters;
  a.err = err;
  // control[0] group cursor, [1] deepest stack; [2] (group count) is written
  // by the build
  cudaMemsetAsync(mb.control, 0, 2 * sizeof(int32_t), st);
  const bool L = learned != nullptr && learned->packed != nullptr &&
                 learned->f_prev != nullptr;
  a.packed = L ? learned->packed : nullptr;
  a.fmin = L ? learned->fmin : nullptr;
  a.fmax = L ? learned->fmax : nullptr;
  a.geom = mb.geom;
  a.mom3 = mb.mom3;
  a.mom4 = mb.mom4;
  a.margins = L ? learned->margins : nullptr;
  a.mac_k = mb.mac_k;
  a.f_prev = L ? learned->f_prev : nullptr;
  a.eta_over_eps = L ? (float)(learned->eta / kEps) : 0.f;
  a.nseg = ens.nseg;
  a.ens_start = ens.start;
  a.roots = ens.roots;
  a.cloud_pk = cloud_pk;
  // warps per SM: kWarpStep per unit of blocks_per_sm, up to what the build
  // holds (a fixed 16 with RDF counts)
  const int bps = tune.blocks_per_sm < 1 ? 1 : (tune.blocks_per_sm > kMaxBlocksPerSm ? kMaxBlocksPerSm : tune.blocks_per_sm);
  const bool r = rdf != nullptr;
  a.team = walk_team(n);
  if (L) k_mac_node_terms<<<mb.sms * 4, 256, 0, st>>>(mb.geom, mb.mom3, tv.tree_bounds,
                                                       learned->margins, 1.f / learned->rho_hi,
                                                       mb.mac_k);
  int dev = 0;
  cudaGetDevice(&dev);
#define TG_LAUNCH(P, R, LL, O, S)                                             \
  do {                                                                        \
    auto kfn = k_walk_mixed<P, R, LL, O, S>;                                  \
    const int most = S ? 16 : walk_warps<R, LL>();                            \
    const int nw = S || R || kWarpStep * bps > most ? most : kWarpStep * bps; \
    const size_t sb = walk_smem_bytes<LL, R>(nw) +                            \
                      (S ? sizeof(TeamSmem) * (nw / a.team) : 0);             \
    static std::atomic<unsigned> attr_set{0}; /* devices with the smem limit raised */ \
    if (dev >= 32 || !(attr_set & (1u << dev))) {                             \
      cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize,  \
                           (int)(walk_smem_bytes<LL, R>(most) + (S ? kTeamBytes : 0))); \
      if (dev < 32) attr_set |= 1u << dev;                                    \
    }                                                                         \
    kfn<<<mb.sms, 32 * nw, sb, st>>>(a);                                      \
  } while (0)
#define TG_LAUNCH_O(P, R, LL)                                                 \
  do {                                                                        \
    if (a.team > 1) TG_LAUNCH_S(P, R, LL, true);                              \
    else TG_LAUNCH_S(P, R, LL, false);                                        \
  } while (0)
#define TG_LAUNCH_S(P, R, LL, S)                                              \
  do {                                                                        \
    if (tune.order >= 4) TG_LAUNCH(P, R, LL, 4, S);                           \
    else if (tune.order == 3) TG_LAUNCH(P, R, LL, 3, S);                      \
    else TG_LAUNCH(P, R, LL, 2, S);                                           \
  } while (0)
  if (wp.physics == 1) {
    if (L) { if (r) TG_LAUNCH_O(1, true, true); else TG_LAUNCH_O(1, false, true); }
    else { if (r) TG_LAUNCH_O(1, true, false); else TG_LAUNCH_O(1, false, false); }
  } else {
    if (L) { if (r) TG_LAUNCH_O(0, true, true); else TG_LAUNCH_O(0, false, true); }
    else { if (r) TG_LAUNCH_O(0, true, false); else TG_LAUNCH_O(0, false, false); }
  }
#undef TG_LAUNCH_O
#undef TG_LAUNCH_S
#undef TG_LAUNCH
  return L ? 2 : 1;
}

}  // namespace tg
