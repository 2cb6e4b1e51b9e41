// walk64.cu -- FP64 per-target tree walk (parity path; compiled -fmad=false,
// fused multiply-adds only where written).
//
// One warp owns T targets, neighbours in sorted order, and walks the electron
// tree, then the ion tree, once for all of them: every target takes its own
// decisions, and an entry of the walk carries the set of targets that are
// still interested in it.  The 32 lanes test the next 32 nodes in pre-order at
// a time and evaluate 32 (interaction, target) pairs at a time; the three sums
// of each target's force are then taken one interaction after the other in
// pre-order, the order of the recursive Search_Tree_ee/_ie/_ei/_ii
// (tree.f90:721-1133).  Decisions, terms and force sums are the reference's to
// the last bit, except where the device exp() differs from the host's by an ulp
// and in one quotient of 10^14 (Divisor): an electron on its ion feels forces
// that cancel to rounding noise, and even that noise is reproduced.  The
// potential is an FP64 sum in another order: each lane adds the terms that it
// evaluates, then the lanes of a target are added (within 1e-12 of the gross
// sum of the reference's).
#include <atomic>
#include "internal.cuh"
#include "pair64.cuh"
#include "walk.h"

namespace tg {

// What bounds it: instruction issue and the latency of dependent operations at
// 16 warps per SM (128 registers, 12 KB of shared memory a warp); the FP64 pipe
// is busy less than half of the time, the memory side is served by L1 and L2.
// At N = 262,144 (theta 0.5, reference laws, RDF) the walk takes 21.7 ms, half of
// it walking and summing, half evaluating: 58.9 ms with one thread per target
// and 20 IEEE divisions per cell (16.5 of 32 lanes active), 25.2 with quotients
// of three operations and sums slot by slot.  At N = 4,096 it takes 0.29 ms against 7.3,
// where a thread per target left one warp per SM.  Per SM, 12 warps (156
// registers) and 20 (96, spills) were slower, 27.7 and 30.6 ms when 16 took 25.2;
// so were blocks of one warp (26.2), a stack of 768 entries (26.2: fewer nodes at
// a time near its limit), and children pushed a lane each by ballots (23.0 when 21.7).
constexpr int kW64Warps = 4;
constexpr int kW64Threads = 32 * kW64Warps;
constexpr int kW64Blocks = 4;    // per SM
constexpr int kW64Ring = 64;     // power of two, > 31 + 32
// Interactions between emission and sum, a power of two.
constexpr int w64_slots(int T) { return T == 1 ? 128 : 64; }
constexpr int kW64Stack = 1024;  // per warp
// Headroom that a depth-first descent from the limit needs: it leaves at most
// 7 siblings per level behind.
constexpr int kW64Reserve = 320;
static_assert(kW64Reserve > 7 * (kMaxLevel + 1), "stack reserve");

// Four targets share a walk when their warps still fill the GPU: the union of
// their interactions is 1.2 times a single target's at N = 262,144 but is
// walked once (21.7 ms against 36.8 with a target per warp).  A target per
// warp | four: N = 2,048 0.127 | 0.211 ms, 4,096 0.283 | 0.358, 8,192 0.612 |
// 0.543, 12,288 1.01 | 0.90, 16,384 1.35 | 1.09.  The line was drawn when
// 8,192 took 0.75 | 0.78; the kernel's later steps moved the crossing to about
// 6,000.
constexpr int kW64Share = 12288;

// Stack entries are a node and a set of targets; one whose node is accepted
// by them, or is a leaf, is only waiting for its place in the sum.
constexpr unsigned kW64Accepted = 0x40, kW64Leaf = 0x80;

template <int T>
struct alignas(16) W64Smem {
  double term[w64_slots(T) * 3 * T];  // per slot and target: force xyz
  double xt[3 * T];                // the targets
  int stack[kW64Stack];            // top = next in pre-order
  unsigned char sset[kW64Stack];
  int m2p[kW64Ring];               // accepted cells, leaves: node, and 256 * slot + targets
  int leaf[kW64Ring];
  unsigned short m2p_at[kW64Ring];
  unsigned short leaf_at[kW64Ring];
};

// The acceptance test w < sqrt(r2) on squares, where rounding (each square is
// within 1e-15) cannot change it: accepted above hi, opened below lo, and by
// the IEEE square root in between.
struct Mac64 {
  double lo, hi;
  __device__ __forceinline__ explicit Mac64(double w) {
    const double w2 = w * w;
    const bool tiny = w2 < 1e-280;  // squares that may have lost bits
    hi = tiny ? 1.1e-280 : w2 * (1.0 + 2e-14);
    lo = tiny ? 0.0 : w2 * (1.0 - 2e-14);
  }
};

// Division by b with a reciprocal of twice the working precision, hi + lo =
// 1/b (1 + d) with |d| < 2^-101: a hi + a lo, rounded once, is the IEEE quotient
// unless that lies within 2^-47 ulp of the middle between two numbers (an ulp
// off in one quotient of 10^14).  The correction of an estimate y by its exact
// residual e = 1 - b y and the series of 1 / (1 - e) are the long division of
// Karp and Markstein ("High-precision division and square root", ACM Trans.
// Math. Softw. 23(4), 1997).  A quotient is two operations, against three with
// a residual of its own (and about 12 for an IEEE division).
struct Divisor {
  double hi, lo;
  // y within 2^-47 of 1/b, relatively
  __device__ __forceinline__ Divisor(double b, double y) : hi(y) {
    const double e = __fma_rn(-b, y, 1.0);
    lo = __fma_rn(e, e, e) * y;
  }
  __device__ __forceinline__ double inv() const { return hi + lo; }
  __device__ __forceinline__ double operator()(double a) const {
    return __fma_rn(a, hi, a * lo);
  }
};

// sqrt(r2) from y = rsqrt(r2), by the same correction.
__device__ __forceinline__ double sqrt_by(double r2, double y) {
  const double g = r2 * y;
  return __fma_rn(__fma_rn(-g, g, r2), 0.5 * y, g);
}

// The far field's divisors r, r^3, r^5, r^7: one rsqrt serves the root and the
// reciprocals of 28 quotients.
struct SharedDivisors {
  Divisor d1, d3, d5, d7;
  __device__ __forceinline__ SharedDivisors(double r2, double r_, double y, double y2,
                                            double y3, double y5)
      : d1(r_, y), d3(r2 * r_, y3), d5((r2 * r_) * r2, y5), d7(((r2 * r_) * r2) * r2, y5 * y2) {}
  __device__ __forceinline__ SharedDivisors(double r2, double y)
      : SharedDivisors(r2, sqrt_by(r2, y), y, y * y, (y * y) * y, ((y * y) * y) * (y * y)) {}
  __device__ __forceinline__ explicit SharedDivisors(double r2)
      : SharedDivisors(r2, rsqrt(r2)) {}
  __device__ __forceinline__ double inv_R3() const { return d3.inv(); }
  __device__ __forceinline__ double r(double a) const { return d1(a); }
  __device__ __forceinline__ double R3(double a) const { return d3(a); }
  __device__ __forceinline__ double R5(double a) const { return d5(a); }
  __device__ __forceinline__ double R7(double a) const { return d7(a); }
};

// The same by IEEE divisions, for distances whose seventh power nears the
// ends of the exponent range (where a residual would not be exact).
struct PlainDivisors {
  double b1, b3, b5, b7;
  __device__ __forceinline__ explicit PlainDivisors(double r2) {
    const double r_ = sqrt(r2);
    b1 = r_;
    b3 = r2 * r_;
    b5 = b3 * r2;
    b7 = b5 * r2;
  }
  __device__ __forceinline__ double inv_R3() const { return 1.0 / b3; }
  __device__ __forceinline__ double r(double a) const { return a / b1; }
  __device__ __forceinline__ double R3(double a) const { return a / b3; }
  __device__ __forceinline__ double R5(double a) const { return a / b5; }
  __device__ __forceinline__ double R7(double a) const { return a / b7; }
};

// One cell's terms: far field of tree.f90:744-779 (identical in the four walks).
template <class Div>
__device__ __forceinline__ void m2p64(const double2* __restrict__ mm, double xr0, double xr1,
                                      double xr2, double r2, double ff, double& f0,
                                      double& f1, double& f2, double& ep) {
  double2 m0 = __ldg(mm + 0), m1 = __ldg(mm + 1), m2 = __ldg(mm + 2),
          m3 = __ldg(mm + 3), m4 = __ldg(mm + 4);
  const Div dv(r2);
  const double qeff = m0.x, PD0 = m0.y, PD1 = m1.x, PD2 = m1.y;
  const double PQ0 = m2.x, PQ1 = m2.y, PQ2 = m3.x, PQQ0 = m3.y, PQQ1 = m4.x,
               PQQ2 = m4.y;
  double D0 = -dv.inv_R3() + dv.R5(3.0 * (xr0 * xr0));
  double D1 = -dv.inv_R3() + dv.R5(3.0 * (xr1 * xr1));
  double D2 = -dv.inv_R3() + dv.R5(3.0 * (xr2 * xr2));
  double D3 = dv.R5(3.0 * xr0 * xr1);
  double D4 = dv.R5(3.0 * xr1 * xr2);
  double D5 = dv.R5(3.0 * xr2 * xr0);
  double Q0 = dv.R7(15.0 * ((xr0 * xr0) * xr0)) - dv.R5(9.0 * xr0);
  double Q1 = dv.R7(15.0 * ((xr1 * xr1) * xr1)) - dv.R5(9.0 * xr1);
  double Q2 = dv.R7(15.0 * ((xr2 * xr2) * xr2)) - dv.R5(9.0 * xr2);
  double Q3 = dv.R7(15.0 * (xr0 * xr0) * xr1) - dv.R5(3.0 * xr1);
  double Q4 = dv.R7(15.0 * (xr0 * xr0) * xr2) - dv.R5(3.0 * xr2);
  double Q5 = dv.R7(15.0 * (xr1 * xr1) * xr0) - dv.R5(3.0 * xr0);
  double Q6 = dv.R7(15.0 * (xr1 * xr1) * xr2) - dv.R5(3.0 * xr2);
  double Q7 = dv.R7(15.0 * (xr2 * xr2) * xr0) - dv.R5(3.0 * xr0);
  double Q8 = dv.R7(15.0 * (xr2 * xr2) * xr1) - dv.R5(3.0 * xr1);
  double Q9 = dv.R7(15.0 * xr0 * xr1 * xr2);
  ep = 0.5 * ff *
                (dv.r(qeff) + dv.R3(PD0 * xr0 + PD1 * xr1 + PD2 * xr2) +
                 PQ0 * D0 + PQ1 * D1 + PQ2 * D2 + PQQ0 * D3 + PQQ1 * D4 +
                 PQQ2 * D5);
  f0 = ff * (dv.R3(qeff * xr0) + D0 * PD0 + D3 * PD1 + D5 * PD2 +
                  Q0 * PQ0 + Q5 * PQ1 + Q7 * PQ2 + Q3 * PQQ0 + Q4 * PQQ2 +
                  Q9 * PQQ1);
  f1 = ff * (dv.R3(qeff * xr1) + D3 * PD0 + D1 * PD1 + D4 * PD2 +
                  Q3 * PQ0 + Q1 * PQ1 + Q8 * PQ2 + Q5 * PQQ0 + Q9 * PQQ2 +
                  Q6 * PQQ1);
  f2 = ff * (dv.R3(qeff * xr2) + D5 * PD0 + D4 * PD1 + D2 * PD2 +
                  Q4 * PQ0 + Q6 * PQ1 + Q2 * PQ2 + Q9 * PQQ0 + Q7 * PQQ2 +
                  Q8 * PQQ1);
}

__device__ __noinline__ void m2p64_extreme(const double2* __restrict__ mm, double xr0,
                                           double xr1, double xr2, double r2, double ff,
                                           double* t) {
  m2p64<PlainDivisors>(mm, xr0, xr1, xr2, r2, ff, t[0], t[1], t[2], t[3]);
}

// Terms of a pair whose law is plain Coulomb to double precision
// (pair64_far2), as leaf_pair64 evaluates them: there exp() changes no bit.
template <int PHYS>
__device__ __forceinline__ void leaf_pair64_far(double xr0, double xr1, double xr2, double r2,
                                                double ff, double& f0, double& f1, double& f2,
                                                double& ep, double& r) {
  const double y = rsqrt(r2);
  r = sqrt_by(r2, y);
  const Divisor dr(r, y);
  if (PHYS == 1) {
    ep = 0.5 * ff * dr.inv();
    const double fr = Divisor(r2 * r, (y * y) * y)(ff);
    f0 = fr * xr0;
    f1 = fr * xr1;
    f2 = fr * xr2;
  } else {
    const Divisor dr2(r2, y * y);
    ep = dr(0.5 * ff);
    // like charges: ff x / r / r2; unlike: ff x (1/r) / r2
    const bool like = ff > 0.0;
    const double yr = dr.inv(), a0 = ff * xr0, a1 = ff * xr1, a2 = ff * xr2;
    f0 = dr2(like ? dr(a0) : a0 * yr);
    f1 = dr2(like ? dr(a1) : a1 * yr);
    f2 = dr2(like ? dr(a2) : a2 * yr);
  }
}

__device__ __forceinline__ void rdf_add(uint32_t* hist, double r,
                                        double dxbin) {
  // id = INT(r/dx)+1 ; counted when 0 < id <= Ndist+1 (tree.f90:916-919)
  double t = r / dxbin;
  if (!(t < (double)kRdfBins)) return;
  int id = (int)t;
  if (id >= 0) atomicAdd(&hist[id], 1u);
}

// Oldest entry of a ring, as an interaction number (seq when the ring is empty).
__device__ __forceinline__ int w64_oldest(const unsigned short* at, int head, int tail, int done,
                                          int seq, int slots) {
  if (tail == head) return seq;
  return done + (((at[head & (kW64Ring - 1)] >> 8) - done) & (slots - 1));
}

template <int PHYS, bool RDF, int T>
__global__ void __launch_bounds__(kW64Threads, kW64Blocks)
    k_walk64(const double* __restrict__ x, int n, int n_el,
             const uint32_t* __restrict__ order, TreeView tv,
             const int32_t* __restrict__ kids, WalkParams wp,
             double* __restrict__ f, double2* __restrict__ epot_part,
             uint32_t* __restrict__ rdf, unsigned long long* counters,
             int32_t* err) {
  constexpr int E = 32 / T;  // interactions per evaluation
  constexpr int kSlots = w64_slots(T);
  extern __shared__ double2 w64_smem[];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  W64Smem<T>& sm = reinterpret_cast<W64Smem<T>*>(w64_smem)[wib];
  const int p0 = (blockIdx.x * kW64Warps + wib) * T;
  if (p0 < n && !(*((volatile int32_t*)err) & (kErrCapacity | kErrDepth | kErrNonFinite))) {
    // this lane's target of an evaluation, and its entry among the E
    const int mt_ = lane & (T - 1), me = lane / T;
    const int nt = min(T, n - p0);
    const int64_t o = order[min(p0 + mt_, n - 1)];
    const int tsp = o >= n_el;  // target species: 0 electron, 1 ion
    const double xt0 = x[3 * o], xt1 = x[3 * o + 1], xt2 = x[3 * o + 2];
    if (lane < T) {
      sm.xt[3 * lane] = xt0;
      sm.xt[3 * lane + 1] = xt1;
      sm.xt[3 * lane + 2] = xt2;
    }
    // ff for accepted cells: -eps for electron targets, +eps for ions
    const double ffc = tsp == 0 ? -1.0 * kEps : kEps;
    double sum = 0.0;  // lane = 3 target + axis: a running force sum
    // this lane's share of its evaluation target's potential, per source tree
    double ep_tree[2] = {0.0, 0.0};
    unsigned nm2p = 0, np2p = 0;
    for (int ssp = 0; ssp < 2; ++ssp) {
      const int root = tv.tree_bounds[ssp], end = tv.tree_bounds[ssp + 1];
      const bool same = ssp == tsp;
      double ep = 0.0;
      int ssize = 0;
      if (root < end) {
        if (lane == 0) {
          sm.stack[0] = root;
          sm.sset[0] = (unsigned char)((1u << nt) - 1u);
        }
        ssize = 1;
      }
      // every round sums or opens a node, and does each at most once per node:
      // more rounds mean a corrupt tree
      unsigned left = 2u * (unsigned)(end - root) + 64u;
      __syncwarp();
      int mh = 0, mt = 0, lh = 0, ltl = 0;  // ring heads / tails (warp-uniform)
      int seq = 0, done = 0;                // interactions emitted / summed
      while (ssize > 0 || done < seq) {
        if (ssize > 0) {
          // ---- the next (up to 32) entries in pre-order ----
          // near the stack's limit fewer are popped, then one at a time: a
          // popped entry leaves at most 8 entries more than it took
          const int room = (kW64Stack - kW64Reserve - ssize) >> 3;
          const int nb = min(min(32, ssize), max(1, room));
          int node = -1;
          unsigned set = 0, fin_set = 0, open_set = 0;  // fin: accepted, or a leaf
          if (lane < nb) {
            node = sm.stack[ssize - 1 - lane];
            set = sm.sset[ssize - 1 - lane];
          }
          ssize -= nb;
          if (--left == 0u) {
            if (lane == 0) set_error(err, kErrWalk);
            break;
          }
          __syncwarp();
          if (set & (kW64Accepted | kW64Leaf)) {
            fin_set = set;
          } else if (lane < nb) {
            const double4 c = ldg_d4(&tv.node_c[node]);
            if (c.w < 0.0) {
              fin_set = set | kW64Leaf;
            } else {
              const Mac64 mac(c.w);
              unsigned close = 0;
#pragma unroll
              for (int t = 0; t < T; ++t) {
                const double x0 = sm.xt[3 * t] - c.x, x1 = sm.xt[3 * t + 1] - c.y,
                             x2 = sm.xt[3 * t + 2] - c.z;
                const double r2 = __fma_rn(x0, x0, __fma_rn(x1, x1, x2 * x2));
                fin_set |= r2 > mac.hi ? 1u << t : 0u;
                close |= r2 < mac.lo ? 0u : 1u << t;
              }
              close &= set & ~fin_set;
              while (close) {
                const int t = __ffs((int)close) - 1;
                close &= close - 1;
                const double x0 = sm.xt[3 * t] - c.x, x1 = sm.xt[3 * t + 1] - c.y,
                             x2 = sm.xt[3 * t + 2] - c.z;
                if (c.w < sqrt(x0 * x0 + x1 * x1 + x2 * x2)) fin_set |= 1u << t;
              }
              fin_set &= set;
              open_set = set & ~fin_set;
              if (fin_set) fin_set |= kW64Accepted;
            }
          }
          // entries up to the first opened node are next in the sum; the
          // others wait on the stack behind that node's children
          const unsigned open = __ballot_sync(0xffffffffu, open_set != 0);
          const int first_open = open ? __ffs((int)open) - 1 : 32;
          const bool emit = lane <= first_open && fin_set != 0;
          const unsigned be = __ballot_sync(0xffffffffu, emit);
          const unsigned bm = __ballot_sync(0xffffffffu, emit && (fin_set & kW64Accepted));
          if (emit) {
            const bool cell = fin_set & kW64Accepted;
            const unsigned at = (((seq + __popc(be & lt)) & (kSlots - 1)) << 8) | (fin_set & 0x3fu);
            const int q = cell ? mt + __popc(bm & lt) : ltl + __popc(be & ~bm & lt);
            (cell ? sm.m2p : sm.leaf)[q & (kW64Ring - 1)] = node;
            (cell ? sm.m2p_at : sm.leaf_at)[q & (kW64Ring - 1)] = (unsigned short)at;
            if (cell) nm2p += __popc(fin_set & 0x3fu);
          }
          mt += __popc(bm);
          ltl += __popc(be & ~bm);
          seq += __popc(be);
          if (open) {
            int4 k0 = make_int4(-1, -1, -1, -1), k1 = k0;
            if (open_set) {
              const int4* kk = reinterpret_cast<const int4*>(kids + 8 * (int64_t)node);
              k0 = __ldg(kk);
              k1 = __ldg(kk + 1);
            }
            const int kv[8] = {k0.x, k0.y, k0.z, k0.w, k1.x, k1.y, k1.z, k1.w};
            const bool back = fin_set != 0 && !emit;
            int kc = back ? 1 : 0;
#pragma unroll
            for (int j = 0; j < 8; ++j) kc += kv[j] >= 0 ? 1 : 0;
            int inc = kc;
#pragma unroll
            for (int s = 1; s < 32; s <<= 1) {
              const int t = __shfl_up_sync(0xffffffffu, inc, s);
              if (lane >= s) inc += t;
            }
            const int tot = __shfl_sync(0xffffffffu, inc, 31);
            int pos = ssize + tot - 1 - (inc - kc);  // earlier in pre-order: higher
            if (back) {
              sm.stack[pos] = node;
              sm.sset[pos--] = (unsigned char)fin_set;
            }
            if (open_set) {
#pragma unroll
              for (int j = 0; j < 8; ++j)
                if (kv[j] >= 0) {
                  sm.stack[pos] = kv[j];
                  sm.sset[pos--] = (unsigned char)open_set;
                }
            }
            ssize += tot;
          }
          __syncwarp();
        }
        // ---- terms of E interactions at a time, then the sums up to the first
        // interaction still without terms; fewer at a time when the walk has
        // ended, or when the oldest such interaction holds up more slots than
        // the next 32 entries leave free
        const bool fin = ssize == 0;
        bool take_leaf = fin, take_m2p = fin;
        while (true) {
          while (ltl - lh >= E || (take_leaf && ltl > lh)) {
            const int cnt = min(E, ltl - lh);
            if (me < cnt) {
              const int q = (lh + me) & (kW64Ring - 1);
              const int node = sm.leaf[q];
              const unsigned at = sm.leaf_at[q];
              double t0 = 0.0, t1 = 0.0, t2 = 0.0, e = 0.0;
              if ((at >> mt_) & 1u) {
                const double4 c = ldg_d4(&tv.node_c[node]);
                const double x0 = xt0 - c.x, x1 = xt1 - c.y, x2 = xt2 - c.z;
                const double r2 = x0 * x0 + x1 * x1 + x2 * x2;
                double r = 0.0;
                bool counted = true;
                if (r2 > pair64_far2<PHYS>(same, tsp, wp) && r2 > 1e-72 && r2 < 1e72) {
                  leaf_pair64_far<PHYS>(x0, x1, x2, r2, same ? kEps : -1.0 * kEps, t0, t1, t2, e, r);
                } else {
                  const bool self = PHYS == 1 && same && __ldg(&tv.node_pt[node]) == (int)o;
                  counted = leaf_pair64<PHYS>(x0, x1, x2, r2, same, tsp, self, wp, t0, t1, t2, e, r);
                }
                if (counted) {
                  ++np2p;
                  if (RDF) {
                    if (!same) rdf_add(rdf, r, wp.dx_ei);
                    else if (tsp == 1 && (PHYS == 0 || r2 > 0.0))
                      rdf_add(rdf + kRdfBins, r, wp.dx_ii);
                  }
                }
              }
              ep += e;
              double* t = sm.term + 3 * ((at >> 8) * T + mt_);
              t[0] = t0;
              t[1] = t1;
              t[2] = t2;
            }
            lh += cnt;
          }
          while (mt - mh >= E || (take_m2p && mt > mh)) {
            const int cnt = min(E, mt - mh);
            if (me < cnt) {
              const int q = (mh + me) & (kW64Ring - 1);
              const int node = sm.m2p[q];
              const unsigned at = sm.m2p_at[q];
              double v[4] = {0.0, 0.0, 0.0, 0.0};
              if ((at >> mt_) & 1u) {
                const double4 c = ldg_d4(&tv.node_c[node]);
                const double x0 = xt0 - c.x, x1 = xt1 - c.y, x2 = xt2 - c.z;
                const double r2 = x0 * x0 + x1 * x1 + x2 * x2;
                const double2* mm = tv.node_m + 5 * (int64_t)node;
                if (r2 > 1e-72 && r2 < 1e72)
                  m2p64<SharedDivisors>(mm, x0, x1, x2, r2, ffc, v[0], v[1], v[2], v[3]);
                else
                  m2p64_extreme(mm, x0, x1, x2, r2, ffc, v);
              }
              ep += v[3];
              double* t = sm.term + 3 * ((at >> 8) * T + mt_);
              t[0] = v[0];
              t[1] = v[1];
              t[2] = v[2];
            }
            mh += cnt;
          }
          __syncwarp();
          const int m_at = w64_oldest(sm.m2p_at, mh, mt, done, seq, kSlots);
          const int l_at = w64_oldest(sm.leaf_at, lh, ltl, done, seq, kSlots);
          const int pend = min(m_at, l_at);
          // whole blocks of 8 slots, so that their addresses are constants
          const double* tc = sm.term + (lane < 3 * T ? lane : 0);
          for (; done + 8 <= pend; done += 8) {
            const double* tb = tc + 3 * T * (done & (kSlots - 1));
            double v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = tb[3 * T * j];
#pragma unroll
            for (int j = 0; j < 8; ++j) sum = sum + v[j];
          }
          if (fin)
            for (; done < pend; ++done) sum = sum + tc[3 * T * (done & (kSlots - 1))];
          __syncwarp();
          if (fin ? done == seq : seq - done <= kSlots - 32) break;
          take_leaf = fin || l_at < m_at;
          take_m2p = fin || !take_leaf;
        }
      }
      ep_tree[ssp] = ep;
    }
#pragma unroll
    for (int s = T; s < 32; s <<= 1) {
      ep_tree[0] += __shfl_xor_sync(0xffffffffu, ep_tree[0], s);
      ep_tree[1] += __shfl_xor_sync(0xffffffffu, ep_tree[1], s);
    }
    nm2p = __reduce_add_sync(0xffffffffu, nm2p);
    np2p = __reduce_add_sync(0xffffffffu, np2p);
    if (lane < 3 * nt) f[3 * (int64_t)order[p0 + lane / 3] + lane % 3] = sum;
    if (lane < nt)
      // Epot_e = ee + ie + ei ; Epot_i = ii (tree.f90:674-715)
      epot_part[o] = tsp == 0 ? make_double2(ep_tree[0] + ep_tree[1], 0.0)
                              : make_double2(ep_tree[0], ep_tree[1]);
    if (lane == 0) {  // interaction counters
      atomicAdd(&counters[0], (unsigned long long)nm2p);
      atomicAdd(&counters[1], (unsigned long long)np2p);
    }
  }
}

void walk64(const double* x, int n, int n_el, const uint32_t* order,
            const TreeView& tv, const int32_t* kids, const WalkParams& wp, double* f,
            double2* epot_part, uint32_t* rdf, unsigned long long* counters,
            int32_t* err, cudaStream_t st) {
  if (n == 0) return;
  int dev = 0;
  cudaGetDevice(&dev);
#define TG_W64(P, R, TT)                                                                    \
  do {                                                                                      \
    auto kfn = k_walk64<P, R, TT>;                                                          \
    constexpr int kSmem = kW64Warps * (int)sizeof(W64Smem<TT>);                             \
    static std::atomic<unsigned> attr_set{0}; /* devices with the smem limit raised */      \
    if (dev >= 32 || !(attr_set & (1u << dev))) {                                           \
      cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);        \
      if (dev < 32) attr_set |= 1u << dev;                                                  \
    }                                                                                       \
    const int g = (n + kW64Warps * TT - 1) / (kW64Warps * TT);                              \
    kfn<<<g, kW64Threads, kSmem, st>>>(x, n, n_el, order, tv, kids, wp, f, epot_part, rdf,  \
                                       counters, err);                                      \
  } while (0)
#define TG_W64_T(P, R)                    \
  do {                                    \
    if (n >= kW64Share) TG_W64(P, R, 4);  \
    else TG_W64(P, R, 1);                 \
  } while (0)
  if (wp.physics == 0) {
    if (rdf) TG_W64_T(0, true);
    else TG_W64_T(0, false);
  } else {
    if (rdf) TG_W64_T(1, true);
    else TG_W64_T(1, false);
  }
#undef TG_W64_T
#undef TG_W64
}

}  // namespace tg
