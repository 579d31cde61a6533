// wg_exact.cu -- wendy's exact event-driven solver (approx=False) on the GPU.
//
// Between collisions every sheet moves under a constant acceleration (or,
// with a harmonic external potential, on a shifted harmonic orbit), so the
// next crossing of two neighbours in position order is the root of a
// quadratic (or of a sinusoid).  The solver processes crossings one at a
// time in time order: advance the two sheets to the crossing, swap them,
// exchange their accelerations by the mass difference, and recompute the
// crossing times of the three neighbour pairs that changed.  The reference
// keeps the pair times in an unbalanced binary search tree
// (wendy/wendy.c:53-315, wendy/bst.c); here they sit in a 32-ary tournament
// tree (each internal node holds the minimum of its 32 children and where it
// lies), each level of an update one coalesced 32-wide load and a warp
// minimum.  The state lives in position order, in shared memory when it fits
// (a few thousand sheets), in global memory otherwise.
//
// The loop is a strict sequence of crossings, each a chain of dependent FP64
// operations, and an FP64 instruction takes a warp 64 cycles on this part,
// dependent or not, however few of its lanes are active (a division about 600,
// a square root 635).  So:
//  * the four sheets around a crossing sit in four lanes, twice: one group of
//    four follows the velocities while the other follows the positions, so
//    that one instruction does an operation of each (an addition as 1 a + b, a
//    product as a b - 0: the same roundings), and the five divisions of the
//    three new pair times are one;
//  * times are compared as integer keys;
//  * a second warp keeps the tree: while the first one finds the three new
//    pair times it inserts the three before them and finds the smallest pair
//    time outside the pairs that are changing, so that the next crossing is
//    the smallest of four numbers.
// A crossing of 1001 sheets of a sech^2 disk takes 1.9 us (about 160 cycles of
// loads, 1100 to the pair's coefficients, 800 for the division, 1000 for the
// square root, 500 to the next crossing); one lane doing all of it, with the
// tree updated in between, took 5.3 us.
//
// Arithmetic, operation order and the per-sheet clocks follow the
// reference (this file is compiled without FMA contraction, as the
// reference's C is), so trajectories agree to rounding; pair times that are NaN
// (pairs that never meet in the harmonic case) never come first, and among
// equal pair times the lowest pair index comes first.
#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <vector>

#include "../../include/wendy_gb300.h"
#include "wg_blocks.cuh"
#include "wg_internal.cuh"

using namespace wg;

namespace {

constexpr int kTreeFan = 32;
constexpr size_t kExactStatic = 128;  // bound on k_exact_step's static shared memory
constexpr int kMaxLevels = 6;  // 32^6 pair times: more than any N this accepts

struct ExactState {
  double* x;
  double* v;
  double* a;
  double* m;
  double* t;      // each sheet's own clock within the output interval
  int32_t* id;    // the sheet at each position (the arrays above are in
                  // position order while the event loop runs)
  double* tcoll;  // crossing time of the pair at positions (i, i + 1)
};

struct ExactArgs {
  ExactState g;        // the state in global memory, by sheet (id: the position order)
  ExactState p;        // the same by position, where shared memory does not hold it
  int n;
  double omega;        // > 0: harmonic external potential
  double dt;
  long long maxcoll;
  // internal levels of the tournament tree: the order key of the smallest
  // pair time below each node (see time_key) and that pair's index
  uint64_t* tree_key[kMaxLevels];
  int32_t* tree_idx[kMaxLevels];
  int levels;
  int level_n[kMaxLevels + 1];   // entries per level (level 0: the n - 1 pair times)
  int* cindx;          // in/out: pair of the next crossing
  double* next_tcoll;  // in/out: its time
  long long* ncoll;    // out: crossings processed
  int* err;            // out: -2 when maxcoll was reached
  int idx0_global;     // the lowest level's indices stay in global memory
  int use_smem;        // the state is staged in shared memory (after the tree)
  size_t tree_bytes;   // shared memory of the tree's internal levels (16-byte multiple)
};

// The reference's root of the crossing quadratic c2 t^2 + c1 t + c0 = 0
// (wendy/wendy.c:33-38).
__device__ double solve_coll_quad(double c0, double c1, double c2) {
  const double mba = -c1 / c2;
  return 0.5 * (mba + sqrt(mba * mba - 4. * c0 / c2));
}

// The reference's first crossing under harmonic motion (wendy/wendy.c:39-52).
__device__ double solve_coll_harm(double c0, double c1, double c2, double omega) {
  const double A = c0 - c2, B = c1 / omega;
  double out = -asin(c2 / sqrt(B * B + A * A)) - atan2(A, B);
  if (out < 0) out = M_PI + asin(c2 / sqrt(B * B + A * A)) - atan2(A, B);
  return out / omega;
}

// Order key of a pair time: increasing in the time (integer compares, off
// the FP64 pipe), NaN after everything.
__device__ __forceinline__ uint64_t time_key(double t) {
  const uint64_t b = (uint64_t)__double_as_longlong(t);
  return (b << 1) > 0xffe0000000000000ull ? ~0ull : key_of(t);
}
// The time of a key that is not NaN's (+0 for either zero).
__device__ __forceinline__ double time_of_key(uint64_t k) {
  return __longlong_as_double((long long)((k >> 63) ? (k & 0x7FFFFFFFFFFFFFFFull) : ~k));
}

// The smallest key over the warp and the lowest lane that holds it.
__device__ __forceinline__ uint64_t warp_min_key(uint64_t k, int& where) {
  const uint32_t hi = (uint32_t)(k >> 32), lo = (uint32_t)k;
  const uint32_t h = __reduce_min_sync(0xffffffffu, hi);
  const uint32_t l = __reduce_min_sync(0xffffffffu, hi == h ? lo : 0xffffffffu);
  where = __ffs(__ballot_sync(0xffffffffu, hi == h && lo == l)) - 1;
  return ((uint64_t)h << 32) | l;
}

// The smallest key among the children of node g of level lv (all lanes) and
// the pair it belongs to; children ca and cb (-1: none) of the level below
// are taken from (ka, ia) and (kb, ib), and at level 0 the pairs lo .. hi are
// left out.
__device__ __forceinline__ uint64_t node_min(const ExactArgs& A, uint64_t* const* tkey,
                                             int32_t* const* tidx, const double* tcoll, int lv,
                                             int g, int lane, int lo, int hi, int ca, uint64_t ka,
                                             int ia, int cb, uint64_t kb, int ib, int& idx) {
  const int j = g * kTreeFan + lane;
  uint64_t k = ~0ull;
  int i = j;
  if (j < A.level_n[lv]) {
    if (lv == 0) {
      if (j < lo || j > hi) k = time_key(tcoll[j]);
    } else {
      k = tkey[lv - 1][j];
      i = tidx[lv - 1][j];
    }
  }
  if (lv > 0 && j == ca) {
    k = ka;
    i = ia;
  }
  if (lv > 0 && j == cb) {
    k = kb;
    i = ib;
  }
  int where;
  const uint64_t best = warp_min_key(k, where);
  idx = __shfl_sync(0xffffffffu, i, where);
  return best;
}

// Rewrites the tree's path above pair time `leaf` (all lanes of one warp).
__device__ __forceinline__ void tree_update(const ExactArgs& A, uint64_t* const* tkey,
                                            int32_t* const* tidx, const double* tcoll, int leaf,
                                            int lane) {
  int child = -1, idx = 0;
  uint64_t best = 0;
  int g = leaf / kTreeFan;
  for (int lv = 0; lv < A.levels; ++lv) {
    best = node_min(A, tkey, tidx, tcoll, lv, g, lane, 0, -1, child, best, idx, -1, 0, 0, idx);
    if (lane == 0) {
      tkey[lv][g] = best;
      tidx[lv][g] = idx;
    }
    child = g;
    g /= kTreeFan;
  }
  __syncwarp();
}

// The smallest pair time outside the pairs lo .. hi (at most three, in one
// group of leaves or two adjacent ones) and its pair; the tree is left alone.
__device__ __forceinline__ uint64_t tree_min_outside(const ExactArgs& A, uint64_t* const* tkey,
                                                     int32_t* const* tidx, const double* tcoll,
                                                     int lo, int hi, int lane, int& idx) {
  int ca = -1, cb = -1, ia = 0, ib = 0;
  uint64_t ka = 0, kb = 0;
  int ga = lo / kTreeFan, gb = hi / kTreeFan;
  for (int lv = 0; lv < A.levels; ++lv) {
    int na, nb = 0;
    const uint64_t qa = node_min(A, tkey, tidx, tcoll, lv, ga, lane, lo, hi, ca, ka, ia, cb, kb,
                                 ib, na);
    uint64_t qb = 0;
    if (gb != ga)
      qb = node_min(A, tkey, tidx, tcoll, lv, gb, lane, lo, hi, ca, ka, ia, cb, kb, ib, nb);
    ca = ga;
    ka = qa;
    ia = na;
    cb = gb != ga ? gb : -1;
    kb = qb;
    ib = nb;
    ga /= kTreeFan;
    gb /= kTreeFan;
  }
  idx = ia;
  return ka;
}

// -x without an FP64 instruction.
__device__ __forceinline__ double negated(double x) {
  return __longlong_as_double(__double_as_longlong(x) ^ (long long)0x8000000000000000ull);
}

// Advance (x, v) from the sheet's own clock t to time tn (reference
// operation order).
__device__ __forceinline__ void advance(double& x, double& v, double a, double t, double tn,
                                        double omega) {
  const double tdt = tn - t;
  if (omega > 0) {
    const double sinot = sin(omega * tdt);
    const double cosot = sqrt(1. - sinot * sinot);
    const double tmpd = x - a;
    const double xo = tmpd * cosot + v / omega * sinot + a;
    v = -tmpd * omega * sinot + v * cosot;
    x = xo;
  } else {
    const double dv = a * tdt;
    x += dv * tdt / 2. + v * tdt;
    v += dv;
  }
}

template <bool HARM>
__global__ void __launch_bounds__(64, 1) k_exact_step(const ExactArgs A) {
  extern __shared__ __align__(16) unsigned char smem[];
  // the new times of the pairs ci - 1, ci, ci + 1 and the smallest time
  // elsewhere, written before and read after the barrier that ends a
  // crossing; used alternately, so that neither is overwritten while the
  // other warp still reads it
  __shared__ double s_new[2][3];
  __shared__ uint64_t s_newkey[2][3];
  __shared__ uint64_t s_rest[2];
  __shared__ int s_rest_idx[2];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n = A.n;
  ExactState S = A.p;
  // the tree's internal levels: in shared memory always (n / 31 entries)
  uint64_t* tkey[kMaxLevels];
  int32_t* tidx[kMaxLevels];
  {
    unsigned char* p = smem;
    for (int lv = 0; lv < A.levels; ++lv) {
      tkey[lv] = reinterpret_cast<uint64_t*>(p);
      p += 8 * (size_t)A.level_n[lv + 1];
    }
    for (int lv = A.levels - 1; lv >= 0; --lv) {
      tidx[lv] = reinterpret_cast<int32_t*>(p);
      p += 4 * (size_t)A.level_n[lv + 1];
    }
    if (A.idx0_global) tidx[0] = A.tree_idx[0];
    for (int lv = 0; lv < A.levels; ++lv)
      for (int j = tid; j < A.level_n[lv + 1]; j += 64) {
        tkey[lv][j] = A.tree_key[lv][j];
        if (lv > 0 || !A.idx0_global) tidx[lv][j] = A.tree_idx[lv][j];
      }
    p = smem + A.tree_bytes;
    if (A.use_smem) {
      // stage the state in shared memory too: x v a m t tcoll, then id
      double* d = reinterpret_cast<double*>(p);
      S.x = d;
      S.v = d + n;
      S.a = d + 2 * n;
      S.m = d + 3 * n;
      S.t = d + 4 * n;
      S.tcoll = d + 5 * n;
      S.id = reinterpret_cast<int32_t*>(d + 6 * n);
      for (int i = tid; i < n; i += 64) {
        const int s = A.g.id[i];
        S.id[i] = s;
        S.x[i] = A.g.x[s];
        S.v[i] = A.g.v[s];
        S.a[i] = A.g.a[s];
        S.m[i] = A.g.m[s];
        if (i < n - 1) S.tcoll[i] = A.g.tcoll[i];
      }
    }
  }
  for (int i = tid; i < n; i += 64) S.t[i] = 0.;
  __syncthreads();
  const double omega = A.omega, dt = A.dt;
  int cindx = *A.cindx;
  double next = *A.next_tcoll;
  uint64_t knext = time_key(next);
  const uint64_t kdt = key_of(dt);
  long long cnt = 0;
  // warp 0: lanes 0 .. 3, and again lanes 4 .. 7, hold the sheets at positions
  // ci - 1 .. ci + 2 of a crossing of ci and ci + 1 (the other lanes do the
  // same work and write nothing)
  const int role = lane & 3;
  const bool mid = role == 1 || role == 2;
  const bool pos_chain = (lane & 4) != 0;  // follows positions (else velocities)
  // partners in the new pairs: the left neighbour meets the sheet from
  // ci + 1, the right one that from ci, and those two each other
  const int partner = (lane & 28) | (role == 0 ? 2 : role == 3 ? 1 : role ^ 3);
  const double num_scale = mid ? 2.0 : pos_chain ? 4.0 : -1.0;
  const double den_scale = mid ? -1.0 : 0.5;
  int prev = -1;  // pair of the crossing before (its new times await insertion)
  while (knext < kdt && cnt < A.maxcoll) {
    const int buf = (int)(cnt & 1);
    ++cnt;
    const int ci = cindx;
    if (warp == 0) {
      const int pos = ci - 1 + role;
      const bool have = pos >= 0 && pos < n;  // the outer two may not exist
      const int at = have ? pos : ci;
      const double t = S.t[at], v = S.v[at], m = S.m[at];
      double x = S.x[at], a = S.a[at];
      const int32_t id = S.id[at];
      double tn, vn;
      if constexpr (HARM) {
        vn = v;
        advance(x, vn, a, t, next, omega);
        // the two swap places and exchange accelerations by the mass difference
        const double mo = __shfl_xor_sync(0xffffffffu, m, 3);
        const double dm = (role == 1 ? mo : m) - (role == 1 ? m : mo);
        const double ad = a - dm;
        const double ao = __shfl_xor_sync(0xffffffffu, ad, 3);
        if (mid) a = ao;
        const double xp = __shfl_sync(0xffffffffu, x, partner);
        const double vp = __shfl_sync(0xffffffffu, vn, partner);
        const double ap = __shfl_sync(0xffffffffu, a, partner);
        if (mid) {
          double q = (vn - vp) / (ap - a) / omega;
          q *= q;
          q = (1. - q) / (1. + q);
          tn = acos(q) / omega;
        } else {
          tn = solve_coll_harm(x - xp, vn - vp, a - ap, omega);
        }
      } else {
        // to the time of the crossing; the outer two are only extrapolated,
        // in the reference's order of additions ((x + a t^2 / 2) + v t,
        // against x + (a t^2 / 2 + v t)), and keep their state
        const double tdt = next - t;
        const double dv = a * tdt;
        // velocities: v + dv          positions: dv tdt
        const double r3 = __fma_rn(pos_chain ? dv : 1.0, pos_chain ? tdt : dv,
                                   pos_chain ? -0.0 : v);
        // velocities: mass difference   positions: v tdt
        const double mo = __shfl_xor_sync(0xffffffffu, m, 3);
        const double r4 = __fma_rn(pos_chain ? v : 1.0, pos_chain ? tdt : role == 1 ? mo : m,
                                   pos_chain ? -0.0 : negated(role == 1 ? m : mo));
        const double half = r3 * 0.5;
        // velocities: a less that difference   positions: first addition
        const double r5 = (pos_chain ? half : a) +
                          (pos_chain ? (mid ? r4 : x) : negated(r4));
        const double ao = __shfl_xor_sync(0xffffffffu, r5, 3);
        if (mid) a = ao;
        const double ap = __shfl_sync(0xffffffffu, a, partner);
        // velocities: difference of accelerations   positions: second addition
        const double r6 = (pos_chain ? r5 : a) + (pos_chain ? (mid ? x : r4) : negated(ap));
        vn = r3;
        x = r6;
        const double y = pos_chain ? r6 : r3;
        const double c = y - __shfl_sync(0xffffffffu, y, partner);
        const double da = __shfl_sync(0xffffffffu, r6, lane & 27);
        // the outer pairs' quadratic c2 t^2 + c1 t + c0 (wendy/wendy.c:33-38),
        // -c1 / c2 in the velocity lanes and 4 c0 / c2 in the position lanes,
        // and the inner pair's other root
        const double quo = (c * num_scale) / (da * den_scale);
        const double qc = __shfl_xor_sync(0xffffffffu, quo, 4);
        const double disc = quo * quo - qc;
        // (lanes without a root of their own take 1: negative numbers would
        // send the whole warp through the slow path of the square root)
        tn = mid ? quo : 0.5 * (quo + sqrt(mid || pos_chain ? 1.0 : disc));
      }
      if (lane < 8) {
        const int to = mid ? (role == 1 ? ci + 1 : ci) : at;
        const bool moves = mid || (HARM && have);
        if (moves && pos_chain) S.x[to] = x;
        if (moves && !pos_chain) {
          S.v[to] = vn;
          S.t[to] = next;
        }
        if (mid && !pos_chain) {
          S.a[to] = a;
          S.m[to] = m;
          S.id[to] = id;
        }
        // role 0: pair ci - 1, role 1: pair ci, role 3: pair ci + 1
        if (!pos_chain && role != 2) {
          const double when = next + tn;
          s_new[buf][role == 3 ? 2 : role] = when;
          s_newkey[buf][role == 3 ? 2 : role] = have ? time_key(when) : ~0ull;
        }
      }
    } else {
      // the new times of the crossing before enter the tree, then the
      // smallest time outside this crossing's pairs
      if (prev >= 0) {
        const int lo = prev > 0 ? prev - 1 : prev, hi = prev < n - 2 ? prev + 1 : prev;
        if (lane < 3 && prev - 1 + lane >= lo && prev - 1 + lane <= hi)
          S.tcoll[prev - 1 + lane] = s_new[buf ^ 1][lane];
        __syncwarp();
        tree_update(A, tkey, tidx, S.tcoll, lo, lane);
        if (hi / kTreeFan != lo / kTreeFan) tree_update(A, tkey, tidx, S.tcoll, hi, lane);
      }
      int idx;
      const uint64_t rest = tree_min_outside(A, tkey, tidx, S.tcoll, ci > 0 ? ci - 1 : ci,
                                             ci < n - 2 ? ci + 1 : ci, lane, idx);
      if (lane == 0) {
        s_rest[buf] = rest;
        s_rest_idx[buf] = idx;
      }
    }
    __syncthreads();
    // the next crossing: ties to the lower pair; NaN times (pairs that never
    // meet) never come first
    prev = ci;
    knext = s_rest[buf];
    cindx = s_rest_idx[buf];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      const uint64_t k = s_newkey[buf][r];
      if (k < knext || (k == knext && k != ~0ull && ci - 1 + r < cindx)) {
        knext = k;
        cindx = ci - 1 + r;
      }
    }
    next = knext == ~0ull ? INFINITY : time_of_key(knext);
  }
  if (warp == 1 && prev >= 0 && lane < 3 && prev - 1 + lane >= 0 && prev - 1 + lane < n - 1)
    S.tcoll[prev - 1 + lane] = s_new[(int)(cnt & 1) ^ 1][lane];
  __syncthreads();
  // every sheet to the end of the interval, clocks and pending times shifted
  for (int i = tid; i < n; i += 64) {
    double x = S.x[i], v = S.v[i];
    advance(x, v, S.a[i], S.t[i], dt, omega);
    if (A.use_smem) {
      const int s = S.id[i];
      A.g.id[i] = s;
      A.g.x[s] = x;
      A.g.v[s] = v;
      A.g.a[s] = S.a[i];
      if (i < n - 1) A.g.tcoll[i] = S.tcoll[i] - dt;
    } else {
      S.x[i] = x;
      S.v[i] = v;
      if (i < n - 1) S.tcoll[i] -= dt;
    }
  }
  // the tree holds absolute times of this interval: rebuilt by the host's
  // next call (k_exact_tree_level), like the reference rebuilds its BST per call
  if (tid == 0) {
    *A.cindx = cindx;
    *A.next_tcoll = next - dt;
    *A.ncoll = cnt;
    *A.err = cnt == A.maxcoll ? -2 : 0;
  }
}

// The state by position from the state by sheet, and back (simulations
// whose state does not fit in shared memory).
__global__ void k_exact_gather(ExactArgs A) {
  const int stride = gridDim.x * blockDim.x;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < A.n; i += stride) {
    const int s = A.g.id[i];
    A.p.id[i] = s;
    A.p.x[i] = A.g.x[s];
    A.p.v[i] = A.g.v[s];
    A.p.a[i] = A.g.a[s];
    A.p.m[i] = A.g.m[s];
  }
}
__global__ void k_exact_scatter(ExactArgs A) {
  const int stride = gridDim.x * blockDim.x;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < A.n; i += stride) {
    const int s = A.p.id[i];
    A.g.id[i] = s;
    A.g.x[s] = A.p.x[i];
    A.g.v[s] = A.p.v[i];
    A.g.a[s] = A.p.a[i];
  }
}

// Builds the tree over the current pair times (one warp per level-0 group,
// then level by level).
__global__ void k_exact_tree_level(ExactArgs A, int lv) {
  const int lane = threadIdx.x & 31;
  const int g = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int ng = (A.level_n[lv] + kTreeFan - 1) / kTreeFan;
  if (g >= ng) return;
  const int j = g * kTreeFan + lane;
  uint64_t k = ~0ull;
  int i = A.level_n[0] - 1;
  if (j < A.level_n[lv]) {
    if (lv == 0) {
      k = time_key(A.g.tcoll[j]);
      i = j;
    } else {
      k = A.tree_key[lv - 1][j];
      i = A.tree_idx[lv - 1][j];
    }
  }
  int where;
  k = warp_min_key(k, where);
  i = __shfl_sync(0xffffffffu, i, where);
  if (lane == 0) {
    A.tree_key[lv][g] = k;
    A.tree_idx[lv][g] = i;
  }
}

// Initial pair times from the sorted state (the reference computes them in
// Python with its C root finders, wendy/wendy.py:208-238).
__global__ void k_exact_pairs(ExactState S, int n, double omega) {
  const int stride = gridDim.x * blockDim.x;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n - 1; i += stride) {
    const int p = S.id[i], q = S.id[i + 1];
    S.tcoll[i] = omega > 0
                     ? solve_coll_harm(S.x[p] - S.x[q], S.v[p] - S.v[q], S.a[p] - S.a[q], omega)
                     : solve_coll_quad(S.x[p] - S.x[q], S.v[p] - S.v[q], (S.a[p] - S.a[q]) / 2.);
  }
}

thread_local char g_exact_error[256];

int fail(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_exact_error, sizeof(g_exact_error), fmt, ap);
  va_end(ap);
  record_last_error(g_exact_error);
  return code;
}

}  // namespace

struct wg_exact {
  int n = 0;
  double omega = 0;
  void* mem = nullptr;
  ExactArgs args{};
  cudaStream_t stream = nullptr;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  int stream_dev = -1;  // their device
  size_t smem = 0;
  int* h_ret = nullptr;  // page-locked: cindx, err, ncoll (as two ints), next (as two ints)
};

namespace {

void free_exact(wg_exact* e) {
  if (!e) return;
  if (e->stream) cudaStreamSynchronize(e->stream);
  block_free(e->mem);
  host_block_free(e->h_ret);
  StreamSet set;
  set.stream = e->stream;
  set.ev0 = e->ev0;
  set.ev1 = e->ev1;
  set.dev = e->stream_dev;
  stream_set_give(set);
  delete e;
}

size_t al(size_t b) { return (b + 255) & ~(size_t)255; }

// Dynamic shared memory an event loop may ask for on the current device (0: the
// limit could not be raised).  The limit belongs to the kernel, not to a handle:
// raised once to all that a block can have, so that simulations of different sizes
// can be alive at once.
size_t raise_smem_limit() {
  int dev = 0, optin = 0;
  cudaFuncAttributes fa[2];
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) !=
          cudaSuccess ||
      cudaFuncGetAttributes(&fa[0], k_exact_step<true>) != cudaSuccess ||
      cudaFuncGetAttributes(&fa[1], k_exact_step<false>) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  const size_t fixed = std::max(fa[0].sharedSizeBytes, fa[1].sharedSizeBytes);
  const size_t most = (size_t)optin > fixed ? (size_t)optin - fixed : 0;
  if (cudaFuncSetAttribute(k_exact_step<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)most) != cudaSuccess ||
      cudaFuncSetAttribute(k_exact_step<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)most) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return most;
}
size_t smem_limit() {
  static std::once_flag once[kMaxDevices];
  static size_t limit[kMaxDevices];
  const int dev = current_device();
  if (dev < 0 || dev >= kMaxDevices) return raise_smem_limit();
  std::call_once(once[dev], [&] { limit[dev] = raise_smem_limit(); });
  return limit[dev];
}

}  // namespace

extern "C" {

int wg_exact_create(int64_t n, const double* x, const double* v, const double* a,
                    const double* m, const int32_t* sindx, double omega, wg_exact** out) {
  if (!out) return fail(WG_ERR_ARG, "null output handle");
  *out = nullptr;
  if (n < 2 || n > (1 << 24)) return fail(WG_ERR_ARG, "exact solver: n outside [2, 2^24]");
  if (!x || !v || !a || !m || !sindx) return fail(WG_ERR_ARG, "exact solver: null array");
  if (!std::isfinite(omega)) return fail(WG_ERR_ARG, "exact solver: omega not finite");
  for (int64_t i = 0; i < n; ++i) {
    if (!std::isfinite(x[i]) || !std::isfinite(v[i]) || !std::isfinite(a[i]) ||
        !std::isfinite(m[i]) || m[i] < 0)
      return fail(WG_ERR_ARG, "exact solver: sheet %lld has a non-finite value or a negative "
                              "mass", (long long)i);
    if (sindx[i] < 0 || sindx[i] >= n)
      return fail(WG_ERR_ARG, "exact solver: sindx[%lld] out of range", (long long)i);
  }
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev < 1) {
    cudaGetLastError();
    return fail(WG_ERR_NODEV, "no CUDA device visible");
  }
  wg_exact* e = new wg_exact();
  e->n = (int)n;
  e->omega = omega > 0 ? omega : 0.0;
  ExactArgs& A = e->args;
  A.n = (int)n;
  A.omega = e->omega;
  // tree levels over the n - 1 pair times
  A.level_n[0] = (int)n - 1;
  A.levels = 0;
  while (true) {
    const int up = (A.level_n[A.levels] + kTreeFan - 1) / kTreeFan;
    A.level_n[A.levels + 1] = up;
    ++A.levels;
    if (up <= 1 || A.levels == kMaxLevels) break;
  }
  const size_t nd = al(8 * (size_t)n), ni = al(4 * (size_t)n);
  size_t tree_b = 0;
  for (int lv = 0; lv < A.levels; ++lv)
    tree_b += al(8 * (size_t)A.level_n[lv + 1]) + al(4 * (size_t)A.level_n[lv + 1]);
  const size_t smem_tree = [&] {
    size_t b = 0;
    for (int lv = 0; lv < A.levels; ++lv) b += 12 * (size_t)A.level_n[lv + 1];
    return (b + 15) & ~(size_t)15;
  }();
  // the tree's internal levels always live in shared memory; the state too
  // when it fits (6 doubles and an index per sheet)
  const size_t smem = smem_tree + 52 * (size_t)n + 64;
  int dev = 0, optin = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  A.use_smem = smem + kExactStatic <= (size_t)optin;
  const size_t total = 6 * nd + ni + tree_b + al(64) + (A.use_smem ? 0 : 4 * nd + ni);
  StreamSet set;
  const cudaError_t es = stream_set_take(&set);
  e->stream = set.stream;
  e->ev0 = set.ev0;
  e->ev1 = set.ev1;
  e->stream_dev = set.dev;
  if (es != cudaSuccess || host_block_alloc(&e->h_ret, 64) != cudaSuccess) {
    cudaGetLastError();
    free_exact(e);
    return fail(WG_ERR_CUDA, "exact solver: stream set-up failed");
  }
  if (block_alloc(&e->mem, total) != cudaSuccess) {
    cudaGetLastError();
    free_exact(e);
    return fail(WG_ERR_NOMEM, "exact solver: cudaMalloc of %zu bytes failed", total);
  }
  char* p = static_cast<char*>(e->mem);
  A.g.x = reinterpret_cast<double*>(p); p += nd;
  A.g.v = reinterpret_cast<double*>(p); p += nd;
  A.g.a = reinterpret_cast<double*>(p); p += nd;
  A.g.m = reinterpret_cast<double*>(p); p += nd;
  A.g.t = reinterpret_cast<double*>(p); p += nd;
  A.g.tcoll = reinterpret_cast<double*>(p); p += nd;
  A.g.id = reinterpret_cast<int32_t*>(p); p += ni;
  A.p = A.g;
  if (!A.use_smem) {
    // (the clocks and pair times belong to positions and have one copy)
    A.p.x = reinterpret_cast<double*>(p); p += nd;
    A.p.v = reinterpret_cast<double*>(p); p += nd;
    A.p.a = reinterpret_cast<double*>(p); p += nd;
    A.p.m = reinterpret_cast<double*>(p); p += nd;
    A.p.id = reinterpret_cast<int32_t*>(p); p += ni;
  }
  for (int lv = 0; lv < A.levels; ++lv) {
    A.tree_key[lv] = reinterpret_cast<uint64_t*>(p); p += al(8 * (size_t)A.level_n[lv + 1]);
    A.tree_idx[lv] = reinterpret_cast<int32_t*>(p); p += al(4 * (size_t)A.level_n[lv + 1]);
  }
  A.tree_bytes = smem_tree;
  A.cindx = reinterpret_cast<int*>(p);
  A.err = A.cindx + 1;
  A.ncoll = reinterpret_cast<long long*>(A.cindx + 2);
  A.next_tcoll = reinterpret_cast<double*>(A.cindx + 4);
  e->smem = A.use_smem ? smem : A.tree_bytes;
  bool fits = e->smem <= (size_t)optin;
  // the kernel's own shared variables come on top: within that of the limit,
  // the lowest level's indices (the last part of the tree) stay outside
  A.idx0_global = fits && e->smem + kExactStatic > (size_t)optin;
  if (A.idx0_global) e->smem -= 4 * (size_t)A.level_n[1];
  if (!fits || e->smem > smem_limit()) {
    free_exact(e);
    return fail(WG_ERR_ARG, "exact solver: %lld sheets need more shared memory for the pair-time "
                            "tree than a block has", (long long)n);
  }
  cudaStream_t s = e->stream;
  cudaError_t ce = cudaSuccess;
  auto up = [&](void* d, const void* h, size_t b) {
    if (ce == cudaSuccess) ce = cudaMemcpyAsync(d, h, b, cudaMemcpyHostToDevice, s);
  };
  up(A.g.x, x, 8 * n);
  up(A.g.v, v, 8 * n);
  up(A.g.a, a, 8 * n);
  up(A.g.m, m, 8 * n);
  up(A.g.id, sindx, 4 * n);
  if (ce == cudaSuccess) {
    k_exact_pairs<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(A.g, (int)n, A.omega);
    ce = cudaGetLastError();
  }
  if (ce == cudaSuccess) ce = cudaStreamSynchronize(s);
  if (ce != cudaSuccess) {
    free_exact(e);
    return fail(WG_ERR_CUDA, "exact solver: set-up failed: %s", cudaGetErrorString(ce));
  }
  // the first crossing, as the reference's argmin (lowest index on ties; a
  // NaN pair time never comes first)
  std::vector<double> tc((size_t)n - 1);
  cudaMemcpy(tc.data(), A.g.tcoll, 8 * (size_t)(n - 1), cudaMemcpyDeviceToHost);
  int ci = -1;
  for (int i = 0; i < (int)n - 1; ++i)
    if (!std::isnan(tc[(size_t)i]) && (ci < 0 || tc[(size_t)i] < tc[(size_t)ci])) ci = i;
  const double nxt = ci < 0 ? INFINITY : tc[(size_t)ci];
  if (ci < 0) ci = 0;
  int hret[2] = {ci, 0};
  cudaMemcpy(A.cindx, hret, 8, cudaMemcpyHostToDevice);
  cudaMemcpy(A.next_tcoll, &nxt, 8, cudaMemcpyHostToDevice);
  *out = e;
  return WG_OK;
}

int wg_exact_step(wg_exact* e, double dt, int64_t maxcoll, int64_t* ncoll,
                  double* time_elapsed) {
  if (!e || !(dt > 0) || !std::isfinite(dt) || maxcoll < 0)
    return fail(WG_ERR_ARG, "exact solver: needs a handle, dt > 0 and maxcoll >= 0");
  ExactArgs& A = e->args;
  A.dt = dt;
  A.maxcoll = (long long)maxcoll;
  cudaStream_t s = e->stream;
  // the tree over this interval's pair times
  for (int lv = 0; lv < A.levels; ++lv) {
    const int groups = (A.level_n[lv] + kTreeFan - 1) / kTreeFan;
    k_exact_tree_level<<<(unsigned)((groups + 7) / 8), 256, 0, s>>>(A, lv);
  }
  const unsigned blocks = (unsigned)((e->n + 255) / 256);
  cudaEventRecord(e->ev0, s);
  if (!A.use_smem) k_exact_gather<<<blocks, 256, 0, s>>>(A);
  if (A.omega > 0)
    k_exact_step<true><<<1, 64, e->smem, s>>>(A);
  else
    k_exact_step<false><<<1, 64, e->smem, s>>>(A);
  if (!A.use_smem) k_exact_scatter<<<blocks, 256, 0, s>>>(A);
  cudaEventRecord(e->ev1, s);
  // (a launch that was refused leaves the state, and what is read back, as it was)
  cudaError_t ce = cudaGetLastError();
  if (ce == cudaSuccess)
    ce = cudaMemcpyAsync(e->h_ret, A.cindx, 24, cudaMemcpyDeviceToHost, s);
  const cudaError_t cw = cudaStreamSynchronize(s);
  if (ce == cudaSuccess) ce = cw;
  if (ce != cudaSuccess) return fail(WG_ERR_CUDA, "exact solver: %s", cudaGetErrorString(ce));
  long long nc = 0;
  std::memcpy(&nc, e->h_ret + 2, 8);
  if (ncoll) *ncoll = nc;
  float ms = 0;
  cudaEventElapsedTime(&ms, e->ev0, e->ev1);
  if (time_elapsed) *time_elapsed = ms * 1e-3;
  if (e->h_ret[1] == -2) return fail(WG_ERR_MAXCOLL, "Maximum number of collisions per time "
                                                     "step exceeded");
  return WG_OK;
}

int wg_exact_download(wg_exact* e, double* x, double* v, double* a, int32_t* sindx) {
  if (!e) return fail(WG_ERR_ARG, "null handle");
  const ExactArgs& A = e->args;
  cudaStream_t s = e->stream;
  cudaError_t ce = cudaSuccess;
  auto down = [&](void* h, const void* d, size_t b) {
    if (h && ce == cudaSuccess) ce = cudaMemcpyAsync(h, d, b, cudaMemcpyDeviceToHost, s);
  };
  down(x, A.g.x, 8 * (size_t)e->n);
  down(v, A.g.v, 8 * (size_t)e->n);
  down(a, A.g.a, 8 * (size_t)e->n);
  down(sindx, A.g.id, 4 * (size_t)e->n);
  if (ce == cudaSuccess) ce = cudaStreamSynchronize(s);
  if (ce != cudaSuccess) return fail(WG_ERR_CUDA, "exact solver: %s", cudaGetErrorString(ce));
  return WG_OK;
}

int wg_exact_destroy(wg_exact* e) {
  free_exact(e);
  return WG_OK;
}

}  // extern "C"
