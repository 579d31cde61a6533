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
// (wendy/wendy.c:53-315, wendy/bst.c); here one warp owns the whole event
// loop and keeps them in a 32-ary tournament tree (each internal node holds
// the minimum of its 32 children and where it lies), so the next event is a
// read of the root and an update rewrites three leaves and their paths, each
// level one coalesced 32-wide load and a warp minimum.  The state lives in
// position order, in shared memory when it fits (a few thousand sheets), in
// global memory otherwise.
//
// The loop is a strict sequence of crossings, each a chain of dependent FP64
// operations, so what bounds it is that chain's latency.  The four sheets
// around a crossing sit in four lanes: they are advanced at once, the five
// divisions of the three new pair times are one division of five lanes (a
// second group of four lanes takes the constant terms), the two square roots
// one square root, and a minimum is two warp-reduce instructions.  Measured
// at 1001 sheets of a sech^2 disk: EXACT_NUMBERS
//
// Arithmetic, operation order and the per-sheet clocks follow the
// reference (this file is compiled without FMA contraction, as the
// reference's C is), so trajectories agree to rounding; pair times that are NaN
// (pairs that never meet in the harmonic case) never come first, and among
// equal pair times the lowest pair index comes first.
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <vector>

#include "../../include/wendy_gb300.h"
#include "wg_internal.cuh"

using namespace wg;

namespace {

constexpr int kTreeFan = 32;
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
  return isnan(t) ? ~0ull : key_of(t);
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

// Recomputes the tree path above pair time `leaf` (all lanes); returns the
// root's pair index and key.
__device__ __forceinline__ int tree_update(const ExactArgs& A, uint64_t* const* tkey,
                                           int32_t* const* tidx, const double* tcoll, int leaf,
                                           int lane, uint64_t& root) {
  int g = leaf / kTreeFan;  // group at level 0
  int j = g * kTreeFan + lane;
  uint64_t k = j < A.level_n[0] ? time_key(tcoll[j]) : ~0ull;
  int where;
  uint64_t best = warp_min_key(k, where);
  int idx = g * kTreeFan + where;
  if (idx >= A.level_n[0]) idx = A.level_n[0] - 1;  // a group of NaN times only
  for (int lv = 1;; ++lv) {
    if (lane == 0) {
      tkey[lv - 1][g] = best;
      tidx[lv - 1][g] = idx;
    }
    if (lv == A.levels) break;
    const int child = g;
    g /= kTreeFan;
    j = g * kTreeFan + lane;
    // the child just rewritten comes from registers
    k = j == child ? best : j < A.level_n[lv] ? tkey[lv - 1][j] : ~0ull;
    int i = j == child ? idx : j < A.level_n[lv] ? tidx[lv - 1][j] : 0;
    best = warp_min_key(k, where);
    idx = __shfl_sync(0xffffffffu, i, where);
  }
  root = best;
  return idx;
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

__global__ void __launch_bounds__(32, 1) k_exact_step(const ExactArgs A) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x;
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
    for (int lv = 0; lv < A.levels; ++lv) {
      tidx[lv] = reinterpret_cast<int32_t*>(p);
      p += 4 * (size_t)A.level_n[lv + 1];
    }
    for (int lv = 0; lv < A.levels; ++lv)
      for (int j = lane; j < A.level_n[lv + 1]; j += 32) {
        tkey[lv][j] = A.tree_key[lv][j];
        tidx[lv][j] = A.tree_idx[lv][j];
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
      for (int i = lane; i < n; i += 32) {
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
  for (int i = lane; i < n; i += 32) S.t[i] = 0.;
  __syncwarp();
  const double omega = A.omega, dt = A.dt;
  int cindx = *A.cindx;
  double next = *A.next_tcoll;
  long long cnt = 0;
  // lanes 0 .. 3 (and 4 .. 7 again, for the second divisions) hold the
  // sheets at positions ci - 1 .. ci + 2 of a crossing of ci and ci + 1
  const int role = lane & 3;
  const bool mid = role == 1 || role == 2, first = lane < 4;
  while (next < dt && cnt < A.maxcoll) {
    ++cnt;
    const int ci = cindx;
    const int pos = ci - 1 + role;
    const bool have = pos >= 0 && pos < n;  // the outer two may not exist
    const int at = have ? pos : ci;
    double x = S.x[at], v = S.v[at], a = S.a[at], t = S.t[at];
    const double m = S.m[at];
    const int32_t id = S.id[at];
    // to the time of the crossing.  Without a harmonic potential the outer
    // two are only extrapolated, in the reference's order of additions
    // ((x + a t^2 / 2) + v t, against x + (a t^2 / 2 + v t)), and keep their
    // clocks
    if (omega > 0) {
      advance(x, v, a, t, next, omega);
    } else {
      const double tdt = next - t;
      const double dv = a * tdt;
      const double p = dv * tdt / 2., q = v * tdt;
      x = (p + (mid ? q : x)) + (mid ? x : q);
      v += dv;
    }
    // the two swap places and exchange accelerations by the mass difference
    {
      const double mo = __shfl_xor_sync(0xffffffffu, m, 3);
      const double dm = role == 1 ? mo - m : m - mo;
      const double ad = a - dm;
      const double ao = __shfl_xor_sync(0xffffffffu, ad, 3);
      if (mid) a = ao;
    }
    // partners of the new pairs: the left neighbour meets the sheet from
    // ci + 1, the right one that from ci, and those two each other
    const int partner = (lane & 4) | (role == 0 ? 2 : role == 3 ? 1 : role ^ 3);
    const double xp = __shfl_sync(0xffffffffu, x, partner);
    const double vp = __shfl_sync(0xffffffffu, v, partner);
    const double ap = __shfl_sync(0xffffffffu, a, partner);
    double tn;
    if (omega > 0) {
      if (mid) {
        double q = (v - vp) / (ap - a) / omega;
        q *= q;
        q = (1. - q) / (1. + q);
        tn = acos(q) / omega;
      } else {
        tn = solve_coll_harm(x - xp, v - vp, a - ap, omega);
      }
    } else {
      // the outer pairs' quadratic c2 t^2 + c1 t + c0 (wendy/wendy.c:33-38)
      // and the inner pair's other root, one division per lane
      const double c0 = x - xp, c1 = v - vp, c2 = 0.5 * (a - ap);
      const double num = mid ? 2. * c1 : first ? -c1 : 4. * c0;
      const double quo = num / (mid ? ap - a : c2);
      const double qc = __shfl_xor_sync(0xffffffffu, quo, 4);
      tn = mid ? quo : 0.5 * (quo + sqrt(quo * quo - qc));
    }
    if (first) {
      if (mid) {
        const int to = role == 1 ? ci + 1 : ci;
        S.x[to] = x;
        S.v[to] = v;
        S.a[to] = a;
        S.m[to] = m;
        S.t[to] = next;
        S.id[to] = id;
      } else if (have && omega > 0) {
        S.x[at] = x;
        S.v[at] = v;
        S.t[at] = next;
      }
      // role 0: pair ci - 1, role 1: pair ci, role 3: pair ci + 1
      if (role != 2 && have) S.tcoll[role == 3 ? ci + 1 : ci - 1 + role] = next + tn;
    }
    __syncwarp();
    // the three pair times that changed, and their paths up the tree; the
    // next crossing is the root
    const int lo = ci > 0 ? ci - 1 : ci, hi = ci < n - 2 ? ci + 1 : ci;
    uint64_t root;
    cindx = tree_update(A, tkey, tidx, S.tcoll, lo, lane, root);
    if (hi / kTreeFan != lo / kTreeFan) {
      __syncwarp();
      cindx = tree_update(A, tkey, tidx, S.tcoll, hi, lane, root);
    }
    next = root == ~0ull ? INFINITY : time_of_key(root);
    __syncwarp();
  }
  // every sheet to the end of the interval, clocks and pending times shifted
  for (int i = lane; i < n; i += 32) {
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
  // next call (k_exact_tree), like the reference rebuilds its BST per call
  if (lane == 0) {
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
  size_t smem = 0;
  int* h_ret = nullptr;  // page-locked: cindx, err, ncoll (as two ints), next (as two ints)
};

namespace {

void free_exact(wg_exact* e) {
  if (!e) return;
  if (e->stream) cudaStreamSynchronize(e->stream);
  if (e->mem) cudaFree(e->mem);
  if (e->h_ret) cudaFreeHost(e->h_ret);
  if (e->ev0) cudaEventDestroy(e->ev0);
  if (e->ev1) cudaEventDestroy(e->ev1);
  if (e->stream) cudaStreamDestroy(e->stream);
  delete e;
}

size_t al(size_t b) { return (b + 255) & ~(size_t)255; }

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
  A.use_smem = smem <= (size_t)optin;
  const size_t total = 6 * nd + ni + tree_b + al(64) + (A.use_smem ? 0 : 4 * nd + ni);
  if (cudaStreamCreateWithFlags(&e->stream, cudaStreamNonBlocking) != cudaSuccess ||
      cudaEventCreate(&e->ev0) != cudaSuccess || cudaEventCreate(&e->ev1) != cudaSuccess ||
      cudaMallocHost(&e->h_ret, 64) != cudaSuccess) {
    cudaGetLastError();
    free_exact(e);
    return fail(WG_ERR_CUDA, "exact solver: stream set-up failed");
  }
  if (cudaMalloc(&e->mem, total) != cudaSuccess) {
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
  if (e->smem > (size_t)optin ||
      cudaFuncSetAttribute(k_exact_step, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)e->smem) != cudaSuccess) {
    cudaGetLastError();
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
  k_exact_step<<<1, 32, e->smem, s>>>(A);
  if (!A.use_smem) k_exact_scatter<<<blocks, 256, 0, s>>>(A);
  cudaEventRecord(e->ev1, s);
  cudaMemcpyAsync(e->h_ret, A.cindx, 24, cudaMemcpyDeviceToHost, s);
  const cudaError_t ce = cudaStreamSynchronize(s);
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
