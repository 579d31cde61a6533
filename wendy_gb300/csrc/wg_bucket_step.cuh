// wg_bucket_step.cuh -- the fused sub-step kernel on bucketed state, a template
// over the kinds of launch, instantiated by wg_bucket.cu (no external force),
// wg_bucket_closed.cu and wg_bucket_expr.cu, which compile side by side.
//
// Between sub-steps the sheets of a simulation live in B buckets of fixed
// capacity; bucket b holds exactly the sheets whose (position key, index)
// lies in [Q_b, Q_{b+1}), in arbitrary order inside the bucket.  One kernel
// launch per sub-step then does, per bucket (one CTA, persistent over a list
// of (simulation, bucket) tasks):
//
//   claim the task one bucket ahead (warp 0, while the other warps write out
//     the previous bucket): the bucket's sheet count and exact fixed-point
//     mass were summed by the writers of the previous sub-step, so the
//     look-back over the earlier buckets of the same simulation for the
//     exclusive (mass, count) prefix never has to wait for a load
//   load the bucket into shared memory (optionally applying the half drift
//     a call starts with)
//   sort the bucket by (key, index) in shared memory: the bounded-window
//     fix-up, since a bucket only ever receives sheets from nearby buckets
//     (one counting-sort pass on a 12-bit order-preserving offset, equal
//     offsets ordered by the full key; a multi-pass radix sort when the keys
//     are too clustered for that)
//   exact prefix of the masses in sorted order, a = [ext(x,t) +]
//     (totmass - 2 C - m [- omega^2 x]); kick; drift
//   publish new splitters: the keys at global ranks j*T (quantiles)
//   route every sheet to the bucket of the next layout that covers its new
//     key (splitters computed by the previous sub-step), add the bucket's
//     count and mass to that layout's aggregates and append the sheet there
//     (the sheets of one warp bound for one bucket take consecutive slots)
//
// so a sub-step reads and writes each sheet once (28 B in, 28 B out).  A
// bucket that would overflow its capacity sends the sheet to an overflow
// list and flags the simulation, whose host side then re-sorts from scratch;
// no sheet is ever lost.  Simulations never interact: every sum, sort and
// splitter is per simulation, so a simulation gives the same bits alone and
// in an ensemble.
//
// Reference: _nbody_force and leapfrog_leappq, wendy/wendy.c:324-384; the
// argsort at wendy/wendy.c:341-357 is what the bucket sort replaces.
#pragma once
#include <cstdint>

#include "wg_bucket.cuh"

namespace wg {

namespace {

constexpr int BT = kBucketThreads;  // 256
constexpr int CAP = kBucketCap;     // 2048
constexpr int MAXI = CAP / BT;      // 8 sheets per thread at most
constexpr int WARPS = BT / 32;
constexpr int RWIN = kSplitterWindow;
constexpr int QB_MIN = 11, QB_MAX = 12;  // counting-sort bits the kernel uses
constexpr int NBIN = 1 << QB_MAX;        // bins the shared memory is sized for
constexpr int SHLIST = 64;               // shared bins a warp can list
constexpr int CTAS = 3;                  // resident CTAs per SM
constexpr int MAXBIN = 48;          // a fuller bin sends the bucket to the radix sort
// Big buckets are cut into chunks of at most CAP sheets along 4096 key bins:
// a chunk starts at every bin whose exclusive count passes a multiple of
// CHUNK, so a chunk holds at most CHUNK + (its last bin) <= CAP sheets as long
// as no bin holds more than CAP - CHUNK.
constexpr int BIGBINS = 4096;
constexpr int CHUNK = CAP / 2;
constexpr int kMaxChunks = kBucketCapBig / CHUNK + 1;
// Two 16-bit bin counters (later offsets) per 32-bit word: bin b lives in the
// half (b & 1) of word b / 2.  The scan takes each thread's consecutive words
// with 16-byte loads, so the words need no padding against bank conflicts
// (a quarter warp's loads of 32-byte pieces conflict twice, not eight times).
constexpr int NWORD = NBIN / 2;
// Offset (or count) of bin b in the packed words.
__device__ __forceinline__ uint32_t bin_get(const uint32_t* bins, int b) {
  return (bins[b >> 1] >> ((b & 1) << 4)) & 0xffffu;
}
// Most splitters that one pass over CAP sheets can publish: a bucket may have
// grown to CAP whatever its target.
constexpr int SAMPLES = CAP / kSmallestTarget + 1;
// Cells of the routing table over a splitter window (see route_table).
constexpr int LUTN = 256;

struct LsdSmem {
  uint16_t p[CAP];           // the other slot permutation (S.perm is the first)
  uint16_t hist[WARPS][256];
};

struct __align__(16) StepSmem {
  double x[CAP];
  double v[CAP];
  double m[CAP];
  int32_t idx[CAP];
  uint16_t perm[CAP];  // sorted position -> slot
  union {
    struct {
      uint32_t bins[NWORD + 4];              // (+ the offset past the last bin)
      uint16_t shared_bin[WARPS][SHLIST];    // per warp: bins its sheets found occupied once
      uint32_t nlong;                        // bins too full for their owner to order
    } srt;
    LsdSmem lsd;
    // destination (window entry << 16 | rank among its sheets) of each sorted
    // position, then (window entry << 16 | slot) grouped by destination; the
    // entry is the window length for a bucket outside the window
    uint32_t dest[CAP];
  } u;
  // splitter window of the next layout
  uint64_t wkey[2 * RWIN + 2];
  int32_t widx[2 * RWIN + 2];
  uint32_t dcount[2 * RWIN + 2];  // sheets bound for each window entry (+ outside the window)
  uint32_t dstart[2 * RWIN + 3];  // their exclusive prefix: segments of the grouped order
  uint32_t dbase[2 * RWIN + 2];   // first slot of each window bucket taken by this bucket
  uint8_t lut[LUTN + 4];          // routing table over the window (route_table)
  uint32_t cell_cnt[LUTN / 4];    // splitters of the window in each of its cells (bytes)
  float lut_x0, lut_scale;
  unsigned next_ticket;              // the next task's ticket and entry, read ahead
  BucketTask next_tk;
  u128 warp_mass[WARPS];
  uint32_t scan_tmp[WARPS];
  u128 prefix_mass;
  int eq;
  uint32_t prefix_cnt;
  uint64_t red_min[WARPS], red_max[WARPS];
  TaskMeta next;
  int win_lo, win_hi;
  int amp_sim;            // simulation whose time factor warp 0 has at hand (-1: none) ...
  double amp_kept, inv_h_kept;  // ... and the factor
  double amp, inv_h;
  unsigned long long maxv;
  unsigned maxc;  // largest destination count this task saw after its reservations
  float vsum[WARPS];      // per warp: sum of the new velocities (predicted splitters)
  unsigned nsamp;         // splitter samples of this task
  double samp_x[SAMPLES];
  int32_t samp_idx[SAMPLES];
  uint32_t samp_q[SAMPLES];
  uint64_t mbar;  // completion of the bucket's bulk copies
  int big_head;   // first of the big buckets this CTA has claimed (-1: none)
  // a big bucket (process_big): its chunks as ranges of key bins
  int chunk_lo[kMaxChunks + 1];
  int nchunks;
  unsigned load_cnt;  // sheets of the current chunk gathered so far
  unsigned splittable;
};

// CTAS CTAs per SM: 228 KiB of shared memory per SM, 1 KiB reserved per CTA.
// Three (24 warps at 80 registers) rather than two with more of the work kept
// in shared memory (fixed-point masses, 64-bit sort keys): the kernel is
// bound by latency and issue, and the third CTA hides more of it than the
// recomputed conversions cost.
static_assert(CTAS * (sizeof(StepSmem) + 1024) <= 228 * 1024, "StepSmem too large");
static_assert(2 * RWIN + 2 <= BT, "one window entry per thread");
static_assert(LUTN == BT, "one routing-table cell per thread");
// process_big keeps its histogram where its chunks' positions go later
static_assert(sizeof(double) * CAP >= 4 * BIGBINS, "big-bucket histogram");

__device__ __forceinline__ bool pair_less(uint64_t k1, int32_t i1, uint64_t k2, int32_t i2) {
  return k1 < k2 || (k1 == k2 && i1 < i2);
}

// Block-wide exclusive scan of one value per thread; returns the exclusive
// prefix and (through total) the block total.  Contains one barrier; the
// caller passes another before the next call (scan_tmp is reused).
__device__ __forceinline__ uint32_t block_excl_scan(StepSmem& S, uint32_t v, uint32_t& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) S.scan_tmp[warp] = incl;
  __syncthreads();
  uint32_t pre = 0;
  total = 0;
#pragma unroll
  for (int w = 0; w < WARPS; ++w) {
    const uint32_t t = S.scan_tmp[w];
    pre += (w < warp) ? t : 0u;
    total += t;
  }
  return pre + incl - v;
}

// Multi-pass fallback: stable LSD radix sort of the slots by 32-bit
// order-preserving offsets (recomputed from the positions), 8 bits per pass
// over the bits that differ, then exact tie order.
__device__ __forceinline__ void lsd_sort(StepSmem& S, int n, uint64_t kmin, uint64_t kmax) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint64_t span = kmax - kmin;
  const int bits = span ? 64 - __clzll((long long)span) : 0;
  const int shift = bits > 32 ? bits - 32 : 0;
  const int passes = (bits - shift + 7) / 8;
  LsdSmem& L = S.u.lsd;
  auto offset = [&](int slot) { return (uint32_t)((key_of(S.x[slot]) - kmin) >> shift); };
  __syncthreads();  // the union was just used as counting-sort bins
  // an even number of permutation moves ends in S.perm
  uint16_t* src = (passes & 1) ? L.p : S.perm;
  uint16_t* dst = (passes & 1) ? S.perm : L.p;
  for (int j = tid; j < n; j += BT) src[j] = (uint16_t)j;
  __syncthreads();
  for (int pass = 0; pass < passes; ++pass) {
    const int ds = 8 * pass;
    for (int i = lane; i < 256; i += 32) L.hist[warp][i] = 0;
    __syncwarp();
    uint16_t rank[MAXI], slot[MAXI];
    uint8_t dig[MAXI];
#pragma unroll
    for (int i = 0; i < MAXI; ++i) {
      const int j = warp * (32 * MAXI) + i * 32 + lane;
      const bool ok = j < n;
      unsigned d = 256u + lane;
      if (ok) {
        slot[i] = src[j];
        d = (offset(slot[i]) >> ds) & 255u;
      }
      dig[i] = (uint8_t)d;
      const unsigned peers = __match_any_sync(0xffffffffu, d);
      uint32_t old = 0;
      if (ok) {
        old = L.hist[warp][d];
        rank[i] = (uint16_t)(old + __popc(peers & lanemask_lt()));
      }
      __syncwarp();
      if (ok && lane == __ffs(peers) - 1) L.hist[warp][d] = (uint16_t)(old + __popc(peers));
      __syncwarp();
    }
    __syncthreads();
    uint32_t run = 0;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) {
      const uint32_t c = L.hist[w][tid];
      L.hist[w][tid] = (uint16_t)run;
      run += c;
    }
    uint32_t total;
    const uint32_t base = block_excl_scan(S, run, total);
#pragma unroll
    for (int w = 0; w < WARPS; ++w) L.hist[w][tid] += (uint16_t)base;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < MAXI; ++i) {
      const int j = warp * (32 * MAXI) + i * 32 + lane;
      if (j < n) dst[L.hist[warp][dig[i]] + rank[i]] = slot[i];
    }
    __syncthreads();
    uint16_t* const t = src;
    src = dst;
    dst = t;
  }
  // equal offsets: order by the full (key, idx)
  for (int j = tid; j + 1 < n; j += BT) {
    const uint32_t qj = offset(S.perm[j]);
    if (qj != offset(S.perm[j + 1]) || (j > 0 && offset(S.perm[j - 1]) == qj)) continue;
    int e = j + 1;
    while (e + 1 < n && offset(S.perm[e + 1]) == qj) ++e;
    for (int a = j + 1; a <= e; ++a) {
      const uint16_t s = S.perm[a];
      const uint64_t ks = key_of(S.x[s]);
      const int32_t is = S.idx[s];
      int b = a - 1;
      while (b >= j && pair_less(ks, is, key_of(S.x[S.perm[b]]), S.idx[S.perm[b]])) {
        S.perm[b + 1] = S.perm[b];
        --b;
      }
      S.perm[b + 1] = s;
    }
  }
  __syncthreads();
}

// Inverse of key_of (of the canonical key: +0 for the zeros).
__device__ __forceinline__ double pos_of_key(uint64_t k) {
  return __longlong_as_double((long long)((k >> 63) ? (k & 0x7FFFFFFFFFFFFFFFull) : ~k));
}

// The smallest and largest key of a warp: the upper halves first, then the
// lower halves among the lanes that share the extreme upper half (four
// warp-reduce instructions instead of five rounds of 64-bit shuffles).
__device__ __forceinline__ uint64_t warp_min_u64(uint64_t k) {
  const uint32_t hi = (uint32_t)(k >> 32);
  const uint32_t h = __reduce_min_sync(0xffffffffu, hi);
  const uint32_t l = __reduce_min_sync(0xffffffffu, hi == h ? (uint32_t)k : 0xffffffffu);
  return ((uint64_t)h << 32) | l;
}
__device__ __forceinline__ uint64_t warp_max_u64(uint64_t k) {
  const uint32_t hi = (uint32_t)(k >> 32);
  const uint32_t h = __reduce_max_sync(0xffffffffu, hi);
  const uint32_t l = __reduce_max_sync(0xffffffffu, hi == h ? (uint32_t)k : 0u);
  return ((uint64_t)h << 32) | l;
}

// A position in single precision, truncated, on the integer pipe (a conversion
// would be one of the four to six FP64 instructions a sheet costs, on the pipe
// that is nearest to its limit).  Non-decreasing in x; magnitudes below the
// normal single-precision range become zero, above it its end.
__device__ __forceinline__ float float_of_pos(double x) {
  const uint32_t h = (uint32_t)__double2hiint(x), l = (uint32_t)__double2loint(x);
  const uint32_t a = h & 0x7fffffffu;
  const uint32_t c = min(a, 0x47efffffu);
  const uint32_t f = __funnelshift_l(c == a ? l : 0xffffffffu, c, 3) + 0x40000000u;
  return a < 0x38100000u ? 0.f : __uint_as_float(f | (h & 0x80000000u));
}

// Cell of a position in the routing table.  Every step (rounding to single
// precision, subtraction, product with a non-negative scale, truncation,
// clamping) is non-decreasing, so a splitter in a lower cell than a position
// lies below it, whatever the rounding.
__device__ __forceinline__ int lut_cell(float x, float x0, float scale) {
  return (int)fminf(fmaxf((x - x0) * scale, 0.f), (float)(LUTN - 1));
}

// Routing table over the splitter window [lo, hi] of the next layout (wlen =
// hi - lo buckets): lut[c] is the largest window entry whose splitter lies in
// a cell below c, so the entry of a position in cell c is one of lut[c] ..
// lut[c + 1] -- one or two candidates where the window's splitters are spread
// over the cells, against the six or seven rounds of a search of the window.
// Cells are cut in position, not in key, space (keys are logarithmic about
// zero).  Here the cell of this thread's splitter (threads 1 .. wlen - 1;
// -1 for the others); the sort counts the splitters per cell and sums the
// counts along with its own bins.
// wk: the window's keys; first, last: it begins or ends with the layout (and
// with an infinite splitter).
__device__ __forceinline__ int route_cell(StepSmem& S, const uint64_t* wk, int wlen, bool first,
                                          bool last) {
  const int j = threadIdx.x;
  if (j < LUTN / 4) S.cell_cnt[j] = 0u;
  if (j >= wlen) return -1;
  // the first and last finite splitters of the window
  const int j0 = first ? 1 : 0, j1 = last ? wlen - 1 : wlen;
  float x0 = 0.f, scale = 0.f;
  if (j1 > j0) {
    x0 = float_of_pos(pos_of_key(wk[j0]));
    const float w = float_of_pos(pos_of_key(wk[j1])) - x0;
    if (w > 1e-30f && w < 1e30f) scale = (float)LUTN / w;
  }
  if (j == 0) {
    S.lut_x0 = x0;
    S.lut_scale = scale;
    return -1;
  }
  return lut_cell(float_of_pos(pos_of_key(wk[j])), x0, scale);
}

// The splitters in this thread's cell (at most 128 in all: a byte holds them).
__device__ __forceinline__ uint32_t cell_count(const StepSmem& S) {
  return reinterpret_cast<const uint8_t*>(S.cell_cnt)[threadIdx.x];
}

// (key, idx) of the sheet in slot a precedes that of slot b.
__device__ __forceinline__ bool slot_less(const StepSmem& S, uint64_t ka, int a, uint64_t kb,
                                          int b) {
  if (ka != kb) return ka < kb;
  return S.idx[a] < S.idx[b];
}

// Puts the places [lo, hi) of one bin in (key, idx) order (one thread).  Up
// to four sheets -- nearly every shared bin -- are ranked by comparing all
// pairs, their loads in flight together; more by insertion.
__device__ __forceinline__ void order_bin(StepSmem& S, uint32_t lo, uint32_t hi) {
  const uint32_t c = hi - lo;
  if (c <= 4) {
    int p[4];
    uint64_t k[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) p[a] = S.perm[lo + ((uint32_t)a < c ? (uint32_t)a : 0u)];
#pragma unroll
    for (int a = 0; a < 4; ++a) k[a] = key_of(S.x[p[a]]);
    uint32_t r[4] = {0, 0, 0, 0};
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = a + 1; b < 4; ++b)
        if ((uint32_t)b < c) {
          const bool ba = slot_less(S, k[b], p[b], k[a], p[a]);
          r[a] += ba ? 1u : 0u;
          r[b] += ba ? 0u : 1u;
        }
#pragma unroll
    for (int a = 0; a < 4; ++a)
      if ((uint32_t)a < c) S.perm[lo + r[a]] = (uint16_t)p[a];
    return;
  }
  for (uint32_t a = lo + 1; a < hi; ++a) {
    const uint16_t pa = S.perm[a];
    const uint64_t ka = key_of(S.x[pa]);
    uint32_t b = a;
    while (b > lo) {
      const uint16_t pb = S.perm[b - 1];
      if (!slot_less(S, ka, pa, key_of(S.x[pb]), pb)) break;
      S.perm[b] = pb;
      --b;
    }
    S.perm[b] = pa;
  }
}

// Sort the n <= CAP sheets of the bucket by (key, idx) into S.perm, with
// 2^qb bins (QB_MIN <= qb <= QB_MAX).  The bin words are zero on entry (cleared while
// the bucket loads).  pre != 0: the opening half drift of a call, applied to
// the positions on the way.
// Returns false, having changed nothing, if some thread did not see the
// sheets arrive.
__device__ __forceinline__ bool bucket_sort(StepSmem& S, int n, int ipt, int qb, bool arrived,
                                            double pre, int rcell) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nbin = 1 << qb;
  uint32_t* bins = S.u.srt.bins;
  // ---- keys (held in registers until they are counted) and their range
  uint64_t key[MAXI];
  uint64_t kmin = ~0ull, kmax = 0;
#pragma unroll
  for (int i = 0; i < MAXI; ++i) {
    const int j = tid + i * BT;
    key[i] = 0;
    if (arrived && i < ipt && j < n) {
      double x = S.x[j];
      if (pre != 0.0) {
        x = fma(pre, S.v[j], x);
        S.x[j] = x;
      }
      key[i] = key_of(x);
      kmin = key[i] < kmin ? key[i] : kmin;
      kmax = key[i] > kmax ? key[i] : kmax;
    }
  }
  kmin = warp_min_u64(kmin);
  kmax = warp_max_u64(kmax);
  if (lane == 0) {
    S.red_min[warp] = kmin;
    S.red_max[warp] = kmax;
  }
  if (tid == 0) S.u.srt.nlong = 0;  // read after the barriers below
  if (__syncthreads_or(!arrived)) return false;
  if (rcell >= 0) atomicAdd(&S.cell_cnt[rcell >> 2], 1u << (8 * (rcell & 3)));
  kmin = warp_min_u64(S.red_min[lane & (WARPS - 1)]);
  kmax = warp_max_u64(S.red_max[lane & (WARPS - 1)]);
  // Bin of a key: the top 32 bits of its offset in the range, times scale /
  // 2^32, which is non-decreasing in the key and spreads the bucket's key
  // range over all nbin bins (a shift alone would leave up to half of them
  // empty).  The scale is a single-precision quotient shrunk by 2^-20, so
  // the largest key still lands below nbin; a range narrower than nbin keys
  // maps one key per bin.
  const uint64_t span = kmax - kmin;
  int ksh = (span >> 32) ? 32 - __clz((int)(uint32_t)(span >> 32)) : 0;
  const uint32_t span32 = (uint32_t)(span >> ksh);
  bool narrow = span32 < (uint32_t)nbin;
  const uint32_t scale =
      narrow ? 0u
             : (uint32_t)((float)nbin / ((float)span32 + 1.0f) * 4294967296.0f *
                          (1.0f - 9.5367431640625e-07f));
  // Keys are logarithmic in the position: a range of more than two binades --
  // a bucket about x = 0, in the far tail, or a whole small simulation -- would
  // crowd most sheets into a few of its bins.  Such a bucket is cut linearly
  // in position instead (difference, conversion, product and truncation are
  // each non-decreasing); elsewhere the integer map is the cheaper one.
  if (span > (2ull << 52)) {
    const double xmin = pos_of_key(kmin);
    const float w = (float)(pos_of_key(kmax) - xmin);
    const float wscale = w > 1e-30f && w < 1e30f ? (float)nbin / w : 0.f;
#pragma unroll
    for (int i = 0; i < MAXI; ++i) {
      const int j = tid + i * BT;
      if (i < ipt && j < n)
        key[i] = kmin + (uint32_t)fminf((float)(S.x[j] - xmin) * wscale, (float)(nbin - 1));
    }
    ksh = 0;
    narrow = true;
  }
  uint32_t qr[MAXI];     // bin << 16 | rank in it
  uint32_t nshared = 0;  // this warp's entries of shared_bin
  bool full = false;
#pragma unroll
  for (int i = 0; i < MAXI; ++i) {
    if (i < ipt) {
      const int j = tid + i * BT;
      uint32_t rk = 0;
      qr[i] = 0;
      if (j < n) {
        const uint32_t d = (uint32_t)((key[i] - kmin) >> ksh);
        const uint32_t q = narrow ? d : __umulhi(d, scale);
        const int sh = (int)(q & 1u) << 4;
        rk = (atomicAdd(&bins[q >> 1], 1u << sh) >> sh) & 0xffffu;
        qr[i] = (q << 16) | rk;
        full |= rk >= MAXBIN;
      }
      // The order inside a bin comes from atomics.  A bin holds two or more
      // sheets exactly when one of them took rank 1 in it: the bins found
      // that way are listed per warp (a fifth as many as sheets), so that
      // ordering them below takes each lane about one bin.
      const unsigned sm = __ballot_sync(0xffffffffu, rk == 1);
      const uint32_t at = nshared + __popc(sm & lanemask_lt());
      if (rk == 1 && at < SHLIST) S.u.srt.shared_bin[warp][at] = (uint16_t)(qr[i] >> 16);
      nshared += __popc(sm);
    }
  }
  full |= nshared > SHLIST;  // more than the list holds: crowded keys
  if (__syncthreads_or(full)) {
    uint32_t total;
    S.lut[tid] = (uint8_t)block_excl_scan(S, cell_count(S), total);
    if (tid == 0) S.lut[LUTN] = (uint8_t)total;
    lsd_sort(S, n, kmin, kmax);
    return true;
  }
  // exclusive scan of the bins: thread t owns w4 groups of four words
  const int w4 = nbin / (8 * BT);  // 1 or 2
  uint4* const b4 = reinterpret_cast<uint4*>(bins) + tid * w4;
  uint32_t run = 0;
  for (int k = 0; k < w4; ++k) {
    const uint4 c = b4[k];
    const uint32_t s = c.x + c.y + c.z + c.w;
    run += (s & 0xffffu) + (s >> 16);
  }
  // (the routing table's counts ride in the upper half: at most 128 splitters)
  uint32_t total;
  const uint32_t both = block_excl_scan(S, run | (cell_count(S) << 16), total);
  S.lut[tid] = (uint8_t)(both >> 16);
  if (tid == 0) S.lut[LUTN] = (uint8_t)(total >> 16);
  uint32_t off = both & 0xffffu;
  for (int k = 0; k < w4; ++k) {
    uint4 c = b4[k];
    // a word (lo, hi) becomes (off, off + lo)
    uint32_t t = c.x;
    c.x = off * 0x10001u + (t << 16);
    off += (t & 0xffffu) + (t >> 16);
    t = c.y;
    c.y = off * 0x10001u + (t << 16);
    off += (t & 0xffffu) + (t >> 16);
    t = c.z;
    c.z = off * 0x10001u + (t << 16);
    off += (t & 0xffffu) + (t >> 16);
    t = c.w;
    c.w = off * 0x10001u + (t << 16);
    off += (t & 0xffffu) + (t >> 16);
    b4[k] = c;
  }
  if (tid == 0) bins[nbin >> 1] = (uint32_t)n;  // offset of bin nbin
  __syncthreads();
#pragma unroll
  for (int i = 0; i < MAXI; ++i) {
    const int j = tid + i * BT;
    if (i < ipt && j < n) S.perm[bin_get(bins, (int)(qr[i] >> 16)) + (qr[i] & 0xffffu)] = (uint16_t)j;
  }
  __syncthreads();
  // the shared bins, each ordered by one lane of the warp that listed it; bins
  // of more than kOwnerSort sheets (rare) are counted and then ordered by the
  // whole block (owners never touch those bins)
  constexpr uint32_t kOwnerSort = 8;
  for (uint32_t e = (uint32_t)lane; e < nshared; e += 32) {
    const int q = S.u.srt.shared_bin[warp][e];
    const uint32_t lo = bin_get(bins, q), hi = bin_get(bins, q + 1);
    if (hi - lo <= kOwnerSort)
      order_bin(S, lo, hi);
    else
      atomicAdd(&S.u.srt.nlong, 1u);
  }
  __syncthreads();
  if (S.u.srt.nlong == 0) return true;
  // the full bins: each of their sheets counts the sheets of its bin that
  // precede it, then takes that place (slots read-only here)
  uint32_t place[MAXI];
#pragma unroll
  for (int i = 0; i < MAXI; ++i) {
    place[i] = 0xffffffffu;
    const int j = tid + i * BT;
    if (i < ipt && j < n) {
      const int q = (int)(qr[i] >> 16);
      const uint32_t lo = bin_get(bins, q), hi = bin_get(bins, q + 1);
      if (hi - lo > kOwnerSort) {
        const uint64_t kj = key_of(S.x[j]);
        uint32_t r = 0;
        for (uint32_t b = lo; b < hi; ++b) {
          const int sb = S.perm[b];
          r += slot_less(S, key_of(S.x[sb]), sb, kj, j) ? 1u : 0u;
        }
        place[i] = lo + r;
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < MAXI; ++i)
    if (place[i] != 0xffffffffu) S.perm[place[i]] = (uint16_t)(tid + i * BT);
  __syncthreads();
  return true;
}

// Bucket of the next layout covering (k, i): the largest j with Q_j <= (k, i).
// (k, i) >= splitter j of the window (keys first; indices only on a tie)
__device__ __forceinline__ bool win_ge(const uint64_t* wk, const int32_t* wi, int j, uint64_t k,
                                       int32_t i) {
  const uint64_t K = wk[j];
  return k > K || (k == K && i >= wi[j]);
}

__device__ __forceinline__ int dest_bucket(const uint64_t* wk, const int32_t* wi, int lo, int w,
                                           const uint64_t* qk, const int32_t* qi, int64_t nb,
                                           uint64_t k, int32_t i) {
  if (win_ge(wk, wi, 0, k, i) && !win_ge(wk, wi, w, k, i)) {
    int l = 0, len = w;  // Q_{lo+l} <= (k,i) < Q_{lo+l+len}
    while (len > 1) {
      const int half = len >> 1;
      const bool ge = win_ge(wk, wi, l + half, k, i);
      l = ge ? l + half : l;
      len = ge ? len - half : half;
    }
    return lo + l;
  }
  int l = 0, h = (int)nb;  // Q_0 = -inf <= (k,i) < Q_nb = +inf
  while (h - l > 1) {
    const int mid = (l + h) >> 1;
    if (pair_less(k, i, __ldg(&qk[mid]), __ldg(&qi[mid])))
      h = mid;
    else
      l = mid;
  }
  return l;
}

__device__ __forceinline__ u128 mass_of_limbs(const unsigned long long* l) {
  return (u128)l[0] + ((u128)l[1] << 32) + ((u128)l[2] << 64) + ((u128)l[3] << 96);
}

// What the look-back reads of one earlier bucket.
struct PredLoad {
  unsigned c;          // its aggregate count ...
  u128 m;              // ... and mass
  ulonglong2 r0, r1;   // its look-back record
};

__device__ __forceinline__ PredLoad load_pred(const unsigned* cnt, const unsigned long long* mass,
                                              const BucketRec* recs, int64_t jj, bool eq) {
  PredLoad p;
  if (jj >= 0) {
    p.c = cnt[jj];
    p.m = eq ? (u128)0 : mass_of_limbs(mass + 4 * jj);
    const ulonglong2* r = reinterpret_cast<const ulonglong2*>(recs + jj);
    p.r0 = __ldcg(r);
    p.r1 = __ldcg(r + 1);
  } else {
    p.c = 0;
    p.m = 0;
    p.r0 = make_ulonglong2(0ull, 0ull);
    p.r1 = p.r0;
  }
  return p;
}

// Prepares task t (task-list entry tk) for processing; all lanes of one warp.
//
// Reads the simulation's abort word, its arrays for this sub-step, the
// bucket's aggregate and the splitter window of the next layout around the
// bucket, clears the bucket's aggregate slot two sub-steps on, and resolves
// the bucket's exclusive (mass, count) prefix by looking back over the
// earlier buckets of the simulation: a bucket whose inclusive prefix is
// published for this sub-step ends the walk, every other one contributes its
// aggregate.  Aggregates were completed by the previous launch, so the walk
// never waits; the bucket then publishes its own inclusive prefix.  The
// loads of the first look-back group are issued together with all the others.
template <int FORCE, int MASS>
__device__ __forceinline__ void prepare_task(const StepLaunch& L, int sub, unsigned ep, int lane,
                                             unsigned t, BucketTask tk, StepSmem& S) {
  TaskMeta& out = S.next;
  if (lane == 0) out.task = t;
  if (t >= (unsigned)L.ntasks) return;
  const SimDev& D = L.sims[tk.sim];
  const int64_t b = tk.bucket;
  const int cs = (D.cs0 + sub) % kAggSlots;
  const unsigned* cnt = D.bcnt[cs];
  const unsigned long long* mass = D.bmass[cs];
  const BucketRec* recs = D.recs;
  const int rw = D.window;
  const int64_t nbk = D.nb;
  const int wlo = (int)(b > rw ? b - rw : 0);
  const int whi = (int)((b + rw + 1) < nbk ? (b + rw + 1) : nbk);
  // ---- one round of loads
  const unsigned ab = __ldcg(D.ocount + 1);
  const bool eq = MASS == kMassEqual ||
                  (MASS == kMassMixed &&
                   (D.eq == kEqYes || (D.eq == kEqWord && __ldcg(D.eq_word) == 0u)));
  const unsigned own_c = cnt[b];
  const u128 own_m = eq ? (u128)0 : mass_of_limbs(mass + 4 * b);
  int64_t j = b - 1;
  PredLoad pl = load_pred(cnt, mass, recs, j - lane, eq);
  double amp = 0.0, inv_h = 0.0;
  if (FORCE != kForceNone && lane == 0 && D.ext.kind == EXT_PULSE_TANH) {
    // (an exponential and three divisions in FP64, 64 cycles an instruction:
    // once per simulation, not per bucket)
    if (S.amp_sim != tk.sim) {
      S.amp_sim = tk.sim;
      S.amp_kept = pulse_amplitude(D.ext, D.t_seq[sub]);
      S.inv_h_kept = 1.0 / D.ext.p[3];
    }
    amp = S.amp_kept;
    inv_h = S.inv_h_kept;
  }
  // an earlier sub-step of this call overflowed the simulation: its host
  // side finishes the call on the compact path
  if (ab != 0 && (int)ab <= sub) {
    if (lane == 0) out.n = -1;
    return;
  }
  const int capg = D.capg;
  const int n = own_c < (unsigned)capg ? (int)own_c : capg;
  const int lay = (D.lay0 + sub) & 1;
  if (lane == 0 && n > 0) {
    // the bucket is loaded after the current one: bring it into L2 now
    const uint32_t n4 = (uint32_t)((min(n, CAP) + 3) & ~3);
    const int64_t base = b * capg;
    bulk_prefetch_l2(D.bx[lay] + base, n4 * 8u);
    bulk_prefetch_l2(D.bv[lay] + base, n4 * 8u);
    if (!eq) bulk_prefetch_l2(D.bm[lay] + base, n4 * 8u);
    bulk_prefetch_l2(D.bi[lay] + base, n4 * 4u);
  }
  {
    const int cz = (cs + 2) % kAggSlots;
    if (lane == 0) D.bcnt[cz][b] = 0u;
    if (lane < 4) D.bmass[cz][4 * b + lane] = 0ull;
  }
  // ---- look-back
  const uint64_t tag = (uint64_t)(ep & kEpochLimit) << 40;
  constexpr uint64_t PAY = (1ull << 40) - 1;
  u128 pm = 0;
  uint32_t pc = 0;
  while (j >= 0) {
    const bool inc = (j - lane >= 0) && ((pl.r0.x & ~PAY) == tag) &&
                     ((pl.r0.y & ~PAY) == tag) && ((pl.r1.x & ~PAY) == tag) &&
                     ((pl.r1.y & ~PAY) == tag);
    const u128 vm = inc ? ((u128)(pl.r0.x & PAY) | ((u128)(pl.r0.y & PAY) << 40) |
                           ((u128)(pl.r1.x & PAY) << 80) |
                           ((u128)((pl.r1.y >> 32) & 0x7Full) << 120))
                        : pl.m;
    const uint32_t vcl = inc ? (uint32_t)pl.r1.y : pl.c;
    const unsigned pmask = __ballot_sync(0xffffffffu, inc);
    const int stop = pmask ? (__ffs(pmask) - 1) : 31;
    const bool take = lane <= stop;
    if (!eq) pm += warp_sum_u128(take ? vm : (u128)0);
    pc += __reduce_add_sync(0xffffffffu, take ? vcl : 0u);
    if (pmask) break;
    j -= 32;
    if (j >= 0) pl = load_pred(cnt, mass, recs, j - lane, eq);
  }
  if (lane == 0) {
    const u128 im = pm + own_m;
    const uint32_t ic = pc + own_c;
    ulonglong2* r = reinterpret_cast<ulonglong2*>(D.recs + b);
    __stcg(r, make_ulonglong2(tag | ((uint64_t)im & PAY), tag | ((uint64_t)(im >> 40) & PAY)));
    __stcg(r + 1, make_ulonglong2(tag | ((uint64_t)(im >> 80) & PAY),
                                  tag | (((uint64_t)(im >> 120) & 0x7Full) << 32) | ic));
    out.sim = tk.sim;
    out.wlo = wlo;
    out.whi = whi;
    out.bucket = b;
    out.lay = lay;
    out.x = D.bx[lay] + b * capg;
    out.v = D.bv[lay] + b * capg;
    out.m = D.bm[lay] + b * capg;
    out.idx = D.bi[lay] + b * capg;
    out.n = n;
    out.amp = amp;
    out.inv_h = inv_h;
    if constexpr (MASS == kMassMixed) out.eq = eq;
    out.pm_lo = (uint64_t)pm;
    out.pm_hi = (uint64_t)(pm >> 64);
    out.pcnt = pc;
  }
}

// Claims a ticket and prepares its task; all lanes of one warp.
template <int FORCE, int MASS>
__device__ __forceinline__ void claim_task(const StepLaunch& L, int sub, unsigned ep, int lane,
                                           StepSmem& S) {
  unsigned t = 0;
  if (lane == 0) t = atomicAdd(L.ticket, 1u);
  t = __shfl_sync(0xffffffffu, t, 0);
  BucketTask tk{0, 0};
  if (t < (unsigned)L.ntasks) tk = L.tasks[t];
  prepare_task<FORCE, MASS>(L, sub, ep, lane, t, tk, S);
}

// Counting-sort bits of a simulation as the kernel uses them: at least four
// bin words per thread, at most what the shared memory has room for.
__device__ __forceinline__ int step_sort_bits(const SimDev& D) {
  return min(max(D.sort_bits, QB_MIN), QB_MAX);
}
__device__ __forceinline__ void clear_bins(StepSmem& S, int qb) {
  uint4* const b4 = reinterpret_cast<uint4*>(S.u.srt.bins);
  const int nw = 1 << (qb - 3);
  for (int j = threadIdx.x; j < nw; j += BT) b4[j] = make_uint4(0u, 0u, 0u, 0u);
}

// Sort, scan, force, kick, drift, route and write out the n <= CAP sheets of
// a bucket (or of one chunk of a big bucket) that sit in shared memory, with
// their bins cleared; S.prefix_mass / S.prefix_cnt hold the exclusive (mass,
// count) prefix of the first of them, the splitter window of the next layout
// is in S.wkey and its routing table in S.lut.  arrived: this
// thread saw the sheets' copies complete; returns false, having done nothing,
// if some thread did not.  rcell: from route_cell.  pre: the opening half drift still to be applied.
// PREP: warp 0 prepares the next task (ticket nt of thread 0) during the
// grouping, as the main kernel's pipeline does; otherwise (chunks of a big
// bucket) the prefix base is advanced past these sheets at the end.
template <bool LAST, int FORCE, int MASS, bool PREP>
__device__ __forceinline__ bool process_bucket(const StepLaunch& L, StepSmem& S, const SimDev& D,
                                               const int64_t b, const int lay, const int n,
                                               const int sub, const unsigned ep,
                                               const bool arrived, const double pre,
                                               const int rcell, const unsigned nt) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ipt = (n + BT - 1) / BT;
  const int E = D.E;
  // ---- sort the bucket
  if (!bucket_sort(S, n, ipt, step_sort_bits(D), arrived, pre, rcell)) return false;
  BucketTask ntk{0, 0};
  if (PREP && tid == 0 && nt < (unsigned)L.ntasks) ntk = L.tasks[nt];
  const uint64_t* const wk = S.wkey;
  const int32_t* const wi = S.widx;

  // ---- exact prefix of the masses in sorted order: thread tid holds the
  // sorted positions [tid * ipt, tid * ipt + ipt)
  const int j0 = tid * ipt;
  const int nmine = (j0 < n) ? ((n - j0) < ipt ? (n - j0) : ipt) : 0;
  u128 tot = 0;
  u128 incl = 0;
  const bool eq = MASS == kMassMixed ? S.eq != 0 : MASS == kMassEqual;
  const u128 Meq = ((u128)D.meq_hi << 64) | D.meq_lo;
  if (!eq) {
#pragma unroll 2
    for (int i = 0; i < nmine; ++i) tot += mass_to_fixed(S.m[S.perm[j0 + i]], E);
    incl = warp_inclusive_scan_u128(tot, lane);
    if (lane == 31) S.warp_mass[warp] = incl;
  }
  // (the barrier below also ends the use of the bins)
  if (PREP && tid == 0) {
    S.next_ticket = nt;
    S.next_tk = ntk;
  }
  __syncthreads();
  const uint32_t rank0 = S.prefix_cnt + (uint32_t)j0;
  u128 C;
  if (eq) {
    C = Meq * rank0;
  } else {
    C = S.prefix_mass;
    for (int w = 0; w < warp; ++w) C += S.warp_mass[w];
    C += incl - tot;
  }

  // ---- splitters of the layout after next: keys at global ranks j*T
  uint64_t* qnk = D.qk[1 - ((D.qsel0 + sub) & 1)];
  int32_t* qni = D.qi[1 - ((D.qsel0 + sub) & 1)];
  if (b == 0 && tid == 0) {
    qnk[0] = 0ull;
    qni[0] = (int32_t)0x80000000;
    qnk[D.nb] = ~0ull;
    qni[D.nb] = 0x7fffffff;
  }
  // descriptor fields used per sheet, held in registers (the descriptor is
  // in global memory and the compiler cannot prove the stores below leave it alone)
  const int has_omega = D.has_omega;
  const double omega2 = D.omega2;
  const ExtForce ext = D.ext;
  // an expression force: its time phase, once per task and thread
  double xr[FORCE == kForceExpr ? kExprRegs : 1];
  double t_ev = 0.0;
  if constexpr (FORCE == kForceExpr) {
    if (ext.kind == EXT_EXPR) {
      t_ev = D.t_seq[sub];
      expr_time(ext, t_ev, xr);
    }
  }
  const uint32_t target = (uint32_t)D.target;
  const int64_t nbk = D.nb;
  // ---- force, kick, drift, routing; new x, v go back to their slots and
  // the destination of every sorted position to the (now free) sort area
  const double dt = L.profile ? 0.0 : D.dt;
  const double dt_drift = LAST ? dt / 2. : dt;
  const double dest_dt = (LAST && !L.profile) ? dt / 2. : 0.0;
  unsigned long long maxv = 0;
  StateTable* const ptab = D.ptab;  // predicted splitters this sub-step

  // the first rank >= rank0 that is a positive multiple of the target
  // starts the next splitter (one per thread at most: ipt <= 8 < target)
  uint32_t qnext = (rank0 + target - 1) / target;
  qnext = qnext ? qnext : 1u;
  const uint32_t rnext = qnext * target;
  const int wlen = S.win_hi - S.win_lo;
  const float lut_x0 = S.lut_x0, lut_scale = S.lut_scale;
  // the acceleration of the sheet at position j is A_j = T - 2 C_j - M_j with
  // C_j the mass before it; from one sheet to the next A falls by M_j + M_j+1
  i128 A = (i128)(((((u128)D.T_hi) << 64) | D.T_lo) - 2 * C);
#pragma unroll 1
  for (int i = 0; i < nmine; ++i) {
    const int sidx = S.perm[j0 + i];
    const int32_t idv = S.idx[sidx];
    const uint32_t r = rank0 + (uint32_t)i;
    const double x = S.x[sidx], v = S.v[sidx];
    if (r == rnext) {
      qnk[qnext] = key_of(x);
      qni[qnext] = idv;
      if (ptab) {
        const unsigned k = atomicAdd(&S.nsamp, 1u);
        if (k < (unsigned)SAMPLES) {
          S.samp_x[k] = x;
          S.samp_idx[k] = idv;
          S.samp_q[k] = qnext;
        }
      }
    }
    const u128 M = eq ? Meq : mass_to_fixed(S.m[sidx], E);
    A -= (i128)M;
    double acc = fixed_to_double(A, E);
    A -= (i128)M;
    if (has_omega) acc = fma(-omega2, x, acc);
    if constexpr (FORCE == kForceExpr) {
      if (ext.kind == EXT_EXPR)
        acc = expr_space(ext, xr, x, t_ev) + acc;
      else if (ext.kind != EXT_NONE)
        acc = ext_force_at(ext, S.amp, S.inv_h, x) + acc;
    } else if (FORCE == kForceClosed && ext.kind != EXT_NONE) {
      acc = ext_force_at(ext, S.amp, S.inv_h, x) + acc;
    }
    const double vn = fma(dt, acc, v);
    const double xn = fma(dt_drift, vn, x);
    S.x[sidx] = xn;
    S.v[sidx] = vn;

    const unsigned long long av =
        (unsigned long long)__double_as_longlong(vn) & 0x7FFFFFFFFFFFFFFFull;
    maxv = av > maxv ? av : maxv;
    if (LAST && !L.profile) {
      OutRec* const ro = D.rec_out;
      if (ro) {
        double2* const r2 = reinterpret_cast<double2*>(ro + idv);
        r2[0] = make_double2(xn, vn);
        r2[1] = make_double2(acc, 0.0);
      } else {
        D.x_out[idv] = xn;
        D.v_out[idv] = vn;
        double* const a_out = D.a_out;
        if (a_out) a_out[idv] = acc;
      }
      SheetRec* const xi_out = D.xi_out;
      if (xi_out) {
        SheetRec rec;
        rec.idx = idv;
        rec.pad = 0;
        rec.val = xn;
        xi_out[r] = rec;
      }
    }
    const double xd = LAST && dest_dt != 0.0 ? fma(dest_dt, vn, xn) : xn;
    // routing: the window entry among the table's candidates
    const uint64_t kd = key_of(xd);
    const int c = lut_cell(float_of_pos(xd), lut_x0, lut_scale);
    int a = S.lut[c], z = S.lut[c + 1];
    // a position in an end cell may lie outside the window (or on its end):
    // unless it is strictly inside, its bucket is found by the search over
    // all splitters where it is needed.  The cells between lie inside.
    bool inw = true;
    if (c == 0 || c == LUTN - 1) inw = kd > wk[0] && kd < wk[wlen];
    // the largest entry with key Q <= key (entry a of the table lies below
    // the position's cell); then splitters with an equal key and a larger
    // index step back (pair order)
    bool tie = false;
    while (a < z) {
      const int mid = (a + z + 1) >> 1;
      const uint64_t K = wk[mid];
      if (K <= kd) {
        a = mid;
        tie = K == kd;
      } else {
        z = mid - 1;
      }
    }
    if (tie)
      while (a > 0 && wk[a] == kd && wi[a] > idv) --a;
    // destination: window entry a, or wlen for a bucket outside the window
    const int w = inw ? a : wlen;
    S.u.dest[j0 + i] = ((uint32_t)w << 16) | atomicAdd(&S.dcount[w], 1u);
  }
  if (ptab) {
    // the new velocities of this thread's sheets (back from shared memory:
    // a register held across the force loop would spill)
    float vsum = 0.f;
    for (int i = 0; i < nmine; ++i) vsum += (float)S.v[S.perm[j0 + i]];
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) vsum += __shfl_xor_sync(0xffffffffu, vsum, o);
    if (lane == 0) S.vsum[warp] = vsum;
  }
  maxv = warp_max_u64(maxv);
  if (lane == 0 && maxv) atomicMax(&S.maxv, maxv);
  __syncthreads();
  if (ptab && tid < (int)min(S.nsamp, (unsigned)SAMPLES)) {
    // the sample's position moved on by two drifts at the bucket's mean
    // velocity: where the bucket is heading.  The mean, not the sample's
    // own velocity: in a warm region single velocities would scatter the
    // splitters by more than a bucket, while the mean follows the bulk flow
    // of a collapsing or breathing slab (single precision is plenty for a
    // splitter, which only has to be near the quantile)
    float vs = 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) vs += S.vsum[w];
    const StateRef c = ptab->cur;
    const uint32_t q = S.samp_q[tid];
    c.x[q - 1] = fma(2.0 * dt, (double)(vs / (float)n), S.samp_x[tid]);
    c.idx[q - 1] = S.samp_idx[tid];
  }
  // ---- warp 0 prepares the next task, which takes it about as long as the
  // others take for the rest of this one: they group the sheets by destination
  // bucket of the next layout and write them out, synchronising among
  // themselves (named barrier 1)
  bool overflow = false;
  if (PREP && warp == 0) {
    prepare_task<FORCE, MASS>(L, sub, ep, lane, S.next_ticket, S.next_tk, S);
  } else {
    constexpr int nw = PREP ? BT - 32 : BT;
    constexpr int MAXD = (CAP + nw - 1) / nw;
    const int t0 = PREP ? tid - 32 : tid, w0 = t0 >> 5;
    auto sync_out = [] {
      if constexpr (PREP)
        asm volatile("bar.sync 1, %0;" ::"n"(BT - 32) : "memory");
      else
        __syncthreads();
    };
    const int cw = (D.cs0 + sub + 1) % kAggSlots;
    unsigned* const cnt_out = D.bcnt[cw];
    unsigned long long* const mass_out = D.bmass[cw];
    const uint64_t* const qfar = D.qk[(D.qsel0 + sub) & 1];
    const int32_t* const ifar = D.qi[(D.qsel0 + sub) & 1];
    // slots: one atomic per window bucket, its round trip overlapping the
    // grouping (the second of these warps on; the first forms the segments)
    uint32_t db = 0, dcn = 0;
    const int wt = t0 - 32;
    if (wt >= 0 && wt < wlen) {
      dcn = S.dcount[wt];
      if (dcn) db = atomicAdd(&cnt_out[S.win_lo + wt], dcn);
    }
    // the destinations go through registers: the same array then holds the
    // grouped order
    uint32_t dest[MAXD];
#pragma unroll
    for (int i = 0; i < MAXD; ++i)
      if (t0 + i * nw < n) dest[i] = S.u.dest[t0 + i * nw];
    if (w0 == 0) {
      // segments: exclusive prefix of the counts of the wlen + 1 entries
      constexpr int E5 = (2 * RWIN + 2 + 31) / 32;
      uint32_t cv[E5];
      uint32_t sum = 0;
#pragma unroll
      for (int k = 0; k < E5; ++k) {
        const int j = lane * E5 + k;
        cv[k] = j <= wlen ? S.dcount[j] : 0u;
        sum += cv[k];
      }
      uint32_t incl2 = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl2, o);
        if (lane >= o) incl2 += y;
      }
      uint32_t ex = incl2 - sum;
#pragma unroll
      for (int k = 0; k < E5; ++k) {
        const int j = lane * E5 + k;
        if (j <= wlen) S.dstart[j] = ex;
        ex += cv[k];
      }
      if (lane == 31) S.dstart[wlen + 1] = incl2;
    }
    sync_out();
#pragma unroll
    for (int i = 0; i < MAXD; ++i)
      if (t0 + i * nw < n) {
        const uint32_t w = dest[i] >> 16;
        S.u.dest[S.dstart[w] + (dest[i] & 0xffffu)] = (w << 16) | S.perm[t0 + i * nw];
      }
    if (dcn) {
      S.dbase[wt] = db;
      atomicMax(&S.maxc, db + dcn);
    }
    sync_out();
    // write-out grouped by destination: consecutive positions of a segment
    // take consecutive slots, so a warp's stores coalesce
    double* const xout = D.bx[1 - lay];
    double* const vout = D.bv[1 - lay];
    double* const mout = D.bm[1 - lay];
    int32_t* const iout = D.bi[1 - lay];
    const unsigned capg = (unsigned)D.capg;
    for (int q = t0; q < n; q += nw) {
      const uint32_t e = S.u.dest[q];
      const int w = (int)(e >> 16), sl = (int)(e & 0xffffu);
      const double xn = S.x[sl], vn = S.v[sl], mn = eq ? D.meq : S.m[sl];
      const int32_t in = S.idx[sl];
      int d;
      uint32_t slot;
      if (w < wlen) {
        d = S.win_lo + w;
        slot = S.dbase[w] + (uint32_t)q - S.dstart[w];
      } else {
        // outside the window: its bucket is found among all splitters, its
        // slot and mass are added one by one
        const uint64_t kf = key_of(LAST && dest_dt != 0.0 ? fma(dest_dt, vn, xn) : xn);
        d = dest_bucket(wk, wi, S.win_lo, wlen, qfar, ifar, nbk, kf, in);
        slot = atomicAdd(&cnt_out[d], 1u);
        atomicMax(&S.maxc, slot + 1u);
        if (!eq) {
          const u128 M = mass_to_fixed(mn, E);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const unsigned long long limb = (unsigned long long)(uint32_t)(M >> (32 * k));
            if (limb) atomicAdd(&mass_out[4 * (int64_t)d + k], limb);
          }
        }
      }
      if (slot < capg) {
        const int64_t o = (int64_t)d * capg + slot;
        xout[o] = xn;
        vout[o] = vn;
        if (!eq) mout[o] = mn;  // (equal masses are read from D.meq everywhere)
        iout[o] = in;
      } else {
        const uint32_t o = atomicAdd(D.ocount, 1u);
        D.ox[o] = xn;
        D.ov[o] = vn;
        D.om[o] = mn;
        D.oi[o] = in;
        overflow = true;
      }
    }
    // ---- masses of the next layout: a warp sums the fixed-point masses of
    // a window bucket's segment and adds them to that bucket's accumulators
    for (int w = eq ? wlen : w0; w < wlen; w += nw / 32) {
      const int q0 = (int)S.dstart[w], q1 = (int)S.dstart[w + 1];
      if (q0 == q1) continue;
      u128 P = 0;
      for (int q = q0 + lane; q < q1; q += 32)
        P += mass_to_fixed(S.m[S.u.dest[q] & 0xffffu], E);
      P = warp_sum_u128(P);
      if (lane < 4) {
        const unsigned long long limb = (unsigned long long)(uint32_t)(P >> (32 * lane));
        if (limb) atomicAdd(&mass_out[4 * (int64_t)(S.win_lo + w) + lane], limb);
      }
    }
  }
  if (overflow) atomicCAS(D.ocount + 1, 0u, (unsigned)(sub + 1));
  __syncthreads();
  if (tid == 0 && S.maxv) atomicMax(&D.flags[sub + 1].max_v, S.maxv);
  if (tid == 0 && S.maxc) atomicMax(&D.flags[sub + 1].max_cnt, S.maxc);
  if (!PREP && tid == 0) {
    // the next chunk of a big bucket starts where this one ended
    u128 tot_all = 0;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) tot_all += S.warp_mass[w];
    S.prefix_mass += tot_all;
    S.prefix_cnt += (uint32_t)n;
  }
  return true;
}

// Bin of a key in [kmin, kmin + span] among BIGBINS (non-decreasing in the
// key; the same multiplicative map as the in-bucket counting sort).
__device__ __forceinline__ int big_bin(uint64_t k, uint64_t kmin, uint64_t span, uint64_t scale) {
  const uint64_t dk = k - kmin;
  return span < (uint64_t)BIGBINS ? (int)dk : (int)__umul64hi(dk, scale);
}

// Position (with the opening half drift of a call applied) of slot j.
__device__ __forceinline__ double big_pos(const double* gx, const double* gv, int j, double pre) {
  const double x = gx[j];
  return pre != 0.0 ? fma(pre, gv[j], x) : x;
}

// Block-wide minimum and maximum of per-thread key ranges (all threads).
__device__ __forceinline__ void block_range(StepSmem& S, uint64_t& kmin, uint64_t& kmax) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
#pragma unroll
  for (int d = 16; d >= 1; d >>= 1) {
    const uint64_t o1 = __shfl_xor_sync(0xffffffffu, kmin, d);
    const uint64_t o2 = __shfl_xor_sync(0xffffffffu, kmax, d);
    kmin = o1 < kmin ? o1 : kmin;
    kmax = o2 > kmax ? o2 : kmax;
  }
  if (lane == 0) {
    S.red_min[warp] = kmin;
    S.red_max[warp] = kmax;
  }
  __syncthreads();
  kmin = ~0ull;
  kmax = 0;
#pragma unroll
  for (int w = 0; w < WARPS; ++w) {
    kmin = S.red_min[w] < kmin ? S.red_min[w] : kmin;
    kmax = S.red_max[w] > kmax ? S.red_max[w] : kmax;
  }
  __syncthreads();  // red_min / red_max are free again
}

// Puts a big bucket's task on this CTA's list (one thread; entries by bucket,
// chained from S.big_head).  Kept out of line: inlined, its fields stayed live
// across the bucket loop and pushed the kernel into register spills.
static __device__ __noinline__ void list_big(StepSmem& S, TaskMeta* big_list, int* big_next,
                                             unsigned* big_count) {
  const int b = (int)S.next.bucket;
  big_list[b] = S.next;
  big_next[b] = S.big_head;
  S.big_head = b;
  atomicAdd(big_count, 1u);
}

// A big bucket (kBucketCap < n <= capg sheets): cut by key into chunks that
// fit in shared memory -- a histogram of its keys over BIGBINS bins, chunks
// along the bins -- each chunk gathered from the layout and processed like a
// bucket, the chunks in key order with the mass and rank prefix carried from
// one to the next.  A bucket whose keys crowd into one bin beyond CAP - CHUNK
// cannot be cut this way: the simulation is flagged (ocount[2]) and its host
// side re-sorts the layout this sub-step read, which the sub-step leaves
// intact.  A CTA keeps the big buckets it has claimed for when it has no other
// task left; a second launch per sub-step for buckets that are rarely there
// cost 3.3 us and the gap before it, empty.
template <bool LAST, int FORCE, int MASS>
__device__ __forceinline__ void process_big(const StepLaunch& L, StepSmem& S, const TaskMeta& bt,
                                            int sub, unsigned ep) {
  const int tid = threadIdx.x;
  const SimDev& D = L.sims[bt.sim];
  const int n = bt.n;
  const double* gx = bt.x;
  const double* gv = bt.v;
  const double* gm = bt.m;
  const int32_t* gi = bt.idx;
  const double pre = sub == 0 ? D.pre_dt : 0.0;
  const bool eq = MASS == kMassMixed ? bt.eq != 0 : MASS == kMassEqual;
  // the splitter window of the next layout around the bucket
  {
    const int qs = (D.qsel0 + sub) & 1;
    for (int j = tid; j <= bt.whi - bt.wlo; j += BT) {
      S.wkey[j] = D.qk[qs][bt.wlo + j];
      S.widx[j] = D.qi[qs][bt.wlo + j];
    }
  }
  if (tid == 0) {
    S.win_lo = bt.wlo;
    S.win_hi = bt.whi;
    S.maxv = 0;
    S.maxc = 0;
    S.nsamp = 0;
    S.prefix_mass = (((u128)bt.pm_hi) << 64) | bt.pm_lo;
    S.prefix_cnt = bt.pcnt;
    if constexpr (MASS == kMassMixed) S.eq = bt.eq;
    S.amp = bt.amp;
    S.inv_h = bt.inv_h;
    S.nchunks = 0;
    S.splittable = 1u;
    for (int c = 0; c <= kMaxChunks; ++c) S.chunk_lo[c] = BIGBINS;
  }
  // ---- the bucket's key range and the histogram of its keys
  uint64_t kmin = ~0ull, kmax = 0;
  for (int j = tid; j < n; j += BT) {
    const uint64_t k = key_of(big_pos(gx, gv, j, pre));
    kmin = k < kmin ? k : kmin;
    kmax = k > kmax ? k : kmax;
  }
  // BIGBINS 32-bit counters where the chunks' positions go later
  uint32_t* hist = reinterpret_cast<uint32_t*>(S.x);
  for (int j = tid; j < BIGBINS; j += BT) hist[j] = 0u;
  block_range(S, kmin, kmax);
  const uint64_t span = kmax - kmin;
  uint64_t scale = 0;
  if (span >= (uint64_t)BIGBINS)
    scale = (uint64_t)((float)BIGBINS / ((float)span + 1.0f) * 18446744073709551616.0f *
                       (1.0f - 9.5367431640625e-07f));
  for (int j = tid; j < n; j += BT) {
    const int bin = big_bin(key_of(big_pos(gx, gv, j, pre)), kmin, span, scale);
    atomicAdd(&hist[bin], 1u);
  }
  __syncthreads();
  // ---- chunks: thread tid owns bins [16 tid, 16 tid + 16)
  {
    constexpr int BPT = BIGBINS / BT;
    uint32_t c[BPT], sum = 0, mx = 0;
#pragma unroll
    for (int k = 0; k < BPT; ++k) {
      c[k] = hist[tid * BPT + k];
      sum += c[k];
      mx = c[k] > mx ? c[k] : mx;
    }
    uint32_t tot;
    uint32_t ex = block_excl_scan(S, sum, tot);
    if (mx > (uint32_t)(CAP - CHUNK)) atomicAnd(&S.splittable, 0u);
    // non-empty bin i belongs to chunk floor(ex_i / CHUNK), ex_i the
    // sheets in earlier bins; a chunk starts at its first bin.  With no
    // bin above CHUNK, consecutive non-empty bins differ by at most one
    // chunk, and a chunk holds fewer than 2 CHUNK = CAP sheets.
#pragma unroll
    for (int k = 0; k < BPT; ++k) {
      if (c[k]) {
        const uint32_t chunk = ex / CHUNK;
        if (chunk < (uint32_t)kMaxChunks) atomicMin(&S.chunk_lo[chunk], tid * BPT + k);
        atomicMax(&S.nchunks, (int)chunk + 1);
      }
      ex += c[k];
    }
  }
  __syncthreads();
  const int nchunks = S.nchunks;
  if (!S.splittable || nchunks > kMaxChunks) {
    // keys crowded into one bin: the host re-sorts the layout read here
    if (tid == 0) {
      atomicCAS(D.ocount + 2, 0u, (unsigned)(sub + 1));
      atomicCAS(D.ocount + 1, 0u, (unsigned)(sub + 1));
    }
    return;
  }
  if (tid == 0) {
    S.chunk_lo[0] = 0;  // bins below the first non-empty one are empty
    S.chunk_lo[nchunks] = BIGBINS;
  }
  __syncthreads();
  // ---- the chunks in key order
  for (int ch = 0; ch < nchunks; ++ch) {
    const int blo = S.chunk_lo[ch], bhi = S.chunk_lo[ch + 1];
    clear_bins(S, step_sort_bits(D));
    for (int j = tid; j <= S.win_hi - S.win_lo; j += BT) S.dcount[j] = 0;
    if (tid == 0) {
      S.load_cnt = 0;
      S.nsamp = 0;  // splitter samples of this chunk
    }
    __syncthreads();
    for (int j = tid; j < n; j += BT) {
      const double x = big_pos(gx, gv, j, pre);
      const uint64_t k = key_of(x);
      const int bin = big_bin(k, kmin, span, scale);
      if (bin >= blo && bin < bhi) {
        const unsigned slot = atomicAdd(&S.load_cnt, 1u);
        if (slot < (unsigned)CAP) {
          S.x[slot] = x;
          S.v[slot] = gv[j];
          if (!eq) S.m[slot] = gm[j];
          S.idx[slot] = gi[j];
        }
      }
    }
    __syncthreads();
    const int nc = (int)S.load_cnt;
    if (nc > CAP) {  // cannot happen with the chunk rule; never write past the arrays
      if (tid == 0) atomicOr(L.err, DEV_ERR_BAD_STATE);
      break;
    }
    if (nc == 0) continue;
    const int rcell = route_cell(S, S.wkey, bt.whi - bt.wlo, bt.wlo == 0, bt.whi == (int)D.nb);
    process_bucket<LAST, FORCE, MASS, false>(L, S, D, bt.bucket, bt.lay, nc, sub, ep, true, 0.0, rcell,
                                      0u);
  }
}

// The fused sub-step.  LAST: the call's last sub-step (half drift, outputs).
// FORCE: the external forces of the launch's simulations -- none, closed forms
// (and none), or expressions among them (the interpreter).  MASS: their masses
// -- any, all equal, or decided per task.  What a launch does not need costs it
// registers: the choice of masses per task 4 %, the unused force 1.6 %.
template <bool LAST, int FORCE, int MASS>
__global__ void __launch_bounds__(BT, CTAS) k_bucket_step(const __grid_constant__ StepLaunch L) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  StepSmem& S = *reinterpret_cast<StepSmem*>(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int sub = L.sub;
  if (tid == 0) {
    S.big_head = -1;
    S.amp_sim = -1;
    mbar_init(&S.mbar, 1);
    fence_proxy_async_smem();
  }
  chain_begin();
  const unsigned ep = L.epochs[sub];
  if (warp == 0) claim_task<FORCE, MASS>(L, sub, ep, lane, S);
  unsigned parity = 0;
  for (;;) {
    __syncthreads();
    const TaskMeta tm = S.next;  // claimed during the previous task
    if (tm.task >= (unsigned)L.ntasks) break;
    if (tm.n < 0 || tm.n > CAP) {
      // n < 0: the simulation has aborted this call.  n > CAP: more sheets
      // than shared memory holds (a simulation whose layout has room for
      // them), taken in chunks after the others
      if (tm.n > CAP && tid == 0) list_big(S, L.big_list, L.big_next, L.big_count);
      __syncthreads();  // every thread has read S.next
      if (warp == 0) claim_task<FORCE, MASS>(L, sub, ep, lane, S);
      continue;
    }
    const SimDev& D = L.sims[tm.sim];
    const int64_t b = tm.bucket;
    const int lay = tm.lay;
    const int n = tm.n;
    // ---- load: the bucket's four arrays arrive by bulk copy (sizes rounded
    // up to 4 sheets, which stays inside the bucket's capacity), then its
    // keys and key range are formed from shared memory
    const int n4 = (n + 3) & ~3;
    const bool eq = MASS == kMassMixed ? tm.eq != 0 : MASS == kMassEqual;
    if (n4 > 0 && tid == 0) {
      fence_proxy_async_smem();  // earlier generic accesses to these buffers are done
      mbar_expect_tx(&S.mbar, (uint32_t)n4 * (eq ? 20u : 28u));
      bulk_g2s(S.x, tm.x, (uint32_t)n4 * 8u, &S.mbar);
      bulk_g2s(S.v, tm.v, (uint32_t)n4 * 8u, &S.mbar);
      if (!eq) bulk_g2s(S.m, tm.m, (uint32_t)n4 * 8u, &S.mbar);
      bulk_g2s(S.idx, tm.idx, (uint32_t)n4 * 4u, &S.mbar);
    }
    // the next task's ticket and task-list entry are read ahead (thread 0)
    // and the task is prepared by warp 0 during the write-out
    unsigned nt = 0;
    if (tid == 0) nt = atomicAdd(L.ticket, 1u);
    const double pre = sub == 0 ? D.pre_dt : 0.0;
    // the splitter window of the next layout around this bucket (wlen + 1
    // entries, at most one per thread); the per-destination counters are cleared
    const int wlen = tm.whi - tm.wlo;
    const int qs = (D.qsel0 + sub) & 1;
    const uint64_t* const qk = D.qk[qs] + tm.wlo;
    if (tid <= wlen) {
      S.wkey[tid] = qk[tid];
      S.widx[tid] = D.qi[qs][tm.wlo + tid];
      S.dcount[tid] = 0;
    }
    if (tid == 0) {
      S.win_lo = tm.wlo;
      S.win_hi = tm.whi;
      S.maxv = 0;
      S.maxc = 0;
      S.nsamp = 0;
      S.prefix_mass = (((u128)tm.pm_hi) << 64) | tm.pm_lo;
      S.prefix_cnt = tm.pcnt;
      if constexpr (MASS == kMassMixed) S.eq = tm.eq;
      S.amp = tm.amp;
      S.inv_h = tm.inv_h;
    }
    // while the copies are in flight: the counting-sort bins are cleared and
    // the window's splitters take their cells of the routing table
    clear_bins(S, step_sort_bits(D));
    const int rcell = route_cell(S, qk, wlen, tm.wlo == 0, tm.whi == (int)D.nb);
    // the copies' completion: a thread that did not see it within the bounded
    // wait leaves the data alone, and the first barrier of the sort (which
    // every thread reaches) decides for the whole CTA
    const bool arrived = n4 > 0 ? mbar_wait(&S.mbar, parity) : true;
    if (!process_bucket<LAST, FORCE, MASS, true>(L, S, D, b, lay, n, sub, ep, arrived, pre, rcell,
                                          nt)) {
      // the bucket's copies did not complete within the bounded wait: its
      // contents are unknown, so this CTA writes nothing more.  It gives the
      // copies a second bounded wait and stops; the host sees the error word
      // (the call fails and the simulation is given up).
      if (tid == 0) atomicOr(L.err, DEV_ERR_COPY_TIMEOUT);
      mbar_wait(&S.mbar, parity);
      return;
    }
    if (n4 > 0) parity ^= 1u;
  }
  // ---- the big buckets this CTA claimed
  for (int b = S.big_head; b >= 0;) {
    const TaskMeta bt = L.big_list[b];
    b = L.big_next[b];
    process_big<LAST, FORCE, MASS>(L, S, bt, sub, ep);
    __syncthreads();
  }
}

}  // namespace

}  // namespace wg
