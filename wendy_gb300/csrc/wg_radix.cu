// wg_radix.cu -- full on-device re-sort of the sheets: a least-significant-
// digit radix sort of the leading bytes of the 64-bit position keys, 8 bits a
// pass, each pass a single read and write of (key, slot) pairs whose tile
// offsets come from a decoupled look-back over per-tile digit counts
// ("onesweep"), and then the few sheets that share those bytes put in order
// by their whole keys.  It replaces the serial argsort of the reference
// (wendy/wendy.c:341-357) when the order cannot be repaired locally.
//
// Positions of N sheets are told apart by about log2 N bits, not by 64: the
// leading five bytes of a key (sign, exponent, 28 bits of the mantissa) leave
// one pair in a hundred together at 1e6 sheets, four bytes one in thirty at
// 65536; above 2^22 sheets, whose crowded states would leave runs of many, six
// bytes are sorted by.  A pass costs a launch and about 10 us at least, and what
// the passes after byte 3 need fits in 32 bits, so five passes move 80 bytes
// per sheet, six 104, where eight of 64-bit keys moved 190.
// A sort of 20011 sheets with its force evaluation 205 -> 126 us, of 2^21 in a
// diagnostics call 560 -> 350 us.
//
//   hist   one read of the positions: the digit histograms; its last block
//          forms the exclusive digit offsets; passes whose digit is the same
//          for every key are skipped (decided on the device)
//   pass   persistent: bulk-copy the tile into shared memory (the next
//          tile's copy overlaps this one's write-out), rank within the tile
//          (bit-plane ballots + per-warp shared-memory counters, stable),
//          publish the tile's digit counts, stage in digit order, look back
//          for the tile's global digit offsets, write out
//   gather permute x, v, m, idx into the other state set; notes in small sorts
//          whether any sheet precedes its predecessor in (key, index)
//   ties   (unless none does) runs of equal leading bytes are ordered by key and
//          original index: short runs in place, longer ones by one warp or one
//          CTA each, whose last block makes the other set the current one; where
//          longer runs hold too much -- positions far from the origin against their spread, or
//          crowded about a few places -- all sheets are sorted by their whole keys
//          instead, by the same launch
//
// Keys that differ in their low bytes only (ranks packed into the bits of a
// double) are sorted whole: first_byte = 0, eight passes of 64-bit keys.
//
// Every kernel first reads the sub-step's `unsorted` flag and returns at once
// when the sheets are already in order, so the sequence can be captured in a
// CUDA graph and still cost nothing when no sort is needed.
#include <cstdint>
#include <functional>
#include <mutex>
#include <type_traits>

#include "wg_internal.cuh"

namespace wg {

namespace {

constexpr int R = 256;
// Look-back status words: top two bits 0 = not yet published, kStatA = the
// tile's own count, kStatP = inclusive count, kStatX = poisoned (a wait of
// this tile or of one it depends on expired: its offsets are unknown).
constexpr unsigned kStatA = 1u << 30, kStatP = 2u << 30, kStatX = 3u << 30,
                   kCountMask = (1u << 30) - 1;

// plan layout (uint32 words)
constexpr int kPlanActive = 0;   // [8]
constexpr int kPlanSrc = 8;      // [8]
constexpr int kPlanDst = 16;     // [8]
constexpr int kPlanFinal = 24;   // [1]
constexpr int kPlanStarts = 32;  // [8 * 256]
constexpr int kPlanWords = kPlanStarts + 8 * R;

// counters (uint32 words, cleared before each sort)
constexpr int kCntClaim = 0;   // [8] next tile of each pass
constexpr int kCntTie = 8;     // some sheet may be out of (key, index) order
constexpr int kCntHist = 10;   // histogram blocks done
constexpr int kCntLong = 11;   // k_radix_long_ties blocks done
constexpr int kCntRuns = 12;   // longer runs listed and, in the upper half of 64 bits,
constexpr int kCntSheets = 13;  // ... the sheets in those of more than a warp's lanes
constexpr int kCntMaxRun = 9;   // the longest of these
constexpr int kCntInv = 14;     // neighbours of one run whose keys were out of order
constexpr int kCntMixed = 15;   // the current set is not in the order of the indices
constexpr int kCntStage = 16;   // [2 x 16] whole sort: tiles claimed and done of each stage
constexpr int kCounters = 48;
// rows of the digit histogram: the eight bytes of the keys, then the four of the
// indices (whole sort)
constexpr int kHistRows = 12;

struct PassArgs {
  const StateTable* table;
  int64_t n;
  int pass;            // byte of the key
  int first;           // the first pass's byte
  int64_t n_tiles;
  void* keys0;         // u64 (whole keys) or u32 (their upper halves)
  void* keys1;
  uint32_t* pos0;
  uint32_t* pos1;
  const uint32_t* plan;
  uint32_t* status;
  uint32_t* counters;
  const StepFlags* flag;
  unsigned* err;
};

// Digit histograms of bytes first .. 7; the last block to finish turns them
// into the plan.  halve: the pass that halves the keys, which is never skipped.
// Four positions per thread, their loads in flight together, and as many blocks
// as that takes: a chain of 16 or more dependent rounds in a few blocks took
// 16 us at 20011 sheets and 22 us at 150001, of a sort of 48 and 62 us.
constexpr int kHistThreads = 256, kHistUnroll = 4;
__global__ void __launch_bounds__(kHistThreads) k_radix_hist(
    const StateTable* table, int64_t n, int first, int halve, uint32_t* hist, uint32_t* plan,
    uint32_t* counters, const StepFlags* flag) {
  chain_begin();
  if (!flag->unsorted) return;
  __shared__ uint32_t sh[8 * R];
  __shared__ int s_last;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < 8 * R; i += kHistThreads) sh[i] = 0;
  __syncthreads();
  const double* x = table->cur.x;
  const int64_t stride = (int64_t)gridDim.x * kHistThreads;
  for (int64_t b0 = (int64_t)blockIdx.x * kHistThreads + (tid & ~31); b0 < n;
       b0 += kHistUnroll * stride) {
    double xs[kHistUnroll];
#pragma unroll
    for (int u = 0; u < kHistUnroll; ++u)
      xs[u] = b0 + u * stride + lane < n ? x[b0 + u * stride + lane] : 0.0;
#pragma unroll
    for (int u = 0; u < kHistUnroll; ++u) {
      const int64_t i0 = b0 + u * stride;
      if (i0 >= n) break;  // (the same for the whole warp)
      const bool ok = i0 + lane < n;
      const uint64_t k = key_of(xs[u]);
      if (ok) {
#pragma unroll
        for (int p = 0; p < 8; ++p)
          if (p >= first) atomicAdd(&sh[p * R + ((k >> (8 * p)) & 255u)], 1u);
      }
    }
  }
  __syncthreads();
  for (int i = first * R + tid; i < 8 * R; i += kHistThreads)
    if (sh[i]) atomicAdd(&hist[i], sh[i]);
  __threadfence();
  __syncthreads();
  if (tid == 0) s_last = atomicAdd(&counters[kCntHist], 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  // ---- the plan: warp w takes byte w, eight digits per lane
  __threadfence();
  if (warp >= first) {
    uint32_t c[8], sum = 0;
    bool triv = false;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      c[q] = __ldcg(&hist[warp * R + lane * 8 + q]);
      sum += c[q];
      triv |= c[q] == (uint32_t)n;
    }
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    uint32_t ex = incl - sum;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      plan[kPlanStarts + warp * R + lane * 8 + q] = ex;
      ex += c[q];
    }
    const unsigned t = __ballot_sync(0xffffffffu, triv);
    if (lane == 0) sh[warp] = t != 0u;
  }
  __syncthreads();
  if (tid == 0) {
    int cur = 0;
    plan[kPlanActive + first] = 1;
    plan[kPlanSrc + first] = 0;
    plan[kPlanDst + first] = 0;
    for (int p = first + 1; p < 8; ++p) {
      const int act = !sh[p] || p == halve;
      plan[kPlanActive + p] = act;
      plan[kPlanSrc + p] = cur;
      plan[kPlanDst + p] = act ? 1 - cur : cur;
      if (act) cur = 1 - cur;
    }
    plan[kPlanFinal] = cur;
  }
}
constexpr int kHistWarps = kHistThreads / 32;
static_assert(kHistWarps == 8, "one warp per byte, one thread per digit");

// What a pass reads and writes: the first one reads positions (double); whole
// keys or their upper halves after that.
template <typename IN>
struct KeyWord {
  typedef IN type;
};
template <>
struct KeyWord<double> {
  typedef uint64_t type;
};

template <int THREADS, int ITEMS, typename KEY>
struct PassSmem {
  static constexpr int TILE = THREADS * ITEMS;
  static constexpr int WARPS = THREADS / 32;
  KEY keys[2][TILE];       // tile k lands in keys[k & 1] (positions on the first pass) ...
  uint32_t vals[2][TILE];  // ... and is staged in digit order in the same buffer
  uint32_t whist[WARPS][R];
  uint32_t tile_excl[R];
  uint32_t gbase[R];
  uint32_t tmp[R / 32];
  uint64_t mbar[2];
  int64_t tile[2];
  int64_t bad;  // 1 + the tile whose offsets are unknown (a bounded wait expired)
  int stop;     // a copy of this CTA never completed: claim no further tile
};

// Persistent: each CTA claims its next tile once the current one's global
// offsets are known and bulk-copies it into its other shared-memory buffer
// during the current write-out.  Claiming that late keeps claim order close
// to processing order, which keeps look-backs short; publishing the counts
// before staging, and looking back only after it, gives the tiles ahead the
// staging time to finish.  Claims are dynamic, so only running CTAs ever
// hold a tile and the look-back always progresses: the smallest tile in work
// has every predecessor finished.
template <int THREADS, int ITEMS, typename IN, typename OUT>
__global__ void __launch_bounds__(THREADS, 512 / THREADS) k_radix_pass(const PassArgs a) {
  // what a tile is read and staged as
  using KEY = typename KeyWord<IN>::type;
  constexpr bool FIRST = std::is_same<IN, double>::value;
  constexpr bool HALVE = sizeof(KEY) > sizeof(OUT);
  using Smem = PassSmem<THREADS, ITEMS, KEY>;
  constexpr int TILE = Smem::TILE;
  constexpr int WARPS = Smem::WARPS;
  constexpr int DW = R / 32;  // warps with a digit per thread
  static_assert(THREADS % R == 0, "a thread per digit");
  extern __shared__ __align__(128) unsigned char smem_raw[];
  Smem& S = *reinterpret_cast<Smem*>(smem_raw);

  chain_begin();
  if (!a.flag->unsorted) return;
  // an earlier pass gave up on a wait: its output is incomplete
  if (*a.err & DEV_ERR_RADIX_TIMEOUT) return;
  const int pass = a.pass;
  if (!a.plan[kPlanActive + pass]) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int shift = 8 * (sizeof(KEY) == 8 ? pass : pass - 4);
  const int srcb = (int)a.plan[kPlanSrc + pass], dstb = (int)a.plan[kPlanDst + pass];
  const KEY* ksrc = static_cast<const KEY*>(srcb ? a.keys1 : a.keys0);
  const uint32_t* psrc = srcb ? a.pos1 : a.pos0;
  OUT* kdst = static_cast<OUT*>(dstb ? a.keys1 : a.keys0);
  uint32_t* pdst = dstb ? a.pos1 : a.pos0;
  const double* x = a.table->cur.x;
  const void* kfrom = FIRST ? (const void*)x : (const void*)ksrc;
  const bool bulk_ok = ((uintptr_t)kfrom & 15u) == 0 && (FIRST || ((uintptr_t)psrc & 15u) == 0);
  uint32_t* stat = a.status + ((int64_t)(pass - a.first) * a.n_tiles) * R;
  unsigned* claim = a.counters + kCntClaim + pass;

  // thread 0: start the copy of tile t into buffer b; partial tiles (and
  // unaligned sources) are read with plain loads, their phase completes at once
  auto issue = [&](int64_t t, int b) {
    if (t >= a.n_tiles) return;
    const int64_t base = t * TILE;
    if (bulk_ok && a.n - base >= TILE) {
      constexpr uint32_t kb = TILE * sizeof(KEY), vb = FIRST ? 0u : TILE * 4u;
      mbar_expect_tx(&S.mbar[b], kb + vb);
      bulk_g2s(S.keys[b], static_cast<const char*>(kfrom) + base * (int64_t)sizeof(KEY), kb,
               &S.mbar[b]);
      if (!FIRST) bulk_g2s(S.vals[b], psrc + base, vb, &S.mbar[b]);
    } else {
      mbar_expect_tx(&S.mbar[b], 0u);
    }
  };

  if (tid == 0) {
    S.bad = 0;
    S.stop = 0;
    mbar_init(&S.mbar[0], 1);
    mbar_init(&S.mbar[1], 1);
    fence_proxy_async_smem();
    const int64_t t0 = atomicAdd(claim, 1u);
    S.tile[0] = t0;
    issue(t0, 0);
  }
  for (int i = tid; i < WARPS * R; i += THREADS) (&S.whist[0][0])[i] = 0;
  __syncthreads();

  for (int k = 0;; ++k) {
    const int b = k & 1;
    const int64_t tile = S.tile[b];
    if (tile >= a.n_tiles) break;
    const int64_t base = tile * TILE;
    const int tile_n = (int)((a.n - base) < TILE ? (a.n - base) : TILE);
    const bool via_bulk = bulk_ok && tile_n == TILE;
    if (via_bulk && !mbar_wait(&S.mbar[b], (unsigned)(k >> 1) & 1u)) {
      // the tile never arrived: its keys, counts and offsets are unknown.  The
      // copy gets a second bounded wait; the tile is published as poisoned
      // and this CTA claims no further tile.
      if (lane == 0) atomicOr(a.err, DEV_ERR_RADIX_TIMEOUT);
      mbar_wait(&S.mbar[b], (unsigned)(k >> 1) & 1u);
      S.bad = tile + 1;
      S.stop = 1;
    }
    KEY key[ITEMS];
    uint32_t val[ITEMS];
    uint32_t rank[ITEMS];
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      const int local = warp * (32 * ITEMS) + i * 32 + lane;
      const int64_t e = base + local;
      if (local < tile_n) {
        if constexpr (FIRST) {
          key[i] = key_of(via_bulk ? __longlong_as_double((long long)S.keys[b][local]) : x[e]);
          val[i] = (uint32_t)e;
        } else {
          key[i] = via_bulk ? S.keys[b][local] : ksrc[e];
          val[i] = via_bulk ? S.vals[b][local] : psrc[e];
        }
      } else {
        key[i] = 0;
        val[i] = 0;
      }
    }
    // Stable ranking inside the warp: items in order, lanes in order.
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      const int local = warp * (32 * ITEMS) + i * 32 + lane;
      const bool ok = local < tile_n;
      const unsigned d = ok ? (unsigned)((key[i] >> shift) & 255u) : (0x100u + lane);
      // lanes holding the same digit, from its eight bit planes (one ballot
      // per bit: cheaper than a match instruction over 32 mostly distinct
      // digits)
      unsigned peers = __ballot_sync(0xffffffffu, ok);
      if (!ok) peers = ~peers;
#pragma unroll
      for (int bit = 0; bit < 8; ++bit) {
        const unsigned bal = __ballot_sync(0xffffffffu, (d >> bit) & 1u);
        peers &= ((d >> bit) & 1u) ? bal : ~bal;
      }
      uint32_t old = 0;
      if (ok) {
        old = S.whist[warp][d];
        rank[i] = old + __popc(peers & lanemask_lt());
      }
      __syncwarp();
      if (ok && lane == __ffs(peers) - 1) S.whist[warp][d] = old + __popc(peers);
      __syncwarp();
    }
    __syncthreads();
    // Column of digit `tid`: exclusive offsets of the warps, tile count;
    // the count is published at once for the tiles behind this one.
    const int d = tid;
    uint32_t count = 0, incl = 0, tex = 0;
    if (warp < DW) {
#pragma unroll
      for (int w = 0; w < WARPS; ++w) {
        const uint32_t c = S.whist[w][d];
        S.whist[w][d] = count;
        count += c;
      }
      if (S.bad == tile + 1)
        st_relaxed_u32(&stat[tile * R + d], kStatX);
      else if (tile == 0)
        st_relaxed_u32(&stat[d], kStatP | count);
      else
        st_relaxed_u32(&stat[tile * R + d], kStatA | count);
      // Exclusive scan of the tile's counts over digits.
      incl = count;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      if (lane == 31) S.tmp[warp] = incl;
    }
    __syncthreads();
    if (warp < DW) {
      uint32_t wpre = 0;
#pragma unroll
      for (int w = 0; w < DW; ++w) wpre += (w < warp) ? S.tmp[w] : 0u;
      tex = wpre + incl - count;
      S.tile_excl[d] = tex;
    }
    __syncthreads();
    // Stage the tile in digit order (over the buffer it arrived in); this
    // needs only the tile's own offsets, and gives the tiles ahead time to
    // finish their look-back before this one starts its own.
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      const int local = warp * (32 * ITEMS) + i * 32 + lane;
      if (local < tile_n) {
        const unsigned dd = (unsigned)((key[i] >> shift) & 255u);
        const uint32_t p = S.tile_excl[dd] + S.whist[warp][dd] + rank[i];
        S.keys[b][p] = key[i];
        S.vals[b][p] = val[i];
      }
    }
    // Decoupled look-back over the same digit of earlier tiles.  Each status
    // word carries its count, so relaxed loads and stores suffice; LB
    // predecessors are read per round, their loads in flight together, and
    // summed in order up to the nearest inclusive one.
    uint32_t excl = 0;
    if (warp < DW && tile != 0 && S.bad != tile + 1) {
      constexpr int LB = 8;
      int64_t j = tile - 1;
      unsigned spins = 0;
      bool poisoned = false;
      for (;;) {
        uint32_t sv[LB];
#pragma unroll
        for (int w = 0; w < LB; ++w) sv[w] = (j - w >= 0) ? ld_relaxed_u32(&stat[(j - w) * R + d]) : 0u;
        bool done = false, blocked = false;
        int w = 0;
        for (; w < LB; ++w) {
          const uint32_t sw = sv[w];
          if ((sw >> 30) == 0u) {
            blocked = true;
            break;
          }
          if ((sw >> 30) == 3u) {  // a predecessor's offsets are unknown
            poisoned = done = true;
            break;
          }
          excl += sw & kCountMask;
          if ((sw >> 30) == 2u || j - w == 0) {
            done = true;
            break;
          }
        }
        if (done) break;
        if (blocked) {
          j -= w;  // resume at the tile that has not published yet
          if (++spins > kSpinLimit) {
            atomicOr(a.err, DEV_ERR_RADIX_TIMEOUT);
            poisoned = true;
            break;
          }
          __nanosleep(16);
          continue;
        }
        j -= LB;
      }
      if (poisoned) {
        // unknown offsets: publish the poison onward and write nothing
        atomicOr(a.err, DEV_ERR_RADIX_TIMEOUT);
        S.bad = tile + 1;
        st_relaxed_u32(&stat[tile * R + d], kStatX);
      } else {
        st_relaxed_u32(&stat[tile * R + d], kStatP | (excl + count));
      }
    }
    if (warp < DW) S.gbase[d] = a.plan[kPlanStarts + pass * R + d] + excl - tex;
    // claim the next tile once this one's offsets are known (claim order
    // then follows processing order) and start its copy into the other buffer
    if (tid == 0) {
      if (S.stop) {
        S.tile[b ^ 1] = a.n_tiles;  // ends the loop after this tile
      } else {
        const int64_t tn = atomicAdd(claim, 1u);
        S.tile[b ^ 1] = tn;
        fence_proxy_async_smem();
        issue(tn, b ^ 1);
      }
    }
    __syncthreads();
    for (int i = tid; i < WARPS * R; i += THREADS) (&S.whist[0][0])[i] = 0;
    const bool skip = S.bad == tile + 1;  // offsets unknown: no write may leave the tile
#pragma unroll
    for (int jj = 0; jj < ITEMS; ++jj) {
      const int p = jj * THREADS + tid;
      if (p < tile_n && !skip) {
        const KEY kk = S.keys[b][p];
        const unsigned dd = (unsigned)((kk >> shift) & 255u);
        const int64_t o = (int64_t)S.gbase[dd] + p;
        kdst[o] = HALVE ? (OUT)((uint64_t)kk >> 32) : (OUT)kk;
        pdst[o] = S.vals[b][p];
      }
    }
    __syncthreads();
  }
}

// Permute x, v, m, idx into the other set; GU sheets per thread with their
// loads in flight together.  The reads are random when the input was (a slab
// whose streams interpenetrate), and bound by the sectors in flight: beyond L2
// sixteen sheets per thread (at 2^26 four take 3.2 ms, eight 2.8, sixteen 2.7); up
// to 2^22 sheets four, which leave enough blocks.  NOTE: notes whether any sheet precedes its
// predecessor in (key, index), which spares small sorts the next kernel's work;
// in large ones some sheet nearly always does, and the looking costs a fifth
// (2^26: 3.75 ms with it, 3.2 without).
constexpr int kGatherThreads = 256;
constexpr int64_t kGatherWideSheets = 1 << 22;
template <int GU, bool NOTE>
__global__ void __launch_bounds__(kGatherThreads) k_radix_gather(
    StateTable* table, int64_t n, const uint32_t* pos0, const uint32_t* pos1,
    const uint32_t* plan, uint32_t* counters, const StepFlags* flag, const unsigned* err) {
  chain_begin();
  // nothing after a pass that gave up on a wait: its slots are incomplete
  if (!flag->unsorted || (*err & DEV_ERR_RADIX_TIMEOUT)) return;
  const int fb = (int)plan[kPlanFinal];
  const uint32_t* __restrict__ pos = fb ? pos1 : pos0;
  const StateRef cur = table->cur, oth = table->other;
  const int lane = threadIdx.x & 31;
  const int64_t chunk = (int64_t)gridDim.x * kGatherThreads * GU;
  bool tie = !NOTE && blockIdx.x == 0;
  for (int64_t b0 = (int64_t)blockIdx.x * kGatherThreads * GU; b0 < n; b0 += chunk) {
    const int64_t p0 = b0 + threadIdx.x;
    uint32_t q[GU], qn[NOTE ? GU : 1];
#pragma unroll
    for (int u = 0; u < GU; ++u) {
      const int64_t p = p0 + (int64_t)u * kGatherThreads;
      q[u] = p < n ? __ldcs(pos + p) : 0u;
      if (NOTE) qn[u] = lane == 31 && p + 1 < n ? __ldg(pos + p + 1) : 0u;
    }
    double xs[GU], vs[GU], ms[GU], xn[NOTE ? GU : 1];
    int32_t is[GU], in[NOTE ? GU : 1];
#pragma unroll
    for (int u = 0; u < GU; ++u) {
      const int64_t p = p0 + (int64_t)u * kGatherThreads;
      if (NOTE) xs[u] = 0.0, is[u] = 0;
      if (p < n) {
        xs[u] = __ldg(cur.x + q[u]);
        vs[u] = __ldg(cur.v + q[u]);
        ms[u] = __ldg(cur.m + q[u]);
        is[u] = __ldg(cur.idx + q[u]);
      }
      if (NOTE) {
        xn[u] = 0.0;
        in[u] = 0;
        if (lane == 31 && p + 1 < n) {  // the first sheet of the next warp
          xn[u] = __ldg(cur.x + qn[u]);
          in[u] = __ldg(cur.idx + qn[u]);
        }
      }
    }
#pragma unroll
    for (int u = 0; u < GU; ++u) {
      const int64_t p = p0 + (int64_t)u * kGatherThreads;
      double xd = 0.0;
      int32_t id = 0;
      if (NOTE) {
        xd = __shfl_down_sync(0xffffffffu, xs[u], 1);
        id = __shfl_down_sync(0xffffffffu, is[u], 1);
        if (lane == 31) {
          xd = xn[u];
          id = in[u];
        }
      }
      if (p < n) {
        oth.x[p] = xs[u];
        oth.v[p] = vs[u];
        oth.m[p] = ms[u];
        oth.idx[p] = is[u];
        if (NOTE && p + 1 < n) {
          const uint64_t k = key_of(xs[u]), kn = key_of(xd);
          tie |= kn < k || (kn == k && id < is[u]);
        }
      }
    }
  }
  if (__syncthreads_or(tie) && threadIdx.x == 0) atomicOr(&counters[kCntTie], 1u);
}

// Runs of equal leading bytes (key >> low_bits): each is ordered by key and
// original index.  The thread at a run's first sheet finds its end by binary
// search over the sorted leading bytes; runs of up to kShortRun sheets are
// insertion-sorted in place, longer ones are listed (start in list_start,
// length in list_len) for k_radix_long_ties, so no thread ever does work quadratic
// in a run.  A warp reads four groups of 32 keys at a time, and a pair in order is passed over on these, before anything
// of its run has moved: one group at a time, each pair's sheets loaded again, took
// 0.44 ms at 2^26 and more than twice that at 2^27; so 0.25 ms.  Threads read the
// leading bytes of sheets that a run's first thread may be moving: moves stay
// inside a run, whose leading bytes are all the same, and both sides use relaxed
// accesses.
constexpr int64_t kShortRun = 8, kWarpRun = 32;
constexpr int kTieUnroll = 4;
__global__ void k_radix_ties(StateTable* table, int64_t n, int low_bits, uint32_t* counters,
                             uint32_t* list_start, uint32_t* list_len, const StepFlags* flag,
                             const unsigned* err) {
  chain_begin();
  if (!flag->unsorted || !counters[kCntTie] || (*err & DEV_ERR_RADIX_TIMEOUT)) return;
  const StateRef oth = table->other;
  auto whole = [&](int64_t p) { return key_of(ld_relaxed_f64(oth.x + p)); };
  auto lead = [&](int64_t p) { return whole(p) >> low_bits; };
  const int lane = threadIdx.x & 31;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  __shared__ unsigned s_inv;
  if (threadIdx.x == 0) s_inv = 0u;
  __syncthreads();
  unsigned inv = 0;  // neighbours of one run out of order
  // the run that starts at sheet p, whose first keys are k0, k1 (and k2, except
  // in the last two lanes)
  auto order_run = [&](int64_t p, uint64_t k0, uint64_t k1, uint64_t k2) {
    const uint64_t kp = k0 >> low_bits;
    // nearly every run is a pair, and most of those are in order already
    if (lane >= 30 && p + 2 < n) k2 = whole(p + 2);
    const bool pair = p + 2 >= n || k2 >> low_bits != kp;
    if (pair && k0 < k1) return;
    // last index e with the same leading bytes
    int64_t lo = p + 1, hi = pair ? p + 1 : n - 1;
    while (lo < hi) {
      const int64_t mid = lo + (hi - lo + 1) / 2;
      if (lead(mid) == kp) lo = mid; else hi = mid - 1;
    }
    const int64_t e = lo;
    if (e - p + 1 > kShortRun) {
      const uint32_t len = (uint32_t)(e - p + 1);
      const uint32_t slot =
          (uint32_t)atomicAdd(reinterpret_cast<unsigned long long*>(&counters[kCntRuns]),
                              ((unsigned long long)(len > kWarpRun ? len : 0u) << 32) | 1ull);
      list_start[slot] = (uint32_t)p;
      list_len[slot] = len;
      if (len > kWarpRun) atomicMax(&counters[kCntMaxRun], len);
      return;
    }
    for (int64_t i = p + 1; i <= e; ++i) {
      const double xi = ld_relaxed_f64(oth.x + i), vi = oth.v[i], mi = oth.m[i];
      const uint64_t ki = key_of(xi);
      const int32_t ii = oth.idx[i];
      int64_t j = i - 1;
      while (j >= p) {
        const double xj = ld_relaxed_f64(oth.x + j);
        const uint64_t kj = key_of(xj);
        if (kj < ki || (kj == ki && oth.idx[j] < ii)) break;
        st_relaxed_f64(oth.x + j + 1, xj);
        oth.v[j + 1] = oth.v[j];
        oth.m[j + 1] = oth.m[j];
        oth.idx[j + 1] = oth.idx[j];
        --j;
      }
      if (j + 1 != i) {
        st_relaxed_f64(oth.x + j + 1, xi);
        oth.v[j + 1] = vi;
        oth.m[j + 1] = mi;
        oth.idx[j + 1] = ii;
      }
    }
  };
  for (int64_t w0 = blockIdx.x * (int64_t)blockDim.x + (threadIdx.x & ~31); w0 < n;
       w0 += kTieUnroll * stride) {
    // keys of kTieUnroll groups of 32 sheets and of their neighbours
    uint64_t ks[kTieUnroll], ke[kTieUnroll];
#pragma unroll
    for (int u = 0; u < kTieUnroll; ++u) {
      const int64_t p = w0 + u * stride + lane;
      const int64_t pe = lane == 31 ? p + 1 : p - 1;
      ks[u] = p < n ? whole(p) : 0ull;
      ke[u] = (lane == 31 || lane == 0) && pe >= 0 && pe < n ? whole(pe) : 0ull;
    }
#pragma unroll
    for (int u = 0; u < kTieUnroll; ++u) {
      const int64_t p = w0 + u * stride + lane;
      const uint64_t k0 = ks[u], kp = k0 >> low_bits;
      uint64_t k1 = __shfl_down_sync(0xffffffffu, k0, 1);
      const uint64_t k2 = __shfl_down_sync(0xffffffffu, k0, 2);
      uint64_t kb = __shfl_up_sync(0xffffffffu, k0, 1);
      if (lane == 31) k1 = ke[u];
      if (lane == 0) kb = ke[u];
      inv += p + 1 < n && kp == k1 >> low_bits && k1 < k0;
      if (p + 1 < n && kp == k1 >> low_bits && (p == 0 || kb >> low_bits != kp))
        order_run(p, k0, k1, k2);
      __syncwarp();
    }
  }
  inv = __reduce_add_sync(0xffffffffu, inv);
  if (lane == 0 && inv) atomicAdd(&s_inv, inv);
  __syncthreads();
  if (threadIdx.x == 0 && s_inv) atomicAdd(&counters[kCntInv], s_inv);
}

constexpr int kLongTieThreads = 256;

// ---- the sort by whole keys --------------------------------------------------
// Positions that share their leading bytes by the thousand (a system of unit width
// at 1e6 has three values of its leading four bytes) leave runs of which one CTA
// takes 3 ms for 1e5 sheets.  Whether that is so is known only after the ties have
// been looked at; the sort by whole keys then runs in the launch that would have
// ordered the runs, so that it costs nothing where it is not needed: a stable radix
// sort of (word, place) pairs by the bytes of the indices and then of the keys, bytes
// that are the same for all sheets left out.  One launch, several passes: tiles of
// all stages are claimed in order, a stage begins when all tiles of the one before
// are done, and those have been claimed by running CTAs, so that every (bounded) wait
// ends however many CTAs are resident.
// Force evaluations on host arrays, a unit-width system about 0 / at 1e6 / at 1e9:
// 307 / 346 / 333 us at 1e5 sheets (309 / 1226 / 3492 with the runs one by one), 2.0 /
// 1.7 / 1.7 ms at 1e6 (2.0 / 2.5 / 19.5), 6.6 / 7.0 / 6.3 ms at 4e6 (6.7 / 8.6 / 134).
// Tiles of 1024 sheets up to 2^17, of 2048 above (20011 sheets 173 -> 153 us a force
// evaluation on device arrays; 1e6 sheets 1.91 -> 1.78 ms on host arrays).
constexpr int kWholeItems = 8, kWholeItemsSmall = 4;
constexpr int64_t kWholeSmallSheets = 1 << 17;
// (the look-back words, two sets used alternately, fit where the passes' were: two
// for every tile against eight for every tile of theirs)
static_assert(2 * kRadixTile <= 8 * kLongTieThreads * kWholeItemsSmall &&
                  2 * kRadixTileSmall <= 8 * kLongTieThreads * kWholeItemsSmall,
              "look-back words");

struct WholeSmem {
  uint64_t word[kLongTieThreads * kWholeItems];
  uint32_t pos[kLongTieThreads * kWholeItems];
  uint32_t whist[kLongTieThreads / 32][R];
  uint32_t tile_excl[R];
  uint32_t gbase[R];
  uint32_t starts[R];
  uint32_t tmp[R / 32];
  int64_t tile;
  int stop;
};

struct WholeArgs {
  StateTable* table;
  int64_t n;
  int first;  // bytes of the keys below this one have not been counted yet
  uint64_t* word[2];
  uint32_t* pos[2];
  uint32_t* hist;
  uint32_t* status;
  uint32_t* counters;
  unsigned* err;
};

// Whether runs of more than a warp's lanes hold more sheets than should be left to
// one CTA per run: more than 2048 (and a 256th of all, at most 30720, more), and not
// just equal positions that are in order already.
__device__ __forceinline__ bool crowded(const uint32_t* counters, int64_t n) {
  const int64_t part = n >> 8;
  const uint32_t most = 2048u + (uint32_t)(part < 30720 ? part : 30720);
  const uint32_t inv = counters[kCntInv];
  return counters[kCntSheets] > most &&
         (inv > most / 8 || (inv && counters[kCntMaxRun] > most));
}

// Exclusive scan of one value per thread over the R threads.
__device__ __forceinline__ uint32_t digit_scan(WholeSmem& S, uint32_t v) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) S.tmp[warp] = incl;
  __syncthreads();
  uint32_t pre = 0;
#pragma unroll
  for (int w = 0; w < R / 32; ++w) pre += w < warp ? S.tmp[w] : 0u;
  __syncthreads();
  return pre + incl - v;
}

// Returns whether the sheets are in the other set (else in the current one).
template <int ITEMS>
__device__ __noinline__ bool sort_whole(const WholeArgs& a, WholeSmem& S) {
  constexpr int T = kLongTieThreads, WARPS = T / 32, TILE = T * ITEMS;
  static_assert(T == R, "a thread per digit");
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t n = a.n, tiles = (n + TILE - 1) / TILE;
  const StateRef oth = a.table->other, cur = a.table->cur;
  auto claim = [&](int stage) {
    __syncthreads();
    if (tid == 0) S.tile = atomicAdd(&a.counters[kCntStage + 2 * stage], 1u);
    __syncthreads();
    return S.tile;
  };
  // `count` tiles of a stage are complete, and what was written for them visible
  auto done = [&](int stage, unsigned count) {
    __threadfence();
    __syncthreads();
    if (tid == 0 && count) atomicAdd(&a.counters[kCntStage + 2 * stage + 1], count);
  };
  auto all_done = [&](int stage) {
    if (tid == 0) {
      unsigned spins = 0;
      S.stop = 0;
      while (ld_relaxed_u32(&a.counters[kCntStage + 2 * stage + 1]) < (unsigned)tiles) {
        if (++spins > kSpinLimit) {
          atomicOr(a.err, DEV_ERR_RADIX_TIMEOUT);
          S.stop = 1;
          break;
        }
        __nanosleep(64);
      }
      __threadfence();
    }
    __syncthreads();
    return S.stop == 0;
  };
  // ---- stage 0: the bytes not counted yet, and clean look-back words
  uint32_t* const sh = &S.whist[0][0];  // rows 0 .. 3: indices; 4 ..: bytes 0 .. first - 1
  static_assert(WARPS >= 8, "rows");
  for (int i = tid; i < 8 * R; i += T) sh[i] = 0u;
  unsigned mine = 0;
  bool mixed = false;
  for (int64_t tile; (tile = claim(0)) < tiles; ++mine) {
    a.status[tile * R + tid] = 0u;
    a.status[(tiles + tile) * R + tid] = 0u;
    for (int i = 0; i < ITEMS; ++i) {
      const int64_t p = tile * TILE + i * T + tid;
      if (p >= n) break;
      const uint32_t id = (uint32_t)oth.idx[p];
      mixed |= p + 1 < n && cur.idx[p + 1] < cur.idx[p];
      const uint64_t k = key_of(oth.x[p]);
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        atomicAdd(&sh[b * R + ((id >> (8 * b)) & 255u)], 1u);
        if (b < a.first) atomicAdd(&sh[(4 + b) * R + ((k >> (8 * b)) & 255u)], 1u);
      }
    }
  }
  __syncthreads();
  for (int i = tid; i < (4 + a.first) * R; i += T)
    if (sh[i]) atomicAdd(&a.hist[i < 4 * R ? 8 * R + i : i - 4 * R], sh[i]);
  if (__syncthreads_or(mixed) && tid == 0) atomicOr(&a.counters[kCntMixed], 1u);
  done(0, mine);
  if (!all_done(0)) return false;
  // from the current set where that is in the order of the indices already (force
  // evaluations, first sorts), which spares the passes by index
  const bool mix = __ldcg(&a.counters[kCntMixed]) != 0u;
  const StateRef from = mix ? oth : cur, to = mix ? cur : oth;
  // ---- the passes: indices (0 .. 3), then keys (4 .. 11)
  int src = -1;        // the buffers that hold the words and places (-1: none yet)
  bool keyed = false;  // ... and whether the words are keys
  int par = 0;         // the look-back words of this pass
  for (int q = mix ? 0 : 4; q < 12; ++q) {
    const int stage = 1 + q, row = q < 4 ? 8 + q : q - 4;
    const int shift = 8 * (q < 4 ? q : q - 4);
    const uint32_t h = __ldcg(&a.hist[row * R + tid]);
    if (__syncthreads_or(h == (uint32_t)n)) continue;
    S.starts[tid] = digit_scan(S, h);
    uint32_t* const stat = a.status + (int64_t)par * tiles * R;
    uint32_t* const next_stat = a.status + (int64_t)(par ^ 1) * tiles * R;
    const int dst = src < 0 ? 0 : src ^ 1;
    for (int64_t tile; (tile = claim(stage)) < tiles;) {
      const int64_t base = tile * TILE;
      const int tile_n = (int)(n - base < TILE ? n - base : TILE);
      uint64_t word[ITEMS];
      uint32_t pos[ITEMS], rank[ITEMS];
#pragma unroll
      for (int i = 0; i < ITEMS; ++i) {
        const int local = warp * (32 * ITEMS) + i * 32 + lane;
        word[i] = 0;
        pos[i] = 0;
        if (local < tile_n) {
          const int64_t e = base + local;
          pos[i] = src < 0 ? (uint32_t)e : __ldcg(a.pos[src] + e);
          if (q >= 4 && !keyed)
            word[i] = key_of(from.x[pos[i]]);
          else
            word[i] = src < 0 ? (uint64_t)(uint32_t)from.idx[e]
                              : ld_cg_u64(a.word[src] + e);
        }
      }
      for (int i = tid; i < WARPS * R; i += T) sh[i] = 0u;
      __syncthreads();
      // stable ranks inside the warp: items in order, lanes in order
#pragma unroll
      for (int i = 0; i < ITEMS; ++i) {
        const bool ok = warp * (32 * ITEMS) + i * 32 + lane < tile_n;
        const unsigned d = ok ? (unsigned)(word[i] >> shift) & 255u : 256u + lane;
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        uint32_t old = 0;
        if (ok) {
          old = S.whist[warp][d];
          rank[i] = old + __popc(peers & lanemask_lt());
        }
        __syncwarp();
        if (ok && lane == __ffs(peers) - 1) S.whist[warp][d] = old + __popc(peers);
        __syncwarp();
      }
      __syncthreads();
      uint32_t count = 0;
#pragma unroll
      for (int w = 0; w < WARPS; ++w) {
        const uint32_t c = S.whist[w][tid];
        S.whist[w][tid] = count;
        count += c;
      }
      st_relaxed_u32(&stat[tile * R + tid], (tile == 0 ? kStatP : kStatA) | count);
      next_stat[tile * R + tid] = 0u;
      const uint32_t tex = digit_scan(S, count);
      S.tile_excl[tid] = tex;
      __syncthreads();
#pragma unroll
      for (int i = 0; i < ITEMS; ++i)
        if (warp * (32 * ITEMS) + i * 32 + lane < tile_n) {
          const unsigned d = (unsigned)(word[i] >> shift) & 255u;
          const uint32_t p = S.tile_excl[d] + S.whist[warp][d] + rank[i];
          S.word[p] = word[i];
          S.pos[p] = pos[i];
        }
      // look-back over the same digit of earlier tiles, LB loads in flight
      constexpr int LB = 4;
      uint32_t excl = 0;
      bool lost = false, found = tile == 0;
      unsigned spins = 0;
      for (int64_t j = tile - 1; !found && !lost;) {
        uint32_t sv[LB];
#pragma unroll
        for (int w = 0; w < LB; ++w)
          sv[w] = j - w >= 0 ? ld_relaxed_u32(&stat[(j - w) * R + tid]) : kStatP;
        int w = 0;
        for (; w < LB && !found; ++w) {
          const uint32_t st = sv[w] >> 30;
          if (st == 0u) break;  // not published yet: resume here
          lost |= st == 3u;
          excl += sv[w] & kCountMask;
          found = st >= 2u;
        }
        if (w < LB && !found) {
          lost |= ++spins > kSpinLimit;
          __nanosleep(16);
        }
        j -= w;
      }
      if (tile > 0)
        st_relaxed_u32(&stat[tile * R + tid], lost ? kStatX : kStatP | (excl + count));
      S.gbase[tid] = S.starts[tid] + excl - tex;
      if (__syncthreads_or(lost)) {
        // offsets unknown: nothing leaves the tile, and the sort is given up
        if (tid == 0) atomicOr(a.err, DEV_ERR_RADIX_TIMEOUT);
        return false;
      }
#pragma unroll
      for (int i = 0; i < ITEMS; ++i) {
        const int p = i * T + tid;
        if (p < tile_n) {
          const uint64_t w = S.word[p];
          const int64_t o = (int64_t)S.gbase[(unsigned)(w >> shift) & 255u] + p;
          a.word[dst][o] = w;
          a.pos[dst][o] = S.pos[p];
        }
      }
      done(stage, 1u);
    }
    if (!all_done(stage)) return false;
    src = dst;
    keyed = q >= 4;
    par ^= 1;
  }
  // ---- the sheets, in order
  for (int64_t p = blockIdx.x * (int64_t)T + tid; p < n; p += (int64_t)gridDim.x * T) {
    const int64_t o = src < 0 ? p : (int64_t)__ldcg(a.pos[src] + p);
    to.x[p] = from.x[o];
    to.v[p] = from.v[o];
    to.m[p] = from.m[o];
    to.idx[p] = from.idx[o];
  }
  return !mix;
}

// Longer runs of equal leading bytes: up to kWarpRun sheets by one warp, ranked by
// comparing all pairs; above that by one CTA, a stable LSD radix sort
// (4-bit digits, each thread a contiguous chunk) of (index, place in run)
// pairs in the key buffers' slots of the run, by index and then by the low
// bits of the key, then the run's sheets are permuted through the current set
// (free until the flip) and copied back.  Runs already in order are left
// alone.  O(run length) work per digit.  Crowded states are sorted whole (sort_whole).
__global__ void __launch_bounds__(kLongTieThreads) k_radix_long_ties(
    const __grid_constant__ WholeArgs a, const StepFlags* flag) {
  chain_begin();
  // after an expired wait the current set stays as it was (unsorted, intact)
  if (!flag->unsorted || (*a.err & DEV_ERR_RADIX_TIMEOUT)) return;
  constexpr int T = kLongTieThreads;
  struct RunSmem {
    uint32_t cnt[16][T + 1];
    uint32_t tot[16];
  };
  __shared__ __align__(16) union {
    RunSmem run;
    WholeSmem whole;
  } sm;
  StateTable* const table = a.table;
  const int64_t n = a.n;
  uint32_t* const counters = a.counters;
  const int tid = threadIdx.x;
  const StateRef oth = table->other, cur = table->cur;
  // the last block to finish makes the other set the current one
  auto flip = [&] {
    __syncthreads();
    if (tid == 0) {
      __threadfence();
      if (atomicAdd(&counters[kCntLong], 1u) == gridDim.x - 1) {
        table->cur = oth;
        table->other = cur;
      }
    }
  };
  if (crowded(counters, n)) {
    if (n <= kWholeSmallSheets ? sort_whole<kWholeItemsSmall>(a, sm.whole)
                               : sort_whole<kWholeItems>(a, sm.whole))
      flip();
    return;
  }
  auto& cnt = sm.run.cnt;
  auto& tot = sm.run.tot;
  const uint32_t* const list_start = a.pos[0];
  const uint32_t* const list_len = a.pos[1];
  const int low_bits = 8 * a.first;
  int bits = 1;
  while (bits < 31 && ((int64_t)1 << bits) < n) ++bits;
  const int ipass = (bits + 3) / 4, npass = ipass + (low_bits + 3) / 4;
  const unsigned nruns = counters[kCntRuns];
  // runs of up to a warp's lanes: each sheet's rank among the others
  const int lane = tid & 31, nw = T / 32;
  for (unsigned r = blockIdx.x * nw + (tid >> 5); r < nruns; r += gridDim.x * nw) {
    const int64_t s = list_start[r];
    const int L = (int)list_len[r];
    if (L > (int)kWarpRun) continue;
    uint64_t k = ~0ull;
    int32_t id = 0x7fffffff;
    double x = 0., v = 0., m = 0.;
    if (lane < L) {
      x = oth.x[s + lane];
      v = oth.v[s + lane];
      m = oth.m[s + lane];
      id = oth.idx[s + lane];
      k = key_of(x);
    }
    int rank = 0;
    for (int j = 0; j < L; ++j) {
      const uint64_t kj = __shfl_sync(0xffffffffu, k, j);
      const int32_t ij = __shfl_sync(0xffffffffu, id, j);
      rank += kj < k || (kj == k && (ij < id || (ij == id && j < lane)));
    }
    if (lane < L && rank != lane) {
      oth.x[s + rank] = x;
      oth.v[s + rank] = v;
      oth.m[s + rank] = m;
      oth.idx[s + rank] = id;
    }
  }
  for (unsigned r = blockIdx.x; r < nruns; r += gridDim.x) {
    const int64_t s = list_start[r], L = list_len[r];
    if (L <= kWarpRun) continue;
    bool unordered = false;
    for (int64_t j = tid; j + 1 < L; j += T) {
      const uint64_t k = key_of(oth.x[s + j]), kn = key_of(oth.x[s + j + 1]);
      unordered |= kn < k || (kn == k && oth.idx[s + j + 1] < oth.idx[s + j]);
    }
    if (!__syncthreads_or(unordered)) continue;
    uint64_t* src = a.word[0] + s;
    uint64_t* dst = a.word[1] + s;
    for (int64_t j = tid; j < L; j += T)
      src[j] = ((uint64_t)(uint32_t)oth.idx[s + j] << 32) | (uint64_t)j;
    const int64_t chunk = (L + T - 1) / T;
    const int64_t c_lo = (int64_t)tid * chunk < L ? (int64_t)tid * chunk : L;
    const int64_t c_hi = c_lo + chunk < L ? c_lo + chunk : L;
    __syncthreads();
    for (int ps = 0; ps < npass; ++ps) {
      auto digit = [&](uint64_t w) {
        return ps < ipass ? (unsigned)(w >> (32 + 4 * ps)) & 15u
                          : (unsigned)(key_of(oth.x[s + (uint32_t)w]) >> (4 * (ps - ipass))) & 15u;
      };
#pragma unroll
      for (int d = 0; d < 16; ++d) cnt[d][tid] = 0;
      for (int64_t j = c_lo; j < c_hi; ++j) ++cnt[digit(src[j])][tid];
      __syncthreads();
      if (tid < 16) {  // digit-major exclusive offsets of each thread's chunk
        uint32_t run = 0;
        for (int t = 0; t < T; ++t) {
          const uint32_t c = cnt[tid][t];
          cnt[tid][t] = run;
          run += c;
        }
        tot[tid] = run;
      }
      __syncthreads();
      if (tid < 16) {
        uint32_t base = 0;
        for (int d = 0; d < tid; ++d) base += tot[d];
        for (int t = 0; t < T; ++t) cnt[tid][t] += base;
      }
      __syncthreads();
      for (int64_t j = c_lo; j < c_hi; ++j) {
        const uint64_t w = src[j];
        dst[cnt[digit(w)][tid]++] = w;
      }
      __syncthreads();
      uint64_t* t2 = src;
      src = dst;
      dst = t2;
    }
    for (int64_t j = tid; j < L; j += T) {
      const int64_t q = s + (int64_t)(uint32_t)src[j];
      cur.x[s + j] = oth.x[q];
      cur.v[s + j] = oth.v[q];
      cur.m[s + j] = oth.m[q];
      cur.idx[s + j] = oth.idx[q];
    }
    __syncthreads();
    for (int64_t j = tid; j < L; j += T) {
      oth.x[s + j] = cur.x[s + j];
      oth.v[s + j] = cur.v[s + j];
      oth.m[s + j] = cur.m[s + j];
      oth.idx[s + j] = cur.idx[s + j];
    }
    __syncthreads();
  }
  flip();
}

size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

// Launch configuration of the radix passes on one device: its SM count and
// the resident pass CTAs per SM, after raising the pass kernels' dynamic
// shared-memory limits on that device.  Set up once per device (thread-safe).
enum { kTilesSmall = 0, kTilesMid = 1, kTilesLarge = 2 };
enum { kPosHalf = 0, kPosWhole = 1, kWhole = 2, kWholeHalf = 3, kHalf = 4 };
struct RadixDevCfg {
  int sms = 1;
  int per_sm[3][5] = {};  // [tiles][what the pass reads and writes]
};

template <int THREADS, int ITEMS, typename IN, typename OUT>
constexpr size_t pass_smem() {
  return sizeof(PassSmem<THREADS, ITEMS, typename KeyWord<IN>::type>);
}
template <int THREADS, int ITEMS, typename IN, typename OUT>
void pass_init(int& per_sm) {
  constexpr size_t dyn = pass_smem<THREADS, ITEMS, IN, OUT>();
  auto* k = k_radix_pass<THREADS, ITEMS, IN, OUT>;
  cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn);
  int c = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&c, k, THREADS, dyn);
  per_sm = c < 1 ? 1 : c;
}
template <int THREADS, int ITEMS, typename IN, typename OUT>
void pass_launch(const PassArgs& a, int per_sm, int sms, cudaStream_t s) {
  int64_t pg = (int64_t)per_sm * sms;
  if (pg > a.n_tiles) pg = a.n_tiles;
  if (pg < 1) pg = 1;
  launch_chained(k_radix_pass<THREADS, ITEMS, IN, OUT>, (unsigned)pg, THREADS,
                 pass_smem<THREADS, ITEMS, IN, OUT>(), s, a);
}

template <int THREADS, int ITEMS>
void pass_init_all(int* per_sm) {
  pass_init<THREADS, ITEMS, double, uint32_t>(per_sm[kPosHalf]);
  pass_init<THREADS, ITEMS, double, uint64_t>(per_sm[kPosWhole]);
  pass_init<THREADS, ITEMS, uint64_t, uint64_t>(per_sm[kWhole]);
  pass_init<THREADS, ITEMS, uint64_t, uint32_t>(per_sm[kWholeHalf]);
  pass_init<THREADS, ITEMS, uint32_t, uint32_t>(per_sm[kHalf]);
}
template <int THREADS, int ITEMS>
void pass_launch_kind(const PassArgs& a, int kind, const int* per_sm, int sms, cudaStream_t s) {
  const int c = per_sm[kind];
  if (kind == kPosHalf) pass_launch<THREADS, ITEMS, double, uint32_t>(a, c, sms, s);
  if (kind == kPosWhole) pass_launch<THREADS, ITEMS, double, uint64_t>(a, c, sms, s);
  if (kind == kWhole) pass_launch<THREADS, ITEMS, uint64_t, uint64_t>(a, c, sms, s);
  if (kind == kWholeHalf) pass_launch<THREADS, ITEMS, uint64_t, uint32_t>(a, c, sms, s);
  if (kind == kHalf) pass_launch<THREADS, ITEMS, uint32_t, uint32_t>(a, c, sms, s);
}

void radix_cfg_init(RadixDevCfg& c, int dev) {
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  c.sms = sms < 1 ? 1 : sms;
  pass_init_all<kRadixThreadsMid, kRadixItemsMid>(c.per_sm[kTilesMid]);
  pass_init_all<kRadixThreads, kRadixItems>(c.per_sm[kTilesLarge]);
  pass_init_all<kRadixThreads, kRadixItemsSmall>(c.per_sm[kTilesSmall]);
}

RadixDevCfg radix_cfg() {
  static std::once_flag once[kMaxDevices];
  static RadixDevCfg cfg[kMaxDevices];
  const int dev = current_device();
  if (dev < 0 || dev >= kMaxDevices) {
    RadixDevCfg c;
    radix_cfg_init(c, dev < 0 ? 0 : dev);
    return c;
  }
  std::call_once(once[dev], radix_cfg_init, std::ref(cfg[dev]), dev);
  return cfg[dev];
}

int64_t tiles_of(int64_t n) {
  const int64_t t = n <= kRadixSmallSheets ? kRadixTileSmall : kRadixTile;
  return (n + t - 1) / t;
}

}  // namespace

size_t radix_bytes(int64_t n) {
  // a workspace for n sheets also serves smaller sorts, whose tiles may be
  // the small ones
  const int64_t small = tiles_of(n < kRadixSmallSheets ? n : kRadixSmallSheets);
  const int64_t tiles = tiles_of(n) > small ? tiles_of(n) : small;
  size_t b = 0;
  b += 2 * align256((size_t)n * 8);
  b += 2 * align256((size_t)n * 4);
  b += align256(kPlanWords * 4);
  b += kHistRows * R * 4 + kCounters * 4;
  b += align256((size_t)8 * tiles * R * 4);
  return b;
}

void radix_bind(RadixWork* w, void* base, int64_t n) {
  char* p = static_cast<char*>(base);
  w->keys[0] = reinterpret_cast<uint64_t*>(p); p += align256((size_t)n * 8);
  w->keys[1] = reinterpret_cast<uint64_t*>(p); p += align256((size_t)n * 8);
  w->pos[0] = reinterpret_cast<uint32_t*>(p); p += align256((size_t)n * 4);
  w->pos[1] = reinterpret_cast<uint32_t*>(p); p += align256((size_t)n * 4);
  w->plan = reinterpret_cast<uint32_t*>(p); p += align256(kPlanWords * 4);
  w->hist = reinterpret_cast<uint32_t*>(p);
  w->counters = w->hist + kHistRows * R;
  w->status = w->counters + kCounters;
}

void radix_sort_state(StateTable* table, int64_t n, RadixWork* w, const StepFlags* flag,
                      unsigned* err, cudaStream_t s, bool whole_keys) {
  const RadixDevCfg cfg = radix_cfg();
  const int sms = cfg.sms;
  // the least significant byte sorted by (kRadixFourSheets, kRadixFiveSheets)
  const int first = radix_first_byte(n, whole_keys);
  // the workspace may be bound for more sheets than this sort has: tiles,
  // look-back words and launches follow n
  const int64_t tiles = tiles_of(n);
  cudaMemsetAsync(w->hist, 0, (kHistRows * R + kCounters + (size_t)(8 - first) * tiles * R) * 4, s);
  constexpr int64_t kHistKeys = kHistUnroll * kHistThreads;
  int64_t hist_grid = (n + kHistKeys - 1) / kHistKeys;
  if (hist_grid > sms * 4) hist_grid = sms * 4;
  launch_chained(k_radix_hist, (unsigned)hist_grid, kHistThreads, 0, s, table, n, first,
                 !whole_keys && first < 3 ? 3 : first, w->hist,
                 w->plan, w->counters, flag);
  PassArgs a;
  a.table = table;
  a.n = n;
  a.first = first;
  a.n_tiles = tiles;
  a.keys0 = w->keys[0];
  a.keys1 = w->keys[1];
  a.pos0 = w->pos[0];
  a.pos1 = w->pos[1];
  a.plan = w->plan;
  a.status = w->status;
  a.counters = w->counters;
  a.flag = flag;
  a.err = err;
  const int kt = n <= kRadixSmallSheets ? kTilesSmall : tiles <= sms ? kTilesMid : kTilesLarge;
  const int* per_sm = cfg.per_sm[kt];
  for (int p = first; p < 8; ++p) {
    a.pass = p;
    // the upper halves of the keys are enough once the bytes left lie in them
    const bool half = !whole_keys && p >= 3;
    const int kind = p == first               ? (half ? kPosHalf : kPosWhole)
                     : whole_keys || p <= 3 ? (half ? kWholeHalf : kWhole)
                                              : kHalf;
    if (kt == kTilesSmall)
      pass_launch_kind<kRadixThreads, kRadixItemsSmall>(a, kind, per_sm, sms, s);
    else if (kt == kTilesMid)
      pass_launch_kind<kRadixThreadsMid, kRadixItemsMid>(a, kind, per_sm, sms, s);
    else
      pass_launch_kind<kRadixThreads, kRadixItems>(a, kind, per_sm, sms, s);
  }
  const bool wide = n > kGatherWideSheets;
  const int64_t per = kGatherThreads * (wide ? 16 : 4);
  int64_t gg = (n + per - 1) / per;
  if (gg > (int64_t)sms * 8) gg = (int64_t)sms * 8;
  if (gg < 1) gg = 1;
  launch_chained(wide ? k_radix_gather<16, false> : k_radix_gather<4, true>, (unsigned)gg, kGatherThreads, 0, s, table, n, w->pos[0], w->pos[1],
                 w->plan, w->counters, flag, err);
  int64_t g = (n + 255) / 256;
  if (g > (int64_t)sms * 16) g = (int64_t)sms * 16;
  if (g < 1) g = 1;
  // pos[] is free once gathered: it holds the list of long runs
  launch_chained(k_radix_ties, (unsigned)g, 256, 0, s, table, n, 8 * first, w->counters, w->pos[0],
                 w->pos[1], flag, err);
  // and the key buffers are scratch for long ones and for the sort by whole keys
  WholeArgs wa;
  wa.table = table;
  wa.n = n;
  wa.first = first;
  for (int k = 0; k < 2; ++k) {
    wa.word[k] = w->keys[k];
    wa.pos[k] = w->pos[k];
  }
  wa.hist = w->hist;
  wa.status = w->status;
  wa.counters = w->counters;
  wa.err = err;
  launch_chained(k_radix_long_ties, (unsigned)sms, kLongTieThreads, 0, s, wa, flag);
}

}  // namespace wg
