// wg_small.cu -- a whole output interval of a small simulation in one launch.
//
// Up to kSmallSheets sheets one CTA holds the simulation in registers, in
// sorted order, through all the sub-steps of a call: per sub-step kick, drift
// and a look at the neighbours' keys.  While no two sheets have crossed, the
// order is still the sorted one, and with it the masses before each sheet and
// the self-gravity acceleration, which is then taken as it is; otherwise the
// order is repaired and the exact mass prefix formed again.  The repair counts,
// for every sheet, the sheets among its 2 x 8 neighbours that are on the wrong
// side of it; the places found that way are checked (all different, and in
// order afterwards).  Sheets that moved further are sorted by counting over
// 4096 bins, or, where they crowd into a few of those, by a bitonic sort.
//
// What bounds it is the latency of a sub-step's dependent FP64 operations (64
// cycles each) and two barriers; launches, the routing between buckets and
// their look-back are gone.  Per sub-step, against the bucket kernel: 0.5 us
// against 20 (64 sheets), 4.3 against 34.9 (1000 sheets, few crossings), 9.9
// against 41.7 (1000 sheets, all moving by several places).
//
// Arithmetic as in k_bucket_step, operation by operation, so results do not
// depend on which of the two ran.
// Reference: _wendy_nbody_approx_onestep, wendy/wendy.c:385-418.
#include <cstdint>
#include <functional>
#include <mutex>

#include "wg_bucket.cuh"
#include "wg_small.cuh"

namespace wg {

namespace {

constexpr int N2 = kSmallSheets;
constexpr int MAXT = kSmallSheets / 2;  // two sheets per thread at most
constexpr int REPAIR = 8;               // neighbours on each side a repair looks at
constexpr unsigned HOLD = 31;           // sub-steps without a repair after one failed
constexpr int kPart = 1 << 15;          // sub-steps of one launch
constexpr int AMPS = 32;                // sub-steps whose force amplitude is computed at once

struct SmallSmem {
  uint64_t key[N2];
  double x[N2], v[N2], m[N2];
  int32_t idx[N2];
  uint16_t slot[N2];
  u128 wtot[MAXT / 32];
  double amp[2][AMPS];  // used alternately: a slow warp may still read the last one
  unsigned long long maxv;
};

template <int K>
struct Own {  // the sheets at sorted positions threadIdx.x * K + (0 .. K - 1)
  double x[K], v[K], m[K];
  uint64_t key[K];
  int32_t idx[K];
};

__device__ __forceinline__ bool less_pair(uint64_t ka, int32_t ia, uint64_t kb, int32_t ib) {
  return ka < kb || (ka == kb && ia < ib);
}

// Whether some sheet of this thread is not in front of the next one (S.key
// and S.idx hold the current order).
template <int K>
__device__ __forceinline__ bool out_of_order(const SmallSmem& S, const Own<K>& o, int n) {
  const int p0 = threadIdx.x * K;
  bool bad = false;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int q = p0 + k + 1;
    if (q < n) {
      const uint64_t kn = k + 1 < K ? o.key[k + 1 < K ? k + 1 : k] : S.key[q];
      if (kn <= o.key[k]) bad |= kn < o.key[k] || S.idx[q] < o.idx[k];
    }
  }
  return bad;
}

// Repair with a window of W neighbours on each side; true if the order is
// right afterwards.  If two sheets claim one place nothing has moved.
template <int K, int W>
__device__ __forceinline__ bool repair(SmallSmem& S, Own<K>& o, int n) {
  const int p0 = threadIdx.x * K;
  int r[K];
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int p = p0 + k;
    r[k] = p;
    if (p < n) {
      const uint64_t ko = o.key[k];
      const int32_t io = o.idx[k];
#pragma unroll 8
      for (int d = 1; d <= W; ++d) {
        if (p + d < n) {
          const uint64_t q = S.key[p + d];
          if (q <= ko) r[k] += q < ko || S.idx[p + d] < io;
        }
        if (p - d >= 0) {
          const uint64_t q = S.key[p - d];
          if (q >= ko) r[k] -= q > ko || S.idx[p - d] > io;
        }
      }
      S.slot[r[k]] = (uint16_t)p;
    }
  }
  __syncthreads();
  bool clash = false;
#pragma unroll
  for (int k = 0; k < K; ++k)
    if (p0 + k < n) clash |= S.slot[r[k]] != (uint16_t)(p0 + k);
  if (__syncthreads_or(clash)) return false;
#pragma unroll
  for (int k = 0; k < K; ++k)
    if (p0 + k < n) {
      S.key[r[k]] = o.key[k];
      S.x[r[k]] = o.x[k];
      S.v[r[k]] = o.v[k];
      S.m[r[k]] = o.m[k];
      S.idx[r[k]] = o.idx[k];
    }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < K; ++k)
    if (p0 + k < n) {
      o.key[k] = S.key[p0 + k];
      o.x[k] = S.x[p0 + k];
      o.v[k] = S.v[p0 + k];
      o.m[k] = S.m[p0 + k];
      o.idx[k] = S.idx[p0 + k];
    }
  return !__syncthreads_or(out_of_order<K>(S, o, n));
}

// Moves every sheet to the position whose slot names it (S.slot; S.key and
// S.idx are rewritten in that order).
template <int K>
__device__ __forceinline__ void take_slots(SmallSmem& S, Own<K>& o, int n) {
  const int p0 = threadIdx.x * K;
#pragma unroll
  for (int k = 0; k < K; ++k)
    if (p0 + k < n) {
      S.x[p0 + k] = o.x[k];
      S.v[p0 + k] = o.v[k];
      S.m[p0 + k] = o.m[k];
    }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < K; ++k)
    if (p0 + k < n) {
      const int s = S.slot[p0 + k];
      o.x[k] = S.x[s];
      o.v[k] = S.v[s];
      o.m[k] = S.m[s];
      o.key[k] = S.key[s];
      o.idx[k] = S.idx[s];
    }
  __syncthreads();
}

// Counting sort over BINS bins cut linearly in position (difference,
// conversion, product and truncation are each non-decreasing), then the
// sheets of a bin by (key, index).  False, with nothing moved, if a bin holds
// more than MAXBIN sheets.
constexpr int BINS = 4096;
constexpr uint32_t MAXBIN = 24;
template <int K>
__device__ __forceinline__ bool bin_sort(SmallSmem& S, Own<K>& o, int n) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, p0 = tid * K;
  const int T = blockDim.x, nw = T >> 5;
  uint32_t* const bins = reinterpret_cast<uint32_t*>(S.v);  // two 16-bit counters per word
  float* const lo = reinterpret_cast<float*>(S.m);          // per warp: range, then scan totals
  float* const hi = lo + 32;
  uint32_t* const wsum = reinterpret_cast<uint32_t*>(hi + 32);
  for (int j = tid; j < BINS / 2; j += T) bins[j] = 0u;
  // range, in single precision (rounded outward by the clamps below)
  float a = INFINITY, b = -INFINITY;
#pragma unroll
  for (int k = 0; k < K; ++k)
    if (p0 + k < n) {
      a = fminf(a, (float)o.x[k]);
      b = fmaxf(b, (float)o.x[k]);
    }
#pragma unroll
  for (int d = 16; d >= 1; d >>= 1) {
    a = fminf(a, __shfl_xor_sync(0xffffffffu, a, d));
    b = fmaxf(b, __shfl_xor_sync(0xffffffffu, b, d));
  }
  if (lane == 0) {
    lo[warp] = a;
    hi[warp] = b;
  }
  __syncthreads();
  a = lane < nw ? lo[lane] : INFINITY;
  b = lane < nw ? hi[lane] : -INFINITY;
#pragma unroll
  for (int d = 16; d >= 1; d >>= 1) {
    a = fminf(a, __shfl_xor_sync(0xffffffffu, a, d));
    b = fmaxf(b, __shfl_xor_sync(0xffffffffu, b, d));
  }
  const float w = b - a;
  const float scale = w > 1e-30f && w < 1e30f ? (float)BINS / w : 0.f;
  const double x0 = (double)a;
  uint32_t q[K], rk[K];
  bool full = false;
#pragma unroll
  for (int k = 0; k < K; ++k)
    if (p0 + k < n) {
      q[k] = (uint32_t)fminf(fmaxf((float)(o.x[k] - x0) * scale, 0.f), (float)(BINS - 1));
      const int sh = (int)(q[k] & 1u) << 4;
      rk[k] = (atomicAdd(&bins[q[k] >> 1], 1u << sh) >> sh) & 0xffffu;
      // (a NaN falls into bin 0, where its key belongs if its sign is set, as
      // arithmetic here leaves it; the order does not rest on that: above
      // infinity's key it is left to the sort by whole keys)
      full |= rk[k] >= MAXBIN || o.key[k] > 0xFFF0000000000000ull;
    }
  if (__syncthreads_or(full)) return false;
  // exclusive scan: thread t owns the words [t wpt, t wpt + wpt)
  const int wpt = (BINS / 2 + T - 1) / T;
  const int w0 = tid * wpt, w1 = min(w0 + wpt, BINS / 2);
  uint32_t run = 0;
  for (int j = w0; j < w1; ++j) run += (bins[j] & 0xffffu) + (bins[j] >> 16);
  uint32_t incl = run;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += y;
  }
  if (lane == 31) wsum[warp] = incl;
  __syncthreads();
  uint32_t off = lane < warp ? wsum[lane] : 0u;
  off = __reduce_add_sync(0xffffffffu, off) + incl - run;
  for (int j = w0; j < w1; ++j) {
    const uint32_t c = bins[j];
    bins[j] = off * 0x10001u + (c << 16);
    off += (c & 0xffffu) + (c >> 16);
  }
  __syncthreads();
  uint32_t at[K];
#pragma unroll
  for (int k = 0; k < K; ++k)
    if (p0 + k < n) {
      at[k] = (bins[q[k] >> 1] >> ((q[k] & 1u) << 4)) & 0xffffu;
      S.slot[at[k] + rk[k]] = (uint16_t)(p0 + k);
    }
  __syncthreads();
  // a bin is shared exactly when one of its sheets took rank 1: that one
  // orders the bin
#pragma unroll
  for (int k = 0; k < K; ++k)
    if (p0 + k < n && rk[k] == 1) {
      const uint32_t end =
          q[k] + 1 < BINS ? (bins[(q[k] + 1) >> 1] >> (((q[k] + 1) & 1u) << 4)) & 0xffffu
                          : (uint32_t)n;
      for (uint32_t i = at[k] + 1; i < end; ++i) {
        const uint16_t si = S.slot[i];
        const uint64_t ki = S.key[si];
        const int32_t ii = S.idx[si];
        uint32_t j = i;
        while (j > at[k]) {
          const uint16_t sj = S.slot[j - 1];
          if (!less_pair(ki, ii, S.key[sj], S.idx[sj])) break;
          S.slot[j] = sj;
          --j;
        }
        S.slot[j] = si;
      }
    }
  __syncthreads();
  take_slots<K>(S, o, n);
  return true;
}

// Full bitonic sort by (key, index); S.key and S.idx hold the present order.
template <int K>
__device__ __forceinline__ void full_sort(SmallSmem& S, Own<K>& o, int n) {
  const int tid = threadIdx.x, p0 = tid * K;
  int P = 1;
  while (P < n) P <<= 1;
#pragma unroll
  for (int k = 0; k < K; ++k)
    if (p0 + k < n) {
      S.x[p0 + k] = o.x[k];
      S.v[p0 + k] = o.v[k];
      S.m[p0 + k] = o.m[k];
    }
  for (int j = tid; j < P; j += blockDim.x) {
    S.slot[j] = (uint16_t)j;
    if (j >= n) {
      S.key[j] = ~0ull;
      S.idx[j] = 0x7fffffff;
    }
  }
  __syncthreads();
  for (int k = 2; k <= P; k <<= 1) {
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int i = tid; i < P; i += blockDim.x) {
        const int l = i ^ j;
        if (l > i) {
          const bool up = (i & k) == 0;
          const uint64_t ki = S.key[i], kl = S.key[l];
          const int32_t ii = S.idx[i], il = S.idx[l];
          if (less_pair(kl, il, ki, ii) == up) {
            S.key[i] = kl;
            S.key[l] = ki;
            S.idx[i] = il;
            S.idx[l] = ii;
            const uint16_t t = S.slot[i];
            S.slot[i] = S.slot[l];
            S.slot[l] = t;
          }
        }
      }
      __syncthreads();
    }
  }
#pragma unroll
  for (int k = 0; k < K; ++k)
    if (p0 + k < n) {
      const int s = S.slot[p0 + k];
      o.key[k] = S.key[p0 + k];
      o.idx[k] = S.idx[p0 + k];
      o.x[k] = S.x[s];
      o.v[k] = S.v[s];
      o.m[k] = S.m[s];
    }
  __syncthreads();
}

template <int K, bool EXPR>
__global__ void __launch_bounds__(MAXT, 1) k_small_run(const SmallArgs A) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  SmallSmem& S = *reinterpret_cast<SmallSmem*>(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n = A.n, p0 = tid * K;
  const StateRef st = A.table->cur;
  const int E = A.E, has_omega = A.has_omega;
  const double omega2 = A.omega2, dt = A.dt;
  const ExtForce ext = A.ext;
  const i128 T = (i128)((((u128)A.T_hi) << 64) | A.T_lo);
  const double inv_h = ext.kind == EXT_PULSE_TANH ? 1.0 / ext.p[3] : 0.0;
  Own<K> o;
  double self[K];  // self-gravity acceleration of each sheet
#pragma unroll
  for (int k = 0; k < K; ++k) {
    self[k] = 0.0;
    o.x[k] = o.v[k] = o.m[k] = 0.0;
    o.idx[k] = 0;
    o.key[k] = ~0ull;
    if (p0 + k < n) {
      o.v[k] = st.v[p0 + k];
      o.m[k] = st.m[p0 + k];
      o.idx[k] = st.idx[p0 + k];
      o.x[k] = A.pre != 0.0 ? fma(A.pre, o.v[k], st.x[p0 + k]) : st.x[p0 + k];
    }
  }
  if (tid == 0) S.maxv = 0;
  bool fresh = true;  // the prefix has to be formed
  unsigned full_sorts = 0, hold = 0;
  double xr[EXPR ? kExprRegs : 1];
  for (int sub = 0; sub < A.nleap; ++sub) {
    // ---- the order of the sheets
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (p0 + k < n) {
        o.key[k] = key_of(o.x[k]);
        S.key[p0 + k] = o.key[k];
        S.idx[p0 + k] = o.idx[k];
      }
    // the time factors of the next sub-steps of a pulsed force, one per lane
    if (ext.kind == EXT_PULSE_TANH && (sub & (AMPS - 1)) == 0 && warp == 0 &&
        sub + lane < A.nleap)
      S.amp[(sub / AMPS) & 1][lane] = pulse_amplitude(ext, A.t_seq[sub + lane]);
    __syncthreads();
    if (__syncthreads_or(out_of_order<K>(S, o, n))) {
      // a repair that failed is not tried again for the next sub-steps
      bool done = false;
      if (hold == 0) {
        done = repair<K, REPAIR>(S, o, n);
        if (!done) hold = HOLD;
      } else {
        --hold;
      }
      if (!done && !bin_sort<K>(S, o, n)) {
        full_sort<K>(S, o, n);
        ++full_sorts;
      }
      fresh = true;
    }
    // ---- exact prefix of the masses and the self-gravity accelerations
    if (fresh) {
      fresh = false;
      u128 M[K], tot = 0;
#pragma unroll
      for (int k = 0; k < K; ++k) {
        M[k] = p0 + k < n ? mass_to_fixed(o.m[k], E) : (u128)0;
        tot += M[k];
      }
      const u128 incl = warp_inclusive_scan_u128(tot, lane);
      if (lane == 31) S.wtot[warp] = incl;
      __syncthreads();
      u128 C = warp_sum_u128(lane < warp ? S.wtot[lane] : (u128)0) + (incl - tot);
#pragma unroll
      for (int k = 0; k < K; ++k) {
        self[k] = fixed_to_double(T - 2 * (i128)C - (i128)M[k], E);
        C += M[k];
      }
    }
    // ---- force, kick, drift
    const bool last = A.ends && sub == A.nleap - 1;
    const double dt_drift = last ? dt / 2. : dt;
    const double amp = ext.kind == EXT_PULSE_TANH ? S.amp[(sub / AMPS) & 1][sub & (AMPS - 1)] : 0.0;
    double t_ev = 0.0;
    if constexpr (EXPR) {
      t_ev = A.t_seq[sub];
      expr_time(ext, t_ev, xr);
    }
    unsigned long long maxv = 0;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      if (p0 + k >= n) continue;
      double acc = self[k];
      if (has_omega) acc = fma(-omega2, o.x[k], acc);
      if constexpr (EXPR)
        acc = expr_space(ext, xr, o.x[k], t_ev) + acc;
      else if (ext.kind != EXT_NONE)
        acc = ext_force_at(ext, amp, inv_h, o.x[k]) + acc;
      o.v[k] = fma(dt, acc, o.v[k]);
      o.x[k] = fma(dt_drift, o.v[k], o.x[k]);
      if (last) {
        const int i = o.idx[k];
        A.x_out[i] = o.x[k];
        A.v_out[i] = o.v[k];
        if (A.a_out) A.a_out[i] = acc;
        if (A.xi_out) {
          SheetRec rec;
          rec.idx = i;
          rec.pad = 0;
          rec.val = o.x[k];
          A.xi_out[p0 + k] = rec;
        }
        const unsigned long long av =
            (unsigned long long)__double_as_longlong(o.v[k]) & 0x7FFFFFFFFFFFFFFFull;
        maxv = av > maxv ? av : maxv;
      }
    }
    if (last && maxv) atomicMax(&S.maxv, maxv);
  }
  // ---- the state for the next call: compact, in the last order
#pragma unroll
  for (int k = 0; k < K; ++k)
    if (p0 + k < n) {
      st.x[p0 + k] = o.x[k];
      st.v[p0 + k] = o.v[k];
      st.m[p0 + k] = o.m[k];
      st.idx[p0 + k] = o.idx[k];
    }
  __syncthreads();
  if (tid == 0) {
    A.flag->unsorted += full_sorts;  // (cleared by the host before the call)
    A.flag->max_cnt = (unsigned)n;
    A.flag->max_v = S.maxv;
  }
}

void small_attr_init() {
  const int b = (int)sizeof(SmallSmem);
  cudaFuncSetAttribute(k_small_run<1, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, b);
  cudaFuncSetAttribute(k_small_run<1, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, b);
  cudaFuncSetAttribute(k_small_run<2, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, b);
  cudaFuncSetAttribute(k_small_run<2, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, b);
}

}  // namespace

static void launch_part(const SmallArgs& a, cudaStream_t s) {
  // one sheet per thread while a CTA has the threads, else two
  const bool two = a.n > MAXT;
  const int t = ((two ? (a.n + 1) / 2 : a.n) + 31) / 32 * 32;
  const size_t b = sizeof(SmallSmem);
  if (a.ext.kind == EXT_EXPR) {
    if (two)
      k_small_run<2, true><<<1, t, b, s>>>(a);
    else
      k_small_run<1, true><<<1, t, b, s>>>(a);
  } else if (two) {
    k_small_run<2, false><<<1, t, b, s>>>(a);
  } else {
    k_small_run<1, false><<<1, t, b, s>>>(a);
  }
}

int launch_small_run(const SmallArgs& a, cudaStream_t s) {
  static std::once_flag once[kMaxDevices];
  const int dev = current_device();
  if (dev < 0 || dev >= kMaxDevices)
    small_attr_init();
  else
    std::call_once(once[dev], small_attr_init);
  // long calls in parts, so that no launch runs for seconds
  SmallArgs b = a;
  int parts = 0;
  for (int done = 0; done < a.nleap; done += kPart, ++parts) {
    b.nleap = a.nleap - done < kPart ? a.nleap - done : kPart;
    b.ends = done + b.nleap == a.nleap;
    b.pre = done == 0 ? a.pre : 0.0;
    b.t_seq = a.t_seq + done;
    launch_part(b, s);
  }
  return parts;
}

}  // namespace wg
