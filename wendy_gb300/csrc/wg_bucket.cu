// wg_bucket.cu -- launches of the fused sub-step (wg_bucket_step.cuh) and the
// kernels around it: layouts from and to compact state, outputs, splitters,
// and the batched re-sort of pool members.
#include <cstdint>
#include <mutex>
#include <utility>
#include <vector>

#include "wg_bucket_step.cuh"

namespace wg {

namespace {

// Compact sorted state -> bucket layout with exactly T sheets per bucket,
// the splitters Q_b = (key, idx) of the sheet at rank b*T, and the buckets'
// aggregates in slot 0 (slots 1 and 2 cleared).  One block per bucket.
__global__ void k_bucketize(const StateTable* table, int64_t n, int target, int64_t nb, int capg,
                            int E,
                            double* x, double* v, double* m, int32_t* idx, unsigned* cnt0,
                            unsigned* cnt1, unsigned* cnt2, unsigned long long* mass0,
                            unsigned long long* mass1, unsigned long long* mass2, uint64_t* qk,
                            int32_t* qi) {
  __shared__ u128 s_mass[32];
  const StateRef st = table->cur;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int64_t b = blockIdx.x; b < nb; b += gridDim.x) {
    const int64_t r0 = b * target;
    const int c = (int)((n - r0) < target ? (n - r0) : target);
    u128 msum = 0;
    for (int j = threadIdx.x; j < c; j += blockDim.x) {
      const int64_t o = b * capg + j;
      const double mj = st.m[r0 + j];
      x[o] = st.x[r0 + j];
      v[o] = st.v[r0 + j];
      m[o] = mj;
      idx[o] = st.idx[r0 + j];
      msum += mass_to_fixed(mj, E);
    }
    msum = warp_sum_u128(msum);
    if (lane == 0) s_mass[warp] = msum;
    __syncthreads();
    if (warp == 0) {
      const u128 t = warp_sum_u128(lane < (int)(blockDim.x >> 5) ? s_mass[lane] : (u128)0);
      if (lane < 4) {
        mass0[4 * b + lane] = (uint32_t)(t >> (32 * lane));
        mass1[4 * b + lane] = 0ull;
        mass2[4 * b + lane] = 0ull;
      }
      if (lane == 0) {
        cnt0[b] = (unsigned)c;
        cnt1[b] = 0u;
        cnt2[b] = 0u;
        if (b > 0) {
          qk[b] = key_of(st.x[r0]);
          qi[b] = st.idx[r0];
        }
      }
    }
    __syncthreads();
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    qk[0] = 0ull;
    qi[0] = (int32_t)0x80000000;
    qk[nb] = ~0ull;
    qi[nb] = 0x7fffffff;
  }
}

// Bucket layout (+ overflow list) -> compact arrays in table->cur, unsorted.
__global__ void k_compact(StateTable* table, int64_t nb, int capg, const double* x, const double* v,
                          const double* m, const int32_t* idx, const unsigned* cnt,
                          const unsigned* offs, const double* ox, const double* ov,
                          const double* om, const int32_t* oi, const unsigned* ocount,
                          int64_t n, EqMass em) {
  const StateRef st = table->cur;
  const bool eq = em.all_equal();
  for (int64_t b = blockIdx.x; b < nb; b += gridDim.x) {
    const unsigned c = cnt[b] < (unsigned)capg ? cnt[b] : (unsigned)capg;
    const int64_t o = offs[b];
    for (unsigned j = threadIdx.x; j < c && o + j < n; j += blockDim.x) {
      const int64_t s = b * capg + j;
      st.x[o + j] = x[s];
      st.v[o + j] = v[s];
      st.m[o + j] = eq ? em.m : m[s];
      st.idx[o + j] = idx[s];
    }
  }
  const unsigned no = *ocount < (unsigned)n ? *ocount : (unsigned)n;
  const int64_t obase = n - no;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < no; k += stride) {
    st.x[obase + k] = ox[k];
    st.v[obase + k] = ov[k];
    st.m[obase + k] = om[k];
    st.idx[obase + k] = oi[k];
  }
}

// Exclusive scan of the clamped bucket counts (single block, any nb).
__global__ void k_count_offsets(const unsigned* cnt, int64_t nb, int capg, unsigned* offs) {
  __shared__ unsigned s_carry;
  __shared__ unsigned s_w[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) s_carry = 0;
  __syncthreads();
  for (int64_t base = 0; base < nb; base += blockDim.x) {
    const int64_t b = base + tid;
    const unsigned c = b < nb ? (cnt[b] < (unsigned)capg ? cnt[b] : (unsigned)capg) : 0u;
    unsigned incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) s_w[warp] = incl;
    __syncthreads();
    unsigned wpre = 0;
    for (int w = 0; w < warp; ++w) wpre += s_w[w];
    if (b < nb) offs[b] = s_carry + wpre + incl - c;
    __syncthreads();
    if (tid == (int)blockDim.x - 1) s_carry += wpre + incl;
    __syncthreads();
  }
}

}  // namespace

int bucket_step_grid(int sm_count, int ctas_per_sm) {
  return sm_count * (ctas_per_sm < 2 ? 1 : CTAS);
}

namespace {
std::mutex g_tune_mu;
std::vector<std::pair<int64_t, BucketTuning>> g_tune;  // rows sorted by n_min
}  // namespace

BucketTuning tuning_for(int64_t n) {
  std::lock_guard<std::mutex> lock(g_tune_mu);
  BucketTuning t;
  for (const auto& row : g_tune)
    if (row.first <= n) t = row.second;
  return t;
}

void set_tuning(const std::vector<std::pair<int64_t, BucketTuning>>& rows) {
  std::lock_guard<std::mutex> lock(g_tune_mu);
  g_tune = rows;
}

StepKernel step_kernel_none(bool last, int mass) {
  if (mass == kMassAny)
    return last ? k_bucket_step<true, kForceNone, kMassAny> : k_bucket_step<false, kForceNone, kMassAny>;
  if (mass == kMassEqual)
    return last ? k_bucket_step<true, kForceNone, kMassEqual> : k_bucket_step<false, kForceNone, kMassEqual>;
  return last ? k_bucket_step<true, kForceNone, kMassMixed> : k_bucket_step<false, kForceNone, kMassMixed>;
}

// The sub-step kernel's dynamic shared-memory limit, raised once per device
// (function attributes belong to the device they were set on).
void bucket_attr_init() {
  for (int mass : {kMassAny, kMassEqual, kMassMixed})
    for (bool last : {false, true})
      for (StepKernel k : {step_kernel_none(last, mass), step_kernel_closed(last, mass),
                           step_kernel_expr(last, mass)})
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(StepSmem));
}

void bucket_step_prepare() {
  static std::once_flag once[kMaxDevices];
  const int dev = current_device();
  if (dev < 0 || dev >= kMaxDevices)
    bucket_attr_init();
  else
    std::call_once(once[dev], bucket_attr_init);
}

__global__ void __launch_bounds__(256) k_split_out(const OutRec* __restrict__ rec, int64_t n,
                                                   double* __restrict__ x_out,
                                                   double* __restrict__ v_out,
                                                   double* __restrict__ a_out) {
  chain_begin();
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += stride) {
    const double2* r2 = reinterpret_cast<const double2*>(rec + i);
    const double2 xv = __ldcs(r2);
    x_out[i] = xv.x;
    v_out[i] = xv.y;
    if (a_out) a_out[i] = __ldcs(r2 + 1).x;
  }
}

void launch_split_out(const OutRec* rec, int64_t n, double* x_out, double* v_out, double* a_out,
                      cudaStream_t s) {
  int64_t g = (n + 255) / 256;
  if (g > 152 * 8) g = 152 * 8;
  if (g < 1) g = 1;
  launch_chained(k_split_out, (unsigned)g, 256, 0, s, rec, n, x_out, v_out, a_out);
}

void launch_bucket_step(const StepLaunch& a, int grid, cudaStream_t s) {
  bucket_step_prepare();
  if (grid > a.ntasks) grid = a.ntasks;
  if (grid < 1) grid = 1;
  const bool last = a.sub == a.nleap - 1;
  const StepKernel k = a.force == kForceNone     ? step_kernel_none(last, a.mass)
                       : a.force == kForceClosed ? step_kernel_closed(last, a.mass)
                                                 : step_kernel_expr(last, a.mass);
  launch_chained(k, (unsigned)grid, BT, sizeof(StepSmem), s, a);
}

__global__ void __launch_bounds__(256) k_member_splitters(const SimDev* devs, const int* list,
                                                          int sub) {
  __shared__ uint64_t sk[kMemberSampleCap];
  __shared__ int32_t si[kMemberSampleCap];
  const SimDev& d = devs[list ? list[blockIdx.x] : (int)blockIdx.x];
  StateTable* const pt = d.ptab;
  if (!pt) return;
  const int64_t m64 = d.nb - 1;
  if (m64 < 1 || m64 > kMemberSampleCap) return;
  const int m = (int)m64;
  int P = 1;
  while (P < m) P <<= 1;
  const StateRef c = pt->cur;
  for (int j = threadIdx.x; j < P; j += blockDim.x) {
    sk[j] = j < m ? key_of(c.x[j]) : ~0ull;
    si[j] = j < m ? c.idx[j] : 0x7fffffff;
  }
  __syncthreads();
  // bitonic sort of (key, idx) pairs, ascending
  for (int k = 2; k <= P; k <<= 1) {
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int i = threadIdx.x; i < P; i += blockDim.x) {
        const int l = i ^ j;
        if (l > i) {
          const bool up = (i & k) == 0;
          const bool gt = sk[i] > sk[l] || (sk[i] == sk[l] && si[i] > si[l]);
          if (gt == up) {
            const uint64_t tk = sk[i];
            sk[i] = sk[l];
            sk[l] = tk;
            const int32_t ti = si[i];
            si[i] = si[l];
            si[l] = ti;
          }
        }
      }
      __syncthreads();
    }
  }
  const int q = 1 - ((d.qsel0 + sub) & 1);
  uint64_t* const qk = d.qk[q];
  int32_t* const qi = d.qi[q];
  for (int j = threadIdx.x; j < m; j += blockDim.x) {
    qk[j + 1] = sk[j];
    qi[j + 1] = si[j];
  }
}

void launch_member_splitters(const SimDev* devs, const int* list, int count, int sub,
                             cudaStream_t s) {
  if (count > 0) k_member_splitters<<<(unsigned)count, 256, 0, s>>>(devs, list, sub);
}

__global__ void k_samples_to_splitters(const StateTable* table, int64_t m, uint64_t* qk,
                                       int32_t* qi) {
  const StateRef c = table->cur;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < m; j += stride) {
    qk[j + 1] = key_of(c.x[j]);
    qi[j + 1] = c.idx[j];
  }
}

// One warp per sample: its rank among all (key, index, place) triples is the
// splitter it becomes.  A quadratic count, but one launch: for the few hundred
// to few thousand buckets that predicted splitters are sorted for after every
// sub-step, the radix sort's fourteen dependent launches took 110 us
// whatever their size, this takes about 4 us at 650 samples (bound by the
// latency of its loads) and 40 at the limit (by issue).
constexpr int kRankThreads = 256;
__global__ void __launch_bounds__(kRankThreads) k_rank_samples(const StateTable* table, int m,
                                                               uint64_t* qk, int32_t* qi) {
  const int lane = threadIdx.x & 31;
  const int j = blockIdx.x * (kRankThreads / 32) + (threadIdx.x >> 5);
  chain_begin();
  if (j >= m) return;
  const StateRef c = table->cur;
  const uint64_t kj = key_of(c.x[j]);
  const int32_t ij = c.idx[j];
  unsigned r = 0;
#pragma unroll 4
  for (int i = lane; i < m; i += 32) {
    const uint64_t k = key_of(c.x[i]);
    if (k <= kj) {
      bool less = k < kj;
      if (!less) {
        const int32_t x = c.idx[i];
        less = x < ij || (x == ij && i < j);
      }
      r += less ? 1u : 0u;
    }
  }
  r = __reduce_add_sync(0xffffffffu, r);
  if (lane == 0) {
    qk[r + 1] = kj;
    qi[r + 1] = ij;
  }
}

void launch_rank_samples(const StateTable* table, int m, uint64_t* qk, int32_t* qi,
                         cudaStream_t s) {
  const int per = kRankThreads / 32;
  launch_chained(k_rank_samples, (unsigned)((m + per - 1) / per), kRankThreads, 0, s, table, m, qk,
                 qi);
}

// Exclusive scan of each batch member's clamped bucket counts (one block per
// member): offs[toff + b] = sheets of the member's buckets before b.
__global__ void k_batch_offsets(const SimDev* devs, const BatchSeg* segs, unsigned* offs) {
  __shared__ unsigned s_carry;
  __shared__ unsigned s_w[32];
  const BatchSeg g = segs[blockIdx.x];
  const SimDev& d = devs[g.k];
  const unsigned* cnt = d.bcnt[g.cslot];
  const int64_t nb = d.nb;
  const unsigned capg = (unsigned)d.capg;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) s_carry = 0;
  __syncthreads();
  for (int64_t base = 0; base < nb; base += blockDim.x) {
    const int64_t b = base + tid;
    const unsigned c = b < nb ? (cnt[b] < capg ? cnt[b] : capg) : 0u;
    unsigned incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) s_w[warp] = incl;
    __syncthreads();
    unsigned wpre = 0;
    for (int w = 0; w < warp; ++w) wpre += s_w[w];
    if (b < nb) offs[g.toff + b] = s_carry + wpre + incl - c;
    __syncthreads();
    if (tid == (int)blockDim.x - 1) s_carry += wpre + incl;
    __syncthreads();
  }
}

// One block per task: bucket b of batch member j into dst, or (b == nb) the
// member's overflow list after its buckets' sheets.
__global__ void k_batch_compact(const SimDev* devs, const BatchSeg* segs, const BucketTask* tasks,
                                StateRef dst, const unsigned* offs, int64_t total) {
  const BucketTask t = tasks[blockIdx.x];
  const BatchSeg g = segs[t.sim];
  const SimDev& d = devs[g.k];
  const int64_t b = t.bucket;
  if (b < d.nb) {
    const unsigned c0 = d.bcnt[g.cslot][b];
    const unsigned c = c0 < (unsigned)d.capg ? c0 : (unsigned)d.capg;
    const int64_t o = g.out + offs[g.toff + b];
    const int64_t base = b * d.capg;
    const double* x = d.bx[g.lay];
    const double* v = d.bv[g.lay];
    const double* m = d.bm[g.lay];
    const int32_t* idx = d.bi[g.lay];
    for (unsigned j = threadIdx.x; j < c && o + j < g.out + g.n && o + j < total;
         j += blockDim.x) {
      dst.x[o + j] = x[base + j];
      dst.v[o + j] = v[base + j];
      dst.m[o + j] = d.eq == kEqYes ? d.meq : m[base + j];
      dst.idx[o + j] = idx[base + j];
    }
  } else {
    // the overflow list fills the member's last slots
    const unsigned no0 = d.ocount[0];
    const unsigned no = no0 < (unsigned)g.n ? no0 : (unsigned)g.n;
    const int64_t o = g.out + g.n - no;
    for (unsigned j = threadIdx.x; j < no && o + j < total; j += blockDim.x) {
      dst.x[o + j] = d.ox[j];
      dst.v[o + j] = d.ov[j];
      dst.m[o + j] = d.om[j];
      dst.idx[o + j] = d.oi[j];
    }
  }
}

void launch_batch_compact(const SimDev* devs, const BatchSeg* segs, int nseg,
                          const BucketTask* tasks, int64_t ntasks, StateRef dst, unsigned* offs,
                          int64_t total, cudaStream_t s) {
  if (nseg < 1 || ntasks < 1) return;
  k_batch_offsets<<<(unsigned)nseg, 1024, 0, s>>>(devs, segs, offs);
  k_batch_compact<<<(unsigned)ntasks, 256, 0, s>>>(devs, segs, tasks, dst, offs, total);
}

// One block per task: bucket b of batch member j from its sorted sheets into
// layout 0, its counts and fixed-point masses (slot 0; slots 1 and 2
// cleared) and splitter b (the first sheet's key and index).
__global__ void k_batch_bucketize(const SimDev* devs, const BatchSeg* segs,
                                  const BucketTask* tasks, StateRef src, int64_t total) {
  __shared__ u128 s_mass[32];
  const BucketTask t = tasks[blockIdx.x];
  const BatchSeg g = segs[t.sim];
  const SimDev& d = devs[g.k];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t b = t.bucket;
  const int64_t r0 = b * d.target;
  int c = (int)((g.n - r0) < d.target ? (g.n - r0) : d.target);
  if (g.out + r0 + c > total) c = (int)(total - g.out - r0 > 0 ? total - g.out - r0 : 0);
  u128 msum = 0;
  for (int j = threadIdx.x; j < c; j += blockDim.x) {
    const int64_t o = b * d.capg + j;
    const int64_t q = g.out + r0 + j;
    const double mj = src.m[q];
    d.bx[0][o] = src.x[q];
    d.bv[0][o] = src.v[q];
    d.bm[0][o] = mj;
    d.bi[0][o] = src.idx[q];
    msum += mass_to_fixed(mj, d.E);
  }
  msum = warp_sum_u128(msum);
  if (lane == 0) s_mass[warp] = msum;
  __syncthreads();
  if (warp == 0) {
    const u128 tm = warp_sum_u128(lane < (int)(blockDim.x >> 5) ? s_mass[lane] : (u128)0);
    if (lane < 4) {
      d.bmass[0][4 * b + lane] = (uint32_t)(tm >> (32 * lane));
      d.bmass[1][4 * b + lane] = 0ull;
      d.bmass[2][4 * b + lane] = 0ull;
    }
    if (lane == 0) {
      d.bcnt[0][b] = (unsigned)c;
      d.bcnt[1][b] = 0u;
      d.bcnt[2][b] = 0u;
      if (b > 0) {
        d.qk[0][b] = key_of(fma(g.pre, src.v[g.out + r0], src.x[g.out + r0]));
        d.qi[0][b] = src.idx[g.out + r0];
      } else {
        d.qk[0][0] = 0ull;
        d.qi[0][0] = (int32_t)0x80000000;
        d.qk[0][d.nb] = ~0ull;
        d.qi[0][d.nb] = 0x7fffffff;
      }
    }
  }
}

void launch_batch_bucketize(const SimDev* devs, const BatchSeg* segs, const BucketTask* tasks,
                            int64_t ntasks, StateRef src, int64_t total, cudaStream_t s) {
  if (ntasks > 0) k_batch_bucketize<<<(unsigned)ntasks, 256, 0, s>>>(devs, segs, tasks, src, total);
}

void launch_samples_to_splitters(const StateTable* table, int64_t m, uint64_t* qk, int32_t* qi,
                                 cudaStream_t s) {
  int64_t g = (m + 255) / 256;
  if (g > 1216) g = 1216;
  k_samples_to_splitters<<<(unsigned)(g < 1 ? 1 : g), 256, 0, s>>>(table, m, qk, qi);
}

void launch_bucketize(const StateTable* table, int64_t n, int target, int64_t nb, int capg, int E,
                      double* x, double* v, double* m, int32_t* idx,
                      unsigned* const cnt[kAggSlots], unsigned long long* const mass[kAggSlots],
                      uint64_t* qk, int32_t* qi, cudaStream_t s) {
  int64_t g = nb < 152 * 8 ? nb : 152 * 8;
  if (g < 1) g = 1;
  k_bucketize<<<(unsigned)g, 256, 0, s>>>(table, n, target, nb, capg, E, x, v, m, idx, cnt[0],
                                           cnt[1], cnt[2], mass[0], mass[1], mass[2], qk, qi);
}

void launch_compact(StateTable* table, int64_t nb, int capg, const double* x, const double* v,
                    const double* m, const int32_t* idx, const unsigned* cnt, unsigned* offs,
                    const double* ox, const double* ov, const double* om, const int32_t* oi,
                    const unsigned* ocount, int64_t n, EqMass em, cudaStream_t s) {
  k_count_offsets<<<1, 1024, 0, s>>>(cnt, nb, capg, offs);
  int64_t g = nb < 152 * 8 ? nb : 152 * 8;
  if (g < 1) g = 1;
  k_compact<<<(unsigned)g, 256, 0, s>>>(table, nb, capg, x, v, m, idx, cnt, offs, ox, ov, om,
                                         oi, ocount, n, em);
}

}  // namespace wg
