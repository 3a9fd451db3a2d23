// egb_direct.cu -- batches of small tasks in three launches.
//
// A task of a few hundred to a few thousand samples is over in microseconds of
// arithmetic; sorting, grid layouts and one launch per step made it a chain of
// thirty operations instead (one pair of 400 samples: 20 launches, 270 us on
// the device).  When every task of a batch is small (run_direct in egb_api.cu
// has the rule), the batch is
//   direct_prep_kernel    one block per task column: gather, the reference's
//                         rescale, FP32 copy of the
//                         distances from a value amid the column (centre_of)
//   direct_search_kernel  one warp per query over all points of its task: the
//                         exact (k+1)-NN distance, then every marginal count
//                         of that query in one more sweep
//   combine_kernel        as for all batches
// The columns stay in L1 / L2; every decision is the exact one of the other
// kernels: FP32 screen with the proven band, FP64 where it cannot settle.
// Tasks with values that rule out the FP32 copy (not finite, or 1e37 from the
// centre) set DIRECT_REDO in their flag word, and the host runs the batch on
// the general path.
#include <algorithm>

#include "egb_list.cuh"
#include "egb_rescale.cuh"
#include "egb_search.cuh"
#include "ennemi_gb.h"

namespace egb {
namespace {

using list_detail::CandidateList;
using list_detail::FULL;
using list_detail::ExactList;
using list_detail::up_band32;

constexpr int DP_THREADS = 256;
constexpr int DP_STAGE = 256;
constexpr int DS_WARPS = 4;

__global__ void __launch_bounds__(DP_THREADS)
direct_prep_kernel(const DirectTask* __restrict__ tasks, const DirectCol* __restrict__ cols,
                   const PwTree* __restrict__ trees, const int2* __restrict__ nodes,
                   const int32_t* __restrict__ levels, const double* __restrict__ noise,
                   uint32_t* __restrict__ flags) {
  __shared__ double v[DIRECT_MAX_N + 1];
  __shared__ double sm[2 * DP_STAGE];   // node sums of the tree, or staged rows
  __shared__ double mean_s, sd_s, rsd_s, centre;
  const DirectCol dc = cols[blockIdx.x];
  const DirectTask& t = tasks[dc.task];
  const int n = t.n, tid = threadIdx.x;
  for (int w = tid; w < n; w += DP_THREADS) {
    const int64_t s = dc.perm ? dc.perm[w] : w;
    v[w] = dc.src[s * dc.stride];
  }
  __syncthreads();
  if (dc.tree >= 0 || dc.group > 1) {  // rescale: the operations of rescale_*_kernel
    // one thread divides: GB300 has few FP64 lanes
    double q;
    PwTree tr{};
    if (dc.group > 1) {
      q = row_sum<DP_STAGE>(v, dc.inv, n, sm, false, 0.0);
    } else {
      tr = trees[dc.tree];
      q = pw_sum_block(v, dc.inv, tr, nodes, levels, sm, false, 0.0);
    }
    if (tid == 0) mean_s = __ddiv_rn(q, (double)n);
    __syncthreads();
    const double mean = mean_s;
    if (dc.group > 1) q = row_sum<DP_STAGE>(v, dc.inv, n, sm, true, mean);
    else q = pw_sum_block(v, dc.inv, tr, nodes, levels, sm, true, mean);
    if (tid == 0) {
      sd_s = __dsqrt_rn(__ddiv_rn(q, (double)n));
      rsd_s = __ddiv_rn(1.0, sd_s);
    }
    __syncthreads();
    const double sd = sd_s, rsd = rsd_s;
    if (fabs(sd) < 1e-20) {  // the reference warns and keeps the column
      if (tid == 0) atomicOr(flags + t.id, RESCALE_CONSTANT);
    } else {
      for (int i = tid; i < n; i += DP_THREADS) {
        const int w = dc.inv ? dc.inv[i] : i;
        v[w] = __dadd_rn(div_rn(__dsub_rn(v[w], mean), sd, rsd), noise[dc.noise_pos + (int64_t)i * dc.group]);
      }
    }
    __syncthreads();
  }
  if (tid < 32) {
    const double m = centre_of(v, n);
    if (tid == 0) centre = m;
  }
  __syncthreads();
  const double c = centre;
  double* x64 = const_cast<double*>(t.x64) + (int64_t)dc.col * t.ld;
  float* x32 = const_cast<float*>(t.x32) + (int64_t)dc.col * t.ld;
  bool bad = false;
  for (int w = tid; w < n; w += DP_THREADS) {
    const double cv = v[w] - c;
    bad |= !(fabs(cv) < 1e37);
    x64[w] = v[w];
    x32[w] = __double2float_rn(cv);
  }
  // the tail of the last 32 candidates: infinitely far from every query
  for (int w = n + tid; w < (int)t.ld; w += DP_THREADS) x32[w] = __builtin_huge_valf();
  if (__syncthreads_or(bad) && tid == 0) atomicOr(flags + t.id, DIRECT_REDO);
}

// Column sets of the count slots of an estimator over D columns (x, y, z ... /
// x ...): bit c of mask(s) is column c; within(s): counted within the query's
// class only.
template <int KIND, int D>
struct Slots {
  static constexpr int N = KIND == EGB_MI ? 2 : (KIND == EGB_CMI || KIND == EGB_CSEMI) ? 3
                           : KIND == EGB_SEMI ? 1 : 0;
  static constexpr __device__ unsigned mask(int s) {
    constexpr unsigned all = (1u << D) - 1u;
    if (KIND == EGB_MI) return s == 0 ? 1u : 2u;
    if (KIND == EGB_CMI) return s == 0 ? all & ~2u : s == 1 ? all & ~1u : all & ~3u;
    if (KIND == EGB_CSEMI) return s == 0 ? all : all & ~1u;
    return all;
  }
  static constexpr __device__ int first(int s) {  // its lowest column
    for (int c = 0; c < D; ++c)
      if ((mask(s) >> c) & 1u) return c;
    return 0;
  }
  static constexpr __device__ bool within(int s) { return KIND == EGB_CSEMI && s == 1; }
  static constexpr bool CLASSES = KIND == EGB_SEMI || KIND == EGB_CSEMI;
};

template <int KIND, int D, int R>
__global__ void __launch_bounds__(DS_WARPS * 32)
direct_search_kernel(const DirectTask* __restrict__ tasks, int ntasks, int part_base, int nparts, int per,
                     uint32_t* __restrict__ crowded) {
  using SL = Slots<KIND, D>;
  constexpr int NS = SL::N;
  constexpr float FINF = __builtin_huge_valf();
  __shared__ __align__(8) uint32_t store[DS_WARPS][CandidateList<R>::WORDS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int part = (int)blockIdx.x * DS_WARPS + warp;
  if (part >= nparts) return;
  int lo_t = 0, hi_t = ntasks;  // the task of this part: the last that starts at or before it
  while (hi_t - lo_t > 1) {
    const int m = (lo_t + hi_t) >> 1;
    if (tasks[m].part0 - part_base <= part) lo_t = m; else hi_t = m;
  }
  const DirectTask& t = tasks[lo_t];
  const int n = t.n, K = t.K;
  const int ld = (int)t.ld;
  const float* __restrict__ g = t.x32;
  const float* __restrict__ gl[D];  // this lane's candidate of each 32
#pragma unroll
  for (int c = 0; c < D; ++c) gl[c] = g + c * ld + lane;
  const double* __restrict__ c64 = t.x64;
  const int q0 = (part - (t.part0 - part_base)) * per, q1 = min(q0 + per, n);
  unsigned over = 0;

  for (int q = q0; q < q1; ++q) {
    float qv[D];
    float am = 0.0f;
#pragma unroll
    for (int c = 0; c < D; ++c) {
      qv[c] = g[c * ld + q];
      am = fmaxf(am, fabsf(qv[c]));
    }
    const float mq = __fmaf_ru(am, 1.0f + 0x1p-22f, 0x1p-148f);  // >= max |q_c - c|
    int b0 = 0, b1 = n;  // the points searched: all, or the query's class
    if constexpr (SL::CLASSES) {
      int a = 0, b = t.nclass;
      while (b - a > 1) {
        const int m = (a + b) >> 1;
        if (t.cls[m] <= q) a = m; else b = m;
      }
      b0 = t.cls[a];
      b1 = t.cls[a + 1];
    }
    auto exact_over = [&](int j, unsigned cols) -> uint64_t {
      uint64_t mx = 0;
#pragma unroll
      for (int c = 0; c < D; ++c)
        if ((cols >> c) & 1u) {
          const uint64_t d = absdiff_bits(c64[c * ld + j], c64[c * ld + q]);
          mx = d > mx ? d : mx;
        }
      return mx;
    };
    auto exact_dist = [&](int j) { return exact_over(j, (1u << D) - 1u); };
    // ---- the K-th distance
    CandidateList<R> list(store[warp], K, mq);
    {
      // 32 candidates at a time, the next ones' loads in flight; positions
      // beyond n hold +inf, those of other classes are left out
      const int j00 = SL::CLASSES ? b0 & ~31 : 0;
      float p[D];
#pragma unroll
      for (int c = 0; c < D; ++c) p[c] = gl[c][j00];
      for (int j0 = j00; j0 < b1 && !list.over; j0 += 32) {
        float dd = fabsf(p[0] - qv[0]);
#pragma unroll
        for (int c = 1; c < D; ++c) dd = fmaxf(dd, fabsf(p[c] - qv[c]));
        const int jn = j0 + 32 < ld ? j0 + 32 : j0;
#pragma unroll
        for (int c = 0; c < D; ++c) p[c] = gl[c][jn];
        if (SL::CLASSES && (j0 + lane < b0 || j0 + lane >= b1)) dd = FINF;
        list.push(dd, j0 + lane);
      }
    }
    uint64_t kth = INF_BITS;
    if (!list.over) {
      kth = list.kth(exact_dist);
    } else if (b1 - b0 >= K) {  // more near ties than the list holds
      ++over;
      ExactList<R> exact(store[warp], K);
      float sb = list.thr;  // the exact distances of the candidates within the bound
      for (int j0 = b0; j0 < b1; j0 += 32) {
        const int j = j0 + lane;
        bool near = false;
        if (j < b1) {
          float dd = 0.0f;
#pragma unroll
          for (int c = 0; c < D; ++c) dd = fmaxf(dd, fabsf(g[c * ld + j] - qv[c]));
          near = dd <= sb;
        }
        if (exact.push(near ? exact_dist(j) : ~0ull))
          sb = fminf(sb, up_band32(f32_up_of_bits(exact.bound), mq));
      }
      kth = exact.kth();
    }
    kth = __shfl_sync(FULL, kth, 0);
    if (lane == 0) t.eps[q] = bits_to_double(kth);
    if constexpr (NS > 0) {
      // ---- the counts within fl64(eps - 1e-12), all slots in one sweep
      const double r = bits_to_double(kth) - 1e-12;
      const int rc = radius_class(r);
      if (rc != 1) {
#pragma unroll
        for (int s = 0; s < NS; ++s)
          if (lane == 0) t.cnt[s][q] = rc == 0 ? 0 : SL::within(s) ? b1 - b0 : n;
        continue;
      }
      const uint64_t rb = (uint64_t)__double_as_longlong(r) & 0x7fffffffffffffffull;
      // inside up to lo, outside beyond hi: band() of egb_internal.cuh, in FP32
      // arithmetic rounded outward
      const float rd = f32_down_of_bits(rb), ru = f32_up_of_bits(rb);
      const float band32 = __fmaf_ru(ru, 0x1p-21f, __fmaf_ru(mq, 0x1p-21f, 0x1p-100f));
      const float lo = __fsub_rd(rd, band32), hi = __fadd_ru(ru, band32);
      // per lane and slot: candidates inside lo; those between lo and hi (the
      // K-th neighbour always is, in the slots that hold its largest
      // coordinate), and the chunk of the last of them
      int acc[NS], mid[NS], at[NS];
#pragma unroll
      for (int s = 0; s < NS; ++s) acc[s] = mid[s] = at[s] = 0;
      auto slot_dist = [&](const float (&a)[D], int s) -> float {
        float dd = a[SL::first(s)];
#pragma unroll
        for (int c = 0; c < D; ++c)
          if (c > SL::first(s) && ((SL::mask(s) >> c) & 1u)) dd = fmaxf(dd, a[c]);
        return dd;
      };
#pragma unroll 4
      for (int j0 = 0; j0 < n; j0 += 32) {
        float a[D];
#pragma unroll
        for (int c = 0; c < D; ++c) a[c] = fabsf(gl[c][j0] - qv[c]);
#pragma unroll
        for (int s = 0; s < NS; ++s) {
          float dd = slot_dist(a, s);
          if (SL::within(s) && (j0 + lane < b0 || j0 + lane >= b1)) dd = FINF;
          if (dd <= lo) {
            ++acc[s];
          } else if (dd <= hi) {
            ++mid[s];
            at[s] = j0;
          }
        }
      }
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        int c0 = (int)__reduce_add_sync(FULL, (unsigned)acc[s]);
        if (!__any_sync(FULL, mid[s] > 1)) {  // at most one per lane: FP64 decides it
          const bool in = mid[s] == 1 && exact_over(at[s] + lane, SL::mask(s)) <= rb;
          c0 += __popc(__ballot_sync(FULL, in));
        } else {
          const int a0 = SL::within(s) ? b0 : 0, a1 = SL::within(s) ? b1 : n;
          for (int j0 = a0; j0 < a1; j0 += 32) {
            const int j = j0 + lane;
            bool in = false;
            if (j < a1) {
              float a[D];
#pragma unroll
              for (int c = 0; c < D; ++c) a[c] = fabsf(g[c * ld + j] - qv[c]);
              const float dd = slot_dist(a, s);
              in = dd > lo && dd <= hi && exact_over(j, SL::mask(s)) <= rb;
            }
            c0 += __popc(__ballot_sync(FULL, in));
          }
        }
        if (lane == 0) t.cnt[s][q] = c0;
      }
    }
  }
  if (lane == 0 && over) atomicAdd(crowded, over);
}

template <int KIND, int D>
void launch_t(const DirectTask* tasks, int ntasks, int kmax, int part_base, int nparts, int per,
              uint32_t* crowded, cudaStream_t st) {
  const int grid = (nparts + DS_WARPS - 1) / DS_WARPS;
  if (kmax <= 16)
    direct_search_kernel<KIND, D, 2><<<grid, DS_WARPS * 32, 0, st>>>(tasks, ntasks, part_base, nparts, per,
                                                                      crowded);
  else
    direct_search_kernel<KIND, D, 4><<<grid, DS_WARPS * 32, 0, st>>>(tasks, ntasks, part_base, nparts, per,
                                                                      crowded);
  count_launch();
}

}  // namespace

// Estimators and column counts with a search kernel.  K <= 64: the list's.
bool direct_supported(int kind, int dx, int dy, int dz, int K) {
  if (K > 64) return false;
  switch (kind) {
    case EGB_MI: return dx == 1 && dy == 1;
    case EGB_CMI: return dx == 1 && dy == 1 && dz <= 3;
    case EGB_SEMI: return dx <= 3;
    case EGB_CSEMI: return dx == 1 && dz <= 2;
    case EGB_ENTROPY: return dx <= 4;
    default: return false;
  }
}

void launch_direct_prep(const DirectTask* tasks_d, const DirectCol* cols_d, int ncols, const PwTree* trees_d,
                        const int2* nodes_d, const int32_t* levels_d, const double* noise, uint32_t* flags,
                        cudaStream_t st) {
  if (ncols <= 0) return;
  direct_prep_kernel<<<ncols, DP_THREADS, 0, st>>>(tasks_d, cols_d, trees_d, nodes_d, levels_d, noise, flags);
  count_launch();
}

void launch_direct_search(int kind, int d, const DirectTask* tasks_d, int ntasks, int kmax, int part_base,
                          int nparts, int per, uint32_t* crowded, cudaStream_t st) {
  if (nparts <= 0) return;
#define EGB_DIRECT(KIND, D)                                                         \
  case KIND * 8 + D:                                                                \
    launch_t<KIND, D>(tasks_d, ntasks, kmax, part_base, nparts, per, crowded, st);  \
    break;
  switch (kind * 8 + d) {
    EGB_DIRECT(EGB_MI, 2)
    EGB_DIRECT(EGB_CMI, 3)
    EGB_DIRECT(EGB_CMI, 4)
    EGB_DIRECT(EGB_CMI, 5)
    EGB_DIRECT(EGB_SEMI, 1)
    EGB_DIRECT(EGB_SEMI, 2)
    EGB_DIRECT(EGB_SEMI, 3)
    EGB_DIRECT(EGB_CSEMI, 2)
    EGB_DIRECT(EGB_CSEMI, 3)
    EGB_DIRECT(EGB_ENTROPY, 1)
    EGB_DIRECT(EGB_ENTROPY, 2)
    EGB_DIRECT(EGB_ENTROPY, 3)
    EGB_DIRECT(EGB_ENTROPY, 4)
    default: break;
  }
#undef EGB_DIRECT
}

}  // namespace egb
