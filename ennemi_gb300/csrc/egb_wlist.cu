// egb_wlist.cu -- kNN distances with one warp per query.
//
// (k+1)-th smallest max-norm distance per point, self included
// (ennemi/_entropy_estimators.py:39, :108, :142, :194, :240), for K <=
// LIST_K_MAX: over the job's grid copy (strips by column 1; nested cells by
// column 2 for d >= 3; column-0 order inside), or over all points of a job
// without one.  The per-lane walks of egb_wwalk.cu need K entries in a lane's
// registers and neighbouring queries that share candidates; here the 32 lanes screen 32 consecutive candidates at a time
// and append those within the query's screen bound to a list in shared
// memory.  When the list is nearly full, and after each range that added to
// it, its K-th smallest FP32 distance t32 (a bisection on the float bits,
// counted by ballots) sets the new bound and the entries beyond it are
// dropped, so the list stays between K and CAP entries whatever the order.
//
// Exactness, with U = up_band32(t32) >= the exact K-th distance (band proven
// in egb_internal.cuh) and S = up_band32(U):
//   * a dropped candidate has FP32 distance > S, hence FP64 distance > U;
//   * strips, cells and column-0 windows are skipped beyond plan_margin(U) on
//     bounds rounded outward, so their points are farther than U;
//   * order statistics move by no more than the values do, so the exact K-th
//     lies in [dn_band32(t32), U]: a listed candidate with up_band32(d) below
//     that range is nearer, one with dn_band32(d) above it farther, and the
//     K-th is the (K - nearer)-th smallest exact distance of the others --
//     usually one candidate, one FP64 evaluation per query.
// A query whose list cannot hold its near ties (rounded data) and the queries
// of jobs whose centred values reach 1e37 sweep the candidates within S (all of
// them) once more, keep the K smallest exact distances and tighten S and U by
// them.  20,000 points on 7 x 7 levels with 1e-10 of noise, K = 21: 0.23 ms,
// against 3.2 with an 8-pass radix select (0.88 of the CTA grid); one far point among
// 20,000: 0.13 against 1.6.
//
// What bounds it: instruction issue and the latency of a query's ranges in
// turn (72 registers, seven blocks an SM: 6.3 -> 5.7 ms for 2.4 million 4-D
// queries, K = 4, against six; eight blocks 5.8, ten 5.9).  First bounds from 128
// neighbours and a bound renewed after two new candidates, against 32 and eight:
// 5.7 -> 5.0 ms (256 neighbours 5.7); 100,000 6-D points, K = 6: 9.5 -> 4.1 ms; but
// 100,000 3-D points, K = 13, 283 -> 324 us, so three columns keep 32 and eight.  20,000 points, K = 51, d = 2: 0.10 ms, against 25.4 ms for the select
// over all points that served K > 32 before; K = 13: 65 us against 252 of the
// CTA grid; d = 4, K = 4, 200,000 points: 1.04 ms against 1.66 of the walks.
#include <algorithm>

#include "egb_leaf.cuh"
#include "egb_list.cuh"

namespace egb {
namespace {

using leaf_detail::QueryBox;
using leaf_detail::coord_above;
using leaf_detail::coord_below;
using leaf_detail::query_ranges;
using list_detail::CandidateList;
using list_detail::FULL;
using list_detail::ExactList;
using list_detail::plan_margin;
using list_detail::up_band32;

constexpr int WL_WARPS = 4;

template <int D, int R, bool GRID, bool NEST>
__global__ void __launch_bounds__(WL_WARPS * 32, 7)
wlist_kernel(const JobDev* __restrict__ jobs, const WorkItem* __restrict__ items, int nitems, int qb,
             int per, int* __restrict__ counter) {
  constexpr int DQ = D ? D : EGB_DMAX;
  // two to four columns: grid copies by point (JobDev::aos)
  constexpr int AOS = GRID && D ? grid_aos(D) : 0;
  // from four columns on a point's neighbours along column 0 are far in the
  // others: more of them for the first bound, and the bound renewed sooner
  constexpr bool DEEP = NEST && D != 3;
  __shared__ __align__(8) uint32_t store[WL_WARPS][CandidateList<R>::WORDS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int split = (qb + per - 1) / per;  // parts of `per` queries of an item

  for (;;) {
    int it = 0;
    if (lane == 0) it = atomicAdd(counter, 1);
    it = __shfl_sync(FULL, it, 0);
    if (it >= nitems * split) break;
    const WorkItem wi = items[it / split];
    const JobDev* __restrict__ J = jobs + wi.job;
    const int d = D ? D : J->sp.d;
    const int len = J->len, K = J->K;
    const int64_t lds = J->lds;
    const double* __restrict__ c64 = GRID ? J->c64g : J->c64;
    const float* __restrict__ g = GRID ? J->c32g : J->c32;
    const int32_t* __restrict__ sst = J->sstart;
    const int32_t* __restrict__ cst = J->cstart;
    const int S2 = NEST ? J->nsub : 1;
    const int sq = NEST ? (wi.strip & 0xffff) : wi.strip;
    const int hc = NEST ? (wi.strip >> 16) : 0;
    const bool unsafe = (*J->jflags & TF_UNSAFE32) != 0u;
    const int qbeg = wi.q0 + (it % split) * per;
    const int qend = min(min(qbeg + per, wi.q0 + qb), GRID ? wi.q1 : len);
    unsigned long long pairs = 0;
    unsigned redone = 0;

    for (int qp = qbeg; qp < qend; ++qp) {
      float qv[DQ];
      float am = 0.0f;
#pragma unroll
      for (int c = 0; c < DQ; ++c) {
        if (D == 0 && c >= d) break;
        qv[c] = AOS ? g[(int64_t)qp * AOS + c] : g[(int64_t)c * lds + qp];
        am = fmaxf(am, fabsf(qv[c]));
      }
      const float mq = __fmaf_ru(am, 1.0f + 0x1p-22f, 0x1p-148f);  // >= max |q_c - c|
      const QueryBox qbox{coord_below(qv[0]), coord_above(qv[0]), coord_below(qv[1]), coord_above(qv[1]),
                          NEST ? coord_below(qv[NEST ? 2 : 0]) : 0.0f,
                          NEST ? coord_above(qv[NEST ? 2 : 0]) : 0.0f};
      CandidateList<R> list(store[warp], K, mq);
      auto exact_dist = [&](int j) -> uint64_t {
        uint64_t mm = 0;
#pragma unroll
        for (int c = 0; c < DQ; ++c) {
          if (D == 0 && c >= d) break;
          const int64_t off = (int64_t)c * lds;
          const uint64_t v = absdiff_bits(c64[off + j], c64[off + qp]);
          mm = v > mm ? v : mm;
        }
        return mm;
      };
      auto dist32 = [&](int j) -> float {
        float dd;
        if constexpr (AOS == 2) {
          const float2 p = reinterpret_cast<const float2*>(g)[j];
          dd = fmaxf(fabsf(p.x - qv[0]), fabsf(p.y - qv[1]));
        } else if constexpr (AOS == 4) {
          const float4 p = reinterpret_cast<const float4*>(g)[j];
          dd = fmaxf(fmaxf(fabsf(p.x - qv[0]), fabsf(p.y - qv[1])), fabsf(p.z - qv[D >= 3 ? 2 : 0]));
          if constexpr (D == 4) dd = fmaxf(dd, fabsf(p.w - qv[D == 4 ? 3 : 0]));
        } else {
          dd = fabsf(g[j] - qv[0]);
#pragma unroll
          for (int c = 1; c < DQ; ++c) {
            if (D == 0 && c >= d) break;
            dd = fmaxf(dd, fabsf(g[(int64_t)c * lds + j] - qv[c]));
          }
        }
        return dd;
      };
      auto screen = [&](int a, int b, int ea, int eb) {  // [a, b) without [ea, eb)
        pairs += (unsigned)(b - a);
        for (int j0 = a; j0 < b && !list.over; j0 += 32) {
          const int j = j0 + lane;
          list.push(j < b && !(j >= ea && j < eb) ? dist32(j) : __builtin_huge_valf(), j);
        }
      };
      // every range of positions within the planning bound, nearest strips
      // first; f may tighten the bound
      auto enumerate = [&](auto&& f) {
        if constexpr (!GRID) f(0, len);
        else query_ranges<NEST, AOS ? AOS : 1>(J, g, sq, qbox, list.tb, f);
      };

      uint64_t kth = INF_BITS;
      if (!unsafe) {
        int e0 = 0, e1 = 0;
        if (GRID) {
          // first bound: the query's neighbours in its own strip or cell
          const int ha = NEST ? cst[sq * S2 + hc] : sst[sq];
          const int hb = NEST ? cst[sq * S2 + hc + 1] : sst[sq + 1];
          const int w = (K + 31) / 32 * (DEEP ? 64 : 16);
          e0 = max(ha, qp - w);
          e1 = min(hb, e0 + 2 * w);
          screen(e0, e1, 0, 0);
          if (list.cnt >= K) list.tighten();
        }
        enumerate([&](int a, int b) {
          if (list.over) return;
          const int had = list.cnt;
          screen(a, b, e0, e1);
          if (list.cnt >= K && (list.cnt - had >= (DEEP ? 2 : 8) || !(list.thr < __builtin_huge_valf()))) list.tighten();
        });
      }
      if (!unsafe && !list.over) {
        kth = list.kth(exact_dist);
      } else if (len >= K) {
        // the exact distances of the candidates within the bounds (set from K
        // listed candidates; none in a job with clamped values)
        ++redone;
        ExactList<R> exact(store[warp], K);
        float sb = list.thr;
        enumerate([&](int a, int b) {
          pairs += (unsigned)(b - a);
          for (int j0 = a; j0 < b; j0 += 32) {
            const int j = j0 + lane;
            const bool near = j < b && (unsafe || dist32(j) <= sb);
            if (exact.push(near ? exact_dist(j) : ~0ull) && !unsafe) {
              const float u = f32_up_of_bits(exact.bound);
              sb = fminf(sb, up_band32(u, mq));
              list.tb = fminf(list.tb, plan_margin(u));
            }
          }
        });
        kth = exact.kth();
        // distances of non-finite data, as the lists and the select rank them
        if (K <= EGB_KREG_MAX && kth > INF_BITS) kth = INF_BITS;
      }
      if (lane == 0) J->eps[GRID ? J->idxg[qp] : J->idx[qp]] = bits_to_double(kth);
    }
    if (lane == 0) {
      atomicAdd(J->stats + 0, pairs);
      if (redone) atomicAdd(J->stats + 2, (unsigned long long)redone);
    }
  }
}

template <int D, int R, bool GRID, bool NEST>
void launch_t(const JobDev* jobs, const WorkItem* items, int nitems, int qb, int* counter, int num_sms,
              cudaStream_t st) {
  auto kern = wlist_kernel<D, R, GRID, NEST>;
  int per_sm = 1;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, WL_WARPS * 32, 0);
  if (per_sm < 1) per_sm = 1;
  const int64_t warps = (int64_t)num_sms * per_sm * WL_WARPS;
  // queries per part: neighbours share cache lines, but a part is one warp's
  // serial work, so small launches take smaller parts (four per warp)
  int per = qb;
  while (per > 1 && (int64_t)nitems * ((qb + per - 1) / per) < 4 * warps) per /= 2;
  const int64_t parts = (int64_t)nitems * ((qb + per - 1) / per);
  const int grid = (int)std::min<int64_t>((int64_t)num_sms * per_sm, (parts + WL_WARPS - 1) / WL_WARPS);
  if (grid < 1) return;
  kern<<<grid, WL_WARPS * 32, 0, st>>>(jobs, items, nitems, qb, per, counter);
  count_launch();
}

template <int R, bool GRID>
void launch_d(int dclass, const JobDev* jobs, const WorkItem* items, int nitems, int qb, int* counter,
              int num_sms, cudaStream_t st) {
  switch (dclass) {
    case 2: launch_t<2, R, GRID, false>(jobs, items, nitems, qb, counter, num_sms, st); break;
    case 3: launch_t<3, R, GRID, GRID>(jobs, items, nitems, qb, counter, num_sms, st); break;
    case 4: launch_t<4, R, GRID, GRID>(jobs, items, nitems, qb, counter, num_sms, st); break;
    default: launch_t<0, R, GRID, GRID>(jobs, items, nitems, qb, counter, num_sms, st); break;
  }
}

}  // namespace

// The list holds CAP = 64, 128, 256 entries (at least K + 16 before it is
// tightened) for K <= 16, 64, 128.
void launch_knn_list(const JobDev* jobs_d, const WorkItem* items_d, int nitems, int qb, int kclass,
                     int dclass, bool grid, int* counter, int num_sms, cudaStream_t st) {
  if (nitems <= 0) return;
  if (grid) {
    if (kclass <= 16) launch_d<2, true>(dclass, jobs_d, items_d, nitems, qb, counter, num_sms, st);
    else if (kclass <= 64) launch_d<4, true>(dclass, jobs_d, items_d, nitems, qb, counter, num_sms, st);
    else launch_d<8, true>(dclass, jobs_d, items_d, nitems, qb, counter, num_sms, st);
  } else {
    if (kclass <= 64) launch_d<4, false>(dclass, jobs_d, items_d, nitems, qb, counter, num_sms, st);
    else launch_d<8, false>(dclass, jobs_d, items_d, nitems, qb, counter, num_sms, st);
  }
}

}  // namespace egb
