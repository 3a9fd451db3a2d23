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
// of jobs whose centred values reach 1e37 take an 8-pass radix select on the
// exact distances of the candidates within U (all candidates).
//
// What bounds it: instruction issue and the latency of a query's ranges in
// turn.  20,000 points, K = 51, d = 2: 0.10 ms, against 25.4 ms for the select
// over all points that served K > 32 before; K = 13: 65 us against 252 of the
// CTA grid; d = 4, K = 4, 200,000 points: 1.04 ms against 1.66 of the walks.
#include <algorithm>

#include "egb_leaf.cuh"

namespace egb {
namespace {

using namespace leaf_detail;

constexpr int WL_WARPS = 4;

// K-th smallest (1-based) of the warp's R x 32 float bit patterns (distances
// >= 0; unused slots +inf), at least K of them finite or +inf alike.
template <int R>
__device__ __forceinline__ uint32_t kth_bits(const uint32_t (&v)[R], int K) {
  uint32_t lo = 0xffffffffu, hi = 0u;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    lo = min(lo, v[r]);
    hi = max(hi, v[r]);
  }
  lo = __reduce_min_sync(FULL, lo);
  if (K <= 8) {  // a few minima in turn are cheaper than a bisection
    uint32_t w[R];
#pragma unroll
    for (int r = 0; r < R; ++r) w[r] = v[r];
    for (int left = K;;) {
      int c = 0;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        c += __popc(__ballot_sync(FULL, w[r] == lo));
        w[r] = w[r] == lo ? 0xffffffffu : w[r];
      }
      left -= c;
      if (left <= 0) return lo;
      uint32_t m = w[0];
#pragma unroll
      for (int r = 1; r < R; ++r) m = min(m, w[r]);
      lo = __reduce_min_sync(FULL, m);
    }
  }
  hi = __reduce_max_sync(FULL, hi);
  while (lo < hi) {
    const uint32_t mid = lo + ((hi - lo) >> 1);
    int c = 0;
#pragma unroll
    for (int r = 0; r < R; ++r) c += __popc(__ballot_sync(FULL, v[r] <= mid));
    if (c == K) {  // the largest of the K values up to mid
      uint32_t m = 0;
#pragma unroll
      for (int r = 0; r < R; ++r) m = max(m, v[r] <= mid ? v[r] : 0u);
      return __reduce_max_sync(FULL, m);
    }
    if (c > K) hi = mid;
    else lo = mid + 1;
  }
  return lo;
}

__device__ __forceinline__ uint64_t warp_min64(uint64_t v) {
  const uint32_t h = __reduce_min_sync(FULL, (uint32_t)(v >> 32));
  const uint32_t l = __reduce_min_sync(FULL, (uint32_t)(v >> 32) == h ? (uint32_t)v : 0xffffffffu);
  return ((uint64_t)h << 32) | l;
}

template <int D, int R, bool GRID, bool NEST>
__global__ void __launch_bounds__(WL_WARPS * 32)
wlist_kernel(const JobDev* __restrict__ jobs, const WorkItem* __restrict__ items, int nitems, int qb,
             int per, int* __restrict__ counter) {
  constexpr int DQ = D ? D : EGB_DMAX;
  constexpr int CAP = 32 * R;
  constexpr float FINF = __builtin_huge_valf();
  struct Entry { float d; int j; };
  constexpr int WORDS = 2 * CAP > 256 ? 2 * CAP : 256;  // the list, or 256 radix counters
  __shared__ __align__(8) uint32_t store[WL_WARPS][WORDS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  Entry* list = reinterpret_cast<Entry*>(store[warp]);
  uint32_t* hist = store[warp];
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
        qv[c] = g[(int64_t)c * lds + qp];
        am = fmaxf(am, fabsf(qv[c]));
      }
      const float mq = __fmaf_ru(am, 1.0f + 0x1p-22f, 0x1p-148f);  // >= max |q_c - c|
      const QueryBox qbox{coord_below(qv[0]), coord_above(qv[0]), coord_below(qv[1]), coord_above(qv[1]),
                          NEST ? coord_below(qv[NEST ? 2 : 0]) : 0.0f,
                          NEST ? coord_above(qv[NEST ? 2 : 0]) : 0.0f};
      float thr = FINF;  // screen bound S
      float tb = FINF;   // planning bound plan_margin(U)
      int cnt = 0;       // listed candidates
      bool over = unsafe;

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
      // New bounds from the list's K-th smallest; entries beyond them leave.
      auto tighten = [&]() {
        __syncwarp();
        uint32_t v[R];
        int ix[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const bool in = r * 32 + lane < cnt;
          const Entry e = in ? list[r * 32 + lane] : Entry{FINF, 0};
          v[r] = __float_as_uint(e.d);
          ix[r] = e.j;
        }
        const float u = up_band32(__uint_as_float(kth_bits<R>(v, K)), mq);
        thr = up_band32(u, mq);
        tb = plan_margin(u);
        __syncwarp();
        int kept = 0;
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const bool keep = r * 32 + lane < cnt && __uint_as_float(v[r]) <= thr;
          const uint32_t m = __ballot_sync(FULL, keep);
          if (keep) list[kept + __popc(m & lt)] = Entry{__uint_as_float(v[r]), ix[r]};
          kept += __popc(m);
        }
        cnt = kept;
        over = over || cnt > CAP - 32;  // more near ties than the list holds
        __syncwarp();
      };
      auto screen = [&](int a, int b, int ea, int eb) {  // [a, b) without [ea, eb)
        pairs += (unsigned)(b - a);
        for (int j0 = a; j0 < b && !over; j0 += 32) {
          const int j = j0 + lane;
          float dd = FINF;
          if (j < b && !(j >= ea && j < eb)) {
            dd = fabsf(g[j] - qv[0]);
#pragma unroll
            for (int c = 1; c < DQ; ++c) {
              if (D == 0 && c >= d) break;
              dd = fmaxf(dd, fabsf(g[(int64_t)c * lds + j] - qv[c]));
            }
          }
          const bool hit = dd <= thr && dd < FINF;
          const uint32_t m = __ballot_sync(FULL, hit);
          if (m) {
            if (hit) list[cnt + __popc(m & lt)] = Entry{dd, j};
            cnt += __popc(m);
            if (cnt > CAP - 32) tighten();
          }
        }
      };
      // Every range of positions within the planning bound, nearest strips
      // first; f may tighten the bound.
      auto enumerate = [&](auto&& f) {
        if constexpr (!GRID) f(0, len);
        else query_ranges<NEST>(J, g, sq, qbox, tb, f);
      };

      uint64_t kth = INF_BITS;
      if (!over) {
        int e0 = 0, e1 = 0;
        if (GRID) {
          // first bound: the query's neighbours in its own strip or cell
          const int ha = NEST ? cst[sq * S2 + hc] : sst[sq];
          const int hb = NEST ? cst[sq * S2 + hc + 1] : sst[sq + 1];
          const int w = (K + 31) / 32 * 16;
          e0 = max(ha, qp - w);
          e1 = min(hb, e0 + 2 * w);
          screen(e0, e1, 0, 0);
          if (cnt >= K) tighten();
        }
        enumerate([&](int a, int b) {
          if (over) return;
          const int had = cnt;
          screen(a, b, e0, e1);
          if (cnt >= K && (cnt - had >= 8 || !(thr < FINF))) tighten();
        });
      }
      if (!over) {
        __syncwarp();
        float v[R];
        int ix[R];
        uint32_t vb[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const bool in = r * 32 + lane < cnt;
          const Entry e = in ? list[r * 32 + lane] : Entry{FINF, 0};
          v[r] = e.d;
          vb[r] = __float_as_uint(e.d);
          ix[r] = e.j;
        }
        if (cnt >= K) {
          const float t32 = __uint_as_float(kth_bits<R>(vb, K));
          const float lo = dn_band32(t32, mq), hi = up_band32(t32, mq);
          int rank = K;
          uint64_t e[R];
#pragma unroll
          for (int r = 0; r < R; ++r) {
            rank -= __popc(__ballot_sync(FULL, up_band32(v[r], mq) < lo));  // false for +inf
            e[r] = ~0ull;
          }
#pragma unroll
          for (int r = 0; r < R; ++r)
            if (v[r] < FINF && !(up_band32(v[r], mq) < lo) && !(dn_band32(v[r], mq) > hi))
              e[r] = exact_dist(ix[r]);
          for (;;) {  // the rank-th smallest of e (ties leave together)
            uint64_t m = ~0ull;
#pragma unroll
            for (int r = 0; r < R; ++r) m = e[r] < m ? e[r] : m;
            m = warp_min64(m);
            int c = 0;
#pragma unroll
            for (int r = 0; r < R; ++r) c += __popc(__ballot_sync(FULL, e[r] == m));
            if (c >= rank || m == ~0ull) {
              kth = m;
              break;
            }
            rank -= c;
#pragma unroll
            for (int r = 0; r < R; ++r) e[r] = e[r] == m ? ~0ull : e[r];
          }
        }
        __syncwarp();
      } else if (len >= K) {
        // radix select on the exact distances, 8 bits a pass, over the
        // candidates within the bound (U was set from K listed candidates)
        ++redone;
        uint64_t prefix = 0, mask = 0;
        uint32_t rank = (uint32_t)K;
        for (int shift = 56; shift >= 0; shift -= 8) {
          __syncwarp();
          for (int b = lane; b < 256; b += 32) hist[b] = 0u;
          __syncwarp();
          enumerate([&](int a, int b) {
            pairs += (unsigned)(b - a);
            for (int j = a + lane; j < b; j += 32) {
              const uint64_t m = exact_dist(j);
              if ((m & mask) == prefix) atomicAdd(&hist[(m >> shift) & 255u], 1u);
            }
            __syncwarp();
          });
          __syncwarp();
          uint32_t s = 0, loc[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            loc[i] = hist[8 * lane + i];
            s += loc[i];
          }
          uint32_t incl = s;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL, incl, o);
            if (lane >= o) incl += y;
          }
          const uint32_t excl = incl - s;
          const unsigned hit = __ballot_sync(FULL, excl < rank && rank <= incl);
          const int src = hit ? __ffs(hit) - 1 : 0;
          uint32_t run = excl, digit = 255, before = excl;
#pragma unroll
          for (int i = 7; i >= 0; --i) {  // the first bucket that reaches the rank
            run = excl;
#pragma unroll
            for (int k = 0; k < i; ++k) run += loc[k];
            if (run < rank && rank <= run + loc[i]) {
              digit = (uint32_t)(8 * lane + i);
              before = run;
            }
          }
          digit = __shfl_sync(FULL, digit, src);
          before = __shfl_sync(FULL, before, src);
          prefix |= (uint64_t)digit << shift;
          mask |= 255ull << shift;
          rank -= before;
        }
        // distances of non-finite data, as the lists and the select rank them
        kth = K <= EGB_KREG_MAX && prefix > INF_BITS ? INF_BITS : prefix;
        __syncwarp();
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
