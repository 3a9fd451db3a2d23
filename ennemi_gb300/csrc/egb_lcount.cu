// egb_lcount.cu -- exact ball counts of three and more columns.
//
// #{j : max_c fl64(|x_cj - x_cq|) <= r_q} per query, as query_ball_point
// (..., p=inf, return_length=True) (ennemi/_entropy_estimators.py:152-154,
// :196, :243-245), on the nested grid copy.
//
// A warp takes an item: up to 32 neighbouring queries, whose points are also
// a leaf with a bounding box (egb_leaf.cuh).  It lists the leaves within the
// item's largest radius once.  For each listed leaf every lane tests its own
// query: a leaf inside the ball counts whole; where some balls' surfaces cut
// it, its points are loaded once, one per lane, and screened for those queries
// in turn.  A query thus looks at the few leaves of its own ball, not at the
// windows of 32 queries, and the loads serve all queries that need them.
//
// Exactness: with band() of egb_internal.cuh, a candidate with FP32 distance
// <= lo = r - band is inside, one beyond hi = r + band outside, and one
// between is decided in FP64; box tests follow the screen's arithmetic
// (egb_leaf.cuh).  Items whose list overflows (far-out queries with wide
// balls) and jobs whose values rule out the FP32 copy take the candidates of
// each query's own windows, the latter in FP64.
//
// What bounds it: instruction issue of the screens (15 cut leaves a query for
// the radii of a 4-D kNN over 20,000 points) and their latency, hence 64
// registers for eight blocks per SM (measured 4.15, 3.33, 3.01 ms at four, six
// and eight).  240 jobs of 20,000 3-D points: 3.0 ms, against 7.1 of the
// warp-wide windows before; 500,000 4-D points: 2.5 against 4.5.
#include <algorithm>

#include "egb_leaf.cuh"

namespace egb {
namespace {

using namespace leaf_detail;

constexpr int LC_WARPS = 4;

// Boxes of the items' points: one warp per item.
__global__ void __launch_bounds__(256)
leaf_box_kernel(const JobDev* __restrict__ jobs, const WorkItem* __restrict__ items, int nitems,
                float* __restrict__ boxes) {
  const int lane = threadIdx.x & 31;
  const int it = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (it >= nitems) return;
  const WorkItem wi = items[it];
  const JobDev* __restrict__ J = jobs + wi.job;
  const int d = J->sp.d;
  const int p = min(wi.q0 + lane, wi.q1 - 1);
  for (int c = 0; c < d; ++c) {
    // order-preserving integer image of the float, for the integer reductions
    const int b = __float_as_int(J->c32g[(int64_t)c * J->lds + p]);
    const int o = b ^ ((b >> 31) & 0x7fffffff);
    const int lo = __reduce_min_sync(FULL, o), hi = __reduce_max_sync(FULL, o);
    if (lane == 0) {
      boxes[(int64_t)(2 * c) * nitems + it] = __int_as_float(lo ^ ((lo >> 31) & 0x7fffffff));
      boxes[(int64_t)(2 * c + 1) * nitems + it] = __int_as_float(hi ^ ((hi >> 31) & 0x7fffffff));
    }
  }
}

template <int D>
__global__ void __launch_bounds__(LC_WARPS * 32, D ? 8 : 1)
lcount_kernel(const JobDev* __restrict__ jobs, const WorkItem* __restrict__ items, int nitems,
              const float* __restrict__ boxes, int per, int* __restrict__ counter) {
  constexpr int DQ = D ? D : EGB_DMAX;
  constexpr float FINF = __builtin_huge_valf();
  __shared__ NearLeaf<D> near_s[LC_WARPS][LEAF_CAP];
  __shared__ float4 query_s[LC_WARPS][D ? 32 : 1];   // coordinates (D <= 4)
  __shared__ float2 bound_s[LC_WARPS][32];           // lo, hi
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  NearLeaf<D>* leaves = near_s[warp];
  const int split = (WG_QB + per - 1) / per;  // parts of `per` queries of an item

  for (;;) {
    int part = 0;
    if (lane == 0) part = atomicAdd(counter, 1);
    part = __shfl_sync(FULL, part, 0);
    if (part >= nitems * split) break;
    const int item = part / split;
    const WorkItem wi = items[item];
    const JobDev* __restrict__ J = jobs + wi.job;
    const int d = D ? D : J->sp.d;
    const int64_t lds = J->lds;
    const double* __restrict__ c64 = J->c64g;
    const float* __restrict__ g = J->c32g;
    const int sq = wi.strip & 0xffff;
    const bool unsafe = (*J->jflags & TF_UNSAFE32) != 0u;
    // one query per lane
    const int q0 = wi.q0 + (part % split) * per;
    const int nq = min(per, wi.q1 - q0);
    if (nq <= 0) continue;
    const bool exists = lane < nq;
    const int qp = q0 + lane;
    float qv[DQ];
    float am = 0.0f;
#pragma unroll
    for (int c = 0; c < DQ; ++c) {
      if (D == 0 && c >= d) break;
      qv[c] = exists ? g[(int64_t)c * lds + qp] : 0.0f;
      am = fmaxf(am, fabsf(qv[c]));
    }
    const float mq = __fmaf_ru(am, 1.0f + 0x1p-22f, 0x1p-148f);
    const int32_t w = exists ? J->idxg[qp] : 0;
    const double qr = exists ? radius_of(J->rad, J->rad_given, w) : -1.0;
    const int rc = exists ? radius_class(qr) : 0;  // 0 none, 1 finite, 2 every point
    const uint64_t rbits = rc == 1 ? (uint64_t)__double_as_longlong(fabs(qr)) : 0ull;
    float lo = -1.0f, hi = -1.0f;  // inside up to lo, outside beyond hi
    if (rc == 1) {
      const double b = band((double)mq, qr);
      lo = unsafe ? -1.0f : __double2float_rd(qr - b);
      hi = unsafe ? FINF : __double2float_ru(qr + b);
    }
    int count = rc == 2 ? J->len : 0;
    unsigned long long pairs = 0, exact = 0;
    const unsigned todo = __ballot_sync(FULL, rc == 1);
    const float T = __uint_as_float(__reduce_max_sync(FULL, rc == 1 ? __float_as_uint(hi) : 0u));
    int nleaf = -1;
    if (todo && !unsafe && T < FINF) nleaf = near_leaves<D>(J, items, boxes, nitems, item, sq, d, T, leaves);

    // the FP64 decision for query i (lanes where `mid`: a candidate j)
    auto exact_in = [&](int i, bool mid, int j) -> unsigned {
      const uint64_t rb = ((uint64_t)__shfl_sync(FULL, (uint32_t)(rbits >> 32), i) << 32) |
                          __shfl_sync(FULL, (uint32_t)rbits, i);
      uint64_t mm = ~0ull;
      if (mid) {
        mm = 0;
#pragma unroll
        for (int c = 0; c < DQ; ++c) {
          if (D == 0 && c >= d) break;
          const uint64_t v = absdiff_bits(c64[(int64_t)c * lds + j], c64[(int64_t)c * lds + q0 + i]);
          mm = v > mm ? v : mm;
        }
      }
      return __ballot_sync(FULL, mid && mm <= rb);
    };

    if (nleaf >= 0) {
      if constexpr (D > 0) {
        query_s[warp][lane] = make_float4(qv[0], qv[1], qv[2], D > 3 ? qv[D > 3 ? 3 : 0] : 0.0f);
        bound_s[warp][lane] = make_float2(lo, hi);
        __syncwarp();
      }
      for (int k = 0; k < nleaf; ++k) {
        const NearLeaf<D> L = leaves[k];
        float near = 0.0f, far = 0.0f;
#pragma unroll
        for (int c = 0; c < DQ; ++c) {
          if (D == 0 && c >= d) break;
          float bl, bh;
          if constexpr (D > 0) {
            bl = L.lo[c];
            bh = L.hi[c];
          } else {
            bl = boxes[(int64_t)(2 * c) * nitems + L.item];
            bh = boxes[(int64_t)(2 * c + 1) * nitems + L.item];
          }
          near = fmaxf(near, fmaxf(bl - qv[c], qv[c] - bh));
          far = fmaxf(far, fmaxf(bh - qv[c], qv[c] - bl));
        }
        const bool whole = far <= lo;  // lo, hi are -1 without a finite radius
        if (whole) count += L.n;
        unsigned cut = __ballot_sync(FULL, near <= hi && !whole);
        if (!cut) continue;
        pairs += 32ull * __popc(cut);
        const bool in = lane < L.n;
        const int j = in ? L.q0 + lane : L.q0;
        float p[DQ];
#pragma unroll
        for (int c = 0; c < DQ; ++c) {
          if (D == 0 && c >= d) break;
          p[c] = g[(int64_t)c * lds + j];
        }
        do {
          const int i = __ffs(cut) - 1;
          cut &= cut - 1u;
          float dd, olo, ohi;
          if constexpr (D > 0) {
            const float4 o = query_s[warp][i];
            const float2 b = bound_s[warp][i];
            dd = fmaxf(fmaxf(fabsf(p[0] - o.x), fabsf(p[1] - o.y)), fabsf(p[2] - o.z));
            if constexpr (D > 3) dd = fmaxf(dd, fabsf(p[D > 3 ? 3 : 0] - o.w));
            olo = b.x;
            ohi = b.y;
          } else {
            dd = 0.0f;
#pragma unroll
            for (int c = 0; c < DQ; ++c) {
              if (c >= d) break;
              dd = fmaxf(dd, fabsf(p[c] - __shfl_sync(FULL, qv[c], i)));
            }
            olo = __shfl_sync(FULL, lo, i);
            ohi = __shfl_sync(FULL, hi, i);
          }
          const unsigned bl = __ballot_sync(FULL, in && dd <= olo);
          const unsigned bh = __ballot_sync(FULL, in && dd <= ohi);
          int c0 = __popc(bl);
          if (bl != bh) {
            c0 += __popc(exact_in(i, ((bh & ~bl) >> lane) & 1u, j));
            exact += __popc(bh & ~bl);
          }
          if (lane == i) count += c0;
        } while (cut);
      }
      __syncwarp();  // the lists are rewritten for the next part
    } else {
      for (unsigned left = todo; left; left &= left - 1u) {
        const int i = __ffs(left) - 1;
        float o[DQ];
#pragma unroll
        for (int c = 0; c < DQ; ++c) {
          if (D == 0 && c >= d) break;
          o[c] = __shfl_sync(FULL, qv[c], i);
        }
        const float olo = __shfl_sync(FULL, lo, i), ohi = __shfl_sync(FULL, hi, i);
        const uint64_t ob = ((uint64_t)__shfl_sync(FULL, (uint32_t)(rbits >> 32), i) << 32) |
                            __shfl_sync(FULL, (uint32_t)rbits, i);
        const QueryBox qb{coord_below(o[0]), coord_above(o[0]), coord_below(o[1]), coord_above(o[1]),
                          coord_below(o[2]), coord_above(o[2])};
        // jobs with clamped values search everything
        const float tb = unsafe ? FINF : plan_margin(f32_up_of_bits(ob));
        int c0 = 0;
        query_ranges<true, 1>(J, g, sq, qb, tb, [&](int a, int b) {
          pairs += (unsigned)(b - a);
          for (int p0 = a; p0 < b; p0 += 32) {
            const bool in = p0 + lane < b;
            const int j = in ? p0 + lane : a;
            float dd = 0.0f;
#pragma unroll
            for (int c = 0; c < DQ; ++c) {
              if (D == 0 && c >= d) break;
              dd = fmaxf(dd, fabsf(g[(int64_t)c * lds + j] - o[c]));
            }
            const unsigned bl = __ballot_sync(FULL, in && dd <= olo);
            const unsigned bh = __ballot_sync(FULL, in && dd <= ohi);
            c0 += __popc(bl);
            if (bl != bh) {
              c0 += __popc(exact_in(i, ((bh & ~bl) >> lane) & 1u, j));
              exact += __popc(bh & ~bl);
            }
          }
        });
        if (lane == i) count += c0;
      }
    }
    if (exists) J->cnt[w] = count;
    if (lane == 0) {
      atomicAdd(J->stats + 0, pairs);
      if (exact) atomicAdd(J->stats + 1, exact);
    }
  }
}

template <int D>
void launch_t(const JobDev* jobs, const WorkItem* items, int nitems, const float* boxes, int* counter,
              int num_sms, cudaStream_t st) {
  auto kern = lcount_kernel<D>;
  int per_sm = 1;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, LC_WARPS * 32, 0);
  if (per_sm < 1) per_sm = 1;
  // queries per part: an item's leaf list serves all of its queries, but a
  // part is one warp's serial work, so small launches take smaller parts
  const int64_t warps = (int64_t)num_sms * per_sm * LC_WARPS;
  int per = WG_QB;
  while (per > 4 && (int64_t)nitems * (WG_QB / per) < 2 * warps) per /= 2;
  const int64_t parts = (int64_t)nitems * (WG_QB / per);
  const int grid = (int)std::min<int64_t>((int64_t)num_sms * per_sm, (parts + LC_WARPS - 1) / LC_WARPS);
  if (grid < 1) return;
  kern<<<grid, LC_WARPS * 32, 0, st>>>(jobs, items, nitems, boxes, per, counter);
  count_launch();
}

}  // namespace

void launch_leaf_boxes(const JobDev* jobs_d, const WorkItem* items_d, int nitems, float* boxes,
                       cudaStream_t st) {
  if (nitems <= 0) return;
  leaf_box_kernel<<<(nitems + 7) / 8, 256, 0, st>>>(jobs_d, items_d, nitems, boxes);
  count_launch();
}

void launch_count_leaf(const JobDev* jobs_d, const WorkItem* items_d, int nitems, const float* boxes,
                       int dclass, int* counter, int num_sms, cudaStream_t st) {
  if (nitems <= 0) return;
  if (dclass == 3) launch_t<3>(jobs_d, items_d, nitems, boxes, counter, num_sms, st);
  else if (dclass == 4) launch_t<4>(jobs_d, items_d, nitems, boxes, counter, num_sms, st);
  else launch_t<0>(jobs_d, items_d, nitems, boxes, counter, num_sms, st);
}

}  // namespace egb
