// egb_leaf.cuh -- leaf boxes of a grid copy, and the ranges of one query.
//
// A work item of a nested grid (up to 32 consecutive positions of one cell,
// in column-0 order) is also a leaf of the job's points: strips split column
// 1, cells column 2, items column 0, as a sort-tile-recursive packing does.
// leaf_box_kernel stores each leaf's bounding box over all d columns, on the
// centred FP32 copy: boxes[(2 c) * nitems + item] the least, [(2 c + 1) *
// nitems + item] the largest value of column c.
//
// The box tests use the screen's own arithmetic.  Rounding is monotone, so
// for a point p of a box [lo, hi] and a query q, fl(|p - q|) >= fl(lo - q) and
// >= fl(q - hi), and <= max(fl(hi - q), fl(q - lo)): a box whose distance
// exceeds a screen bound holds no candidate that the screen would keep, and a
// box whose farthest distance is within a bound holds only candidates within
// it -- no margin is needed.
#pragma once
#include "egb_wgrid.cuh"

namespace egb {
namespace leaf_detail {

using wgrid_detail::dn_band32;
using wgrid_detail::plan_margin;
using wgrid_detail::up_band32;
using wgrid_detail::warp_window;

constexpr unsigned FULL = 0xffffffffu;
constexpr int LEAF_CAP = 128;  // listed leaves of an item

// Planning bounds of a query's coordinates 0..2 (from its FP32 copy: see
// wwalk_kernel).
struct QueryBox {
  float xl, xh, yl, yh, zl, zh;
};
__device__ __forceinline__ float coord_below(float v) {
  return __fsub_rd(v, __fmaf_ru(fabsf(v), 0x1p-22f, 0x1p-148f));
}
__device__ __forceinline__ float coord_above(float v) {
  return __fadd_ru(v, __fmaf_ru(fabsf(v), 0x1p-22f, 0x1p-148f));
}

// Every range of positions within the planning bound tb of one query (warp
// uniform), its strip sq first and then outward; f(a, b) may tighten tb.
// STRIDE: floats from one position's column 0 to the next.
template <bool NEST, int STRIDE, typename F>
__device__ __forceinline__ void query_ranges(const JobDev* __restrict__ J, const float* __restrict__ g,
                                             int sq, const QueryBox& q, const float& tb, F&& f) {
  const int lane = threadIdx.x & 31;
  const int32_t* __restrict__ sst = J->sstart;
  const int32_t* __restrict__ cst = J->cstart;
  const float* __restrict__ ylo = J->sylo32;
  const float* __restrict__ yhi = J->syhi32;
  const int S = J->nstrips, S2 = NEST ? J->nsub : 1;
  auto crange = [&](int a, int b) {
    const float xl = fminf(__fsub_rd(q.xl, tb), 1e37f), xh = fmaxf(__fadd_ru(q.xh, tb), -1e37f);
    int wl, wh;
    if (b - a <= 1024) {
      // whole blocks of 32 positions, from the first value of each: one load
      // and two ballots, and no candidate block is split
      const int p = a + 32 * lane;
      const float x = p < b ? g[(int64_t)p * STRIDE] : __builtin_huge_valf();
      const int nl = __popc(__ballot_sync(FULL, x < xl)), nh = __popc(__ballot_sync(FULL, x <= xh));
      wl = a + 32 * max(nl - 1, 0);
      wh = min(b, a + 32 * nh);
    } else {
      warp_window<float, STRIDE>(g, a, b, xl, xh, wl, wh);
    }
    if (wl < wh) f(wl, wh);
  };
  auto cstrip = [&](int s) {
    if constexpr (NEST) {
      const float* __restrict__ zlo = J->czlo32 + s * S2;
      const float* __restrict__ zhi = J->czhi32 + s * S2;
      int c0 = 0, c1 = 0;
      for (int b = 0; b < S2; b += 32) {
        const int c = b + lane;
        c0 += __popc(__ballot_sync(FULL, c < S2 && __fsub_rd(q.zl, zhi[c]) > tb));
        c1 += __popc(__ballot_sync(FULL, c < S2 && !(__fsub_rd(zlo[c], q.zh) > tb)));
      }
      for (int c = c0; c < c1; ++c) crange(cst[s * S2 + c], cst[s * S2 + c + 1]);
    } else {
      crange(sst[s], sst[s + 1]);
    }
  };
  cstrip(sq);
  for (int up = sq + 1, dn = sq - 1;;) {
    const bool ou = up < S && !(__fsub_rd(ylo[up], q.yh) > tb);
    const bool od = dn >= 0 && !(__fsub_rd(q.yl, yhi[dn]) > tb);
    if (!ou && !od) break;
    cstrip(ou && (!od || (up - sq) <= (sq - dn)) ? up++ : dn--);
  }
}

// A listed leaf: its box (columns beyond four stay in global memory) and its
// points [q0, q0 + n).
template <int D>
struct alignas(16) NearLeaf {
  float lo[D], hi[D];
  int q0, n;
};
template <>
struct alignas(16) NearLeaf<0> {
  int item, q0, n;
};

// The leaves whose boxes lie within T of the box of leaf `home` (the item's
// own), home strip first, into out.  Returns their number, or -1 when out
// cannot hold them.
template <int D>
__device__ __forceinline__ int near_leaves(const JobDev* __restrict__ J,
                                           const WorkItem* __restrict__ items,
                                           const float* __restrict__ boxes, int64_t nitems, int home,
                                           int sq, int d, float T, NearLeaf<D>* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  const uint32_t lt = (1u << lane) - 1u;
  const int S = J->nstrips, S2 = J->nsub;
  const float* __restrict__ ylo = J->sylo32;
  const float* __restrict__ yhi = J->syhi32;
  const int32_t* __restrict__ first = J->leaf0;  // first leaf of each cell
  const float yl = boxes[2 * nitems + home], yh = boxes[3 * nitems + home];
  const float zl = boxes[4 * nitems + home], zh = boxes[5 * nitems + home];
  int n = 0;
  auto strip = [&](int s) {
    const float* __restrict__ zlo = J->czlo32 + s * S2;
    const float* __restrict__ zhi = J->czhi32 + s * S2;
    int c0 = 0, c1 = 0;
    for (int b = 0; b < S2; b += 32) {
      const int c = b + lane;
      c0 += __popc(__ballot_sync(FULL, c < S2 && zl - zhi[c] > T));
      c1 += __popc(__ballot_sync(FULL, c < S2 && !(zlo[c] - zh > T)));
    }
    if (c0 >= c1) return true;
    const int l1 = first[s * S2 + c1];
    for (int b = first[s * S2 + c0]; b < l1; b += 32) {
      const int l = b + lane;
      bool in = l < l1;
      NearLeaf<D> L;
#pragma unroll
      for (int c = 0; c < (D ? D : EGB_DMAX); ++c) {
        if (D == 0 && c >= d) break;
        if (in) {
          const float lo = boxes[(2 * c) * nitems + l], hi = boxes[(2 * c + 1) * nitems + l];
          in = !(lo - boxes[(2 * c + 1) * nitems + home] > T) && !(boxes[(2 * c) * nitems + home] - hi > T);
          if constexpr (D > 0) {
            L.lo[c] = lo;
            L.hi[c] = hi;
          }
        }
      }
      const uint32_t m = __ballot_sync(FULL, in);
      if (n + __popc(m) > LEAF_CAP) return false;
      if (in) {
        if constexpr (D == 0) L.item = l;
        L.q0 = items[l].q0;
        L.n = items[l].q1 - L.q0;
        out[n + __popc(m & lt)] = L;
      }
      n += __popc(m);
    }
    return true;
  };
  if (!strip(sq)) return -1;
  for (int up = sq + 1; up < S && !(ylo[up] - yh > T); ++up)
    if (!strip(up)) return -1;
  for (int dn = sq - 1; dn >= 0 && !(yl - yhi[dn] > T); --dn)
    if (!strip(dn)) return -1;
  __syncwarp();
  return n;
}

}  // namespace leaf_detail
}  // namespace egb
