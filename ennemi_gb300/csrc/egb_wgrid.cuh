// egb_wgrid.cuh -- warp-level form of the grid (strip) kernels in FP64, the
// comparator of the FP32 kernels, and pieces that those share with it.
//
// Same layout and search region as egb_grid.cuh, but every warp works alone:
// it pulls an item of up to 32 consecutive strip positions (one query per
// lane) from the device work counter and plans its windows with ballots and
// shuffles instead of CTA barriers, so planning never stalls other warps, and
// each warp's windows are narrower (32 queries span a quarter of the x-range
// of 128).
//
// Schedule of an item: the queries' own positions, the rest of the home
// strip's window [xa - T, xb + T], then strips sq+1, sq-1, sq+2, ... while
// open for some unfinished query, T being the largest threshold among
// unfinished queries.  Window ends are exact (16-ary warp search).  When at
// most OUTLIER_LANES queries are still unfinished, the warp finishes them one
// at a time with all 32 lanes sharing the candidates of the remaining strips
// (window [q0 - t, q0 + t] of that query alone); for kNN each lane keeps its
// own list and the K-th smallest of the union is taken at the end.
#pragma once
#include "egb_tile.cuh"

namespace egb {
namespace wgrid_detail {

constexpr int WG_WARPS = 4;       // warps per CTA (independent)
constexpr int OUTLIER_LANES = 2;  // switch to cooperative finishing below this

template <int KMAX>
__device__ __forceinline__ void insert_sorted(uint64_t (&top)[KMAX], uint64_t v) {
  top[KMAX - 1] = v;
#pragma unroll
  for (int s = KMAX - 1; s > 0; --s) {
    const uint64_t a = top[s - 1], b = top[s];
    const bool sw = b < a;
    top[s - 1] = sw ? b : a;
    top[s] = sw ? a : b;
  }
}

__device__ __forceinline__ uint64_t warp_max_u64(uint64_t v) {
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    const uint64_t w = __shfl_xor_sync(0xffffffffu, v, o);
    v = w > v ? w : v;
  }
  return v;
}
__device__ __forceinline__ uint64_t warp_min_u64(uint64_t v) {
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    const uint64_t w = __shfl_xor_sync(0xffffffffu, v, o);
    v = w < v ? w : v;
  }
  return v;
}

// Conservative FP32 planning values.  A grid copy holds, per coordinate,
// f(v) = fl32(clamp(fl64(v - c), +-1e37)), monotone in v.  plan_margin(t) >=
// t (1 + 2^-20), so that a candidate skipped because its coordinate gap
// exceeds plan_margin(t) has an FP64 coordinate distance fl64(gap) >= gap (1 - 2^-53) > t.
__device__ __forceinline__ float plan_margin(float t) { return __fmul_ru(t, 1.0f + 0x1p-20f); }

// Exact window of strip [s0, s1) for column-0 values [xlo, xhi]: the lower
// half-warp finds the first position with x >= xlo, the upper half the first
// with x > xhi.
// STRIDE: elements from one position's column 0 to the next.
template <typename V, int STRIDE = 1>
__device__ __forceinline__ void warp_window(const V* x, int s0, int s1, V xlo, V xhi, int& wlo,
                                            int& whi) {
  const int lane = threadIdx.x & 31;
  const bool upper = lane >= 16;
  const int l16 = lane & 15;
  const unsigned m = upper ? 0xffff0000u : 0x0000ffffu;
  // Both halves run the same loop shape; each keeps its own bracket.
  int lo = s0, hi = s1;
  for (int round = 0; round < 40; ++round) {
    const int n = hi - lo;
    const bool small = n <= 16;
    int p = small ? lo + l16 : lo + (int)((int64_t)(l16 + 1) * n / 17);
    const bool inr = p < hi;
    p = inr ? p : s0;
    const V v = x[(int64_t)p * STRIDE];
    const bool t = inr && (upper ? (v <= xhi) : (v < xlo));
    const unsigned b = __ballot_sync(0xffffffffu, t) & m;
    const int c = __popc(b);
    if (small) {
      lo = lo + c;
      hi = lo;
    } else {
      const int nlo = c == 0 ? lo : lo + (int)((int64_t)c * n / 17) + 1;
      const int nhi = c == 16 ? hi : lo + (int)((int64_t)(c + 1) * n / 17);
      lo = nlo;
      hi = nhi;
    }
    const bool done = hi - lo <= 0;
    if (__all_sync(0xffffffffu, done)) break;
  }
  wlo = __shfl_sync(0xffffffffu, lo, 0);
  whi = __shfl_sync(0xffffffffu, lo, 16);
  if (whi < wlo) whi = wlo;
}

// FP32 threshold bounding from above the FP64 distance of any candidate
// whose FP32 distance is t (t >= 0 finite): t + band(mq, t), rounded up.
__device__ __forceinline__ float up_band32(float t, float mq) {
  if (!(t < __int_as_float(0x7f800000))) return __int_as_float(0x7f800000);
  return __fmaf_ru(t, 1.0f + 0x1p-21f, __fmaf_ru(mq, 0x1p-21f, 0x1p-100f));
}
// FP32 value bounding from below the FP64 distance of a candidate whose FP32
// distance is t (t >= 0 finite).  From |t - D| <= 2^-23 (M + D)(1 + 2^-20)
// + 2^-148 (egb_internal.cuh), D >= (t - 2^-23 M (1 + 2^-20) - 2^-148) /
// (1 + 2^-23 (1 + 2^-20)); with mq >= M and the factors taken four times
// over, (t - 2^-21 mq - 2^-100)(1 - 2^-21) rounded down is below that.
__device__ __forceinline__ float dn_band32(float t, float mq) {
  if (!(t < __int_as_float(0x7f800000))) return 0.0f;
  const float a = __fsub_rd(t, __fmaf_ru(mq, 0x1p-21f, 0x1p-100f));
  return a > 0.0f ? __fmul_rd(a, 1.0f - 0x1p-21f) : 0.0f;
}

// Sorted insert of (v, j) into an FP32 list with candidate indices; returns
// the value pushed out of the last slot.
template <int KMAX>
__device__ __forceinline__ float insert_sorted_fi(float (&l)[KMAX], int (&ix)[KMAX], float v,
                                                  int j) {
  const float out = l[KMAX - 1];
  l[KMAX - 1] = v;
  ix[KMAX - 1] = j;
#pragma unroll
  for (int s = KMAX - 1; s > 0; --s) {
    const float a = l[s - 1], b = l[s];
    const int ia = ix[s - 1], ib = ix[s];
    const bool sw = b < a;
    l[s - 1] = sw ? b : a;
    l[s] = sw ? a : b;
    ix[s - 1] = sw ? ib : ia;
    ix[s] = sw ? ia : ib;
  }
  return out;
}

// K-th smallest of the union of per-lane sorted lists (the first KMAX - K
// entries of each list are padding).  Warp-wide; result in every lane.
template <int KMAX, typename V>
__device__ __forceinline__ V warp_kth_of_lists(const V (&lst_in)[KMAX], int K, V inf) {
  const int lane = threadIdx.x & 31;
  V lst[KMAX];
#pragma unroll
  for (int s = 0; s < KMAX; ++s) lst[s] = lst_in[s];
  int h = KMAX - K;
  V kth = inf;
  for (int r = 0; r < K; ++r) {
    V v = h < KMAX ? lst[h] : inf;
    int who = lane;
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      const V ov = __shfl_xor_sync(0xffffffffu, v, o);
      const int ow = __shfl_xor_sync(0xffffffffu, who, o);
      if (ov < v || (ov == v && ow < who)) {
        v = ov;
        who = ow;
      }
    }
    kth = v;
    if (lane == who) ++h;
  }
  return kth;
}

// Blocks per SM the register budget of a variant targets: the K <= 4 kNN
// kernels are latency-bound and gain from occupancy more than they lose to
// a few spilled registers outside the candidate loop.
template <int D, int KMAX, bool COUNT>
constexpr int wgrid_min_blocks() {
  return (!COUNT && KMAX == 4) ? (D == 2 ? 5 : 4) : 1;
}

template <int D, int KMAX, bool COUNT, bool NEST>
__global__ void __launch_bounds__(WG_WARPS * 32, (wgrid_min_blocks<D, KMAX, COUNT>()))
wgrid_kernel(const JobDev* __restrict__ jobs, const WorkItem* __restrict__ items, int nitems,
             int* __restrict__ counter, int dmax) {
  constexpr int DQ = D ? D : EGB_DMAX;
  const int lane = threadIdx.x & 31;
  (void)dmax;

  for (;;) {
    int it = 0;
    if (lane == 0) it = atomicAdd(counter, 1);
    it = __shfl_sync(0xffffffffu, it, 0);
    if (it >= nitems) break;
    const WorkItem wi = items[it];
    const JobDev* __restrict__ J = jobs + wi.job;
    const int d = D ? D : J->sp.d;
    const int len = J->len;
    const int64_t lds = J->lds;
    const double* __restrict__ g = J->c64g;
    const int32_t* __restrict__ sst = J->sstart;      // strip starts
    // strip column-1 bounds and (nested) cell column-2 bounds
    const double* __restrict__ ylo_t = J->sylo;
    const double* __restrict__ yhi_t = J->syhi;
    const int S = J->nstrips;
    // nested grids: cells of strip s are s * S2 .. s * S2 + S2 - 1
    const int S2 = NEST ? J->nsub : 1;
    const int32_t* __restrict__ cst = J->cstart;
    const double* __restrict__ czlo = J->czlo;
    const double* __restrict__ czhi = J->czhi;
    const int K = COUNT ? 1 : J->K;

    const int qp = wi.q0 + lane;
    const bool exists = qp < wi.q1;
    const int nq = wi.q1 - wi.q0;
    double qv[DQ];
#pragma unroll
    for (int c = 0; c < DQ; ++c) {
      if (D == 0 && c >= d) break;
      qv[c] = exists ? g[(int64_t)c * lds + qp] : 0.0;
    }
    const double qx = qv[0], qy = qv[1];
    const double qz = NEST ? qv[NEST ? 2 : 0] : 0.0;

    // ---- per-lane state
    uint64_t top[COUNT ? 1 : KMAX];      // exact list (bit patterns)
    double qr = -1.0;
    uint64_t rbits = 0;
    int cntq = 0;
    bool qok = exists;
    if constexpr (COUNT) {
      qr = exists ? radius_of(J->rad, J->rad_given, J->idxg[qp]) : -1.0;
      qok = exists && (qr >= 0.0);
      rbits = qok ? (uint64_t)__double_as_longlong(qr) : 0ull;
    } else {
#pragma unroll
      for (int s = 0; s < KMAX; ++s) top[s] = (exists && s >= KMAX - K) ? INF_BITS : 0ull;
    }
    // upper bound of what this lane's query still needs (planning threshold)
    auto tq = [&]() -> double {
      if (!qok) return -1.0;
      if constexpr (COUNT) {
        return qr;
      } else {
        return bits_to_double(top[KMAX - 1]);
      }
    };
    // largest planning threshold over the lanes (negative ones count as 0)
    auto wmax = [&](double v) -> double {
      return bits_to_double(warp_max_u64(v >= 0.0 ? (uint64_t)__double_as_longlong(v) : 0ull));
    };
    auto exact_dist = [&](int j, int q) -> uint64_t {
      uint64_t mm = 0;
#pragma unroll
      for (int c = 0; c < DQ; ++c) {
        if (D == 0 && c >= d) break;
        const int64_t off = (int64_t)c * lds;
        const uint64_t v = absdiff_bits(g[off + j], g[off + q]);
        mm = v > mm ? v : mm;
      }
      return mm;
    };

    // Resolve the hits of one group of 4 candidates at g0.
    auto resolve = [&](int g0, uint32_t hits) {
      if constexpr (!COUNT) {
        while (hits) {
          const int j = g0 + __ffs(hits) - 1;
          hits &= hits - 1u;
          const uint64_t mm = exact_dist(j, qp);
          if (mm < top[KMAX - 1]) insert_sorted<KMAX>(top, mm);
        }
      }
    };
    // candidates of the group at g0 inside [ra, rb) and outside [ea, eb)
    auto group_mask = [](int g0, int ra, int rb, int ea, int eb) -> uint32_t {
      uint32_t vmask = 0xFu;
      if (g0 < ra) vmask &= ~((1u << (ra - g0)) - 1u);
      if (g0 + 4 > rb) vmask &= (1u << (rb - g0)) - 1u;
      if (g0 + 4 > ea && g0 < eb) {
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (g0 + u >= ea && g0 + u < eb) vmask &= ~(1u << u);
      }
      return vmask;
    };

    unsigned long long pairs = 0;  // candidate-query pairs screened by this item
    // Screen the candidates [ra, rb) minus [ea, eb) against this lane's query.
    auto scan = [&](int ra, int rb, int ea, int eb) {
      if (rb <= ra) return;
      pairs += (unsigned long long)(rb - ra - max(0, min(rb, eb) - max(ra, ea))) * (unsigned long long)nq;
      for (int g0 = ra & ~3; g0 < rb; g0 += 4) {
        const uint32_t vmask = group_mask(g0, ra, rb, ea, eb);
        uint32_t hits = 0;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int j = g0 + u < len ? g0 + u : len - 1;
          uint64_t mm = 0;
#pragma unroll
          for (int c = 0; c < DQ; ++c) {
            if (D == 0 && c >= d) break;
            const uint64_t v = absdiff_bits(g[(int64_t)c * lds + j], qv[c]);
            mm = v > mm ? v : mm;
          }
          if constexpr (COUNT) cntq += ((vmask >> u) & 1u) && qok && mm <= rbits ? 1 : 0;
          else hits |= (mm < top[KMAX - 1] ? 1u : 0u) << u;
        }
        hits &= vmask;
        if (hits) resolve(g0, hits);
      }
    };

    const int sq = NEST ? (wi.strip & 0xffff) : wi.strip;
    const int hc2 = NEST ? (wi.strip >> 16) : 0;  // home cell within the strip
    const int hs0 = NEST ? cst[sq * S2 + hc2] : sst[sq];
    const int hs1 = NEST ? cst[sq * S2 + hc2 + 1] : sst[sq + 1];
    const double xa = __shfl_sync(0xffffffffu, qx, 0);        // the item's column-0 range
    const double xb = __shfl_sync(0xffffffffu, qx, nq - 1);
    // column-2 centre of the item (nested grids: where other strips start)
    const double zmid = NEST ? __shfl_sync(0xffffffffu, qz, (nq - 1) >> 1) : 0.0;

    // Nested grids: first cell of strip s whose column-2 range reaches z.
    auto start_cell = [&](int s, double z) -> int {
      int c0 = 0;
      for (int b = 0; b < S2; b += 32) {
        const int c = b + lane;
        c0 += __popc(__ballot_sync(0xffffffffu, c < S2 && czhi[s * S2 + c] < z));
      }
      return c0 < S2 ? c0 : S2 - 1;
    };
    // Nested grids: the cells of strip s that some lane still needs, outward
    // in column 2 from cell c0 (cell `skip` already scanned).  A lane needs a
    // cell while the strip's column-1 range and the cell's column-2 range are
    // both within its threshold; cells are ordered by column 2, so each
    // direction ends at the first cell that no lane reaches.
    auto visit_cells = [&](int s, int c0, int skip) {
      const int cb = s * S2;
      int up2 = c0, dn2 = c0 - 1;
      bool tu = true;
      for (;;) {
        const double t = tq();
        const bool reach = qok && !(ylo_t[s] - qy > t) && !(qy - yhi_t[s] > t);
        const bool ou = reach && up2 < S2 && !(czlo[cb + up2] - qz > t);
        const bool od = reach && dn2 >= 0 && !(qz - czhi[cb + dn2] > t);
        const bool any_u = __any_sync(0xffffffffu, ou);
        const bool any_d = __any_sync(0xffffffffu, od);
        if (!any_u && !any_d) break;
        int c;
        if ((tu && any_u) || !any_d) {
          c = up2++;
          tu = false;
        } else {
          c = dn2--;
          tu = true;
        }
        if (c == skip) continue;
        const bool nd = reach && !(czlo[cb + c] - qz > t) && !(qz - czhi[cb + c] > t);
        if (!__any_sync(0xffffffffu, nd)) continue;
        const double Tw = wmax(nd ? t : -1.0);
        int wl, wh;
        warp_window(g, cst[cb + c], cst[cb + c + 1], xa - Tw, xb + Tw, wl, wh);
        scan(wl, wh, 0, 0);
      }
    };

    // ---- own positions (they seed the kNN thresholds), then the rest of
    // the home strip's (cell's) window
    scan(wi.q0, wi.q1, 0, 0);
    {
      const double Tw = wmax(tq());
      int wl, wh;
      warp_window(g, hs0, hs1, xa - Tw, xb + Tw, wl, wh);
      scan(wl, wh, wi.q0, wi.q1);
    }

    // ---- other strips (nested grids: first the other cells of the home strip)
    int up = sq + 1, dn = sq - 1;
    bool turn_up = true;
    bool home_cells = NEST;
    auto unfinished = [&]() -> bool {
      if (!qok) return false;
      const double t = tq();
      const bool u = up >= S || ylo_t[up] - qy > t;
      const bool l = dn < 0 || qy - yhi_t[dn] > t;
      return !(u && l);
    };
    for (;;) {
      if (NEST && home_cells) {
        home_cells = false;
        visit_cells(sq, hc2, hc2);
        continue;
      }
      const bool unf = unfinished();
      const unsigned ub = __ballot_sync(0xffffffffu, unf);
      if (ub == 0u || __popc(ub) <= OUTLIER_LANES) break;
      const double t = tq();
      const bool ou = unf && up < S && !(ylo_t[up] - qy > t);
      const bool od = unf && dn >= 0 && !(qy - yhi_t[dn] > t);
      const bool any_u = __any_sync(0xffffffffu, ou);
      const bool any_d = __any_sync(0xffffffffu, od);
      if (!any_u && !any_d) break;  // an unfinished query always needs a side
      int s;
      if ((turn_up && any_u) || !any_d) {
        s = up++;
        turn_up = false;
      } else {
        s = dn--;
        turn_up = true;
      }
      if constexpr (NEST) {
        visit_cells(s, start_cell(s, zmid), -1);
      } else {
        const double Tw = wmax(unf ? t : -1.0);
        int wl, wh;
        warp_window(g, sst[s], sst[s + 1], xa - Tw, xb + Tw, wl, wh);
        scan(wl, wh, 0, 0);
      }
    }

    // ---- remaining unfinished queries: one at a time, all lanes cooperating
    unsigned rest = __ballot_sync(0xffffffffu, unfinished());
    if (lane == 0 && rest) atomicAdd(J->stats + 1, (unsigned long long)__popc(rest));
    while (rest) {
      const int ol = __ffs(rest) - 1;
      rest &= rest - 1u;
      const double oqx = __shfl_sync(0xffffffffu, qx, ol);
      const double oqy = __shfl_sync(0xffffffffu, qy, ol);
      const double oqz = __shfl_sync(0xffffffffu, qz, ol);
      double oqv[DQ];
#pragma unroll
      for (int c = 0; c < DQ; ++c) {
        if (D == 0 && c >= d) break;
        oqv[c] = __shfl_sync(0xffffffffu, qv[c], ol);
      }
      uint64_t top2[COUNT ? 1 : KMAX];
      int cnt2 = 0;
      uint64_t orbits = 0;
      double tb = __shfl_sync(0xffffffffu, tq(), ol);  // planning bound of what the outlier needs
      if constexpr (COUNT) {
        orbits = __shfl_sync(0xffffffffu, rbits, ol);
      } else {
#pragma unroll
        for (int s2 = 0; s2 < KMAX; ++s2) top2[s2] = s2 >= KMAX - K ? INF_BITS : 0ull;
      }
      auto oscan = [&](int ra, int rb) {
        for (int j0 = ra; j0 < rb; j0 += 32) {
          const int j = j0 + lane;
          if (j >= rb) continue;
          uint64_t mm = 0;
#pragma unroll
          for (int c = 0; c < DQ; ++c) {
            if (D == 0 && c >= d) break;
            const uint64_t v = absdiff_bits(g[(int64_t)c * lds + j], oqv[c]);
            mm = v > mm ? v : mm;
          }
          if constexpr (COUNT) cnt2 += mm <= orbits ? 1 : 0;
          else if (mm < top2[KMAX - 1]) insert_sorted<KMAX>(top2, mm);
        }
      };
      int oup = up, odn = dn;
      for (;;) {
        if constexpr (!COUNT) tb = fmin(tb, bits_to_double(warp_min_u64(top2[KMAX - 1])));
        const bool ou = oup < S && !(ylo_t[oup] - oqy > tb);
        const bool od = odn >= 0 && !(oqy - yhi_t[odn] > tb);
        if (!ou && !od) break;
        const int s = ou && (!od || (oup - sq) <= (sq - odn)) ? oup++ : odn--;
        int wl, wh;
        if constexpr (NEST) {
          // cells with column-2 range meeting [oqz - tb, oqz + tb]: a run
          int clo = 0, chi = 0;
          for (int b = 0; b < S2; b += 32) {
            const int c = b + lane;
            clo += __popc(__ballot_sync(0xffffffffu, c < S2 && oqz - czhi[s * S2 + c] > tb));
            chi += __popc(__ballot_sync(0xffffffffu, c < S2 && !(czlo[s * S2 + c] - oqz > tb)));
          }
          for (int c = clo; c < chi; ++c) {
            warp_window(g, cst[s * S2 + c], cst[s * S2 + c + 1], oqx - tb, oqx + tb, wl, wh);
            pairs += (unsigned long long)(wh > wl ? wh - wl : 0);
            oscan(wl, wh);
          }
        } else {
          warp_window(g, sst[s], sst[s + 1], oqx - tb, oqx + tb, wl, wh);
          pairs += (unsigned long long)(wh > wl ? wh - wl : 0);
          oscan(wl, wh);
        }
      }
      if constexpr (COUNT) {
        const int add = __reduce_add_sync(0xffffffffu, cnt2);
        if (lane == ol) cntq += add;
      } else {
        if (lane == ol) {
#pragma unroll
          for (int s2 = 0; s2 < KMAX; ++s2)
            if (s2 >= KMAX - K && top[s2] < top2[KMAX - 1]) insert_sorted<KMAX>(top2, top[s2]);
        }
        const uint64_t kth = warp_kth_of_lists<KMAX, uint64_t>(top2, K, INF_BITS);
        if (lane == ol) top[KMAX - 1] = kth;
      }
    }

    if (exists) {
      if constexpr (COUNT) J->cnt[J->idxg[qp]] = qok ? cntq : 0;
      else J->eps[J->idxg[qp]] = bits_to_double(top[KMAX - 1]);
    }
    if (lane == 0) atomicAdd(J->stats + 0, pairs);
  }
}

// d >= 3 (D != 2) runs on nested grids.
template <int D, int KMAX, bool COUNT>
void launch_wgrid_t(const JobDev* jobs, const WorkItem* items, int nitems, int* counter, int dmax,
                    int num_sms, cudaStream_t st) {
  auto kern = wgrid_kernel<D, KMAX, COUNT, D != 2>;
  int per_sm = 1;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, WG_WARPS * 32, 0);
  if (per_sm < 1) per_sm = 1;
  int grid = num_sms * per_sm;
  const int need = (nitems + WG_WARPS - 1) / WG_WARPS;
  if (grid > need) grid = need;
  if (grid < 1) return;
  kern<<<grid, WG_WARPS * 32, 0, st>>>(jobs, items, nitems, counter, dmax);
  count_launch();
}

struct WgridDispatch {
  template <int D>
  static void knn_d(int kclass, const JobDev* jobs, const WorkItem* items, int nitems, int* ctr,
                    int dmax, int sms, cudaStream_t st) {
    if (kclass <= 4) launch_wgrid_t<D, 4, false>(jobs, items, nitems, ctr, dmax, sms, st);
    else launch_wgrid_t<D, 8, false>(jobs, items, nitems, ctr, dmax, sms, st);
  }
  static void knn(int kclass, int dclass, const JobDev* jobs, const WorkItem* items, int nitems,
                  int* ctr, int dmax, int sms, cudaStream_t st) {
    switch (dclass) {
      case 2: knn_d<2>(kclass, jobs, items, nitems, ctr, dmax, sms, st); break;
      case 3: knn_d<3>(kclass, jobs, items, nitems, ctr, dmax, sms, st); break;
      case 4: knn_d<4>(kclass, jobs, items, nitems, ctr, dmax, sms, st); break;
      default: knn_d<0>(kclass, jobs, items, nitems, ctr, dmax, sms, st); break;
    }
  }
  static void count(int dclass, const JobDev* jobs, const WorkItem* items, int nitems, int* ctr,
                    int dmax, int sms, cudaStream_t st) {
    switch (dclass) {
      case 2: launch_wgrid_t<2, 4, true>(jobs, items, nitems, ctr, dmax, sms, st); break;
      case 3: launch_wgrid_t<3, 4, true>(jobs, items, nitems, ctr, dmax, sms, st); break;
      case 4: launch_wgrid_t<4, 4, true>(jobs, items, nitems, ctr, dmax, sms, st); break;
      default: launch_wgrid_t<0, 4, true>(jobs, items, nitems, ctr, dmax, sms, st); break;
    }
  }
};

}  // namespace wgrid_detail
}  // namespace egb
