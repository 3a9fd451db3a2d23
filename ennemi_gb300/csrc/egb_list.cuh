// egb_list.cuh -- a query's candidate list, kept by one warp.
//
// The K nearest candidates of one query by FP32 distance, and every other one
// within the screen bound, in shared memory; the exact K-th distance from them
// (egb_wlist.cu has the argument).  All calls are warp-uniform.
#pragma once
#include "egb_wgrid.cuh"

namespace egb {
namespace list_detail {

using wgrid_detail::dn_band32;
using wgrid_detail::plan_margin;
using wgrid_detail::up_band32;

constexpr unsigned FULL = 0xffffffffu;

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

struct Entry {
  float d;
  int j;
};
template <int R>
struct CandidateList {
  static constexpr int CAP = 32 * R;
  static constexpr int WORDS = 2 * CAP;  // 32-bit words of shared memory (an ExactList's too)
  Entry* list;
  int K;
  float mq;    // >= max_c |q_c - c|
  float thr;   // screen bound S: candidates beyond it are not listed
  float tb;    // planning bound plan_margin(U)
  int cnt;
  bool over;   // more near ties than the list holds

  __device__ __forceinline__ CandidateList(uint32_t* store, int K_, float mq_)
      : list(reinterpret_cast<Entry*>(store)), K(K_), mq(mq_), thr(__builtin_huge_valf()),
        tb(__builtin_huge_valf()), cnt(0), over(false) {}

  // New bounds from the K-th smallest of at least K entries; entries beyond
  // them leave.
  __device__ __forceinline__ void tighten() {
    const int lane = threadIdx.x & 31;
    __syncwarp();
    uint32_t v[R];
    int ix[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const bool in = r * 32 + lane < cnt;
      const Entry e = in ? list[r * 32 + lane] : Entry{__builtin_huge_valf(), 0};
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
      if (keep) list[kept + __popc(m & ((1u << lane) - 1u))] = Entry{__uint_as_float(v[r]), ix[r]};
      kept += __popc(m);
    }
    cnt = kept;
    over = over || cnt > CAP - 32;
    __syncwarp();
  }

  // One candidate per lane: j at FP32 distance dd (+inf: none).
  __device__ __forceinline__ void push(float dd, int j) {
    const int lane = threadIdx.x & 31;
    const bool hit = dd <= thr && dd < __builtin_huge_valf();
    const uint32_t m = __ballot_sync(FULL, hit);
    if (m) {
      if (hit) list[cnt + __popc(m & ((1u << lane) - 1u))] = Entry{dd, j};
      cnt += __popc(m);
      if (cnt > CAP - 32) tighten();
    }
  }

  // The exact K-th distance (bits), +inf if fewer than K candidates; exact(j):
  // the FP64 distance of candidate j.
  template <typename F>
  __device__ __forceinline__ uint64_t kth(F&& exact) {
    const int lane = threadIdx.x & 31;
    uint64_t res = INF_BITS;
    __syncwarp();
    if (cnt >= K) {
      float v[R];
      int ix[R];
      uint32_t vb[R];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const bool in = r * 32 + lane < cnt;
        const Entry e = in ? list[r * 32 + lane] : Entry{__builtin_huge_valf(), 0};
        v[r] = e.d;
        vb[r] = __float_as_uint(e.d);
        ix[r] = e.j;
      }
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
        if (v[r] < __builtin_huge_valf() && !(up_band32(v[r], mq) < lo) && !(dn_band32(v[r], mq) > hi))
          e[r] = exact(ix[r]);
      for (;;) {  // the rank-th smallest of e (ties leave together)
        uint64_t m = ~0ull;
#pragma unroll
        for (int r = 0; r < R; ++r) m = e[r] < m ? e[r] : m;
        m = warp_min64(m);
        int c = 0;
#pragma unroll
        for (int r = 0; r < R; ++r) c += __popc(__ballot_sync(FULL, e[r] == m));
        if (c >= rank || m == ~0ull) {
          res = m;
          break;
        }
        rank -= c;
#pragma unroll
        for (int r = 0; r < R; ++r) e[r] = e[r] == m ? ~0ull : e[r];
      }
    }
    __syncwarp();
    return res;
  }
};

// The K smallest of a sequence of exact distances (FP64 bits), kept by one warp:
// for queries whose near ties a CandidateList cannot hold.  Ties need no room
// here: of the distances equal to the K-th, only as many as make K are kept.
// (A radix select, used before, took eight sweeps of FP64 distances.)
template <int R>
struct ExactList {
  static constexpr int CAP = 32 * R;
  uint64_t* list;
  int K;
  int cnt;
  uint64_t bound;  // the K-th of the distances seen at the last tightening

  __device__ __forceinline__ ExactList(uint32_t* store, int K_)
      : list(reinterpret_cast<uint64_t*>(store)), K(K_), cnt(0), bound(~0ull) {}

  // The K-th smallest of the cnt >= K entries v (unused slots ~0).
  __device__ __forceinline__ uint64_t select(const uint64_t (&v)[R]) const {
    uint32_t w[R];
#pragma unroll
    for (int r = 0; r < R; ++r) w[r] = (uint32_t)(v[r] >> 32);
    const uint32_t h = kth_bits<R>(w, K);
    int below = 0;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      below += __popc(__ballot_sync(FULL, w[r] < h));
      w[r] = w[r] == h ? (uint32_t)v[r] : 0xffffffffu;
    }
    return (uint64_t)h << 32 | kth_bits<R>(w, K - below);
  }

  __device__ __forceinline__ void load(uint64_t (&v)[R]) const {
    const int lane = threadIdx.x & 31;
    __syncwarp();
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = r * 32 + lane < cnt ? list[r * 32 + lane] : ~0ull;
    __syncwarp();
  }

  // One distance per lane (~0: none); true if the bound was renewed.
  __device__ __forceinline__ bool push(uint64_t e) {
    const int lane = threadIdx.x & 31;
    const uint32_t lt = (1u << lane) - 1u;
    const uint32_t m = __ballot_sync(FULL, e < bound);
    if (!m) return false;
    if (e < bound) list[cnt + __popc(m & lt)] = e;
    cnt += __popc(m);
    if (cnt <= CAP - 32) return false;
    uint64_t v[R];
    load(v);
    bound = select(v);
    int kept = 0;  // those below the K-th, then copies of it
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const uint32_t k = __ballot_sync(FULL, v[r] < bound);
      if (v[r] < bound) list[kept + __popc(k & lt)] = v[r];
      kept += __popc(k);
    }
    for (int i = kept + lane; i < K; i += 32) list[i] = bound;
    cnt = K;
    return true;
  }

  // The K-th smallest of all, ~0 if there were fewer.
  __device__ __forceinline__ uint64_t kth() const {
    uint64_t res = ~0ull;
    if (cnt >= K) {
      uint64_t v[R];
      load(v);
      res = select(v);
    }
    __syncwarp();
    return res;
  }
};

}  // namespace list_detail
}  // namespace egb
