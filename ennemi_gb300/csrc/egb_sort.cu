// egb_sort.cu -- batched segmented LSD radix sort of FP64 columns, and the
// 1-D estimator kernels that run on the sorted arrays.
//
// Sort.  Every requested (task, column, segment) is one segment of a single
// concatenated key array.  Keys are the order-preserving uint64 image of the
// FP64 value (key_of), the payload is the working index of the point.  The
// batch sort takes stable 8-bit single-sweep LSD passes over the high 48 key
// bits and repairs the rare runs tied there (below), for large batches only
// over what the sort of 32-bit codes leaves (egb_codesort.cu), whose passes
// also order the strip keys of the grid layouts.
//
// 1-D kNN (entropy of one column, Ross MI with 1-D x): for the point at
// sorted position p the (k+1)-th smallest |x_j - x_p| (self included) is
// found by merging outward from p -- the exact FP64 distances, as cKDTree.
//
// 1-D counts (marginal spaces of KSG / CMI): #{j : fl64(|x_j - q|) <= r},
// r = fl64(eps - 1e-12).  fl64(s_j - q) is monotone in s_j (rounding is
// monotone), so on each side of q the predicate holds on one contiguous run
// of sorted positions -- one key range (ball_keys), whose ends are found
// through the segment's samples (egb_search.cuh).
#include <algorithm>

#include "egb_internal.cuh"
#include "egb_search.cuh"
#include "egb_sweep.cuh"

namespace egb {

namespace {

constexpr int SORT_THREADS = 256;
constexpr int SORTED_THREADS = SORTED_BLOCK;

// ------------------------------------------------------- single sweep --
// The batch sort proper: stable 8-bit LSD passes, one launch each,
// after Adinets and Merrill's single-sweep radix sort (Onesweep, 2022).  The
// load kernel computes the digit totals of all the passes per segment at
// once; each pass then needs, per tile and digit, only the count of that
// digit in the segment's earlier tiles.  A tile takes its id from an atomic
// counter (so every earlier tile of its segment has started), publishes its
// own digit counts at once, and looks back over its predecessors' published
// words -- aggregates or inclusive prefixes -- until it meets an inclusive
// one; it then publishes its own inclusive prefix and scatters.  A flag word
// holds the pass + 1 (bits 56-63; other passes' words read as "not yet"),
// an inclusive bit (55) and the count (bits 0-31), and is written and read
// whole, so no other data needs ordering.  Every wait is bounded: past
// OS_SPIN_LIMIT polls the tile records DERR_WAIT_TIMEOUT (the batch then
// reports EGB_ERR_DEVICE) and goes on.
//
// redo (else null): the kernels run after the code sort (egb_codesort.cu), for
// the segments marked REDO_DIGITS there alone -- usually none, so a launch has few blocks
// and each takes many tiles.
__global__ void __launch_bounds__(SORT_THREADS)
onesweep_load_kernel(const BatchCol* __restrict__ slots, const SortSeg* __restrict__ segs,
                     const int32_t* __restrict__ blk_seg, int nblk, uint64_t* __restrict__ keys,
                     int32_t* __restrict__ vals, uint32_t* __restrict__ seg_hist, int first,
                     const uint32_t* __restrict__ redo, int nseg) {
  __shared__ uint32_t h[OS_PASSES * 256];
  if (redo && !(redo[nseg] & REDO_DIGITS)) return;
  for (int b = blockIdx.x; b < nblk; b += gridDim.x) {
    const int si = blk_seg[b];
    if (redo && !(redo[si] & REDO_DIGITS)) continue;
    const SortSeg s = segs[si];
    for (int i = threadIdx.x; i < OS_PASSES * 256; i += SORT_THREADS) h[i] = 0;
    __syncthreads();
    const uint64_t* __restrict__ x = reinterpret_cast<const uint64_t*>(slots[s.slot].x + s.src_begin);
    const int i0 = (b - s.blk0) * SORT_TILE;
    const int i1 = min(i0 + SORT_TILE, s.len);
    for (int i = i0 + threadIdx.x; i < i1; i += SORT_THREADS) {
      const uint64_t k = key_of_bits(x[i]);
      keys[s.out_base + i] = k;
      vals[s.out_base + i] = s.src_begin + i;
#pragma unroll
      for (int p = 0; p < OS_PASSES; ++p)
        if (p >= first) atomicAdd(&h[p * 256 + (uint32_t)((k >> (8 * p)) & 255u)], 1u);
    }
    __syncthreads();
    uint32_t* g = seg_hist + (size_t)si * ALL_PASSES * 256;
    for (int i = threadIdx.x; i < OS_PASSES * 256; i += SORT_THREADS)
      if (h[i]) atomicAdd(g + i, h[i]);
    __syncthreads();
  }
}

// A pass tile is TILE keys on OS_THREADS threads (four or eight keys a thread);
// its staging arrays exceed the 48 KB of static shared memory.
constexpr int OS_THREADS = 512;
constexpr int OS_NW = OS_THREADS / 32;
template <int TILE>
struct OsSmem {
  uint32_t wcnt[OS_NW][256];  // per-warp digit counts, then offsets
  uint32_t dstart[256];       // first tile slot of each digit
  uint32_t gbase[256];        // first output position of each digit
  uint32_t ws[8];             // digit-scan scratch
  int tile;
  uint64_t sk[TILE];
  int32_t sv[TILE];
};

// LOOK tiles at once shorten the passes of a sort with a tile per SM at most
// (six over 400,000 keys: 74 us, 82 with one).  A larger one looks back one at a time,
// which fits in 64 registers, and hides that behind a second block an SM:
// eight passes over 18 million keys 1.32 ms, with 110 registers and one block 1.98.
// REDO: after the code sort, a block takes tiles until none is left.
template <int TILE, int LOOK, bool REDO>
__global__ void __launch_bounds__(OS_THREADS, LOOK > 1 && TILE == OS_TILE ? 1 : 2)
onesweep_pass_kernel(const SortSeg* __restrict__ segs, const int32_t* __restrict__ os_blk_seg, int nblk,
                     const uint64_t* __restrict__ kin, const int32_t* __restrict__ vin,
                     uint64_t* __restrict__ kout, int32_t* __restrict__ vout, int pass,
                     const uint32_t* __restrict__ seg_hist, unsigned long long* flags,
                     int* tile_counter, uint32_t* err, const uint32_t* __restrict__ redo, int nseg) {
  constexpr int CH = TILE / OS_NW;  // keys per warp
  constexpr int R = CH / 32;           // rounds per warp
  static_assert(TILE % OS_NW == 0 && CH % 32 == 0, "whole warp rounds");
  extern __shared__ __align__(16) unsigned char os_raw[];
  OsSmem<TILE>& S = *reinterpret_cast<OsSmem<TILE>*>(os_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (REDO && !(redo[nseg] & REDO_DIGITS)) return;
  do {
    if (tid == 0) S.tile = atomicAdd(tile_counter, 1);
    for (int i = tid; i < OS_NW * 256; i += OS_THREADS) (&S.wcnt[0][0])[i] = 0u;
    __syncthreads();
    const int b = S.tile;
    if (REDO && b >= nblk) break;
    const int si = os_blk_seg[b];
    if constexpr (REDO) {
      __syncthreads();  // S.tile is read before the next tile's id lands
      if (!(redo[si] & REDO_DIGITS)) continue;
    }
    const SortSeg s = segs[si];
    const int lb = b - s.os_blk0;
    const int shift = 8 * pass;
    const int i0 = lb * TILE;
    const int n = min(TILE, s.len - i0);
    const uint32_t lt = (1u << lane) - 1u;
    uint64_t key[R];
    int32_t val[R];
    uint32_t dg[R], rk[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int t = warp * CH + r * 32 + lane;
      const bool valid = t < n;
      key[r] = valid ? kin[s.out_base + i0 + t] : 0ull;
      val[r] = valid ? vin[s.out_base + i0 + t] : 0;
      const uint32_t d = valid ? (uint32_t)(key[r] >> shift) & 255u : 256u + lane;
      dg[r] = d;
      uint32_t peers = 0xffffffffu;  // lanes with the same 9-bit digit
#pragma unroll
      for (int bit = 0; bit < 9; ++bit) {
        const uint32_t bb = __ballot_sync(0xffffffffu, (d >> bit) & 1u);
        peers &= ((d >> bit) & 1u) ? bb : ~bb;
      }
      const uint32_t before = valid ? S.wcnt[warp][d] : 0u;
      __syncwarp();
      if (valid && (peers & lt) == 0) S.wcnt[warp][d] = before + __popc(peers);
      __syncwarp();
      rk[r] = before + __popc(peers & lt);
    }
    __syncthreads();
    uint32_t cnt = 0;  // digit tid: offsets of the warps, then its count in the tile
    if (tid < 256) {
#pragma unroll
      for (int w = 0; w < OS_NW; ++w) {
        const uint32_t c = S.wcnt[w][tid];
        S.wcnt[w][tid] = cnt;
        cnt += c;
      }
    }
    // publish this tile's count of digit tid, then look back for the count of
    // digit tid in the segment's earlier tiles
    const uint32_t excl = tid < 256 ? sweep_look_back<LOOK>(flags, b, s.os_blk0, tid, pass, cnt, err) : 0u;
    // digit tid of the whole segment starts after the smaller digits
    const uint32_t seg_tot = tid < 256 ? seg_hist[((size_t)si * ALL_PASSES + pass) * 256 + tid] : 0u;
    const uint32_t seg_off = digit_excl_scan(seg_tot, S.ws);
    const uint32_t ds = digit_excl_scan(cnt, S.ws);
    if (tid < 256) {
      S.gbase[tid] = seg_off + excl;
      S.dstart[tid] = ds;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int t = warp * CH + r * 32 + lane;
      if (t < n) {
        const uint32_t d = dg[r];
        const uint32_t slot = S.dstart[d] + S.wcnt[warp][d] + rk[r];
        S.sk[slot] = key[r];
        S.sv[slot] = val[r];
      }
    }
    __syncthreads();
    for (int t = tid; t < n; t += OS_THREADS) {
      const uint64_t k = S.sk[t];
      const uint32_t d = (uint32_t)(k >> shift) & 255u;
      const uint32_t pos = S.gbase[d] + ((uint32_t)t - S.dstart[d]);
      if (pos < (uint32_t)s.len) {
        kout[s.out_base + pos] = k;
        vout[s.out_base + pos] = S.sv[t];
      } else {
        atomicOr(err, DERR_BAD_INDEX);
      }
    }
    if (REDO) __syncthreads();
  } while (REDO);
}

// ----------------------------------------------------------- tie repair --
// After the passes over digits 2..7 the keys of a segment are ordered by
// their high 48 bits (sign, exponent and 36 mantissa bits of the value),
// stably.  Keys equal there but not in the low 16 bits -- values within a
// relative 2^-36 of each other -- are rare, and sit in short runs: the first
// thread of a run of at most TIE_RUN keys sorts it by the whole key with an
// insertion sort (stable, so equal keys keep their input order and the
// result is the permutation of the eight-pass sort).  A longer run that is
// out of order is not repaired: its threads set DERR_SORT_TIES and the host
// runs the batch again with all eight passes.  Repairs permute keys only
// within runs, so the high bits read at any position never change while the
// kernel runs: run boundaries are read race-free.
//
// What follows in such a batch is thrown away, and a search relies on the order:
// walks over columns that are not in order ran 70 ms for a pair of 200,000 whole
// numbers, against 1.0 ms in the run that counts.  So the first thread to
// report moves the work counters of all the searches past their last items, and
// they end at once.
constexpr int TIE_RUN = 32;
constexpr int NO_ITEMS = 1 << 30;

__global__ void __launch_bounds__(SORT_THREADS)
tie_fix_kernel(const SortSeg* __restrict__ segs, const int32_t* __restrict__ blk_seg, int nblk,
               uint64_t* keys_all, int32_t* vals_all, uint32_t* __restrict__ err,
               int* __restrict__ counters, int ncounters, const uint32_t* __restrict__ redo, int nseg) {
  if (redo && !redo[nseg]) return;
  for (int b = blockIdx.x; b < nblk; b += gridDim.x) {
    const int si = blk_seg[b];
    if (redo && !redo[si]) continue;
    const SortSeg sg = segs[si];
    const int len = sg.len;
    const int i0 = (b - sg.blk0) * SORT_TILE;
    const int i1 = min(i0 + SORT_TILE, len);
    uint64_t* keys = keys_all + sg.out_base;  // written by run owners: no __restrict__
    int32_t* vals = vals_all + sg.out_base;
    for (int q = i0 + (int)threadIdx.x; q < i1; q += SORT_THREADS) {
      const uint64_t k = keys[q];
      const uint64_t hi = k >> 16;
      const bool starts = q == 0 || (keys[q - 1] >> 16) != hi;
      if (!starts) {
        // inside a run: out of order against the previous key and the run
        // too long to be repaired -> the batch needs the full sort
        if (k < keys[q - 1]) {
          int s = q - 1, e = q + 1;
          while (s > 0 && (keys[s - 1] >> 16) == hi && q - s <= TIE_RUN) --s;
          while (e < len && (keys[e] >> 16) == hi && e - s <= TIE_RUN) ++e;
          if (e - s > TIE_RUN && !(atomicOr(err, (uint32_t)DERR_SORT_TIES) & DERR_SORT_TIES))
            for (int c = 0; c < ncounters; c += 2) counters[c] = NO_ITEMS;
        }
        continue;
      }
      if (q + 1 >= len || (keys[q + 1] >> 16) != hi) continue;  // a run of one
      int e = q + 1;
      while (e < len && (keys[e] >> 16) == hi && e - q <= TIE_RUN) ++e;
      if (e - q > TIE_RUN) continue;
      for (int i = q + 1; i < e; ++i) {  // stable insertion sort of [q, e)
        const uint64_t ki = keys[i];
        if (ki >= keys[i - 1]) continue;
        const int32_t vi = vals[i];
        int j = i;
        while (j > q && keys[j - 1] > ki) {
          keys[j] = keys[j - 1];
          vals[j] = vals[j - 1];
          --j;
        }
        keys[j] = ki;
        vals[j] = vi;
      }
    }
  }
}

// --------------------------------------------------------- sorted jobs ----
// the job of this block: last j with jobs[j].blk0 <= blockIdx.x
__device__ __forceinline__ int sorted_job_of(const SortedJob* __restrict__ jobs, int njobs) {
  int lo = 0, hi = njobs;
  while (hi - lo > 1) {
    const int m = (lo + hi) >> 1;
    if (jobs[m].blk0 <= (int)blockIdx.x) lo = m; else hi = m;
  }
  return lo;
}

// 1-D kNN distances: one thread per sorted position.
__global__ void sorted_jobs_kernel(const TaskDev* __restrict__ tasks,
                                   const SortedJob* __restrict__ jobs, int njobs,
                                   const KeyIndex kx, const int32_t* __restrict__ perm_all) {
  const SortedJob jb = jobs[sorted_job_of(jobs, njobs)];
  const int64_t p = (int64_t)((int)blockIdx.x - jb.blk0) * SORTED_THREADS + threadIdx.x;
  const int64_t len = jb.len;
  if (p >= len) return;
  const uint64_t* __restrict__ keys = kx.keys + jb.base;
  const double q = value_of(keys[p]);
  const double INF = __longlong_as_double((long long)INF_BITS);
  // (k+1)-NN distance, self included; +inf if too few
  int64_t L = p - 1, R = p + 1;
  double d = (jb.K <= len) ? 0.0 : INF;
  if (jb.K <= len) {
    for (int s = 1; s < jb.K; ++s) {
      const double dl = L >= 0 ? q - value_of(keys[L]) : INF;
      const double dr = R < len ? value_of(keys[R]) - q : INF;
      if (dl <= dr) { d = dl; --L; } else { d = dr; ++R; }
    }
  }
  tasks[jb.task].eps[perm_all[jb.base + p]] = d;
}

// 1-D ball counts.  A block takes BALL_SPAN consecutive sorted
// positions and searches the ends of their balls in the FP32 values of those
// positions and BALL_HALF to either side, held in shared memory (21 KB).
//
// Bound by the latency of the search (12 dependent shared loads, both ends at
// once) and of the two gathers by working index (radius in, count out), with
// the L1 pipe about half busy, so what counts is warps in flight: 32
// registers, 8 blocks an SM.  784 jobs of 180,000 points: 11.5 ms with
// galloping searches over global samples, one position per thread; 8.1 ms
// from the window at 5 or 6 blocks an SM; 6.5 ms at 8.  2016 pairs of 50,000:
// 7.8 -> 4.3 ms.  BALL_HALF: with 4096 five or six blocks fit (8.1 / 5.4 ms);
// with 1024 too many ends fall outside (10.5 / 6.3 ms at 5 blocks against 8.7
// / 5.6).  Blocks of 512 threads: 7.6 / 5.2 ms.
constexpr int BALL_THREADS = 256;
constexpr int BALL_HALF = 2048;
template <int PER>
__global__ void __launch_bounds__(BALL_THREADS, 8)
ball_jobs_kernel(const TaskDev* __restrict__ tasks, const SortedJob* __restrict__ jobs, int njobs,
                 const KeyIndex kx, const int32_t* __restrict__ perm_all) {
  constexpr int SPAN = BALL_THREADS * PER;
  constexpr int WIN = SPAN + 2 * BALL_HALF + 4;
  __shared__ __align__(16) float win[WIN];
  const SortedJob& jb = jobs[sorted_job_of(jobs, njobs)];
  const int64_t base = jb.base;
  const int len = jb.len;
  const int p0 = ((int)blockIdx.x - jb.blk0) * SPAN;
  const TaskDev& t = tasks[jb.task];

  int32_t idx[PER];
  double rad[PER];
#pragma unroll
  for (int s = 0; s < PER; ++s) {
    const int p = p0 + s * BALL_THREADS + (int)threadIdx.x;
    idx[s] = p < len ? __ldg(perm_all + base + p) : -1;
  }
  // the window of FP32 keys, from a position whose address is 16-byte aligned
  const int off = (int)(base & 3);
  const int w0 = p0 - BALL_HALF - off;
  const float* fk = kx.fkeys + base;
  for (int j = (int)threadIdx.x; j < WIN / 4; j += BALL_THREADS) {
    const int g = w0 + 4 * j;
    float4 v;
    if (g >= 0 && g + 4 <= len) {
      v = __ldg((const float4*)(fk + g));
    } else {
      const float INF = __int_as_float(0x7f800000);
      auto at = [&](int p) { return p < 0 ? -INF : p < len ? __ldg(fk + p) : INF; };
      v = make_float4(at(g), at(g + 1), at(g + 2), at(g + 3));
    }
    *(float4*)(win + 4 * j) = v;
  }
#pragma unroll
  for (int s = 0; s < PER; ++s) rad[s] = idx[s] >= 0 ? radius_of(t.rad, t.rad_given, idx[s]) : 0.0;
  __syncthreads();

  const SegView v = seg_view(kx, base, jb.s1_base, jb.s2_base, len);
  int32_t* __restrict__ cnt = t.cnt[jb.slot];
  int2* __restrict__ ranges = jb.ranges;
#pragma unroll
  for (int s = 0; s < PER; ++s) {
    if (idx[s] < 0) break;
    const int at = off + BALL_HALF + s * BALL_THREADS + (int)threadIdx.x;
    const int p = w0 + at;
    const int rc = radius_class(rad[s]);
    int32_t count;
    if (rc == 0) {
      count = 0;
    } else if (rc == 2) {
      count = len;
    } else {
      int lo, hi;
      ball_positions_at<BALL_HALF>(v, win, at, p, rad[s], lo, hi);
      count = hi - lo;
      if (ranges) ranges[idx[s]] = make_int2(lo, hi);
    }
    cnt[idx[s]] = count;
  }
}

// ----------------------------------------------------------- grid keys ----
// inv[out + (w_B - seg_begin)] = p_B for the column-1 order of each grid job.
__global__ void grid_inv_kernel(const JobDev* __restrict__ jobs,
                                const int32_t* __restrict__ grid_jobs, int ngrid,
                                const SortSeg* __restrict__ gsegs,
                                const int32_t* __restrict__ sorted_vals,
                                const SortSeg* __restrict__ segs, int32_t* __restrict__ inv) {
  for (int g = blockIdx.y; g < ngrid; g += gridDim.y) {
    const JobDev& J = jobs[grid_jobs[g]];
    const int64_t out = gsegs[J.gseg].out_base;
    const int32_t* vb = sorted_vals + segs[J.sort_seg_b].out_base;
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < J.len;
         p += (int64_t)gridDim.x * blockDim.x)
      inv[out + (vb[p] - J.seg_begin)] = (int32_t)p;
  }
}

// Points per value of the digit threadIdx.x (256 threads), for keys that are
// positions in a table of count + 1 starts.
__device__ __forceinline__ uint32_t low_digit_total(const int32_t* __restrict__ starts, int count) {
  uint32_t n = 0;
  for (int k = (int)threadIdx.x; k < count; k += 256) n += (uint32_t)(starts[k + 1] - starts[k]);
  return n;
}
__device__ __forceinline__ uint32_t high_digit_total(const int32_t* __restrict__ starts, int count) {
  const int k = 256 * (int)threadIdx.x;
  return (uint32_t)(starts[min(k + 256, count)] - starts[min(k, count)]);
}

// words[out + i] = (label, i), with the digit totals from the class sizes.
__global__ void __launch_bounds__(256)
label_word_kernel(const LabelJob* __restrict__ jobs, int njobs, uint64_t* __restrict__ words,
                  uint32_t* __restrict__ seg_hist) {
  for (int g = blockIdx.y; g < njobs; g += gridDim.y) {
    const LabelJob& J = jobs[g];
    if (blockIdx.x == 0) {
      uint32_t* h = seg_hist + ((size_t)g * ALL_PASSES + GRID_PASS) * 256 + threadIdx.x;
      h[0] = low_digit_total(J.starts, J.nclass);
      h[256] = high_digit_total(J.starts, J.nclass);
    }
    const int32_t* __restrict__ labels = J.labels;
    uint64_t* __restrict__ out = words + J.out_base;
    for (int i = blockIdx.x * 256 + threadIdx.x; i < J.n; i += gridDim.x * 256)
      out[i] = (uint64_t)(uint32_t)labels[i] << 32 | (uint32_t)i;
  }
}
__global__ void __launch_bounds__(256)
label_perm_kernel(const LabelJob* __restrict__ jobs, int njobs, const uint64_t* __restrict__ words) {
  for (int g = blockIdx.y; g < njobs; g += gridDim.y) {
    const LabelJob& J = jobs[g];
    for (int i = blockIdx.x * 256 + threadIdx.x; i < J.n; i += gridDim.x * 256)
      J.perm[i] = (int32_t)(uint32_t)words[J.out_base + i];
  }
}

// words[out + p_A] = cell key of the point at column-0 position p_A, and p_A.
// The first block of a job writes its digit totals: the sizes of the cells.
__global__ void __launch_bounds__(256)
grid_key_kernel(const JobDev* __restrict__ jobs, const int32_t* __restrict__ grid_jobs, int ngrid,
                const SortSeg* __restrict__ gsegs, const int32_t* __restrict__ sorted_vals,
                const SortSeg* __restrict__ segs, const int32_t* __restrict__ inv,
                const int32_t* __restrict__ sub, uint64_t* __restrict__ words,
                uint32_t* __restrict__ seg_hist) {
  for (int g = blockIdx.y; g < ngrid; g += gridDim.y) {
    const JobDev& J = jobs[grid_jobs[g]];
    const int64_t out = gsegs[J.gseg].out_base;
    const int32_t* va = sorted_vals + segs[J.sort_seg].out_base;
    const int64_t len = J.len;
    const int nsub = J.nsub;
    if (blockIdx.x == 0) {
      const int32_t* starts = nsub > 0 ? J.cstart : J.sstart;
      const int count = nsub > 0 ? J.nstrips * nsub : J.nstrips;
      uint32_t* h = seg_hist + ((size_t)J.gseg * ALL_PASSES + GRID_PASS) * 256 + threadIdx.x;
      h[0] = low_digit_total(starts, count);
      h[256] = high_digit_total(starts, count);
    }
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < len;
         p += (int64_t)gridDim.x * blockDim.x) {
      const int64_t w = va[p] - J.seg_begin;
      const int64_t strip = (int64_t)inv[out + w] * J.nstrips / len;
      words[out + p] = (uint64_t)(nsub > 0 ? strip * nsub + sub[out + w] : strip) << 32 | (uint32_t)p;
    }
  }
}

// words[out + r] = strip of the point at column-2 position r, and its offset.
__global__ void __launch_bounds__(256)
nest_key_kernel(const JobDev* __restrict__ jobs, const int32_t* __restrict__ grid_jobs, int ngrid,
                const SortSeg* __restrict__ gsegs, const int32_t* __restrict__ sorted_vals,
                const SortSeg* __restrict__ segs, const int32_t* __restrict__ inv,
                uint64_t* __restrict__ words, uint32_t* __restrict__ seg_hist) {
  for (int g = blockIdx.y; g < ngrid; g += gridDim.y) {
    const JobDev& J = jobs[grid_jobs[g]];
    const int64_t out = gsegs[J.gseg].out_base;
    const int64_t len = J.len;
    const bool nested = J.nsub > 0;
    const int32_t* vc = nested ? sorted_vals + segs[J.sort_seg_c].out_base : nullptr;
    if (blockIdx.x == 0)
      seg_hist[((size_t)J.gseg * ALL_PASSES + NEST_PASS) * 256 + threadIdx.x] =
          nested ? low_digit_total(J.sstart, J.nstrips) : threadIdx.x == 0 ? (uint32_t)len : 0u;
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < len;
         r += (int64_t)gridDim.x * blockDim.x) {
      const int32_t w = nested ? vc[r] - J.seg_begin : (int32_t)r;
      const uint64_t strip = nested ? (uint64_t)((int64_t)inv[out + w] * J.nstrips / len) : 0u;
      words[out + r] = strip << 32 | (uint32_t)w;
    }
  }
}

// After the strip pass over the column-2 order: position p2 of strip s1
// holds within-strip column-2 rank p2 - sstart[s1].
__global__ void nest_sub_kernel(const TaskDev* __restrict__ tasks,
                                const JobDev* __restrict__ jobs,
                                const int32_t* __restrict__ grid_jobs, int ngrid,
                                const SortSeg* __restrict__ gsegs,
                                const uint64_t* __restrict__ words, int32_t* __restrict__ sub) {
  for (int g = blockIdx.y; g < ngrid; g += gridDim.y) {
    const JobDev& J = jobs[grid_jobs[g]];
    if (J.nsub <= 0) continue;
    const TaskDev& t = tasks[J.task];
    const int64_t out = gsegs[J.gseg].out_base;
    const int nsub = J.nsub;
    const double* z = t.col[J.sp.cols[2]] + J.seg_begin;
    for (int64_t p2 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p2 < J.len;
         p2 += (int64_t)gridDim.x * blockDim.x) {
      const uint64_t word = words[out + p2];
      const int s1 = (int)(word >> 32);
      const int32_t w = (int32_t)(uint32_t)word;
      const int32_t s0 = J.sstart[s1];
      const int32_t L = J.sstart[s1 + 1] - s0;
      const int c2 = (int)((p2 - s0) * nsub / L);
      sub[out + w] = c2;
      const int cell = s1 * nsub + c2;
      if (p2 == J.cstart[cell]) {
        J.czlo[cell] = z[w];
        J.czlo32[cell] = __double2float_rd(__dsub_rd(z[w], J.center[2]));
      }
      if (p2 == J.cstart[cell + 1] - 1) {
        J.czhi[cell] = z[w];
        J.czhi32[cell] = __double2float_ru(__dsub_ru(z[w], J.center[2]));
      }
    }
  }
}

dim3 grid_of(int ngrid, int64_t max_len) {
  int gx = (int)((max_len + 255) / 256);
  if (gx > 1024) gx = 1024;
  if (gx < 1) gx = 1;
  return dim3(gx, ngrid > 65535 ? 65535 : ngrid);
}

}  // namespace

void launch_grid_inv(const JobDev* jobs_d, const int32_t* grid_jobs_d, int ngrid,
                     const SortSeg* gsegs_d, const int32_t* sorted_vals, const SortSeg* segs_d,
                     int32_t* inv_scratch, int64_t max_len, cudaStream_t st) {
  if (ngrid <= 0) return;
  grid_inv_kernel<<<grid_of(ngrid, max_len), 256, 0, st>>>(jobs_d, grid_jobs_d, ngrid, gsegs_d,
                                                           sorted_vals, segs_d, inv_scratch);
  count_launch();
}

void launch_label_order(const LabelJob* jobs_d, int njobs, int max_classes, int64_t max_n,
                        const SortSeg* segs_d, const int32_t* os_blk_seg_d, int os_nblk, int os_tile,
                        uint64_t* words_a, uint64_t* words_b, const Sweep& w, uint32_t* err, cudaStream_t st) {
  if (njobs <= 0) return;
  label_word_kernel<<<grid_of(njobs, max_n), 256, 0, st>>>(jobs_d, njobs, words_a, w.seg_hist);
  count_launch();
  launch_word_pass(segs_d, os_blk_seg_d, os_nblk, os_tile, words_a, words_b, 0, GRID_PASS, w, err, st);
  uint64_t* sorted = words_b;
  if (max_classes > 256) {
    launch_word_pass(segs_d, os_blk_seg_d, os_nblk, os_tile, words_b, words_a, 1, GRID_PASS + 1, w, err, st);
    sorted = words_a;
  }
  label_perm_kernel<<<grid_of(njobs, max_n), 256, 0, st>>>(jobs_d, njobs, sorted);
  count_launch();
}

void launch_grid_key(const JobDev* jobs_d, const int32_t* grid_jobs_d, int ngrid,
                     const SortSeg* gsegs_d, const int32_t* sorted_vals, const SortSeg* segs_d,
                     const int32_t* inv_scratch, const int32_t* sub, uint64_t* words, const Sweep& w,
                     int64_t max_len, cudaStream_t st) {
  if (ngrid <= 0) return;
  grid_key_kernel<<<grid_of(ngrid, max_len), 256, 0, st>>>(jobs_d, grid_jobs_d, ngrid, gsegs_d, sorted_vals,
                                                           segs_d, inv_scratch, sub, words, w.seg_hist);
  count_launch();
}

void launch_nest_key(const JobDev* jobs_d, const int32_t* grid_jobs_d, int ngrid,
                     const SortSeg* gsegs_d, const int32_t* sorted_vals, const SortSeg* segs_d,
                     const int32_t* inv_scratch, uint64_t* words, const Sweep& w, int64_t max_len,
                     cudaStream_t st) {
  if (ngrid <= 0) return;
  nest_key_kernel<<<grid_of(ngrid, max_len), 256, 0, st>>>(jobs_d, grid_jobs_d, ngrid, gsegs_d, sorted_vals,
                                                           segs_d, inv_scratch, words, w.seg_hist);
  count_launch();
}

void launch_nest_sub(const TaskDev* tasks_d, const JobDev* jobs_d, const int32_t* grid_jobs_d,
                     int ngrid, const SortSeg* gsegs_d, const uint64_t* words, int32_t* sub,
                     int64_t max_len, cudaStream_t st) {
  if (ngrid <= 0) return;
  nest_sub_kernel<<<grid_of(ngrid, max_len), 256, 0, st>>>(tasks_d, jobs_d, grid_jobs_d, ngrid, gsegs_d, words,
                                                           sub);
  count_launch();
}

int init_sort_kernels() {
  int rc = init_code_sort();
  auto allow = [&](auto kernel) {
    if (!rc)
      rc = (int)cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(OsSmem<OS_TILE>));
  };
  allow(onesweep_pass_kernel<OS_TILE, 1, false>);
  allow(onesweep_pass_kernel<OS_TILE, 8, false>);
  allow(onesweep_pass_kernel<OS_TILE, 1, true>);
  return rc;
}

size_t sort_sweep_bytes(int os_nblk, int nseg) { return sweep_layout(nullptr, os_nblk, nseg, nullptr) + 64; }

void launch_sort(const BatchCol* slots_d, const SortSeg* segs_d,
                 const int32_t* blk_seg_d, int nblk, const int32_t* os_blk_seg_d, int os_nblk,
                 int os_tile, int nseg, uint64_t* keys_a, uint64_t* keys_b, int32_t* vals_a, int32_t* vals_b,
                 const KeyIndexOut& ko, void* sweep, int first, bool codes, int num_sms,
                 uint32_t* err, int* counters, int ncounters, cudaStream_t st, cudaEvent_t* pass_events) {
  if (nblk <= 0 || os_nblk <= 0) {
    if (pass_events) cudaEventRecord(pass_events[0], st), cudaEventRecord(pass_events[1], st);
    return;
  }
  Sweep w;
  sweep_layout(sweep, os_nblk, nseg, &w);
  if (codes)
    launch_code_sort(slots_d, segs_d, blk_seg_d, nblk, os_blk_seg_d, os_nblk, nseg, keys_a, keys_b, vals_a, ko, w, num_sms, err,
                     st, pass_events);
  const uint32_t* redo = codes ? w.redo : nullptr;
  const int gl = codes ? std::min(nblk, 8 * num_sms) : nblk;
  const int gp = codes ? std::min(os_nblk, 2 * num_sms) : os_nblk;
  onesweep_load_kernel<<<gl, SORT_THREADS, 0, st>>>(slots_d, segs_d, blk_seg_d, nblk, keys_a, vals_a,
                                                   w.seg_hist, first, redo, nseg);
  count_launch();
  uint64_t* kin = keys_a;
  uint64_t* kout = keys_b;
  int32_t* vin = vals_a;
  int32_t* vout = vals_b;
  if (pass_events && !codes) cudaEventRecord(pass_events[0], st);
  for (int pass = first; pass < OS_PASSES; ++pass) {
    auto run = [&](auto kernel, size_t smem) {
      kernel<<<gp, OS_THREADS, smem, st>>>(segs_d, os_blk_seg_d, os_nblk, kin, vin, kout, vout, pass, w.seg_hist,
                                           w.flags, w.counters + pass, err, redo, nseg);
    };
    if (codes) run(onesweep_pass_kernel<OS_TILE, 1, true>, sizeof(OsSmem<OS_TILE>));
    else if (os_tile != OS_TILE) run(onesweep_pass_kernel<OS_TILE_SMALL, 8, false>, sizeof(OsSmem<OS_TILE_SMALL>));
    else if (os_nblk <= num_sms) run(onesweep_pass_kernel<OS_TILE, 8, false>, sizeof(OsSmem<OS_TILE>));
    else run(onesweep_pass_kernel<OS_TILE, 1, false>, sizeof(OsSmem<OS_TILE>));
    count_launch();
    uint64_t* tk = kin; kin = kout; kout = tk;
    int32_t* tv = vin; vin = vout; vout = tv;
  }
  if (pass_events && !codes) cudaEventRecord(pass_events[1], st);
  // an even number of passes: the sorted keys and values are back in
  // keys_a / vals_a
  if (first > 0) {
    tie_fix_kernel<<<gl, SORT_THREADS, 0, st>>>(segs_d, blk_seg_d, nblk, keys_a, vals_a, err, counters, ncounters, redo,
                                                 nseg);
    count_launch();
  }
  launch_samples(segs_d, blk_seg_d, nblk, gl, keys_a, ko, redo, nseg, st);
}

void launch_sorted_jobs(const TaskDev* tasks_d, const SortedJob* jobs_d, int njobs,
                        int total_blocks, const KeyIndex& kx, const int32_t* perm, cudaStream_t st) {
  if (njobs <= 0 || total_blocks <= 0) return;
  sorted_jobs_kernel<<<(unsigned)total_blocks, SORTED_THREADS, 0, st>>>(tasks_d, jobs_d, njobs, kx,
                                                                        perm);
  count_launch();
}

void launch_ball_jobs(const TaskDev* tasks_d, const SortedJob* jobs_d, int njobs, int total_blocks,
                      int span, const KeyIndex& kx, const int32_t* perm, cudaStream_t st) {
  if (njobs <= 0 || total_blocks <= 0) return;
  const unsigned nb = (unsigned)total_blocks;
  if (span == BALL_THREADS)
    ball_jobs_kernel<1><<<nb, BALL_THREADS, 0, st>>>(tasks_d, jobs_d, njobs, kx, perm);
  else
    ball_jobs_kernel<4><<<nb, BALL_THREADS, 0, st>>>(tasks_d, jobs_d, njobs, kx, perm);
  count_launch();
}

}  // namespace egb
