// egb_codesort.cu -- the batch sort of large batches: four passes over 32-bit
// codes instead of six over 64-bit keys.
//
// A value's code is the order-preserving image of its FP32 distance from the
// median of 32 values of its segment, rounded to nearest.  Subtraction and
// rounding are monotone, so codes never order two values wrongly, whatever the
// centre; values that FP32 cannot tell apart share one.  A centre amid the
// values gives the most of them distances of their own also in columns with an
// offset or long tails (from the midrange, half of what one outlier reaches,
// they would share few).  A pass moves one 8-byte word per point (code, working
// index), 16 bytes of traffic against the 24 of key and index apart, and four
// digits stand for six.  The last kernel reads each point's value through its
// index (the column lies in L2), orders the runs of equal codes by the full
// key, and writes keys, indices and the samples of the searches
// (egb_search.cuh): the stable order of the full keys, exactly.
//
// A run of more than TIE_RUN equal codes that is out of order (rounded values,
// which the noise of 1e-10 sets apart in FP64 alone: every level is one; a value
// repeated in a column) marks its segment in Sweep::redo with REDO_RUNS, and
// run_fix_kernel sorts the segment's long runs, up to RUN_CAP points, by their high
// 48 key bits in shared memory.  Longer ones, and any other pair out of order
// (NaNs), mark it with REDO_DIGITS, and the passes over the keys' own digits
// (egb_sort.cu) run for it.  Either way the tie repair and the samples of egb_sort.cu
// follow for the segment.  All of these are launched always and return at once
// when nothing is marked, so nothing waits for the host.  Exact duplicates are in
// order as they come and mark nothing.  100 columns of 180,000 normals (0.77 ms)
// rounded to 0.001: 1.37 ms, 3.01 when all of them took the digits after the codes,
// 1.30 with digits alone; 0.1 % of each column one value: 0.94, 2.55 and 1.20.
//
// 785 segments of 180,000 keys: load, passes, repair and samples 0.54 + 7.60 +
// 0.35 + 0.28 ms with the keys' digits; here load, passes and unpack 0.57 + 3.23
// + 1.19.  Eleven columns of a million: 0.81 -> 0.50 ms; 126 of 50,000: 0.45 ->
// 0.28.  A pass moves 16 bytes a point at 2.8 TB/s and is bound by the chain
// from digit counts to slots: barriers and shared-memory latency.  Blocks of
// 256 threads, one per digit and sixteen words each, five to an SM (with a few
// spills): 3.23 ms; four 3.27; 512 threads, three to an SM: 3.65; two: 4.48.
// The unpack is bound by its gathers from L2: 512 threads 1.19 ms, 256 1.30.
#include <algorithm>
#include <type_traits>

#include "egb_internal.cuh"
#include "egb_search.cuh"
#include "egb_sweep.cuh"

namespace egb {

namespace {

constexpr int LOAD_THREADS = 256;
constexpr int UNPACK_THREADS = 512;
constexpr int PASS_THREADS = 256;          // one per digit
constexpr int PASS_NW = PASS_THREADS / 32;
constexpr int TIE_RUN = 32;
constexpr int RUN_CAP = 2048;              // its places take 16 bits beside 48 of the key
constexpr int RUN_THREADS = 256;
constexpr int RUN_WARP = RUN_CAP / (RUN_THREADS / 32);  // longest run that one warp sorts
constexpr int RUN_COUNT = 128;             // and ranks by counting

__device__ __forceinline__ uint32_t code_of(double x, double c) {
  uint32_t b = __float_as_uint(f32_nearest(x - c));
  if (b == 0x80000000u) b = 0u;  // -0 and +0 are one value
  return (b >> 31) ? ~b : (b | 0x80000000u);
}

__global__ void __launch_bounds__(LOAD_THREADS)
code_load_kernel(const BatchCol* __restrict__ slots, const SortSeg* __restrict__ segs,
                 const int32_t* __restrict__ blk_seg, uint64_t* __restrict__ words,
                 uint32_t* __restrict__ seg_hist) {
  __shared__ uint32_t h[CODE_PASSES * 256];
  __shared__ double centre;
  const int si = blk_seg[blockIdx.x];
  const SortSeg& s = segs[si];
  const double* __restrict__ x = slots[s.slot].x + s.src_begin;
  for (int i = threadIdx.x; i < CODE_PASSES * 256; i += LOAD_THREADS) h[i] = 0;
  if (threadIdx.x < 32) {
    const double m = centre_of(x, s.len);
    if (threadIdx.x == 0) centre = m;
  }
  __syncthreads();
  const double c = centre;
  uint64_t* __restrict__ out = words + s.out_base;
  const int i0 = ((int)blockIdx.x - s.blk0) * SORT_TILE;
  const int i1 = min(i0 + SORT_TILE, s.len);
  const int w0 = s.src_begin;
  for (int i = i0 + (int)threadIdx.x; i < i1; i += LOAD_THREADS) {
    const uint32_t code = code_of(__ldg(x + i), c);
    out[i] = (uint64_t)code << 32 | (uint32_t)(w0 + i);
#pragma unroll
    for (int p = 0; p < CODE_PASSES; ++p) atomicAdd(&h[p * 256 + ((code >> (8 * p)) & 255u)], 1u);
  }
  __syncthreads();
  uint32_t* g = seg_hist + ((size_t)si * ALL_PASSES + OS_PASSES) * 256;
  for (int i = threadIdx.x; i < CODE_PASSES * 256; i += LOAD_THREADS)
    if (h[i]) atomicAdd(g + i, h[i]);
}

// One digit of the codes: the single-sweep pass of egb_sort.cu on words.  A
// tile's missing words read as the largest digit, behind all others.
template <int TILE>
struct PassSmem {
  uint32_t wcnt[PASS_NW][256];  // per-warp digit counts, then offsets
  uint32_t dstart[256];         // first tile slot of each digit
  uint32_t gbase[256];          // first output position of each digit, less dstart
  uint2 warp_sum[PASS_NW];      // of the two digit scans
  int tile;
  uint64_t sk[TILE];
};

template <int TILE, int LOOK>
__global__ void __launch_bounds__(PASS_THREADS, 5)
code_pass_kernel(const SortSeg* __restrict__ segs, const int32_t* __restrict__ os_blk_seg,
                 const uint64_t* __restrict__ in, uint64_t* __restrict__ out, int digit, int pass,
                 const uint32_t* __restrict__ seg_hist, unsigned long long* flags, int* tile_counter,
                 uint32_t* err) {
  constexpr int PASS_CH = TILE / PASS_NW;  // words per warp
  constexpr int PASS_R = PASS_CH / 32;     // rounds per warp
  extern __shared__ __align__(16) unsigned char raw[];
  PassSmem<TILE>& S = *reinterpret_cast<PassSmem<TILE>*>(raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) S.tile = atomicAdd(tile_counter, 1);
  for (int i = tid; i < PASS_NW * 256; i += PASS_THREADS) (&S.wcnt[0][0])[i] = 0u;
  __syncthreads();
  const int b = S.tile;
  const int si = os_blk_seg[b];
  const int64_t base = segs[si].out_base;
  const int len = segs[si].len, first = segs[si].os_blk0;
  const int i0 = (b - first) * TILE;
  const int n = min(TILE, len - i0);
  const int shift = 8 * digit;
  const uint32_t lt = (1u << lane) - 1u;
  uint64_t key[PASS_R];
  const uint64_t* __restrict__ src = in + base + i0 + warp * PASS_CH + lane;
#pragma unroll
  for (int r = 0; r < PASS_R; ++r)
    key[r] = warp * PASS_CH + r * 32 + lane < n ? __ldg(src + r * 32) : ~0ull;
  uint32_t rk[PASS_R];
#pragma unroll
  for (int r = 0; r < PASS_R; ++r) {
    const uint32_t d = ((uint32_t)(key[r] >> 32) >> shift) & 255u;
    uint32_t peers = 0xffffffffu;  // lanes with the same digit
#pragma unroll
    for (int bit = 0; bit < 8; ++bit) {
      const uint32_t bb = __ballot_sync(0xffffffffu, (d >> bit) & 1u);
      peers &= ((d >> bit) & 1u) ? bb : ~bb;
    }
    const uint32_t before = S.wcnt[warp][d];
    __syncwarp();
    if ((peers & lt) == 0) S.wcnt[warp][d] = before + __popc(peers);
    __syncwarp();
    rk[r] = before + __popc(peers & lt);
  }
  __syncthreads();
  uint32_t cnt = 0;  // digit tid: offsets of the warps, then its count in the tile
#pragma unroll
  for (int w = 0; w < PASS_NW; ++w) {
    const uint32_t c = S.wcnt[w][tid];
    S.wcnt[w][tid] = cnt;
    cnt += c;
  }
  if (tid == 255) cnt -= (uint32_t)(TILE - n);
  // exclusive scans over the digits of the tile's counts and of the segment's
  const uint32_t tot = seg_hist[((size_t)si * ALL_PASSES + pass) * 256 + tid];
  uint2 sum = make_uint2(cnt, tot);
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t a = __shfl_up_sync(0xffffffffu, sum.x, o), c = __shfl_up_sync(0xffffffffu, sum.y, o);
    if (lane >= o) sum.x += a, sum.y += c;
  }
  if (lane == 31) S.warp_sum[warp] = sum;
  const uint32_t excl = sweep_look_back<LOOK>(flags, b, first, tid, pass, cnt, err);
  __syncthreads();
  for (int w = 0; w < warp; ++w) sum.x += S.warp_sum[w].x, sum.y += S.warp_sum[w].y;
  S.gbase[tid] = (sum.y - tot) + excl - (sum.x - cnt);
  S.dstart[tid] = sum.x - cnt;
  __syncthreads();
#pragma unroll
  for (int r = 0; r < PASS_R; ++r) {
    const uint32_t d = ((uint32_t)(key[r] >> 32) >> shift) & 255u;
    S.sk[S.dstart[d] + S.wcnt[warp][d] + rk[r]] = key[r];
  }
  __syncthreads();
  for (int t = tid; t < n; t += PASS_THREADS) {
    const uint64_t k = S.sk[t];
    const uint32_t d = ((uint32_t)(k >> 32) >> shift) & 255u;
    const uint32_t pos = S.gbase[d] + (uint32_t)t;
    if (pos < (uint32_t)len)
      out[base + pos] = k;
    else
      atomicOr(err, DERR_BAD_INDEX);
  }
}

// Sorted words -> keys, indices and samples.  A block takes SORT_TILE
// positions and 32 to either side: enough to see all of a run of TIE_RUN.
// Warps with no inversion in sight write their positions as they are.
__global__ void __launch_bounds__(UNPACK_THREADS, 4)
code_unpack_kernel(const BatchCol* __restrict__ slots, const SortSeg* __restrict__ segs,
                   const int32_t* __restrict__ blk_seg, const uint64_t* __restrict__ words,
                   uint64_t* __restrict__ keys, int32_t* __restrict__ vals, KeyIndexOut ko,
                   uint32_t* redo, int nseg) {
  constexpr int SPAN = SORT_TILE + 64;
  __shared__ uint64_t sk[SPAN];
  __shared__ uint32_t sc[SPAN];
  __shared__ uint32_t inv[SPAN / 32];  // bit: below its predecessor
  const int si = blk_seg[blockIdx.x];
  const SortSeg& s = segs[si];
  const int len = s.len;
  const int i0 = ((int)blockIdx.x - s.blk0) * SORT_TILE;
  const int64_t base = s.out_base;
  const double* __restrict__ x = slots[s.slot].x;
  const int lane = threadIdx.x & 31;
  const int w0 = s.src_begin;
  constexpr int R = SORT_TILE / UNPACK_THREADS;
  uint32_t idx[R];
#pragma unroll
  for (int r = 0; r <= R; ++r) {  // the last round: the positions to either side
    const int u = r < R ? 32 + r * UNPACK_THREADS + (int)threadIdx.x
                        : (int)threadIdx.x < 32 ? (int)threadIdx.x : SORT_TILE + (int)threadIdx.x;
    if (r == R && threadIdx.x >= 64) break;
    const int p = i0 - 32 + u;
    if (p >= 0 && p < len) {
      const uint64_t w = __ldg(words + base + p);
      const uint32_t i = min(max((int)(uint32_t)w, w0), w0 + len - 1);
      if (r < R) idx[r] = i;
      sk[u] = key_of_bits((uint64_t)__double_as_longlong(__ldg(x + i)));
      sc[u] = (uint32_t)(w >> 32);
    }
  }
  __syncthreads();
  bool bad = false, runs = false;
  for (int u = threadIdx.x; u < SPAN; u += UNPACK_THREADS) {
    const int p = i0 - 32 + u;
    const bool below = u > 0 && p > 0 && p < len && sk[u] < sk[u - 1];
    bad |= below && sc[u] != sc[u - 1];
    const uint32_t m = __ballot_sync(0xffffffffu, below);
    if (lane == 0) inv[u / 32] = m;
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int u = 32 + r * UNPACK_THREADS + (int)threadIdx.x;
    const int p = i0 - 32 + u;
    const uint64_t k = sk[u];
    int pos = p;
    if (inv[u / 32 - 1] | inv[u / 32] | inv[u / 32 + 1]) {  // the same for the whole warp
      // points of the run before and after this one (32: that many, or more), from
      // the positions that start another run: those at u - 31 .. u from the top, at
      // u + 1 .. u + 32 from the bottom
      auto starts = [&](int w) {
        const int q = i0 - 32 + w;
        return w > 0 && (q <= 0 || q >= len || sc[w] != sc[w - 1]);
      };
      const uint32_t b0 = __ballot_sync(0xffffffffu, starts(u - 32));
      const uint32_t b1 = __ballot_sync(0xffffffffu, starts(u));
      const uint32_t b2 = __ballot_sync(0xffffffffu, starts(u + 32));
      const uint32_t before = __funnelshift_rc(b0, b1, lane + 1), after = __funnelshift_rc(b1, b2, lane + 1);
      const int l = __clz((int)before), g = after ? __ffs((int)after) - 1 : TIE_RUN;
      if (p >= len) {
      } else if (l + g + 1 <= TIE_RUN) {  // the rank among the run
        int below = 0;
        for (int j = u - l; j < u; ++j) below += sk[j] <= k;
        for (int j = u + 1; j <= u + g; ++j) below += sk[j] < k;
        pos = p - l + below;
      } else {
        runs |= l > 0 && k < sk[u - 1];
      }
    }
    if (p < len) {
      keys[base + pos] = k;
      vals[base + pos] = (int32_t)idx[r];
      put_samples(ko, s, pos, k);
    }
  }
  const uint32_t mark = (bad ? REDO_DIGITS : 0u) | (runs ? REDO_RUNS : 0u);
  if (mark && (*(volatile uint32_t*)(redo + si) & mark) != mark) {
    atomicOr(redo + si, mark);
    atomicOr(redo + nseg, mark);
  }
}

// The m words of buf (a power of two) in order, by the threads i0, i0 + step, ...
// of a warp or a block that sync() joins.
template <typename F>
__device__ __forceinline__ void bitonic_words(uint64_t* buf, int m, int i0, int step, F&& sync) {
  for (int k = 2; k <= m; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int i = i0; i < m / 2; i += step) {
        const int a = ((i & ~(j - 1)) << 1) | (i & (j - 1)), b = a | j;
        const uint64_t u = buf[a], v = buf[b];
        if ((u > v) == ((a & k) == 0)) {
          buf[a] = v;
          buf[b] = u;
        }
      }
      sync();
    }
}

// The runs of more than TIE_RUN equal codes that start in a tile, each stably by
// the high 48 bits of its keys: a word is those and the point's place in the run.
// Runs of up to RUN_WARP points take a warp each -- up to RUN_COUNT, the place is
// the number of smaller words, each read by all lanes at once; sorting networks there
// are bound by their shared-memory accesses (18 million points in runs of 50: the
// sort takes 1.88 ms with them, 1.37 so) -- and then the block takes the longer ones.
__global__ void __launch_bounds__(RUN_THREADS, 6)
run_fix_kernel(const SortSeg* __restrict__ segs, const int32_t* __restrict__ blk_seg, int nblk,
               const uint64_t* __restrict__ words, uint64_t* keys, int32_t* vals, uint32_t* redo, int nseg) {
  constexpr int NW = RUN_THREADS / 32;
  __shared__ uint64_t word[RUN_CAP];
  __shared__ int32_t idx[RUN_CAP];     // of the run's points, in the order they came
  __shared__ uint16_t low[RUN_CAP];    // and the low bits of their keys
  __shared__ int starts[SORT_TILE / TIE_RUN], lens[SORT_TILE / TIE_RUN];
  __shared__ int nrun;
  if (!(redo[nseg] & REDO_RUNS)) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int b = blockIdx.x; b < nblk; b += gridDim.x) {
    const int si = blk_seg[b];
    if (threadIdx.x == 0) nrun = 0;
    // REDO_RUNS is not written any more; a segment with REDO_DIGITS is sorted anew
    if (!(*(volatile uint32_t*)(redo + si) & REDO_RUNS)) continue;
    __syncthreads();
    const SortSeg& s = segs[si];
    const int len = s.len, i0 = (b - s.blk0) * SORT_TILE;
    const uint64_t* __restrict__ w = words + s.out_base;
    uint64_t* key = keys + s.out_base;
    int32_t* val = vals + s.out_base;
    auto code = [&](int p) { return (uint32_t)(__ldg(w + p) >> 32); };
    for (int p = i0 + (int)threadIdx.x; p < min(i0 + SORT_TILE, len); p += RUN_THREADS) {
      const uint32_t c = code(p);
      if (p + TIE_RUN < len && code(p + TIE_RUN) == c && (p == 0 || code(p - 1) != c)) starts[atomicAdd(&nrun, 1)] = p;
    }
    __syncthreads();
    const int n = nrun;
    if ((int)threadIdx.x < n) {
      const int p = starts[threadIdx.x];
      const uint32_t c = code(p);
      int lo = p + TIE_RUN, hi = lo + 1;  // codes ascend: code(lo) == c; steps that double, then halves
      for (int step = TIE_RUN; hi < len && hi <= p + RUN_CAP && code(hi) == c; step <<= 1) {
        lo = hi;
        hi = min(hi + step, len);
      }
      while (hi - lo > 1) {
        const int m = (lo + hi) >> 1;
        if (code(m) == c) lo = m; else hi = m;
      }
      lens[threadIdx.x] = hi - p;
      if (hi - p > RUN_CAP) {
        atomicOr(redo + si, REDO_DIGITS);
        atomicOr(redo + nseg, REDO_DIGITS);
      }
    }
    __syncthreads();
    // n points from p on, staged from slot o on, by threads t, t + step, ...
    auto sort_run = [&](int o, int p, int n, int t, int step, auto&& sync) {
      int m = 64;
      while (m < n) m <<= 1;
      for (int i = t; i < m; i += step) {
        const uint64_t k = i < n ? key[p + i] : 0ull;
        word[o + i] = i < n ? (k & ~0xffffull) | (uint32_t)i : ~0ull;
        if (i < n) {
          idx[o + i] = val[p + i];
          low[o + i] = (uint16_t)k;
        }
      }
      sync();
      bitonic_words(word + o, m, t, step, sync);
      for (int i = t; i < n; i += step) {
        const uint64_t k = word[o + i];
        const int from = o + (int)(k & 0xffffull);
        key[p + i] = (k & ~0xffffull) | low[from];
        val[p + i] = idx[from];
      }
      sync();
    };
    auto count_run = [&](auto words_a_lane, int o, int p, int n) {
      constexpr int R = decltype(words_a_lane)::value;
      uint64_t w[R];
      int32_t v[R];
      uint32_t lo[R];
      int place[R];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int i = r * 32 + lane;
        const uint64_t k = i < n ? key[p + i] : ~0ull;
        v[r] = i < n ? val[p + i] : 0;
        w[r] = (k & ~0xffffull) | (uint32_t)i;
        lo[r] = (uint32_t)k & 0xffffu;
        place[r] = 0;
        if (i < n) word[o + i] = w[r];
      }
      __syncwarp();
#pragma unroll 4
      for (int j = 0; j < n; ++j) {
        const uint64_t x = word[o + j];
#pragma unroll
        for (int r = 0; r < R; ++r) place[r] += x < w[r];
      }
      __syncwarp();
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (r * 32 + lane < n) {
          key[p + place[r]] = (w[r] & ~0xffffull) | lo[r];
          val[p + place[r]] = v[r];
        }
    };
    for (int r = warp; r < n; r += NW)
      if (lens[r] <= RUN_COUNT / 2)
        count_run(std::integral_constant<int, RUN_COUNT / 64>{}, warp * RUN_WARP, starts[r], lens[r]);
      else if (lens[r] <= RUN_COUNT)
        count_run(std::integral_constant<int, RUN_COUNT / 32>{}, warp * RUN_WARP, starts[r], lens[r]);
      else if (lens[r] <= RUN_WARP)
        sort_run(warp * RUN_WARP, starts[r], lens[r], lane, 32, [] { __syncwarp(); });
    __syncthreads();
    for (int r = 0; r < n; ++r)
      if (lens[r] > RUN_WARP && lens[r] <= RUN_CAP)
        sort_run(0, starts[r], lens[r], (int)threadIdx.x, RUN_THREADS, [] { __syncthreads(); });
    __syncthreads();
  }
}
static_assert(PASS_THREADS == 256, "one thread per digit");
static_assert((SORT_TILE + 64) % 32 == 0 && TIE_RUN == 32, "words of bits");

}  // namespace

int init_code_sort() {
  return (int)cudaFuncSetAttribute(code_pass_kernel<OS_TILE, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)sizeof(PassSmem<OS_TILE>));
}

void launch_word_pass(const SortSeg* segs_d, const int32_t* os_blk_seg_d, int os_nblk, int os_tile,
                      const uint64_t* in, uint64_t* out, int digit, int pass, const Sweep& w, uint32_t* err,
                      cudaStream_t st) {
  if (os_nblk <= 0) return;
  auto run = [&](auto kernel, size_t smem) {
    kernel<<<os_nblk, PASS_THREADS, smem, st>>>(segs_d, os_blk_seg_d, in, out, digit, pass, w.seg_hist, w.flags,
                                                w.counters + pass, err);
  };
  if (os_tile == OS_TILE) run(code_pass_kernel<OS_TILE, 1>, sizeof(PassSmem<OS_TILE>));
  else run(code_pass_kernel<OS_TILE_SMALL, 4>, sizeof(PassSmem<OS_TILE_SMALL>));
  count_launch();
}

void launch_code_sort(const BatchCol* slots_d, const SortSeg* segs_d, const int32_t* blk_seg_d, int nblk,
                      const int32_t* os_blk_seg_d, int os_nblk, int nseg, uint64_t* keys, uint64_t* words,
                      int32_t* vals, const KeyIndexOut& ko, const Sweep& w, int num_sms, uint32_t* err, cudaStream_t st,
                      cudaEvent_t* pass_events) {
  code_load_kernel<<<nblk, LOAD_THREADS, 0, st>>>(slots_d, segs_d, blk_seg_d, words, w.seg_hist);
  count_launch();
  if (pass_events) cudaEventRecord(pass_events[0], st);
  uint64_t* in = words;  // an even number of passes: back in words
  uint64_t* out = keys;
  for (int d = 0; d < CODE_PASSES; ++d) {
    launch_word_pass(segs_d, os_blk_seg_d, os_nblk, OS_TILE, in, out, d, OS_PASSES + d, w, err, st);
    uint64_t* t = in; in = out; out = t;
  }
  if (pass_events) cudaEventRecord(pass_events[1], st);
  code_unpack_kernel<<<nblk, UNPACK_THREADS, 0, st>>>(slots_d, segs_d, blk_seg_d, words, keys, vals, ko, w.redo,
                                                   nseg);
  count_launch();
  run_fix_kernel<<<std::min(nblk, 6 * num_sms), RUN_THREADS, 0, st>>>(segs_d, blk_seg_d, nblk, words, keys, vals, w.redo,
                                                                     nseg);
  count_launch();
}

}  // namespace egb
