// egb_strips.cu -- grid copies of two-column jobs, one block per strip.
//
// A strip holds consecutive positions [s0, s1) of the column-1 order, and its
// points stand in column-0 order in the grid copy.  The block reads the
// points' column-0 ranks through the inverse of that order (one inverse per
// sorted segment, however many jobs read it), puts them in order in shared
// memory and writes the strip: values, centred FP32 values, working indices
// and column-1 bounds.
//
// Ordering: the ranks are distinct integers, spread over as many buckets as the
// strip has points; a point's place is its bucket's start plus the smaller
// ranks in the bucket.  A strip whose ranks crowd into few buckets (columns
// that are functions of each other) is sorted bitonically instead.
//
// What bounds it: L2 sector throughput of the two gathers per point.  784 jobs
// of 180,000 points: 8.1 ms as a radix pass over strip keys and a gather by
// job (inverse, keys, histogram, three scans, scatter, copy), 2.6 ms here.
#include <algorithm>

#include "egb_internal.cuh"

namespace egb {
namespace {

constexpr int SB_CROWD = 24;   // largest bucket ranked by counting

// inv[w - src_begin] = position of working index w in the segment's order
__global__ void seg_inv_kernel(const InvSeg* __restrict__ segs, int nsegs,
                               const int32_t* __restrict__ sorted_vals) {
  for (int g = blockIdx.y; g < nsegs; g += gridDim.y) {
    const InvSeg s = segs[g];
    const int32_t* v = sorted_vals + s.base;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < s.len; p += gridDim.x * blockDim.x)
      s.inv[v[p] - s.src_begin] = p;
  }
}

// Shared memory of a strip of up to cap points (a power of two).
struct StripSmem {
  uint32_t* rank;    // [cap] column-0 rank of the strip's i-th point (column-1 order)
  uint32_t* start;   // [cap] bucket counts, then bucket ends
  uint32_t* brank;   // [cap] ranks in bucket order   (with bidx: 64-bit keys of the
  uint32_t* bidx;    // [cap] their points             bitonic sort)
  uint32_t* order;   // [cap] point at each place
};

// THREADS: about four points a thread.
template <int THREADS>
__global__ void __launch_bounds__(THREADS, 1536 / THREADS)
strip_build_kernel(const JobDev* __restrict__ jobs, const StripJob* __restrict__ sjobs, int nsjobs, int cap,
                   const uint64_t* __restrict__ keys, const int32_t* __restrict__ vals) {
  extern __shared__ __align__(8) uint32_t raw[];
  const StripSmem M{raw + 2 * cap, raw + 3 * cap, raw, raw + cap, raw + 4 * cap};
  uint64_t* key64 = reinterpret_cast<uint64_t*>(raw);
  __shared__ uint32_t wsum[THREADS / 32];
  __shared__ uint32_t rmin_s, rmax_s, crowd_s;
  int lo = 0, hi = nsjobs;  // the job of this block: the last that starts at or before it
  while (hi - lo > 1) {
    const int m = (lo + hi) >> 1;
    if (sjobs[m].blk0 <= (int)blockIdx.x) lo = m; else hi = m;
  }
  const StripJob sj = sjobs[lo];
  const JobDev& J = jobs[sj.job];
  const int s = (int)blockIdx.x - sj.blk0;
  const int s0 = J.sstart[s], n = J.sstart[s + 1] - s0;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint64_t* __restrict__ ka = keys + sj.base_a;
  const uint64_t* __restrict__ kb = keys + sj.base_b + s0;
  const int32_t* __restrict__ vb = vals + sj.base_b + s0;
  const int sb = J.seg_begin;
  if (tid == 0) {
    rmin_s = 0xffffffffu;
    rmax_s = crowd_s = 0u;
  }
  for (int i = tid; i < n; i += THREADS) M.start[i] = 0u;
  __syncthreads();
  uint32_t mn = 0xffffffffu, mx = 0u;
  for (int i = tid; i < n; i += THREADS) {
    const uint32_t r = (uint32_t)__ldg(sj.inv + (vb[i] - sb));
    M.rank[i] = r;
    mn = min(mn, r);
    mx = max(mx, r);
  }
  mn = __reduce_min_sync(0xffffffffu, mn);
  mx = __reduce_max_sync(0xffffffffu, mx);
  if (lane == 0) {
    atomicMin(&rmin_s, mn);
    atomicMax(&rmax_s, mx);
  }
  __syncthreads();
  // bucket of a rank: monotone in it
  const uint32_t r0 = rmin_s;
  const float scale = (float)n / (float)(rmax_s - r0 + 1u);
  auto bucket = [&](uint32_t r) { return min((int)((float)(r - r0) * scale), n - 1); };
  for (int i = tid; i < n; i += THREADS) atomicAdd(&M.start[bucket(M.rank[i])], 1u);
  __syncthreads();
  // exclusive scan of the counts; the largest
  const int per = (n + THREADS - 1) / THREADS;
  const int a = min(tid * per, n), b = min(a + per, n);
  uint32_t sum = 0, most = 0;
  for (int i = a; i < b; ++i) {
    sum += M.start[i];
    most = max(most, M.start[i]);
  }
  uint32_t x = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  most = __reduce_max_sync(0xffffffffu, most);
  if (lane == 31) wsum[warp] = x;
  if (lane == 0) atomicMax(&crowd_s, most);
  __syncthreads();
  if (crowd_s <= SB_CROWD) {
    uint32_t run = x - sum;
    for (int w = 0; w < warp; ++w) run += wsum[w];
    for (int i = a; i < b; ++i) {
      const uint32_t c = M.start[i];
      M.start[i] = run;
      run += c;
    }
    __syncthreads();
    for (int i = tid; i < n; i += THREADS) {
      const uint32_t r = M.rank[i];
      const uint32_t p = atomicAdd(&M.start[bucket(r)], 1u);  // start becomes the bucket's end
      M.brank[p] = r;
      M.bidx[p] = (uint32_t)i;
    }
    __syncthreads();
    for (int p = tid; p < n; p += THREADS) {
      const uint32_t r = M.brank[p];
      const int k = bucket(r);
      const int q0 = k ? (int)M.start[k - 1] : 0, q1 = (int)M.start[k];
      int place = q0;
      for (int q = q0; q < q1; ++q) place += M.brank[q] < r;
      M.order[place] = M.bidx[p];
    }
    __syncthreads();
  } else {  // bitonic sort of (rank, point)
    int m = 1;
    while (m < n) m <<= 1;
    for (int i = tid; i < m; i += THREADS)
      key64[i] = i < n ? ((uint64_t)M.rank[i] << 32) | (uint32_t)i : ~0ull;
    __syncthreads();
    for (int k = 2; k <= m; k <<= 1)
      for (int j = k >> 1; j > 0; j >>= 1) {
        for (int i = tid; i < m; i += THREADS) {
          const int l = i ^ j;
          if (l > i) {
            const uint64_t u = key64[i], v = key64[l];
            if ((u > v) == ((i & k) == 0)) {
              key64[i] = v;
              key64[l] = u;
            }
          }
        }
        __syncthreads();
      }
    for (int i = tid; i < n; i += THREADS) M.order[i] = (uint32_t)key64[i];
    __syncthreads();
  }
  const double c0 = J.center[0], c1 = J.center[1];
  bool bad = false;
  for (int t = tid; t < n; t += THREADS) {
    const int i = (int)M.order[t];
    const double x0 = value_of(__ldg(ka + M.rank[i])), x1 = value_of(kb[i]);
    double d0 = x0 - c0, d1 = x1 - c1;
    if (!fits32(d0) || !fits32(d1)) {
      bad = true;  // clamped so that FP32 distances stay finite (such jobs decide in FP64)
      d0 = fmin(fmax(d0, -1e37), 1e37);
      d1 = fmin(fmax(d1, -1e37), 1e37);
    }
    const int64_t p = s0 + t;
    J.idxg[p] = vb[i];
    J.c64g[p] = x0;
    J.c64g[J.lds + p] = x1;
    const float f0 = f32_nearest(d0), f1 = f32_nearest(d1);
    if (J.aos) {
      reinterpret_cast<float2*>(J.c32g)[p] = make_float2(f0, f1);
    } else {
      J.c32g[p] = f0;
      J.c32g[J.lds + p] = f1;
    }
  }
  if (s == J.nstrips - 1)  // the padding behind the last point
    for (int64_t p = J.len + tid; p < J.lds; p += THREADS) {
      J.idxg[p] = sb;
      for (int c = 0; c < 2; ++c) {
        J.c64g[c * J.lds + p] = 0.0;
        J.c32g[J.aos ? 2 * p + c : c * J.lds + p] = 0.0f;
      }
    }
  if (tid == 0) {
    const double yl = value_of(kb[0]), yh = value_of(kb[n - 1]);
    J.sylo[s] = yl;
    J.syhi[s] = yh;
    J.sylo32[s] = __double2float_rd(__dsub_rd(yl, c1));
    J.syhi32[s] = __double2float_ru(__dsub_ru(yh, c1));
  }
  if (__syncthreads_or(bad) && tid == 0) atomicOr(J.jflags, (uint32_t)TF_UNSAFE32);
}

}  // namespace

int init_strip_kernels() {
  return (int)cudaFuncSetAttribute(strip_build_kernel<512>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   5 * STRIP_CAP * (int)sizeof(uint32_t));
}

void launch_seg_inv(const InvSeg* segs_d, int nsegs, int64_t max_len, const int32_t* sorted_vals,
                    cudaStream_t st) {
  if (nsegs <= 0) return;
  const dim3 grid((unsigned)std::min<int64_t>((max_len + 255) / 256, 1024), (unsigned)std::min(nsegs, 65535));
  seg_inv_kernel<<<grid, 256, 0, st>>>(segs_d, nsegs, sorted_vals);
  count_launch();
}

void launch_strip_build(const JobDev* jobs_d, const StripJob* sjobs_d, int nsjobs, int nstrips, int largest,
                        const uint64_t* keys, const int32_t* vals, cudaStream_t st) {
  if (nsjobs <= 0) return;
  int cap = 64;
  while (cap < largest) cap <<= 1;
  const size_t smem = 5 * (size_t)cap * sizeof(uint32_t);
  if (cap <= 512)
    strip_build_kernel<128><<<nstrips, 128, smem, st>>>(jobs_d, sjobs_d, nsjobs, cap, keys, vals);
  else if (cap <= 1024)
    strip_build_kernel<256><<<nstrips, 256, smem, st>>>(jobs_d, sjobs_d, nsjobs, cap, keys, vals);
  else
    strip_build_kernel<512><<<nstrips, 512, smem, st>>>(jobs_d, sjobs_d, nsjobs, cap, keys, vals);
  count_launch();
}

}  // namespace egb
