// egb_prep.cu -- data movement around the search kernels.
//
// gather       caller columns (strided, optionally class-permuted) -> the
//              batch's working FP64 columns, zero padded up to ld;
// centres      per job column a value amid its values (centre_of);
// materialize  per multi-D job: its columns copied into one SoA block in
//              working or sorted order, with the FP32 centred copy and the
//              job's "FP32 unsafe" flag (a centred value >= 1e37 or not
//              finite: every candidate of that job is then decided in FP64);
// combine      per-sample estimator term summed in fixed 4096-sample chunks
//              (deterministic order), plus per-slot "a count was zero" flags.
//              Terms, from ennemi/_entropy_estimators.py:
//                MI     psi(nx) + psi(ny)                       (:113)
//                CMI    psi(nxz) + psi(nyz) - psi(nz)           (:156)
//                SEMI   psi(n)                                  (:200)
//                CSEMI  psi(nxz) + psi(nyz) - psi(nz)           (:247)
//                ENT    log(eps)                                (:42)
//              psi comes from an FP64 table indexed by the integer count.
#include <cooperative_groups.h>

#include <algorithm>

#include "egb_internal.cuh"
#include "egb_rescale.cuh"
#include "ennemi_gb.h"

namespace egb {

namespace {

constexpr int PREP_THREADS = 256;

int grid_x_for(int64_t n) {
  int64_t b = (n + PREP_THREADS - 1) / PREP_THREADS;
  if (b > 2048) b = 2048;
  return (int)(b < 1 ? 1 : b);
}
int grid_y_for(int n) { return n > 65535 ? 65535 : (n < 1 ? 1 : n); }

// n clusters of CL blocks each
template <int CL, typename... P, typename... A>
void launch_clusters(void (*kern)(P...), int n, int threads, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = CL;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)(n * CL));
  cfg.blockDim = dim3((unsigned)threads);
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kern, P(args)...);
}

// Four loads in flight per thread before its stores: columns read in place
// from host memory cross the CPU-GPU link, where throughput follows the
// requests outstanding.
constexpr int GATHER_UNROLL = 4;
__global__ void gather_kernel(const BatchCol* __restrict__ slots, int nslots) {
  for (int g = blockIdx.y; g < nslots; g += gridDim.y) {
    const BatchCol bc = slots[g];
    const int64_t step = (int64_t)gridDim.x * blockDim.x;
    for (int64_t w0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w0 < bc.ld;
         w0 += GATHER_UNROLL * step) {
      double v[GATHER_UNROLL];
#pragma unroll
      for (int u = 0; u < GATHER_UNROLL; ++u) {
        const int64_t w = w0 + u * step;
        v[u] = 0.0;
        if (w < bc.n) {
          const int64_t s = bc.perm ? (int64_t)bc.perm[w] : w;
          v[u] = bc.src[s * bc.stride];
        }
      }
#pragma unroll
      for (int u = 0; u < GATHER_UNROLL; ++u) {
        const int64_t w = w0 + u * step;
        if (w < bc.ld) bc.x[w] = v[u];
      }
    }
  }
}

// ----------------------------------------------------------- rescale --
// The reference's _rescale_data per column (egb_rescale.cuh).

// One leaf of pairwise_sum: fewer than 8 values in order from 0.0; else eight
// running sums over strides of 8, combined ((r0+r1)+(r2+r3))+((r4+r5)+(r6+r7)),
// then the remaining (len % 8) values in order.
// (a, inv: the column with the leaf's first sample at index 0)
__device__ double pw_leaf(const double* a, const int32_t* inv, int len, bool sq, double m) {
  if (len < 8) {
    double r = 0.0;
    for (int i = 0; i < len; ++i) r = __dadd_rn(r, pw_value(a, inv, i, sq, m));
    return r;
  }
  double r0 = pw_value(a, inv, 0, sq, m), r1 = pw_value(a, inv, 1, sq, m), r2 = pw_value(a, inv, 2, sq, m),
         r3 = pw_value(a, inv, 3, sq, m), r4 = pw_value(a, inv, 4, sq, m), r5 = pw_value(a, inv, 5, sq, m),
         r6 = pw_value(a, inv, 6, sq, m), r7 = pw_value(a, inv, 7, sq, m);
  const int end = len - (len % 8);
  int i = 8;
  for (; i < end; i += 8) {
    r0 = __dadd_rn(r0, pw_value(a, inv, i + 0, sq, m));
    r1 = __dadd_rn(r1, pw_value(a, inv, i + 1, sq, m));
    r2 = __dadd_rn(r2, pw_value(a, inv, i + 2, sq, m));
    r3 = __dadd_rn(r3, pw_value(a, inv, i + 3, sq, m));
    r4 = __dadd_rn(r4, pw_value(a, inv, i + 4, sq, m));
    r5 = __dadd_rn(r5, pw_value(a, inv, i + 5, sq, m));
    r6 = __dadd_rn(r6, pw_value(a, inv, i + 6, sq, m));
    r7 = __dadd_rn(r7, pw_value(a, inv, i + 7, sq, m));
  }
  double res = __dadd_rn(__dadd_rn(__dadd_rn(r0, r1), __dadd_rn(r2, r3)),
                         __dadd_rn(__dadd_rn(r4, r5), __dadd_rn(r6, r7)));
  for (; i < len; ++i) res = __dadd_rn(res, pw_value(a, inv, i, sq, m));
  return res;
}

// The pairwise sum of x[0, n) (sq: of (x - m)^2) by a cluster of CL blocks:
// leaves in parallel -- on one lane each (CL = 1: fewest FP64 operations) or
// on eight (CL > 1: the shortest chain) -- then the first block one height at
// a time, in shared memory where the tree fits.  Node sums pass through ns
// (global, read back through L2); the first block returns the sum.
constexpr int PW_SMEM_NODES = 4096;  // trees of n up to 180,000 and more
template <int CL>
__device__ double pw_sum(const double* x, const int32_t* inv, const PwTree& tr,
                         const int2* __restrict__ nodes, const int32_t* __restrict__ levels,
                         double* ns, double* sm, bool sq, double m) {
  if constexpr (CL == 1) {
    for (int i = threadIdx.x; i < tr.nleaf; i += blockDim.x) {
      const int2 L = nodes[tr.node0 + i];
      ns[i] = inv ? pw_leaf(x, inv + L.x, L.y, sq, m) : pw_leaf(x + L.x, nullptr, L.y, sq, m);
    }
    __syncthreads();
  } else {
    auto cl = cooperative_groups::this_cluster();
    const int rank = (int)cl.block_rank(), r = threadIdx.x & 7, per = blockDim.x >> 3;
    for (int i0 = rank * per; i0 < tr.nleaf; i0 += CL * per) {
      const int i = i0 + (threadIdx.x >> 3);
      const int2 L = i < tr.nleaf ? nodes[tr.node0 + i] : make_int2(0, 0);
      const double s = inv ? pw_leaf8(x, inv + L.x, L.y, r, sq, m)
                           : pw_leaf8(x + L.x, nullptr, L.y, r, sq, m);
      if (r == 0 && i < tr.nleaf) ns[i] = s;
    }
    cl.sync();  // orders the leaf sums for the cluster
    if (rank != 0) return 0.0;
  }
  const bool fits = CL > 1 && tr.nnode <= PW_SMEM_NODES;
  if (fits) {
    for (int i = threadIdx.x; i < tr.nleaf; i += blockDim.x) sm[i] = __ldcg(ns + i);
    __syncthreads();
  }
  for (int h = 0; h < tr.nlvl; ++h) {
    const int a = levels[tr.lvl0 + h], b = levels[tr.lvl0 + h + 1];
    for (int i = a + threadIdx.x; i < b; i += blockDim.x) {
      const int2 c = nodes[tr.node0 + i];
      if (fits) sm[i] = __dadd_rn(sm[c.x], sm[c.y]);
      else ns[i] = __dadd_rn(__ldcg(ns + c.x), __ldcg(ns + c.y));
    }
    __syncthreads();
  }
  return fits ? sm[tr.nnode - 1] : __ldcg(ns + tr.nnode - 1);
}

// One column per cluster of CL blocks.  A column's sums are FP64-bound on one
// SM (two operations a clock), so a handful of columns takes CL = 8 and more
// columns CL = 1 (785 columns of 180,000: 1.42 ms).
constexpr int STATS_FEW = 16, STATS_CLUSTER = 8;
constexpr int ROW_STAGE = 1024;  // rows staged at a time
template <int CL>
__global__ void __launch_bounds__(PREP_THREADS)
rescale_stats_kernel(const BatchCol* __restrict__ slots, const RescaleStat* __restrict__ stats,
                     const PwTree* __restrict__ trees, const int2* __restrict__ nodes,
                     const int32_t* __restrict__ levels, double* __restrict__ scratch,
                     double2* __restrict__ ms) {
  __shared__ double sm[CL > 1 ? PW_SMEM_NODES : 2 * ROW_STAGE];
  __shared__ double mean_s;
  const int stat = blockIdx.x / CL;
  const RescaleStat rs = stats[stat];
  const int len = slots[rs.slot].n;
  const double* x = slots[rs.slot].x;
  const double n = (double)len;
  if (rs.group > 1) {  // axis-0 reduction of an (n, group) array: in row order
    if (blockIdx.x % CL) return;
    const double mean = __ddiv_rn(row_sum<ROW_STAGE>(x, rs.inv, len, sm, false, 0.0), n);
    const double q = row_sum<ROW_STAGE>(x, rs.inv, len, sm, true, mean);
    if (threadIdx.x == 0) ms[stat] = make_double2(mean, __dsqrt_rn(__ddiv_rn(q, n)));
    return;
  }
  const PwTree tr = trees[rs.tree];
  double* ns = scratch + rs.scratch;
  double mean = __ddiv_rn(pw_sum<CL>(x, rs.inv, tr, nodes, levels, ns, sm, false, 0.0), n);
  if constexpr (CL > 1) {  // the first block's mean for all
    auto cl = cooperative_groups::this_cluster();
    if (cl.block_rank() == 0 && threadIdx.x == 0) mean_s = mean;
    cl.sync();
    mean = *cl.map_shared_rank(&mean_s, 0);
  } else {
    __syncthreads();  // every thread has read the root before the slots are reused
  }
  const double q = pw_sum<CL>(x, rs.inv, tr, nodes, levels, ns, sm, true, mean);
  if (threadIdx.x == 0 && blockIdx.x % CL == 0) ms[stat] = make_double2(mean, __dsqrt_rn(__ddiv_rn(q, n)));
}

// x = RN(RN(RN(x - mean) / sd) + noise) per sample of a task column (one
// y-row of blocks per column, four samples in flight per thread)
__global__ void __launch_bounds__(PREP_THREADS)
rescale_apply_kernel(const BatchCol* __restrict__ slots, const RescaleCol* __restrict__ cols,
                     const double2* __restrict__ ms, const double* __restrict__ noise,
                     uint32_t* __restrict__ const_flags) {
  const RescaleCol rc = cols[blockIdx.y];
  const int n = slots[rc.slot].n;
  double* x = slots[rc.slot].x;
  const double2 m = ms[rc.stat];
  const double mean = m.x, sd = m.y;
  if (fabs(sd) < 1e-20) {  // np.abs(std) < 1e-20: the reference warns and keeps x
    if (blockIdx.x == 0 && threadIdx.x == 0) const_flags[rc.slot] = 1u;
    return;
  }
  __shared__ double rsd_s;  // RN(1 / sd), once per block
  if (threadIdx.x == 0) rsd_s = __ddiv_rn(1.0, sd);
  __syncthreads();
  const double rsd = rsd_s;
  const double* nz = noise + rc.noise_pos;
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i0 < n; i0 += 4 * step) {
    int w[4];
    double v[4], z[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {  // sample i0 + u * step
      const int64_t i = i0 + u * step;
      w[u] = -1;
      if (i < n) {
        w[u] = rc.inv ? rc.inv[i] : (int)i;
        v[u] = x[w[u]];
        z[u] = nz[i * rc.group];
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (w[u] >= 0) x[w[u]] = __dadd_rn(div_rn(__dsub_rn(v[u], mean), sd, rsd), z[u]);
  }
}

// egb_debug_divide: div_rn over n pairs (one thread per pair)
__global__ void divide_kernel(const double* __restrict__ a, const double* __restrict__ b, int64_t n,
                              double* __restrict__ out) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    out[i] = div_rn(a[i], b[i], __ddiv_rn(1.0, b[i]));
}

// The centre of every column of every job: a warp each.  (The midrange, used
// before, took a pass over every column -- 0.55 ms for 785 of 180,000 -- and one
// outlier moves it away from all other values: FP32 distances then tie and
// queries are decided in FP64.  Four pairs of 500,000 Cauchy values took 1.18 s
// a call and two take 0.85 ms; pairs of normals with one value at 1e6 in each
// column, 0.47 s for four against 9 ms for two.)
__global__ void __launch_bounds__(256)
centre_kernel(const TaskDev* __restrict__ tasks, const JobDev* __restrict__ jobs, int njobs) {
  for (int g = (int)((blockIdx.x * 256 + threadIdx.x) >> 5); g < njobs; g += (int)(gridDim.x * 8)) {
    const JobDev& J = jobs[g];
    const TaskDev& t = tasks[J.task];
    for (int c = 0; c < J.sp.d; ++c) {
      const double m = centre_of(t.col[J.sp.cols[c]] + J.seg_begin, J.len);
      if ((threadIdx.x & 31) == 0) J.center[c] = m;
    }
  }
}

__device__ __forceinline__ bool materialize_copy(const TaskDev& t, const JobDev& J, int d,
                                                 double* c64, float* c32, int32_t* idx,
                                                 const int32_t* sv) {
  bool bad = false;
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < J.lds;
       p += (int64_t)gridDim.x * blockDim.x) {
    if (p < J.len) {
      const int32_t w = sv ? sv[p] : J.seg_begin + (int32_t)p;
      idx[p] = w;
      for (int c = 0; c < d; ++c) {
        const int tc = J.sp.cols[c];
        const double v = t.col[tc][w];
        double cv = v - J.center[c];
        if (!fits32(cv)) {
          bad = true;
          cv = fmin(fmax(cv, -1e37), 1e37);
        }
        c64[(int64_t)c * J.lds + p] = v;
        // clamped so that FP32 distances stay finite; a job with a clamped
        // value never trusts its FP32 copy (TF_UNSAFE32)
        c32[(int64_t)c * J.lds + p] = f32_nearest(cv);
      }
    } else {
      idx[p] = J.seg_begin;
      for (int c = 0; c < d; ++c) {
        c64[(int64_t)c * J.lds + p] = 0.0;
        c32[(int64_t)c * J.lds + p] = 0.0f;
      }
    }
  }
  return bad;
}

__global__ void materialize_kernel(const TaskDev* __restrict__ tasks,
                                   const JobDev* __restrict__ jobs, int njobs,
                                   const int32_t* __restrict__ sorted_vals,
                                   const SortSeg* __restrict__ segs) {
  for (int jb = blockIdx.y; jb < njobs; jb += gridDim.y) {
    const JobDev J = jobs[jb];
    const TaskDev t = tasks[J.task];
    const int d = J.sp.d;
    if (J.c64 == nullptr) continue;  // grid copy only (materialize_grid_kernel)
    const int32_t* sv = J.slab ? sorted_vals + segs[J.sort_seg].out_base : nullptr;
    bool bad = materialize_copy(t, J, d, J.c64, J.c32, J.idx, sv);
    if (J.c64b != nullptr)  // second copy, sorted by column 1 (same values)
      materialize_copy(t, J, d, J.c64b, J.c32b, J.idxb, sorted_vals + segs[J.sort_seg_b].out_base);
    if (__syncthreads_or(bad) && threadIdx.x == 0) atomicOr(J.jflags, (uint32_t)TF_UNSAFE32);
  }
}

// Grid copy: position p_G of the strip order takes the point at column-0
// position p_A, the lower half of the sorted word at p_G.
__global__ void materialize_grid_kernel(const TaskDev* __restrict__ tasks,
                                        const JobDev* __restrict__ jobs,
                                        const int32_t* __restrict__ grid_jobs, int ngrid,
                                        const int32_t* __restrict__ sorted_vals,
                                        const SortSeg* __restrict__ segs,
                                        const uint64_t* __restrict__ words,
                                        const SortSeg* __restrict__ gsegs) {
  for (int g = blockIdx.y; g < ngrid; g += gridDim.y) {
    const JobDev J = jobs[grid_jobs[g]];
    const TaskDev t = tasks[J.task];
    const int d = J.sp.d;
    const int32_t* va = sorted_vals + segs[J.sort_seg].out_base;
    const uint64_t* gv = words + gsegs[J.gseg].out_base;
    // column-1 bounds of each strip, from the column-1 sort
    const int32_t* vb = sorted_vals + segs[J.sort_seg_b].out_base;
    const double* x1 = t.col[J.sp.cols[1]];
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < J.nstrips; s += gridDim.x * blockDim.x) {
      const double lo = x1[vb[J.sstart[s]]];
      const double hi = x1[vb[J.sstart[s + 1] - 1]];
      J.sylo[s] = lo;
      J.syhi[s] = hi;
      J.sylo32[s] = __double2float_rd(__dsub_rd(lo, J.center[1]));
      J.syhi32[s] = __double2float_ru(__dsub_ru(hi, J.center[1]));
    }
    bool bad = false;  // a centred value too large for the FP32 copy
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < J.lds;
         p += (int64_t)gridDim.x * blockDim.x) {
      if (p < J.len) {
        const int32_t pa = (int32_t)(uint32_t)gv[p];
        const int32_t w = va[pa];
        if (J.posg) J.posg[p] = pa;
        J.idxg[p] = w;
        for (int c = 0; c < d; ++c) {
          const int tc = J.sp.cols[c];
          const double v = t.col[tc][w];
          if (J.kform) {
            const uint64_t k = raw_key((uint64_t)__double_as_longlong(v));
            uint32_t* kw = reinterpret_cast<uint32_t*>(J.c64g);
            kw[(int64_t)(2 * c) * J.lds + p] = (uint32_t)(k >> 32);
            kw[(int64_t)(2 * c + 1) * J.lds + p] = (uint32_t)k;
          } else {
            double cv = v - J.center[c];
            if (!fits32(cv)) {
              bad = true;
              cv = fmin(fmax(cv, -1e37), 1e37);
            }
            J.c64g[(int64_t)c * J.lds + p] = v;
            J.c32g[J.aos ? p * grid_aos(d) + c : (int64_t)c * J.lds + p] = f32_nearest(cv);
          }
        }
      } else {
        if (J.posg) J.posg[p] = 0;
        J.idxg[p] = J.seg_begin;
        for (int c = 0; c < d; ++c) {
          if (J.kform) {
            uint32_t* kw = reinterpret_cast<uint32_t*>(J.c64g);
            kw[(int64_t)(2 * c) * J.lds + p] = 0u;
            kw[(int64_t)(2 * c + 1) * J.lds + p] = 0u;
          } else {
            J.c64g[(int64_t)c * J.lds + p] = 0.0;
            J.c32g[J.aos ? p * grid_aos(d) + c : (int64_t)c * J.lds + p] = 0.0f;
          }
        }
      }
    }
    if (__syncthreads_or(bad) && threadIdx.x == 0) atomicOr(J.jflags, (uint32_t)TF_UNSAFE32);
  }
}

__device__ __forceinline__ double psi_of(const double* __restrict__ tab, int64_t len, int32_t n,
                                         uint32_t& bad) {
  if (n < 0 || n >= len) {
    bad = 1u;
    return 0.0;
  }
  return tab[n];  // entry 0 is a placeholder; zero counts are flagged
}

// The sample's term of a combine job, with its zero-count flags.
__device__ __forceinline__ double combine_term(const TaskDev& t, int kind, int64_t i,
                                               const double* __restrict__ psi_tab, int64_t psi_len,
                                               uint32_t& zf, uint32_t& bad) {
  double term;
  switch (kind) {
    case EGB_MI: {
      const int32_t a = t.cnt[0][i], b = t.cnt[1][i];
      zf |= (a == 0 ? 1u : 0u) | (b == 0 ? 2u : 0u);
      term = psi_of(psi_tab, psi_len, a, bad) + psi_of(psi_tab, psi_len, b, bad);
      break;
    }
    case EGB_CMI:
    case EGB_CSEMI: {
      const int32_t a = t.cnt[0][i], b = t.cnt[1][i], c = t.cnt[2][i];
      zf |= (a == 0 ? 1u : 0u) | (b == 0 ? 2u : 0u) | (c == 0 ? 4u : 0u);
      term = (psi_of(psi_tab, psi_len, a, bad) + psi_of(psi_tab, psi_len, b, bad)) -
             psi_of(psi_tab, psi_len, c, bad);
      break;
    }
    case EGB_SEMI: {
      const int32_t a = t.cnt[0][i];
      zf |= (a == 0 ? 1u : 0u);
      term = psi_of(psi_tab, psi_len, a, bad);
      break;
    }
    case EGB_DISCRETE_ENTROPY: {   // log(c / N)
      term = log((double)t.cnt[0][i] / (double)t.n);
      break;
    }
    case EGB_DISCRETE_MI: {        // log(N c_xy / (c_x c_y)), integer products exact
      const int64_t num = (int64_t)t.n * t.cnt[0][i];
      const int64_t den = (int64_t)t.cnt[1][i] * t.cnt[2][i];
      term = log((double)num / (double)den);
      break;
    }
    case EGB_DISCRETE_CMI: {       // log(c_z c_xyz / (c_xz c_yz))
      const int64_t num = (int64_t)t.cnt[3][i] * t.cnt[0][i];
      const int64_t den = (int64_t)t.cnt[1][i] * t.cnt[2][i];
      term = log((double)num / (double)den);
      break;
    }
    default: {  // EGB_ENTROPY: log(0) = -inf propagates exactly as in NumPy
      const double e = t.eps[i];
      zf |= (e == 0.0 ? 1u : 0u);
      term = log(e);
      break;
    }
  }
  return term;
}

// Sum of a chunk's terms in a fixed order: term(j) = the chunk's j-th, thread
// i the terms i, i + 256, ..., then warp shuffles, then warp 0 over the warps.
constexpr int COMBINE_THREADS = 256;
template <typename F>
__device__ __forceinline__ void chunk_sum(int cnt, F term, double* out) {
  __shared__ double wsum[COMBINE_THREADS / 32];
  double acc = 0.0;
  for (int j = threadIdx.x; j < cnt; j += COMBINE_THREADS) acc += term(j);
#pragma unroll
  for (int o = 16; o; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) wsum[warp] = acc;
  __syncthreads();
  if (warp == 0) {
    double v = lane < COMBINE_THREADS / 32 ? wsum[lane] : 0.0;
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) *out = v;
  }
}

// CL blocks (a cluster) share a chunk of COMBINE_CHUNK samples: each evaluates
// 1 / CL of its terms and leaves them in the first block's shared memory,
// which adds them -- the same order, so the same bits, for every CL.  CL = 8
// while chunks are fewer than a third of the SMs (the loads, or an entropy's
// FP64 logarithms, are then the time): 3 chunks of an MI 11.6 -> 6 us, 49 of an
// entropy 41 -> 21 us; CL = 1 beyond (125 chunks: 25 us against 31).
template <int CL>
__global__ void __launch_bounds__(COMBINE_THREADS)
combine_kernel(const TaskDev* __restrict__ tasks, const CombineJob* __restrict__ jobs,
               const int32_t* __restrict__ chunk_job, const double* __restrict__ psi_tab,
               int64_t psi_len, double* __restrict__ partial, uint32_t* __restrict__ zero_flags,
               uint32_t* __restrict__ err) {
  __shared__ double terms[CL > 1 ? COMBINE_CHUNK : 1];
  const int chunk = blockIdx.x / CL;
  const CombineJob jb = jobs[chunk_job[chunk]];
  const TaskDev t = tasks[jb.task];
  const int64_t p0 = (int64_t)(chunk - jb.chunk0) * COMBINE_CHUNK;
  const int cnt = (int)min((int64_t)COMBINE_CHUNK, (int64_t)t.n - p0);
  uint32_t zf = 0, bad = 0;
  auto flags = [&]() {
    zf = __reduce_or_sync(0xffffffffu, zf);
    bad = __reduce_or_sync(0xffffffffu, bad);
    if ((threadIdx.x & 31) == 0 && zf) atomicOr(&zero_flags[jb.task], zf);
    if ((threadIdx.x & 31) == 0 && bad) atomicOr(err, (uint32_t)DERR_BAD_INDEX);
  };
  if constexpr (CL == 1) {
    chunk_sum(cnt, [&](int j) { return combine_term(t, jb.kind, p0 + j, psi_tab, psi_len, zf, bad); },
              partial + chunk);
    flags();
  } else {
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    double* first = cl.map_shared_rank(terms, 0);
    cl.sync();  // every block of the cluster has started
    for (int j = (int)cl.block_rank() * COMBINE_THREADS + threadIdx.x; j < cnt; j += CL * COMBINE_THREADS)
      first[j] = combine_term(t, jb.kind, p0 + j, psi_tab, psi_len, zf, bad);
    flags();
    cl.sync();
    if (cl.block_rank() == 0) chunk_sum(cnt, [&](int j) { return terms[j]; }, partial + chunk);
  }
}

}  // namespace

void launch_gather(const BatchCol* slots_d, int nslots, int64_t max_ld, cudaStream_t st) {
  if (nslots <= 0) return;
  dim3 grid(grid_x_for((max_ld + GATHER_UNROLL - 1) / GATHER_UNROLL), grid_y_for(nslots));
  gather_kernel<<<grid, PREP_THREADS, 0, st>>>(slots_d, nslots);
  count_launch();
}

void launch_rescale(const BatchCol* slots_d, const RescaleStat* stats_d, int nstats,
                    const RescaleCol* cols_d, int ncols, const PwTree* trees_d,
                    const int2* nodes_d, const int32_t* levels_d, double* scratch, double2* ms,
                    const double* noise, uint32_t* const_flags, int64_t max_n, cudaStream_t st) {
  if (ncols <= 0 || nstats <= 0) return;
  if (nstats <= STATS_FEW)
    launch_clusters<STATS_CLUSTER>(rescale_stats_kernel<STATS_CLUSTER>, nstats, PREP_THREADS, st, slots_d,
                                   stats_d, trees_d, nodes_d, levels_d, scratch, ms);
  else
    rescale_stats_kernel<1><<<nstats, PREP_THREADS, 0, st>>>(slots_d, stats_d, trees_d, nodes_d, levels_d,
                                                             scratch, ms);
  count_launch();
  // 32 samples a thread where the columns fill the GPU (one division per
  // block), down to 4 where they do not: two columns of 10,000 samples took
  // 16 us on two blocks each
  const int gx = std::min(grid_x_for((max_n + 3) / 4),
                          std::max(grid_x_for((max_n + 31) / 32), 2048 / std::min(ncols, 2048)));
  for (int c0 = 0; c0 < ncols; c0 += 65535) {  // as many columns as a grid has rows
    const dim3 agrid(gx, grid_y_for(ncols - c0));
    rescale_apply_kernel<<<agrid, PREP_THREADS, 0, st>>>(slots_d, cols_d + c0, ms, noise, const_flags);
    count_launch();
  }
}

void launch_divide(const double* a_d, const double* b_d, int64_t n, double* out_d, cudaStream_t st) {
  if (n <= 0) return;
  divide_kernel<<<grid_x_for(n), PREP_THREADS, 0, st>>>(a_d, b_d, n, out_d);
  count_launch();
}

void launch_centres(const TaskDev* tasks_d, const JobDev* jobs_d, int njobs, cudaStream_t st) {
  if (njobs <= 0) return;
  centre_kernel<<<std::min((njobs + 7) / 8, 4096), 256, 0, st>>>(tasks_d, jobs_d, njobs);
  count_launch();
}

void launch_materialize(const TaskDev* tasks_d, const JobDev* jobs_d, int njobs,
                        const int32_t* sorted_vals, const SortSeg* segs_d, int64_t max_lds,
                        cudaStream_t st) {
  if (njobs <= 0) return;
  dim3 grid(grid_x_for(max_lds), grid_y_for(njobs));
  materialize_kernel<<<grid, PREP_THREADS, 0, st>>>(tasks_d, jobs_d, njobs, sorted_vals, segs_d);
  count_launch();
}

namespace {
// One thread per item: its run (the last whose first item is <= it), then
// its cell within the run, both by binary search over the item offsets.
__global__ void emit_items_kernel(const JobDev* __restrict__ jobs, const ItemRun* __restrict__ runs,
                                  int nruns, const int32_t* __restrict__ cum, int64_t nitems,
                                  WorkItem* __restrict__ items) {
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < nitems;
       t += (int64_t)gridDim.x * blockDim.x) {
    int lo = 0, hi = nruns;
    while (hi - lo > 1) {
      const int m = (lo + hi) >> 1;
      if (cum[runs[m].cum0] <= t) lo = m; else hi = m;
    }
    const ItemRun r = runs[lo];
    int c0 = 0, c1 = r.ncell;  // the last cell whose first item is <= t
    while (c1 - c0 > 1) {
      const int m = (c0 + c1) >> 1;
      if (cum[r.cum0 + m] <= t) c0 = m; else c1 = m;
    }
    const JobDev& J = jobs[r.job];
    int a, b, code;
    if (J.nsub > 0) {
      a = J.cstart[c0];
      b = J.cstart[c0 + 1];
      code = (c0 / J.nsub) | ((c0 % J.nsub) << 16);
    } else {
      a = J.sstart[c0];
      b = J.sstart[c0 + 1];
      code = c0;
    }
    const int q0 = a + (int)(t - cum[r.cum0 + c0]) * r.qb;
    items[t] = WorkItem{r.job, q0, min(q0 + r.qb, b), code};
  }
}
}  // namespace

void launch_emit_items(const JobDev* jobs_d, const ItemRun* runs_d, int nruns, const int32_t* cum_d,
                       int64_t nitems, WorkItem* items_d, cudaStream_t st) {
  if (nruns <= 0 || nitems <= 0) return;
  int grid = (int)((nitems + 255) / 256);
  if (grid > 8192) grid = 8192;
  emit_items_kernel<<<grid, 256, 0, st>>>(jobs_d, runs_d, nruns, cum_d, nitems, items_d);
  count_launch();
}

void launch_materialize_grid(const TaskDev* tasks_d, const JobDev* jobs_d,
                             const int32_t* grid_jobs_d, int ngrid, const int32_t* sorted_vals,
                             const SortSeg* segs_d, const uint64_t* words,
                             const SortSeg* gsegs_d, int64_t max_lds, cudaStream_t st) {
  if (ngrid <= 0) return;
  dim3 grid(grid_x_for(max_lds), grid_y_for(ngrid));
  materialize_grid_kernel<<<grid, PREP_THREADS, 0, st>>>(tasks_d, jobs_d, grid_jobs_d, ngrid,
                                                         sorted_vals, segs_d, words, gsegs_d);
  count_launch();
}

void launch_combine(const TaskDev* tasks_d, const CombineJob* jobs_d, const int32_t* chunk_job_d,
                    int nchunks, const double* psi_tab, int64_t psi_len, double* partial,
                    uint32_t* zero_flags, uint32_t* err, int num_sms, cudaStream_t st) {
  if (nchunks <= 0) return;
  if (3 * nchunks >= num_sms) {
    combine_kernel<1><<<nchunks, COMBINE_THREADS, 0, st>>>(tasks_d, jobs_d, chunk_job_d, psi_tab,
                                                           psi_len, partial, zero_flags, err);
  } else {
    constexpr int CL = 8;
    launch_clusters<CL>(combine_kernel<CL>, nchunks, COMBINE_THREADS, st, tasks_d, jobs_d, chunk_job_d,
                        psi_tab, psi_len, partial, zero_flags, err);
  }
  count_launch();
}

}  // namespace egb
