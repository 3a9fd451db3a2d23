// egb_rescale.cuh -- the arithmetic of the reference's _rescale_data
// (_driver.py:871-902), bit for bit, shared by the batch kernels (egb_prep.cu)
// and the small-batch path (egb_direct.cu): mean = pairwise_sum(x) / n, std =
// sqrt(pairwise_sum((x - mean)^2) / n), x = (x - mean) / std + noise -- every
// operation one IEEE double rounding (explicit _rn intrinsics: no contraction),
// the sums in NumPy's order.
#pragma once
#include "egb_internal.cuh"

namespace egb {

// Sample i of the column: x[i], or x[inv[i]] for a class-ordered task.
__device__ __forceinline__ double pw_value(const double* a, const int32_t* inv, int i, bool sq,
                                           double m) {
  const double v = inv ? a[inv[i]] : a[i];
  if (!sq) return v;
  const double d = __dsub_rn(v, m);
  return __dmul_rn(d, d);
}

// One leaf of pairwise_sum on eight lanes: fewer than 8 values in order from
// 0.0; else eight running sums over strides of 8 -- lane r of the group keeps
// r_r -- combined ((r0+r1)+(r2+r3))+((r4+r5)+(r6+r7)) by three exchanges
// (addition commutes, so every lane holds the same bits), then the remaining
// (len % 8) values in order.  Every lane of the warp
// calls it (len 0 where a group has no leaf).
__device__ __forceinline__ double pw_leaf8(const double* a, const int32_t* inv, int len, int r, bool sq, double m) {
  const int end = len >= 8 ? len - (len % 8) : 0;
  double s = r < end ? pw_value(a, inv, r, sq, m) : 0.0;
  int i = 8 + r;
  for (; i + 24 < end; i += 32) {  // four loads in flight, added in order
    const double v0 = pw_value(a, inv, i, sq, m), v1 = pw_value(a, inv, i + 8, sq, m);
    const double v2 = pw_value(a, inv, i + 16, sq, m), v3 = pw_value(a, inv, i + 24, sq, m);
    s = __dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn(s, v0), v1), v2), v3);
  }
  for (; i < end; i += 8) s = __dadd_rn(s, pw_value(a, inv, i, sq, m));
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) s = __dadd_rn(s, __shfl_xor_sync(0xffffffffu, s, o));
  if (end == 0) s = 0.0;
  for (i = end; i < len; ++i) s = __dadd_rn(s, pw_value(a, inv, i, sq, m));
  return s;
}

// The block's pairwise sum of x[0, n) (sq: of (x - m)^2) for a tree whose node
// sums fit into sm: leaves in parallel, then one height at a time.
__device__ __forceinline__ double pw_sum_block(const double* x, const int32_t* inv, const PwTree& tr,
                                               const int2* __restrict__ nodes,
                                               const int32_t* __restrict__ levels, double* sm, bool sq,
                                               double m) {
  const int r = threadIdx.x & 7, per = blockDim.x >> 3;
  for (int i0 = 0; i0 < tr.nleaf; i0 += per) {
    const int i = i0 + (threadIdx.x >> 3);
    const int2 L = i < tr.nleaf ? nodes[tr.node0 + i] : make_int2(0, 0);
    const double s = inv ? pw_leaf8(x, inv + L.x, L.y, r, sq, m)
                         : pw_leaf8(x + L.x, nullptr, L.y, r, sq, m);
    if (r == 0 && i < tr.nleaf) sm[i] = s;
  }
  __syncthreads();
  for (int h = 0; h < tr.nlvl; ++h) {
    const int a = levels[tr.lvl0 + h], b = levels[tr.lvl0 + h + 1];
    for (int i = a + threadIdx.x; i < b; i += blockDim.x) {
      const int2 c = nodes[tr.node0 + i];
      sm[i] = __dadd_rn(sm[c.x], sm[c.y]);
    }
    __syncthreads();
  }
  return sm[tr.nnode - 1];
}

// s + x_0 + x_1 + ... in order, each addition rounded, for the 32 values of
// the warp's lanes (the first cnt of them; lane i holds x_i).
//
// While the running sum stays inside one binade it is an integer multiple
// M u of the binade's ulp u, and RN(M u + x) = u (M + rint(x / u)): rounding
// to the grid u does not depend on M unless x / u lies exactly between two
// integers (the tie goes to the even sum).  So the additions up to the first
// one that ties or leaves the binade's interior are a sum of integers, exact
// and order-free; that one addition is done in FP64, and the rest follow on
// the new grid.  Integer instructions only, FP64 having few lanes here: a
// chain of dependent FP64 additions takes 79 cycles each with the loads off
// it (1.53 ms for two columns of 20,000 rows, mean and deviation).
__device__ __forceinline__ double ordered_add(double s, double x, int cnt) {
  constexpr int64_t ONE = (int64_t)1 << 52;
  const int lane = threadIdx.x & 31;
  const uint64_t ux = (uint64_t)__double_as_longlong(x);
  const int ex = (int)((ux >> 52) & 0x7ffu);
  const uint64_t mx = (ux & (uint64_t)(ONE - 1)) | (ex ? (uint64_t)ONE : 0ull);
  int i0 = 0;  // values before lane i0 are in s
  while (i0 < cnt) {
    const uint64_t us = (uint64_t)__double_as_longlong(s);
    const int e = (int)((us >> 52) & 0x7ffu);
    int f = i0;  // first value to add in FP64
    if (e != 0 && e != 0x7ff) {
      // q = rint(|x| / u): |x| = mx 2^(max(ex, 1) - 1075), u = 2^(e - 1075)
      const bool mine = lane >= i0 && lane < cnt;
      const int sh = e - max(ex, 1);
      const int sr = min(max(sh, 1), 55);  // mx < 2^53: 0 and no tie from 54 on
      const uint64_t half = 1ull << (sr - 1), rem = mx & ((half << 1) - 1ull);
      uint64_t q = sh <= 0 ? mx : (mx >> sr) + (rem > half ? 1u : 0u);
      const bool ok = sh >= 0 && !(sh > 0 && rem == half);  // x below s's binade's end, no tie
      if (!mine || !ok) q = 0;
      const bool neg = ((ux ^ us) >> 63) != 0;  // towards zero, with s as positive
      const int64_t M = (int64_t)((us & (uint64_t)(ONE - 1)) | (uint64_t)ONE);
      // all at once while |M| +- the sum of q stays inside (q < 2^54, split
      // at bit 28 for 32-bit reductions)
      const uint32_t top = __reduce_add_sync(0xffffffffu, (uint32_t)(q >> 28) + 1u);
      const int64_t reach = (int64_t)top << 28;  // > the sum of q
      const bool simple = !__any_sync(0xffffffffu, mine && !ok) && M - reach > ONE && M + reach < 2 * ONE;
      int64_t am;
      if (simple) {
        const int hi = neg ? -(int)(q >> 28) : (int)(q >> 28);
        const int lo = (int)(q & 0xfffffffull);
        const int64_t shi = __reduce_add_sync(0xffffffffu, hi);
        // 28 bits in two halves of 14: 32 of them stay within an int
        const int64_t slo0 = __reduce_add_sync(0xffffffffu, neg ? -(lo & 0x3fff) : (lo & 0x3fff));
        const int64_t slo1 = __reduce_add_sync(0xffffffffu, neg ? -(lo >> 14) : (lo >> 14));
        am = M + shi * ((int64_t)1 << 28) + slo1 * ((int64_t)1 << 14) + slo0;
        f = cnt;
      } else {
        int64_t p = neg ? -(int64_t)q : (int64_t)q;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int64_t y = __shfl_up_sync(0xffffffffu, p, o);
          if (lane >= o) p += y;
        }
        const int64_t m = M + p;  // the magnitude after this lane's value, in u
        const unsigned b = __ballot_sync(0xffffffffu, mine && !(ok && m > ONE && m < 2 * ONE));
        f = b ? __ffs(b) - 1 : cnt;
        am = __shfl_sync(0xffffffffu, m, f > i0 ? f - 1 : 0);
      }
      if (f > i0)  // ONE < am < 2 ONE: the mantissa of a double of exponent e
        s = __longlong_as_double((long long)((us & 0xfff0000000000000ull) | ((uint64_t)am & (uint64_t)(ONE - 1))));
    }
    // the addition that leaves the grid; a sum that leaves it at once (values
    // that cancel, subnormal sums) takes eight, so that such data costs no
    // more than the plain chain
    const int g = min(cnt, f == i0 ? f + 8 : f + 1);
    for (; f < g; ++f) s = __dadd_rn(s, __shfl_sync(0xffffffffu, x, f));
    i0 = g;
  }
  return s;
}

// Sum of x (sq: of (x - m)^2) row by row from the first row, as NumPy reduces
// axis 0 of an (n, group) array.  The other warps stage the terms of the next
// rows in shared memory while warp 0 adds.  sm: 2 STAGE doubles.
template <int ROW_STAGE>
__device__ __forceinline__ double row_sum(const double* x, const int32_t* inv, int n, double* sm, bool sq, double m) {
  auto stage = [&](int c) {
    double* d = sm + (c & 1) * ROW_STAGE;
    const int i0 = c * ROW_STAGE, cnt = min(ROW_STAGE, n - i0);
    for (int i = (int)threadIdx.x - 32; i < cnt; i += (int)blockDim.x - 32)
      d[i] = pw_value(x, inv, i0 + i, sq, m);
  };
  const int nc = (n + ROW_STAGE - 1) / ROW_STAGE;
  double s = 0.0;
  if (threadIdx.x >= 32) stage(0);
  __syncthreads();
  for (int c = 0; c < nc; ++c) {
    if (threadIdx.x >= 32) {
      if (c + 1 < nc) stage(c + 1);
    } else {
      const double* d = sm + (c & 1) * ROW_STAGE;
      const int cnt = min(ROW_STAGE, n - c * ROW_STAGE);
      int i = 0;
      if (c == 0) s = d[i++];
      for (; i < cnt; i += 32) {
        const int k = min(32, cnt - i);
        s = ordered_add(s, (int)threadIdx.x < k ? d[i + threadIdx.x] : 0.0, k);
      }
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) sm[0] = s;
  __syncthreads();
  s = sm[0];
  __syncthreads();
  return s;
}

// RN(a / b) without a division per element.  q = RN(a * rb) (rb = RN(1/b))
// is within two ulps of the quotient; the remainder a - q b from one FMA is
// exact once q is within one ulp (the remainder of a faithful quotient is
// representable: Boldo and Daumas, 2003), and the quotient lies above the
// midpoint between q and its successor exactly when that remainder exceeds
// half an ulp of q times b -- a power-of-two multiple of b, built by integer
// exponent arithmetic.  q steps one ulp at a time until the remainder lies
// between the two midpoints; a remainder equal to one of them is a tie,
// rounded to the even neighbour.  Magnitudes throughout, the sign applied at
// the end (round to nearest is symmetric).  Operands outside the exponent
// range where no step can underflow or overflow take the division itself.
// One FP64 multiply and one or two FMAs per element, against the FP64 pipe's
// few operations per clock per SM.
__device__ __forceinline__ double div_rn(double a, double b, double rb) {
  const uint64_t ua = (uint64_t)__double_as_longlong(a), ub = (uint64_t)__double_as_longlong(b);
  const uint64_t sign = (ua ^ ub) & 0x8000000000000000ull;
  const uint64_t ma = ua & 0x7fffffffffffffffull, mb = ub & 0x7fffffffffffffffull;
  const int ea = (int)(ma >> 52), eb = (int)(mb >> 52);
  if (ea < 1023 - 900 || ea > 1023 + 900 || eb < 1023 - 900 || eb > 1023 + 900 ||
      abs(ea - eb) > 1000)
    return __ddiv_rn(a, b);
  const double A = __longlong_as_double((long long)ma), B = __longlong_as_double((long long)mb);
  const int64_t half_b = (int64_t)mb - ((int64_t)1 << 52);  // bits of B / 2
  double q = __dmul_rn(A, fabs(rb));
  for (int it = 0; it < 4; ++it) {
    const double e = __fma_rn(-q, B, A);  // A - q B
    const uint64_t uq = (uint64_t)__double_as_longlong(q);
    const int eq = (int)(uq >> 52);
    // half an ulp of q above (and below: half that at a power of two) times B
    const uint64_t h_up = (uint64_t)(half_b + ((int64_t)(eq - 1075) << 52));
    const uint64_t h_dn = (uq & 0xfffffffffffffull) ? h_up : h_up - (1ull << 52);
    const uint64_t ue = (uint64_t)__double_as_longlong(e);
    const uint64_t me = ue & 0x7fffffffffffffffull;
    const bool neg = (ue >> 63) != 0 && me != 0;
    if (!neg && me > h_up) { q = __longlong_as_double((long long)(uq + 1)); continue; }
    if (neg && me > h_dn) { q = __longlong_as_double((long long)(uq - 1)); continue; }
    if (!neg && me == h_up) q = __longlong_as_double((long long)((uq & 1) ? uq + 1 : uq));
    else if (neg && me == h_dn) q = __longlong_as_double((long long)((uq & 1) ? uq - 1 : uq));
    return __longlong_as_double((long long)((uint64_t)__double_as_longlong(q) | sign));
  }
  return __ddiv_rn(a, b);  // not settled in four steps (not met in the fast range)
}

}  // namespace egb
