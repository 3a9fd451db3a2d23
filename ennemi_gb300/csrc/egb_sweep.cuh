// egb_sweep.cuh -- the pieces that the single-sweep radix passes share: the
// look-back over a segment's tiles, the digit scan, the layout of the sweep
// buffer.
#pragma once
#include "egb_internal.cuh"

namespace egb {

constexpr int OS_PASSES = 8;        // digits of a 64-bit key
constexpr int CODE_PASSES = 4;      // digits of a 32-bit code, numbered 8 .. 11
constexpr int ALL_PASSES = OS_PASSES + CODE_PASSES;
// passes over the strip keys of the grid layouts, in a sweep buffer of their
// own: the two digits of a cell, the strip of a nested job's column-2 order
constexpr int GRID_PASS = OS_PASSES;
constexpr int NEST_PASS = OS_PASSES + 2;
constexpr int OS_SPIN_LIMIT = 1 << 22;

// The sweep buffer (zeroed before the sort): flag words, digit totals per
// segment and pass, a tile counter per pass, and per segment (then for all
// of them) what the code sort left to do.
constexpr uint32_t REDO_DIGITS = 1u;  // the passes over the keys' digits
constexpr uint32_t REDO_RUNS = 2u;    // long runs of equal codes to be put in order
struct Sweep {
  unsigned long long* flags;  // [256 tiles]
  uint32_t* seg_hist;         // [nseg][ALL_PASSES][256]
  int* counters;              // [ALL_PASSES]
  uint32_t* redo;             // [nseg + 1]
};
inline size_t sweep_layout(void* base, int os_nblk, int nseg, Sweep* out) {
  const size_t nt = (size_t)(os_nblk > 0 ? os_nblk : 1), ns = (size_t)(nseg > 0 ? nseg : 1);
  Sweep w;
  w.flags = (unsigned long long*)base;
  w.seg_hist = (uint32_t*)(w.flags + 256 * nt);
  w.counters = (int*)(w.seg_hist + (size_t)ALL_PASSES * 256 * ns);
  w.redo = (uint32_t*)(w.counters + ALL_PASSES);
  if (out) *out = w;
  return sizeof(unsigned long long) * 256 * nt +
         sizeof(uint32_t) * ((size_t)ALL_PASSES * 256 * ns + ALL_PASSES + ns + 1);
}

#ifdef __CUDACC__
__device__ __forceinline__ uint64_t key_of_bits(uint64_t u) {
  u = u == 0x8000000000000000ull ? 0ull : u;  // -0 -> +0
  return (u >> 63) ? ~u : (u | 0x8000000000000000ull);
}

// Publishes the count of one digit in tile b and returns its count in the
// segment's earlier tiles (first: the segment's first tile).
template <int LOOK>
__device__ __forceinline__ uint32_t sweep_look_back(unsigned long long* flags, int b, int first, int digit,
                                                    int pass, uint32_t cnt, uint32_t* err) {
  const unsigned long long tag = (unsigned long long)(pass + 1) << 56;
  const unsigned long long INCL = 1ull << 55;
  unsigned long long* mine = flags + (size_t)b * 256 + digit;
  if (b == first) {
    atomicExch(mine, tag | INCL | cnt);
    return 0;
  }
  atomicExch(mine, tag | cnt);
  uint32_t excl = 0;
  int pb = b - 1;
  for (bool more = true; more; pb -= LOOK) {  // LOOK tiles at once: one latency
    unsigned long long w[LOOK];
#pragma unroll
    for (int i = 0; i < LOOK; ++i) w[i] = *(volatile unsigned long long*)(flags + (size_t)max(pb - i, first) * 256 + digit);
#pragma unroll
    for (int i = 0; i < LOOK; ++i) {
      if (!more) break;
      int spins = 0;
      while ((w[i] >> 56) != (unsigned long long)(pass + 1)) {
        if (++spins > OS_SPIN_LIMIT) {
          atomicOr(err, DERR_WAIT_TIMEOUT);
          w[i] = tag | INCL;
          break;
        }
        w[i] = *(volatile unsigned long long*)(flags + (size_t)(pb - i) * 256 + digit);
      }
      excl += (uint32_t)w[i];
      more = !(w[i] & INCL) && pb - i > first;
    }
  }
  atomicExch(mine, tag | INCL | (excl + cnt));
  return excl;
}

// Exclusive scan over the 256 digits, one value per digit thread (tid <
// 256: warps 0-7); every thread of the block calls it.
__device__ __forceinline__ uint32_t digit_excl_scan(uint32_t v, uint32_t* ws) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint32_t x = v;
  if (tid < 256) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) ws[warp] = x;
  }
  __syncthreads();
  if (warp == 0) {
    uint32_t w = lane < 8 ? ws[lane] : 0u;
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    if (lane < 8) ws[lane] = w;
  }
  __syncthreads();
  const uint32_t r = tid < 256 ? (warp ? ws[warp - 1] : 0u) + x - v : 0u;
  __syncthreads();
  return r;
}
#endif

}  // namespace egb
