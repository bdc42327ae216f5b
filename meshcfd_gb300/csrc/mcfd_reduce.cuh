// The sum s = ((0 + p0) + p1) + ... of non-negative doubles, every addition
// rounded to nearest even in that order, computed by one warp with the bits of
// the sequential loop.
//
// The loop is a chain of dependent FP64 additions at 64 cycles each (608 block
// partials: 39,000 cycles, 32 us with its loads), and its order cannot change:
// a last place of the finite-difference step moves the products it divides.
// While the sum stays in one binade, though, its spacing u is fixed, and adding
// p rounds to s + u round(p / u) (s being a multiple of u): the rounded
// integers do not depend on s and add up in any order.  So 32 terms are
// rounded to multiples of u at once and added by an integer prefix sum, up to
// the first one that leaves the binade, is a tie (whose rounding depends on
// the parity of s) or is larger than s or not an ordinary non-negative number;
// that one is added by the FP64 unit, and the next 32 start after it.
#pragma once

#include "mcfd_arith.cuh"

namespace mcfd {

// p: the terms (shared memory), term i at p[i * stride].  All 32 lanes call;
// every lane returns the sum.
__device__ __forceinline__ double ordered_sum_warp(const double* p, int n, int stride) {
  const int lane = threadIdx.x & 31;
  double s = 0.0;
  int i = 0;
  while (i < n) {
    const double x = i + lane < n ? p[(size_t)(i + lane) * stride] : 0.0;
    const unsigned long long bs = ia::bits(s), bx = ia::bits(x);
    const int es = (int)(bs >> 52);  // s >= 0
    int bad = 0;                     // first term of the 32 that the integers do not cover
    if (es >= 1 && es <= 2046) {
      const unsigned long long m = (bs & ia::kMant) | ia::kImpl;
      const int ex = (int)(bx >> 52);  // with the sign bit
      unsigned long long r = 0;
      bool ok = (bx << 1) == 0ull;  // +-0 adds nothing
      if (!ok && ex >= 1 && ex <= es && es <= 2046) {
        const unsigned long long mx = (bx & ia::kMant) | ia::kImpl;
        const int d = es - ex;
        if (d == 0) {
          r = mx;
          ok = true;
        } else if (d > 54) {
          ok = true;  // below half a spacing
        } else {
          const unsigned long long rem = mx & ((1ull << d) - 1ull), half = 1ull << (d - 1);
          r = (mx >> d) + (rem > half ? 1ull : 0ull);
          ok = rem != half;
        }
      }
      unsigned long long sum = r;  // inclusive prefix; at most 32 2^53
      for (int off = 1; off < 32; off <<= 1) {
        const unsigned long long o = __shfl_up_sync(0xffffffffu, sum, off);
        if (lane >= off) sum += o;
      }
      const bool good = ok && m + sum < (ia::kImpl << 1);
      const unsigned wrong = __ballot_sync(0xffffffffu, !good);
      bad = wrong ? __ffs((int)wrong) - 1 : 32;
      if (bad > 0) {
        const unsigned long long t = m + __shfl_sync(0xffffffffu, sum, bad - 1);
        s = ia::from_bits(((unsigned long long)es << 52) | (t & ia::kMant));
      }
    }
    if (bad < 32) {
      if (i + bad < n) s = s + __shfl_sync(0xffffffffu, x, bad);
      i += bad + 1;
    } else {
      i += 32;
    }
  }
  return s;
}

// The same from global memory: the block copies n * stride doubles into sh
// first; warp w < stride sums column w and its lane 0 stores out[w].
__device__ __forceinline__ void ordered_sums_block(const double* __restrict__ p, int n, int stride, double* sh,
                                                   double* out) {
  for (int i = threadIdx.x; i < n * stride; i += blockDim.x) sh[i] = p[i];
  __syncthreads();
  const int w = threadIdx.x >> 5;
  if (w < stride) {
    const double s = ordered_sum_warp(sh + w, n, stride);
    if ((threadIdx.x & 31) == 0) out[w] = s;
  }
}

}  // namespace mcfd
