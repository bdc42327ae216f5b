// Exterior states of pressure-inlet, mass-flow-inlet and mass-flow-outlet
// faces (solver.py:4412-4577): a block per 128 faces of a boundary patch, one
// for a mass-flow inlet.
//
// * pressure inlet (_pressure_inlet_boundary_states): per face, the Mach
//   number by 64 bisection steps on the outgoing Riemann invariant, then the
//   isentropic static state from the total conditions;
//   (both bisections: see known_side below for the steps they skip)
// * mass-flow inlet (_mass_flow_inlet_boundary_states): one speed per patch by
//   80 bisection steps on the patch's integrated flow rate; a step computes
//   the face terms density * speed * projection * length in parallel and adds
//   them in NumPy's pairwise order (np.sum), whose eight interleaved sums per
//   128 terms run on eight lanes;
//   density p / (R T) per face, velocity speed * direction on every face (the
//   reference builds a one-row velocity array there, which only works for
//   single-face patches, solver.py:4552-4554);
// * mass-flow outlet (_mass_flow_outlet_boundary_states): per face, the
//   normal velocity from the patch flow rate, tangential velocity kept.
// Checks set the reference's error bits and the lowest failing patch index.
// Python's scalar x**2 is libm pow and NumPy's array power its own SIMD code;
// both are reproduced only to the last place (x * x and mode_pow here).
#include "mcfd_device.cuh"
#include "mcfd_internal.h"

namespace mcfd {
namespace {

constexpr int kBlock = kBcThreads;

__device__ __forceinline__ void flag_patch(DevStatus* st, int bits, int patch) {
  atomicOr(&st->code, bits);
  atomicMin(&st->first_patch, patch);
}

// NumPy's pairwise summation (np.add.reduce of a contiguous float64 array):
// fewer than 8 terms add in order, up to 128 terms use eight interleaved
// partial sums combined as ((r0+r1)+(r2+r3))+((r4+r5)+(r6+r7)) followed by
// the remainder, longer arrays split at n/2 rounded down to a multiple of 8.
//
// The splits, walked without recursion (a device stack would have to be sized
// for it): leaf(first, terms) gives each leaf's sum, left to right.  2^30
// terms are 24 levels deep.
__host__ __device__ __forceinline__ int pairwise_half(int m) {
  const int h = m / 2;
  return h - h % 8;
}
template <typename Leaf>
__host__ __device__ __forceinline__ double pairwise_walk(int n, Leaf leaf) {
  int need[28], stage[28];  // stage 1: in its left half, 2: in its right half
  double left[28];
  double total = 0.0;
  int top = 0, first = 0;
  if (n <= 0) return 0.0;
  need[0] = n;
  stage[0] = 0;
  top = 1;
  bool have = false;  // total holds the sum of the half just finished
  while (top > 0) {
    const int k = top - 1, m = need[k];
    if (m <= 128) {  // a leaf is always a new entry
      total = leaf(first, m);
      first += m;
      have = true;
      --top;
    } else if (!have) {
      stage[k] = 1;
      need[top] = pairwise_half(m);
      stage[top++] = 0;
    } else if (stage[k] == 1) {
      left[k] = total;
      stage[k] = 2;
      need[top] = m - pairwise_half(m);
      stage[top++] = 0;
      have = false;
    } else {
      total = left[k] + total;
      --top;
    }
  }
  return total;
}

// A leaf of m <= 128 terms at a, by the eight lanes of an aligned group
// (mask: the participating lanes of the warp); every lane returns the sum.
__device__ __forceinline__ double pairwise_leaf(const double* a, int m, unsigned mask) {
  const int lane = (int)threadIdx.x & 7;
  double r = 0.0;
  if (m < 8) {
    for (int i = 0; i < m; ++i) r += a[i];
    return r;
  }
  const int whole = m - m % 8;
  r = a[lane];
  for (int i = 8; i < whole; i += 8) r += a[i + lane];
  r += __shfl_down_sync(mask, r, 1, 8);  // lanes 0, 2, 4, 6: r0 + r1, ...
  r += __shfl_down_sync(mask, r, 2, 8);  // lanes 0, 4: (r0 + r1) + (r2 + r3), ...
  r += __shfl_down_sync(mask, r, 4, 8);
  r = __shfl_sync(mask, r, 0, 8);
  for (int i = whole; i < m; ++i) r += a[i];
  return r;
}

// Which side of a bisection's root a midpoint lies on, where that needs no
// evaluation: -1 below, 1 above, 0 too close to tell.  The bisections take
// 64 and 80 steps of a function that is monotone up to the rounding of its
// evaluation, and most of their midpoints are nowhere near the root.  With
// the root known to within `margin` (rounding of the evaluation over the
// slope, and of the root itself, both with a factor of eight to spare), the
// sign of f(mid) - target there is that of the exact function, so the
// evaluated step would have gone the same way: the same interval, bit for
// bit.  Only midpoints within the margin are evaluated, about ten of 64, and
// once the interval is two neighbouring doubles the midpoint is one of its
// ends, whose side is known, and nothing changes any more.
// Both were a serial chain: 64 evaluations of some 1,450 cycles per face, 80
// block-wide evaluations of some 9,000 per patch.  Residual and time steps of
// two 19,440-cell ducts (160 x 81, half split), four such launches of 209 us
// on average before, 41 us now.
__device__ __forceinline__ int known_side(double mid, double root, double margin) {
  return mid < root - margin ? -1 : mid > root + margin ? 1 : 0;
}

__device__ __forceinline__ St4 interior_state(const DevGeom& g, const double* P, const double* recon, int f) {
  return recon ? ld4(recon + 4 * (size_t)g.ff_lslot[f]) : ld4(P + 4 * (size_t)g.ff_lcell[f]);
}

// outgoing invariant at Mach m: a0 / sqrt(1 + (gamma-1)/2 m^2) (dn m + 2/(gamma-1))
__device__ __forceinline__ double invariant_at(double m, double dn, double a0, double gamma) {
  const double ratio = 1.0 + 0.5 * (gamma - 1.0) * (m * m);
  const double sound = div_rn(a0, sqrt_rn(ratio));
  return sound * (dn * m + div_rn(2.0, gamma - 1.0));
}

template <bool LIBRARY>
__device__ void pressure_inlet(const DevGeom& g, const double* P, const double* recon, double gamma, double R,
                               const BcBlock& b, double* ext) {
  const int base = g.seg_begin[SEG_BCX];
  const double pt = b.value[0], tt = b.value[1], dx = b.value[2], dy = b.value[3];
  const double a0 = sqrt_rn(gamma * R * tt);
  for (int j = b.first + b.part * kBlock + (int)threadIdx.x; j < b.last; j += b.parts * kBlock) {
    const int f = base + j;
    const St4 q = interior_state(g, P, recon, f);
    const double2 n = g.ff_normal[f];
    const double dn = g.bc_dn[j];
    int bits = 0;
    if (dn >= -1e-12) bits |= MCFD_S_PIN_DIRECTION;
    const double c = sqrt_rn(div_rn(gamma * q.d, q.a));
    const double un = q.b * n.x + q.c * n.y;
    const double mach_in = div_rn(un, c);
    if (mach_in >= 1.0) bits |= MCFD_S_PIN_SUPERSONIC_OUT;
    if (mach_in <= -1.0) bits |= MCFD_S_PIN_SUPERSONIC_IN;
    const double outgoing = un + div_rn(2.0 * c, gamma - 1.0);
    if (!bits) {
      const double lo_v = invariant_at(0.0, dn, a0, gamma), hi_v = invariant_at(1.0, dn, a0, gamma);
      if (!(hi_v <= outgoing && outgoing <= lo_v)) bits |= MCFD_S_PIN_INCOMPATIBLE;
    }
    St4 out = q;
    if (!bits) {
      // The root of a0 (dn m + g) / sqrt(1 + k m^2) = outgoing, k = (gamma -
      // 1) / 2 and g = 1 / k: a quadratic, then one Newton step with the
      // slope a0 (dn - m) (1 + k m^2)^(-3/2), which is negative (dn < 0).
      const double k = 0.5 * (gamma - 1.0), ig = div_rn(1.0, k), c = div_rn(outgoing, a0);
      const double qa = dn * dn - c * c * k, qb = dn * ig, qc = ig * ig - c * c;
      const double disc = qb * qb - qa * qc;
      double root = div_rn(qc, sqrt_rn(disc > 0.0 ? disc : 0.0) - qb);  // -qb > 0: the sum has no cancellation
      root = root > 0.0 ? (root < 1.0 ? root : 1.0) : 0.0;
      const double ratio = 1.0 + k * (root * root);
      root = root + div_rn((invariant_at(root, dn, a0, gamma) - outgoing) * (ratio * sqrt_rn(ratio)), a0 * (root - dn));
      // values of the invariant over a0 stay below g + 1, evaluated within ten
      // roundings; the slope over a0 is above (m - dn) / ratio^(3/2), ratio <= 1 + k
      double margin = div_rn(0x1p-46 * (ig + 1.0) * ((1.0 + k) * (1.0 + k)), (root > 0.0 ? root : 0.0) - dn);
      if (!(root >= 0.0 && root <= 1.0 && margin < 0.01)) root = 0.0, margin = 2.0;  // no root to trust: every step evaluates
      double low = 0.0, high = 1.0;
      for (int it = 0; it < 64; ++it) {
        const double mid = 0.5 * (low + high);
        int side = known_side(mid, root, margin);
        if (side == 0) {
          if (mid == low && it > 0 && low > 0.0) break;  // neighbouring doubles: both ends' sides are known
          if (mid == high && high < 1.0) break;
          side = invariant_at(mid, dn, a0, gamma) > outgoing ? -1 : 1;
        }
        if (side < 0) low = mid;
        else high = mid;
      }
      const double m = 0.5 * (low + high);
      const double t = div_rn(tt, 1.0 + 0.5 * (gamma - 1.0) * (m * m));
      const double p = pt * mode_pow<LIBRARY>(div_rn(t, tt), div_rn(gamma, gamma - 1.0));
      const double rho = div_rn(p, R * t);
      const double speed = m * sqrt_rn(gamma * R * t);
      out = St4{rho, speed * dx, speed * dy, p};
      const bool finite = isfinite(out.a) && isfinite(out.b) && isfinite(out.c) && isfinite(out.d);
      if (!finite || !(rho > 0.0) || !(p > 0.0)) bits |= MCFD_S_PIN_STATE;
    }
    if (bits) flag_patch(g.status, bits, b.patch);
    st4(ext + 4 * (size_t)j, out);
  }
}

constexpr int kSharedTerms = 1024;  // faces of a mass-flow inlet patch summed in shared memory

__device__ void mass_flow_inlet(const DevGeom& g, const double* P, const double* recon, double gamma, double R,
                                const BcBlock& blk, double* ext) {
  __shared__ int s_bad;
  __shared__ int s_below;
  __shared__ int s_leaves;
  __shared__ int s_leaf[kSharedTerms / 64 + 2];  // first term of each leaf of the pairwise sum, and the end
  __shared__ double s_terms[kSharedTerms], s_weight[kSharedTerms], s_pressure[kSharedTerms], s_sum[kSharedTerms / 64 + 2];
  __shared__ double s_part[kBlock];
  const int base = g.seg_begin[SEG_BCX];
  const int patch = blk.patch, j0 = blk.first, j1 = blk.last, n = j1 - j0;
  const bool shared = n <= kSharedTerms;
  const double mdot = blk.value[0], tt = blk.value[1], dx = blk.value[2], dy = blk.value[3];
  if (threadIdx.x == 0) {
    s_bad = 0;
    int count = 0;
    if (shared) {
      pairwise_walk(n, [&](int first, int) {
        s_leaf[count++] = first;
        return 0.0;
      });
      s_leaf[count] = n;
    }
    s_leaves = count;
  }
  __syncthreads();
  int bits = 0;
  double flux = 0.0;  // sum of p proj L
  for (int j = j0 + threadIdx.x; j < j1; j += blockDim.x) {
    const double proj = -g.bc_dn[j];
    if (proj <= 1e-12) bits |= MCFD_S_MFI_DIRECTION;
    const double p = interior_state(g, P, recon, base + j).d;
    if (p <= 0.0 || !isfinite(p)) bits |= MCFD_S_MFI_PRESSURE;
    flux += p * proj * g.ff_len[base + j];
    if (shared) s_pressure[j - j0] = p, s_weight[j - j0] = proj;
  }
  s_part[threadIdx.x] = flux;
  if (bits) {
    flag_patch(g.status, bits, patch);
    atomicOr(&s_bad, 1);
  }
  __syncthreads();
  const double cp = div_rn(gamma * R, gamma - 1.0);
  double speed = 0.0;
  if (!s_bad) {
    double* terms = shared ? s_terms : g.bc_terms + j0;
    // flow_at(s) > or < the configured rate, decided for the block
    auto below = [&](double s) -> bool {
      const double rt = R * (tt - div_rn(s * s, 2.0 * cp));
      const unsigned long long rx = recip_fixed(rt);
      for (int j = threadIdx.x; j < n; j += blockDim.x) {
        const double p = shared ? s_pressure[j] : interior_state(g, P, recon, base + j0 + j).d;
        const double proj = shared ? s_weight[j] : -g.bc_dn[j0 + j];
        terms[j] = div_rn_recip(p, rt, rx) * s * proj * g.ff_len[base + j0 + j];
      }
      __syncthreads();
      if (shared) {
        // every leaf at once, eight lanes each; one thread combines them
        for (int k = (int)threadIdx.x >> 3; k < s_leaves; k += kBlock / 8) {
          const double r = pairwise_leaf(terms + s_leaf[k], s_leaf[k + 1] - s_leaf[k], 0xffu << (threadIdx.x & 24));
          if ((threadIdx.x & 7) == 0) s_sum[k] = r;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
          int k = 0;
          s_below = (0.0 + pairwise_walk(n, [&](int, int) { return s_sum[k++]; })) < mdot;
        }
      } else if (threadIdx.x < 32) {
        const double total = pairwise_walk(n, [&](int first, int m) { return pairwise_leaf(terms + first, m, 0xffffffffu); });
        if (threadIdx.x == 0) s_below = (0.0 + total) < mdot;
      }
      __syncthreads();
      const bool r = s_below != 0;
      __syncthreads();
      return r;
    };
    double low = 0.0, high = sqrt_rn(2.0 * cp * tt) * (1.0 - 1e-12);
    if (below(high)) {
      if (threadIdx.x == 0) flag_patch(g.status, MCFD_S_MFI_FLOW_RATE, patch);
    } else {
      // The root of K s / (R (T - s^2 / (2 cp))) = mdot, K the sum of p proj L
      // (positive terms): s^2 + b s = 2 cp T, b = 2 cp K / (R mdot).  The
      // flow's relative slope in s is at least one, and where its rounding
      // grows (T - s^2 / (2 cp) cancelling) the slope grows with it, so its
      // relative rounding, n + 8 units at most, bounds that of the root.
      if (threadIdx.x < 32) {
        double k = 0.0;
        for (int i = threadIdx.x; i < kBlock; i += 32) k += s_part[i];
        for (int off = 16; off > 0; off >>= 1) k += __shfl_down_sync(0xffffffffu, k, off);
        if (threadIdx.x == 0) s_part[0] = k;
      }
      __syncthreads();
      const double b = div_rn(2.0 * cp * s_part[0], R * mdot), q = 2.0 * cp * tt;
      double root = div_rn(2.0 * q, b + sqrt_rn(b * b + 4.0 * q));
      double margin = root * ((double)(n + 64) * 0x1p-50);
      if (!(b > 0.0 && isfinite(b) && root > 0.0 && root < high)) root = 0.0, margin = 2.0 * high;  // every step evaluates
      for (int it = 0; it < 80; ++it) {
        const double mid = 0.5 * (low + high);
        int side = known_side(mid, root, margin);
        if (side == 0) {
          if ((mid == low && low > 0.0) || mid == high) break;  // neighbouring doubles, both evaluated or known
          side = below(mid) ? -1 : 1;
        }
        if (side < 0) low = mid;
        else high = mid;
      }
    }
    speed = 0.5 * (low + high);
  }
  const double rt = R * (tt - div_rn(speed * speed, 2.0 * cp));
  for (int j = j0 + threadIdx.x; j < j1; j += blockDim.x) {
    const St4 q = interior_state(g, P, recon, base + j);
    st4(ext + 4 * (size_t)j, St4{div_rn(q.d, rt), speed * dx, speed * dy, q.d});
  }
}

__device__ void mass_flow_outlet(const DevGeom& g, const double* P, const double* recon, const BcBlock& b, double* ext) {
  const int base = g.seg_begin[SEG_BCX];
  const double mdot = b.value[0], total_length = b.value[1];
  for (int j = b.first + b.part * kBlock + (int)threadIdx.x; j < b.last; j += b.parts * kBlock) {
    const int f = base + j;
    const St4 q = interior_state(g, P, recon, f);
    if (q.a <= 0.0 || !isfinite(q.a)) flag_patch(g.status, MCFD_S_MFO_DENSITY, b.patch);
    const double2 n = g.ff_normal[f];
    const double vn = div_rn(mdot, total_length * q.a);
    const double tx = -n.y, ty = n.x;
    const double vt = q.b * tx + q.c * ty;
    st4(ext + 4 * (size_t)j, St4{q.a, vn * n.x + vt * tx, vn * n.y + vt * ty, q.d});
  }
}

template <bool LIBRARY>
__global__ void __launch_bounds__(kBlock) k_bc_states(DevGeom g, const double* __restrict__ P,
                                                      const double* __restrict__ recon, double gamma, double R,
                                                      double* __restrict__ ext) {
  const BcBlock b = g.bc_blocks[blockIdx.x];
  if (b.kind == MCFD_BC_PRESSURE_INLET) pressure_inlet<LIBRARY>(g, P, recon, gamma, R, b, ext);
  else if (b.kind == MCFD_BC_MASS_FLOW_OUTLET) mass_flow_outlet(g, P, recon, b, ext);
  else mass_flow_inlet(g, P, recon, gamma, R, b, ext);
}

}  // namespace

cudaError_t launch_bc_states(const DevGeom& g, const mcfd_config& cfg, const double* P, const double* recon,
                             double* ext, cudaStream_t s) {
  if (g.n_bc_patches <= 0) return cudaSuccess;
  count_launch();
  if (cfg.mode == MCFD_MODE_EXACT)
    k_bc_states<true><<<g.n_bc_blocks, kBlock, 0, s>>>(g, P, recon, cfg.gamma, cfg.gas_constant, ext);
  else
    k_bc_states<false><<<g.n_bc_blocks, kBlock, 0, s>>>(g, P, recon, cfg.gamma, cfg.gas_constant, ext);
  return cudaGetLastError();
}

}  // namespace mcfd
