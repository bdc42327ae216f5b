// Exact Jacobian-vector product of the residual (forward mode).
//
// dR = (dR/dU) dU for the residual of mcfd_residual (first order or MUSCL
// linear with the four limiters, all fluxes and boundary kinds), evaluated
// with Dual<1> numbers in the same kernel structure as the residual:
// tangent of the primitive recovery (per cell), of the reconstruction (per
// cell: LSQ gradient, limiter through its minimising entry and the extreme
// neighbours, face states), of the face fluxes (per flux face, ghost states
// included) and of the divergence gather (per cell, reference order).  It is
// the exact counterpart of the reference's finite-difference product
// (solver.py:1532-1567).  Values are recomputed in the exact operation order,
// so the switch decisions (limiter band, extreme neighbour, HLLC region,
// far-field regime) are those of the residual itself.
#include "mcfd_ad.cuh"
#include "mcfd_internal.h"
#include "mcfd_jvp.h"

namespace mcfd {
namespace {

using D1 = ad::Dual<1>;
constexpr int kBlock = 256;
inline int blocks_for(int n) { return (n + kBlock - 1) / kBlock; }

__device__ __forceinline__ D1 dual(double v, double d) {
  D1 x(v);
  x.d[0] = d;
  return x;
}

__device__ __forceinline__ ad::S4<D1> ld4d(const double* p, const double* dp, size_t i) {
  const St4 a = ld4(p + 4 * i), b = ld4(dp + 4 * i);
  return ad::S4<D1>{dual(a.a, b.a), dual(a.b, b.b), dual(a.c, b.c), dual(a.d, b.d)};
}

__global__ void k_prim_tangent(int C, const double* __restrict__ U, const double* __restrict__ dU, double gamma,
                               double* __restrict__ P, double* __restrict__ dP) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= C) return;
  // values in the reference's exact order; tangents from the dual form
  bool ok;
  const St4 p = cons_to_prim(ld4(U + 4 * (size_t)c), gamma, &ok);
  const ad::S4<D1> q = ad::prim(ld4d(U, dU, c), gamma);
  st4(P + 4 * (size_t)c, p);
  st4(dP + 4 * (size_t)c, St4{q.a.d[0], q.b.d[0], q.c.d[0], q.d.d[0]});
}

// derivative of the limiter function g at ratio r (0 where it is capped)
template <int LIMITER>
__device__ __forceinline__ double limiter_slope(double r) {
  if (LIMITER <= 1) return r < 1.0 ? 1.0 : 0.0;
  if (LIMITER == 2) {
    if (!(r > 0.0)) return 0.0;
    const double q = div_rn(2.0 * r, 1.0 + r);
    return q < 1.0 ? div_rn(2.0, (1.0 + r) * (1.0 + r)) : 0.0;
  }
  const double eps = 1e-12;
  const double N = r * r + 2.0 * r + eps, D = r * r + r + 2.0 + eps;
  if (div_rn(N, D) > 1.0) return 0.0;
  return div_rn((2.0 * r + 2.0) * D - N * (2.0 * r + 1.0), D * D);
}

// Face states and their tangents, one thread per (cell, variable): the
// variables of a cell are independent, and the values are those of the exact
// residual's reconstruction (the same expressions in the same order), so one
// pass over the neighbours and limiter entries gives both.  The limiter's
// derivative is taken once, at the first entry of least factor.  Bound by
// FP64 issue: 67 us (values) + 177 us (tangents, one thread per cell, the
// derivative at every entry) before, 111 us now, for 131,327 cells.
template <int LIMITER>
__global__ void __launch_bounds__(kBlock) k_reconstruct_tangent(DevGeom g, const double* __restrict__ P,
                                                                const double* __restrict__ dP,
                                                                double* __restrict__ Q, double* __restrict__ dQ,
                                                                double venkat_k) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = t >> 2, v = t & 3;
  if (i >= g.n_cells) return;
  const int c = g.cell_order[i];
  const double pv = P[4 * (size_t)c + v], dpv = dP[4 * (size_t)c + v];
  double gx = 0.0, gy = 0.0, dgx = 0.0, dgy = 0.0, lo = pv, hi = pv, dlo = dpv, dhi = dpv;
  for (int e = g.grad_ptr[c], e1 = g.grad_ptr[c + 1]; e < e1; ++e) {
    const size_t nb = 4 * (size_t)g.grad_nb[e] + v;
    const double cx = g.grad_cx[e], cy = g.grad_cy[e];
    const double q = P[nb], dq = dP[nb];
    const double d = q - pv;
    gx = gx + cx * d;
    gy = gy + cy * d;
    const double dd = dq - dpv;
    dgx = ia::fma_rn(cx, dd, dgx);
    dgy = ia::fma_rn(cy, dd, dgy);
    if (icmp::lt(q, lo)) { lo = q; dlo = dq; }
    if (icmp::lt(hi, q)) { hi = q; dhi = dq; }
  }
  double phi = 1.0, dphi = 0.0, arg_inc = 0.0, arg_dinc = 0.0;
  bool have = false;
  const int s0 = g.lim_ptr[c], s1 = g.lim_ptr[c + 1];
  if constexpr (LIMITER == MCFD_LIMITER_VENKATAKRISHNAN_K) {
    // the smooth form: the minimising face's factor and its total derivative
    // through d1 (the extreme neighbour or the cell) and d2 (the gradient)
    const double e2 = venkat_k_e2(venkat_k, g.area[c]);
    VenkatK best{};
    for (int s = s0; s < s1; ++s) {
      const double2 r = g.lim_d[s];
      const double inc = gx * r.x + gy * r.y;
      const VenkatK f = venkat_k_face(pv, inc, lo, hi, e2);
      if (s == s0 || icmp::lt(f.f, phi)) {
        phi = f.f;
        best = f;
        arg_inc = inc;
        arg_dinc = ia::fma_rn(dgx, r.x, dgy * r.y);
        have = true;
      }
    }
    if (have) {
      double sa, sb;
      venkat_k_slopes(best, arg_inc, &sa, &sb);
      const double dd1 = (icmp::gt0(arg_inc) ? dhi : dlo) - dpv;
      dphi = sa * dd1 + sb * arg_dinc;
    }
  } else {
    const double tol = limiter_tolerance(pv);
    for (int s = s0; s < s1; ++s) {
      const double2 r = g.lim_d[s];
      const double inc = gx * r.x + gy * r.y;
      const double f = limiter_face_factor<LIMITER>(pv, inc, lo, hi, tol);
      if (icmp::lt_nonneg(f, phi)) {
        phi = f;
        arg_inc = inc;
        arg_dinc = ia::fma_rn(dgx, r.x, dgy * r.y);
        have = true;
      }
    }
    const bool pos = icmp::gt_pos(arg_inc, tol), neg = icmp::neg_gt_pos(arg_inc, tol);
    if (have && (pos || neg)) {
      const double num = pos ? hi - pv : lo - pv;
      const double dnum = pos ? dhi - dpv : dlo - dpv;
      const double ratio = div_rn(num, arg_inc);
      if (icmp::gt0(ratio))
        dphi = div_rn(limiter_slope<LIMITER>(ratio) * ia::fma_rn(-ratio, arg_dinc, dnum), arg_inc);
    }
  }
  for (int s = s0; s < s1; ++s) {
    const double2 r = g.lim_d[s];
    const size_t o = 4 * (size_t)g.lim_slot[s] + v;
    const double inc = gx * r.x + gy * r.y;
    Q[o] = pv + phi * inc;
    dQ[o] = ia::fma_rn(phi, ia::fma_rn(dgx, r.x, dgy * r.y), ia::fma_rn(dphi, inc, dpv));
  }
}

template <int FLUX, int SEG, bool FO, bool KH>
__device__ __forceinline__ void flux_tangent_face(const DevGeom& g, const double* __restrict__ P,
                                                  const double* __restrict__ dP, const double* __restrict__ recon,
                                                  const double* __restrict__ drecon, double* __restrict__ dflux,
                                                  double gamma, int f, int begin) {
  const double2 n = g.ff_normal[f];
  using S = ad::S4<D1>;
  const S L = FO ? ld4d(P, dP, g.ff_lcell[f]) : ld4d(recon, drecon, g.ff_lslot[f]);
  S R;
  if (SEG == SEG_INTERIOR || SEG == SEG_PERIODIC) {
    R = FO ? ld4d(P, dP, g.ff_rcell[f]) : ld4d(recon, drecon, g.ff_rslot[f]);
  } else if (SEG == SEG_WALL) {
    const double2 wv = g.ff_wall_velocity[f - begin];
    D1 un = (L.b - wv.x) * n.x + (L.c - wv.y) * n.y;
    R = S{L.a, L.b - 2.0 * un * n.x, L.c - 2.0 * un * n.y, L.d};
  } else if (SEG == SEG_VIN) {
    const St4 x = ld4(g.ff_vin_state + 4 * (size_t)(f - begin));
    R = S{D1(x.a), D1(x.b), D1(x.c), D1(x.d)};
  } else if (SEG == SEG_POUT) {
    R = S{L.a, L.b, L.c, D1(g.ff_pout_pressure[f - begin])};
  } else {
    const St4 x = ld4(g.ff_far_state + 4 * (size_t)(f - begin));
    R = ad::far_field(L, S{D1(x.a), D1(x.b), D1(x.c), D1(x.d)}, n.x, n.y, gamma);
  }
  D1 out[4];
  ad::numerical_flux<D1>(FLUX, (SEG == SEG_INTERIOR) && KH, L, R, n.x, n.y, gamma, out);
  st4(dflux + 4 * (size_t)f, St4{out[0].d[0], out[1].d[0], out[2].d[0], out[3].d[0]});
}

// Every segment in one launch, the far field's blocks first: its chain of
// powers is the longest.  Bound by FP64 issue on large meshes and by that chain
// on small ones.  A launch per segment was slower at every size, with walls and
// far field (a product with HLLC fluxes and MUSCL on 208 / 59,080 / 457,080 /
// 1,230,080 faces 76 / 133 / 581 / 1,443 us, 49 / 94 / 512 / 1,331 us so) and on a
// periodic box (901,200 faces 1,070 and 1,005 us).
template <int FLUX, bool FO, bool KH>
__global__ void __launch_bounds__(kBlock) k_flux_tangent(DevGeom g, const double* __restrict__ P,
                                                         const double* __restrict__ dP,
                                                         const double* __restrict__ recon,
                                                         const double* __restrict__ drecon,
                                                         double* __restrict__ dflux, double gamma) {
  int b = blockIdx.x;
#define MCFD_SEG(SEGV)                                                                                      \
  {                                                                                                         \
    const int begin = g.seg_begin[SEGV], n = g.seg_begin[SEGV + 1] - begin;                                 \
    const int nb = (n + (int)blockDim.x - 1) / (int)blockDim.x;                                             \
    if (b < nb) {                                                                                           \
      const int k = b * (int)blockDim.x + (int)threadIdx.x;                                                 \
      if (k < n)                                                                                            \
        flux_tangent_face<FLUX, SEGV, FO, KH>(g, P, dP, recon, drecon, dflux, gamma, begin + k, begin);     \
      return;                                                                                               \
    }                                                                                                       \
    b -= nb;                                                                                                \
  }
  MCFD_SEG(SEG_FAR)
  MCFD_SEG(SEG_VIN)
  MCFD_SEG(SEG_POUT)
  MCFD_SEG(SEG_WALL)
  MCFD_SEG(SEG_PERIODIC)
  MCFD_SEG(SEG_INTERIOR)
#undef MCFD_SEG
}

__global__ void __launch_bounds__(kBlock) k_gather_tangent(DevGeom g, const double* __restrict__ P,
                                                           const double* __restrict__ dP,
                                                           const double* __restrict__ dflux, double ax,
                                                           double ay, double* __restrict__ dR) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= g.n_cells) return;
  double r[4] = {0.0, 0.0, 0.0, 0.0};
  for (int j = g.gi_ptr[c]; j < g.gi_ptr[c + 1]; ++j) {
    const double a = g.gi_coef[j];
    const St4 F = ld4(dflux + 4 * (size_t)g.gi_flux[j]);
    r[0] += a * F.a; r[1] += a * F.b; r[2] += a * F.c; r[3] += a * F.d;
  }
  const int jb0 = g.gb_ptr[c], jb1 = g.gb_ptr[c + 1];
  if (jb0 < jb1) {
    const double ia = div_rn(1.0, g.area[c]);
    for (int j = jb0; j < jb1; ++j) {
      const double w = g.gb_len[j] * ia;
      const St4 F = ld4(dflux + 4 * (size_t)g.gb_flux[j]);
      r[0] += w * F.a; r[1] += w * F.b; r[2] += w * F.c; r[3] += w * F.d;
    }
  }
  if (ax != 0.0 || ay != 0.0) {
    const St4 p = ld4(P + 4 * (size_t)c), t = ld4(dP + 4 * (size_t)c);
    r[1] += t.a * ax;
    r[2] += t.a * ay;
    r[3] += t.a * (ax * p.b + ay * p.c) + p.a * (ax * t.b + ay * t.c);
  }
  st4(dR + 4 * (size_t)c, St4{r[0], r[1], r[2], r[3]});
}

template <int FLUX, bool FO, bool KH>
void launch_flux_tangent(const DevGeom& g, const double* P, const double* dP, const double* recon,
                         const double* drecon, double* dflux, double gamma, cudaStream_t s) {
  const int t = seg_threads(g.seg_begin[SEG_BCX]);
  int blocks = 0;
  for (int k = 0; k < SEG_BCX; ++k) blocks += (g.seg_begin[k + 1] - g.seg_begin[k] + t - 1) / t;
  if (blocks == 0) return;
  count_launch();
  k_flux_tangent<FLUX, FO, KH><<<blocks, t, 0, s>>>(g, P, dP, recon, drecon, dflux, gamma);
}

}  // namespace

cudaError_t launch_jvp(const DevGeom& g, const mcfd_config& cfg, const double* U, const double* dU,
                       const JvpWork& w, double* dR, cudaStream_t s) {
  const int C = g.n_cells;
  count_launch();
  k_prim_tangent<<<seg_blocks(C), seg_threads(C), 0, s>>>(C, U, dU, cfg.gamma, w.P, w.dP);
  const bool fo = cfg.reconstruction == MCFD_RECON_FIRST_ORDER;
  if (!fo) {
    const int t = 64, blocks = (int)((4LL * C + t - 1) / t);
    count_launch();
    switch (cfg.limiter) {
      case 0: k_reconstruct_tangent<0><<<blocks, t, 0, s>>>(g, w.P, w.dP, w.recon, w.drecon, 0.0); break;
      case 1: k_reconstruct_tangent<1><<<blocks, t, 0, s>>>(g, w.P, w.dP, w.recon, w.drecon, 0.0); break;
      case 2: k_reconstruct_tangent<2><<<blocks, t, 0, s>>>(g, w.P, w.dP, w.recon, w.drecon, 0.0); break;
      case 3: k_reconstruct_tangent<3><<<blocks, t, 0, s>>>(g, w.P, w.dP, w.recon, w.drecon, 0.0); break;
      default:
        k_reconstruct_tangent<MCFD_LIMITER_VENKATAKRISHNAN_K><<<blocks, t, 0, s>>>(g, w.P, w.dP, w.recon, w.drecon,
                                                                                   cfg.venkat_k);
        break;
    }
  }
  const bool kh = cfg.reconstruction != MCFD_RECON_MUSCL_PARABOLIC;
  switch (cfg.flux) {
    case MCFD_FLUX_RUSANOV:
      if (fo) launch_flux_tangent<0, true, false>(g, w.P, w.dP, w.recon, w.drecon, w.dflux, cfg.gamma, s);
      else launch_flux_tangent<0, false, false>(g, w.P, w.dP, w.recon, w.drecon, w.dflux, cfg.gamma, s);
      break;
    case MCFD_FLUX_HLLC:
      if (fo) launch_flux_tangent<1, true, true>(g, w.P, w.dP, w.recon, w.drecon, w.dflux, cfg.gamma, s);
      else if (kh) launch_flux_tangent<1, false, true>(g, w.P, w.dP, w.recon, w.drecon, w.dflux, cfg.gamma, s);
      else launch_flux_tangent<1, false, false>(g, w.P, w.dP, w.recon, w.drecon, w.dflux, cfg.gamma, s);
      break;
    default:
      if (fo) launch_flux_tangent<2, true, false>(g, w.P, w.dP, w.recon, w.drecon, w.dflux, cfg.gamma, s);
      else launch_flux_tangent<2, false, false>(g, w.P, w.dP, w.recon, w.drecon, w.dflux, cfg.gamma, s);
      break;
  }
  count_launch();
  k_gather_tangent<<<seg_blocks(C), seg_threads(C), 0, s>>>(g, w.P, w.dP, w.dflux, cfg.acceleration_x, cfg.acceleration_y, dR);
  return cudaGetLastError();
}

}  // namespace mcfd

namespace mcfd {
namespace {

// the scales are read from the prepared operator's device copy, so a
// captured GMRES step uses the current ones
__global__ void k_scale_dir(int n4, const double* __restrict__ v, const double* __restrict__ scale,
                            double* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n4) out[i] = scale[i & 3] * v[i];
}

__global__ void k_exact_combine(int n4, const double* __restrict__ v, const double* __restrict__ dR,
                                const double* __restrict__ scale, const double* __restrict__ dt, int dt_per_cell,
                                double* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n4) return;
  const double d = dt_per_cell ? dt[i >> 2] : dt[0];
  out[i] = v[i] - div_rn(d * dR[i], scale[i & 3]);
}

}  // namespace

cudaError_t exact_operator(const DevGeom& g, const mcfd_config& cfg1, const ImplicitState& st, const JvpWork& w,
                           const double* v, double* out, cudaStream_t s) {
  const int n4 = 4 * g.n_cells;
  count_launch();
  k_scale_dir<<<blocks_for(n4), kBlock, 0, s>>>(n4, v, st.scale_dev, w.sv);
  cudaError_t e = launch_jvp(g, cfg1, st.state, w.sv, w, w.dR, s);
  if (e != cudaSuccess) return e;
  count_launch();
  k_exact_combine<<<blocks_for(n4), kBlock, 0, s>>>(n4, v, w.dR, st.scale_dev, st.dt, st.dt_per_cell, out);
  return cudaGetLastError();
}

}  // namespace mcfd
