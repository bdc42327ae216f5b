// MUSCL-parabolic reconstruction and the reference's reconstruction fields.
//
// _parabolic_reconstruction (solver.py:2322-2415).  Per cell, from the mesh
// alone (k_parabolic_plan, once per geometry, one thread per cell):
//   * the stencil scale max(|dx|, |dy|) over the cell's two-ring entries;
//   * the weighted normal equations M (5x5), accumulated over the cell's
//     entries in the reference's entry order (np.add.at is sequential),
//     weights 1 / max(|r/scale|^2, 1e-300);
//   * the rank gate np.linalg.matrix_rank(M) == 5: an LU with partial
//     pivoting gives the Frobenius condition number kappa_F = |M| |M^-1|;
//     below 1e12 the matrix is certainly of full rank (s_min / s_max >=
//     1 / kappa_F, far above the 5 eps threshold), otherwise one-sided
//     Jacobi singular values (Hestenes' method) and the rank rule decide;
//   * that LU's factors (row interchange to the first largest |a_ik|, unit
//     lower factor, right-looking), and per entry the five products weight x
//     basis in the order of the interchanged rows, so that the right-hand
//     side accumulates in its pivoted order.
// Per state (k_reconstruct_parabolic, one thread per cell and variable):
//   * the variable's right-hand side, accumulated over the entries in order;
//   * the solve by the stored LU; np.linalg.solve's LAPACK gesv agrees to
//     rounding (a few 1e-15 relative), not bit for bit;
//   * the limiter on the quadratic increment with two-ring extrema, or, for
//     cells that fail the gate, the linear gradient and limiter of
//     _limited_gradients (identical to the linear kernels, entry order kept).
// The face states are written per limiter slot as P + phi (G . r + the
// curvature term) in _reconstruct's order (solver.py:2418-2434).
//
// Compiled with -fmad=false: every product and sum rounds as the C oracle's
// restatement does, so the two agree bit for bit.
#include "mcfd_device.cuh"
#include "mcfd_internal.h"

namespace mcfd {
namespace {

constexpr int kBlock = 128;
constexpr double kEps = 2.220446049250313e-16;  // DBL_EPSILON

// Row interchange of rows k and p of a 5-column array with compile-time row
// indices only (the array stays in registers).
template <int K, int NC>
__device__ __forceinline__ void swap_rows(double (&A)[5][NC], int p) {
#pragma unroll
  for (int i = K + 1; i < 5; ++i) {
    if (p == i) {
#pragma unroll
      for (int j = 0; j < NC; ++j) {
        const double t = A[K][j];
        A[K][j] = A[i][j];
        A[i][j] = t;
      }
    }
  }
}

// Gaussian elimination with partial pivoting in place; false on a zero or
// non-finite pivot.
__device__ __forceinline__ bool lu5(double (&A)[5][5], int (&piv)[5]) {
  bool ok = true;
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    int p = k;
    double best = fabs(A[k][k]);
#pragma unroll
    for (int i = k + 1; i < 5; ++i) {
      const double a = fabs(A[i][k]);
      if (a > best) {
        best = a;
        p = i;
      }
    }
    piv[k] = p;
    if (!(best > 0.0) || !isfinite(best)) ok = false;
    if (!ok) return false;
    switch (k) {
      case 0: swap_rows<0, 5>(A, p); break;
      case 1: swap_rows<1, 5>(A, p); break;
      case 2: swap_rows<2, 5>(A, p); break;
      case 3: swap_rows<3, 5>(A, p); break;
      default: break;
    }
#pragma unroll
    for (int i = k + 1; i < 5; ++i) {
      const double l = div_rn(A[i][k], A[k][k]);
      A[i][k] = l;
#pragma unroll
      for (int j = k + 1; j < 5; ++j) A[i][j] = A[i][j] - l * A[k][j];
    }
  }
  return ok;
}

template <int M>
__device__ __forceinline__ void lu5_solve(const double (&LU)[5][5], const int (&piv)[5], double (&b)[5][M]) {
  swap_rows<0, M>(b, piv[0]);
  swap_rows<1, M>(b, piv[1]);
  swap_rows<2, M>(b, piv[2]);
  swap_rows<3, M>(b, piv[3]);
#pragma unroll
  for (int i = 1; i < 5; ++i)
#pragma unroll
    for (int j = 0; j < i; ++j)
#pragma unroll
      for (int v = 0; v < M; ++v) b[i][v] = b[i][v] - LU[i][j] * b[j][v];
#pragma unroll
  for (int i = 4; i >= 0; --i) {
#pragma unroll
    for (int j = i + 1; j < 5; ++j)
#pragma unroll
      for (int v = 0; v < M; ++v) b[i][v] = b[i][v] - LU[i][j] * b[j][v];
#pragma unroll
    for (int v = 0; v < M; ++v) b[i][v] = div_rn(b[i][v], LU[i][i]);
  }
}

// Singular values by one-sided Jacobi rotations; returns the rank by the
// rule of np.linalg.matrix_rank (s > max(s) * 5 * eps).
__device__ __noinline__ int jacobi_rank5(const double (&M)[5][5]) {
  double A[5][5];
#pragma unroll
  for (int i = 0; i < 5; ++i)
#pragma unroll
    for (int j = 0; j < 5; ++j) A[i][j] = M[i][j];
  for (int sweep = 0; sweep < 60; ++sweep) {
    bool rotated = false;
#pragma unroll
    for (int p = 0; p < 4; ++p)
#pragma unroll
      for (int q = p + 1; q < 5; ++q) {
        double alpha = 0.0, beta = 0.0, gam = 0.0;
#pragma unroll
        for (int i = 0; i < 5; ++i) {
          alpha += A[i][p] * A[i][p];
          beta += A[i][q] * A[i][q];
          gam += A[i][p] * A[i][q];
        }
        if (!(fabs(gam) > 1e-15 * sqrt_rn(alpha * beta))) continue;
        rotated = true;
        const double zeta = div_rn(beta - alpha, 2.0 * gam);
        const double t = fabs(zeta) > 1e150 ? div_rn(0.5, zeta)
                                            : div_rn(copysign(1.0, zeta), fabs(zeta) + sqrt_rn(1.0 + zeta * zeta));
        const double c = div_rn(1.0, sqrt_rn(1.0 + t * t)), sn = c * t;
#pragma unroll
        for (int i = 0; i < 5; ++i) {
          const double ap = A[i][p], aq = A[i][q];
          A[i][p] = c * ap - sn * aq;
          A[i][q] = sn * ap + c * aq;
        }
      }
    if (!rotated) break;
  }
  double sv[5], smax = 0.0;
#pragma unroll
  for (int j = 0; j < 5; ++j) {
    double n2 = 0.0;
#pragma unroll
    for (int i = 0; i < 5; ++i) n2 += A[i][j] * A[i][j];
    sv[j] = sqrt_rn(n2);
    if (sv[j] > smax) smax = sv[j];
  }
  int rank = 0;
#pragma unroll
  for (int j = 0; j < 5; ++j)
    if (sv[j] > smax * 5.0 * kEps) ++rank;
  return rank;
}

__device__ __forceinline__ bool full_rank5(const double (&M)[5][5], const double (&LU)[5][5], const int (&piv)[5],
                                           bool lu_ok) {
  if (lu_ok) {
    double X[5][5];
#pragma unroll
    for (int i = 0; i < 5; ++i)
#pragma unroll
      for (int j = 0; j < 5; ++j) X[i][j] = i == j ? 1.0 : 0.0;
    lu5_solve<5>(LU, piv, X);
    double na = 0.0, ni = 0.0;
#pragma unroll
    for (int i = 0; i < 5; ++i)
#pragma unroll
      for (int j = 0; j < 5; ++j) {
        na += M[i][j] * M[i][j];
        ni += X[i][j] * X[i][j];
      }
    const double kappa = sqrt_rn(na) * sqrt_rn(ni);
    if (isfinite(kappa) && kappa < 1e12) return true;
  }
  return jacobi_rank5(M) == 5;
}

// Linear gradient and limiter factors of one cell (_kernels.py:240-273 and
// 10-67), the same arithmetic as the exact linear kernel.
template <int LIMITER>
__device__ __forceinline__ void linear_cell(const DevGeom& g, const double* __restrict__ P, int c,
                                            const double (&pv)[4], double (&gx)[4], double (&gy)[4],
                                            double (&phi)[4]) {
  double lo[4], hi[4];
#pragma unroll
  for (int v = 0; v < 4; ++v) {
    gx[v] = gy[v] = 0.0;
    lo[v] = hi[v] = pv[v];
    phi[v] = 1.0;
  }
  const int e0 = g.grad_ptr[c], e1 = g.grad_ptr[c + 1];
  for (int e = e0; e < e1; ++e) {
    const St4 q = ld4(P + 4 * (size_t)g.grad_nb[e]);
    const double qv[4] = {q.a, q.b, q.c, q.d};
    const double cx = g.grad_cx[e], cy = g.grad_cy[e];
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const double d = qv[v] - pv[v];
      gx[v] = gx[v] + cx * d;
      gy[v] = gy[v] + cy * d;
      if (icmp::lt(qv[v], lo[v])) lo[v] = qv[v];
      if (icmp::lt(hi[v], qv[v])) hi[v] = qv[v];
    }
  }
  if (g.n_gradient == 0) return;  // _limited_gradients: zeros and ones (solver.py:2298-2302)
  const int s0 = g.lim_ptr[c], s1 = g.lim_ptr[c + 1];
  for (int s = s0; s < s1; ++s) {
    const double2 d = g.lim_d[s];
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const double inc = gx[v] * d.x + gy[v] * d.y;
      const double f = limiter_face_factor<LIMITER>(pv[v], inc, lo[v], hi[v], limiter_tolerance(pv[v]));
      if (icmp::lt_nonneg(f, phi[v])) phi[v] = f;
    }
  }
}

// The linear fields of the reference (mcfd_reconstruction), one thread per cell.
template <int LIMITER>
__global__ void __launch_bounds__(kBlock) k_linear_fields(DevGeom g, const double* __restrict__ P,
                                                          double* __restrict__ grad_out,
                                                          double* __restrict__ fac_out) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= g.n_cells) return;
  const St4 p = ld4(P + 4 * (size_t)c);
  const double pv[4] = {p.a, p.b, p.c, p.d};
  double gx[4], gy[4], phi[4];
  linear_cell<LIMITER>(g, P, c, pv, gx, gy, phi);
#pragma unroll
  for (int v = 0; v < 4; ++v) {
    grad_out[8 * (size_t)c + 2 * v] = gx[v];
    grad_out[8 * (size_t)c + 2 * v + 1] = gy[v];
    fac_out[4 * (size_t)c + v] = phi[v];
  }
}

// Everything of a cell's fit that depends on the mesh alone.  The normal
// matrix, its LU, the inverse of the rank gate and the weights were some 85 %
// of the former one-kernel reconstruction's operations; they are the same for
// every state, so they are computed once, when the geometry is created.
// fit: [kParFit][C], the LU row by row (25), the fixed-point reciprocals of
// its diagonal (5), the scale, its square and their reciprocals (4); rec:
// [entries][6], the weight x basis products in pivoted row order and the
// neighbour's index; full: whether the cell passes the rank gate.
__global__ void __launch_bounds__(kBlock) k_parabolic_plan(DevGeom g, double* __restrict__ fit,
                                                           double* __restrict__ rec, int* __restrict__ full_out) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= g.n_cells) return;
  const int e0 = g.par_ptr[c], e1 = g.par_ptr[c + 1];
  double scale = 0.0;
  for (int e = e0; e < e1; ++e) {
    const double2 d = g.par_d[e];
    const double a = fabs(d.x), b = fabs(d.y);
    const double m = a >= b ? a : b;
    if (m > scale) scale = m;
  }
  if (!(scale >= 1e-300)) scale = 1e-300;
  auto products = [&](int e, double (&dd)[5], double (&wd)[5]) {
    const double2 d = g.par_d[e];
    const double nx = div_rn(d.x, scale), ny = div_rn(d.y, scale);
    dd[0] = nx;
    dd[1] = ny;
    dd[2] = 0.5 * (nx * nx);
    dd[3] = nx * ny;
    dd[4] = 0.5 * (ny * ny);
    const double r2 = nx * nx + ny * ny;
    const double w = div_rn(1.0, r2 >= 1e-300 ? r2 : 1e-300);
#pragma unroll
    for (int i = 0; i < 5; ++i) wd[i] = w * dd[i];
  };
  double M[5][5];
#pragma unroll
  for (int i = 0; i < 5; ++i)
#pragma unroll
    for (int j = 0; j < 5; ++j) M[i][j] = 0.0;
  for (int e = e0; e < e1; ++e) {
    double dd[5], wd[5];
    products(e, dd, wd);
#pragma unroll
    for (int i = 0; i < 5; ++i)
#pragma unroll
      for (int j = 0; j < 5; ++j) M[i][j] += wd[i] * dd[j];
  }
  double LU[5][5];
#pragma unroll
  for (int i = 0; i < 5; ++i)
#pragma unroll
    for (int j = 0; j < 5; ++j) LU[i][j] = M[i][j];
  int piv[5] = {0, 1, 2, 3, 4};
  const bool ok = lu5(LU, piv);
  full_out[c] = full_rank5(M, LU, piv, ok) ? 1 : 0;
  const size_t C = g.n_cells;
#pragma unroll
  for (int i = 0; i < 5; ++i) {
#pragma unroll
    for (int j = 0; j < 5; ++j) fit[(5 * i + j) * C + c] = LU[i][j];
    fit[(25 + i) * C + c] = __longlong_as_double((long long)recip_fixed(LU[i][i]));
  }
  const double sc2 = scale * scale;
  fit[30 * C + c] = scale;
  fit[31 * C + c] = sc2;
  fit[32 * C + c] = __longlong_as_double((long long)recip_fixed(scale));
  fit[33 * C + c] = __longlong_as_double((long long)recip_fixed(sc2));
  // the products' row of each pivoted row, by the solve's own interchanges
  // (a failed LU leaves no solve: any order)
  for (int e = e0; e < e1; ++e) {
    double dd[5], wd[5], b[5][1];
    products(e, dd, wd);
#pragma unroll
    for (int i = 0; i < 5; ++i) b[i][0] = wd[i];
    swap_rows<0, 1>(b, piv[0]);
    swap_rows<1, 1>(b, piv[1]);
    swap_rows<2, 1>(b, piv[2]);
    swap_rows<3, 1>(b, piv[3]);
    double2* dst = reinterpret_cast<double2*>(rec + 6 * (size_t)e);
    dst[0] = make_double2(b[0][0], b[1][0]);
    dst[1] = make_double2(b[2][0], b[3][0]);
    dst[2] = make_double2(b[4][0], __longlong_as_double((long long)g.par_nb[e]));
  }
}

// Products of the right-hand side that run on the integer pipe (mul_rn, the
// same IEEE product): the first MCFD_PAR_INT_MUL of an entry's five.  RK3 step
// of the 181 x 181 vortex with 0 / 2 / 5 of them: 478 / 437 / 396 us; and with 6
// / 8 / 10 / 11 resident 128-thread blocks 385 / 386 / 392 / 396 us (on 36,100
// cells 412 / 412 / 418 / 446).
#ifndef MCFD_PAR_INT_MUL
#define MCFD_PAR_INT_MUL 5
#endif
#ifndef MCFD_PAR_MIN_BLOCKS
#define MCFD_PAR_MIN_BLOCKS 6
#endif
template <int I>
__device__ __forceinline__ double rhs_mul(double a, double b) {
  if constexpr (I < MCFD_PAR_INT_MUL) return mul_rn(a, b);
  else return a * b;
}

// Limiter factor and face states (or fields) of one variable, its increments
// kept for up to four limiter entries (KEPT; else any count, recomputing the
// increments).  The two sums of the increment associate differently, as the
// reference's limiter and its _reconstruct do; they share their products.
// The entries' loop stays a loop: a warp that mixes triangles and quads runs
// each entry once (bodies compiled for 3 and for 4 entries ran one after the
// other), and the body, some 300 instructions with its fixed-point quotients,
// stays in the instruction cache, which warps at different places of the
// unrolled code kept missing (7 of 24 stall cycles an issue).  FP64
// instructions of a warp are 64 cycles apart either way, so nothing is lost by
// the order.  RK3 step of the 181 x 181 vortex 523 us with the bodies for 3 and
// 4 entries, 514 / 427 / 386 us unrolled by 4 / 2 / 1.
template <int LIMITER, bool KEPT>
__device__ __forceinline__ double parabolic_faces(const DevGeom& g, double* __restrict__ recon, int v, double pv,
                                                  int s0, int s1, double gx, double gy, double kxx, double kxy,
                                                  double kyy, double lo, double hi) {
  const double tol = limiter_tolerance(pv);
  const double hxx = 0.5 * kxx, hyy = 0.5 * kyy;
  double phi = 1.0;
  if constexpr (KEPT) {
    const int n = s1 - s0;
    double o0 = 0.0, o1 = 0.0, o2 = 0.0, o3 = 0.0;
#pragma unroll 1
    for (int k = 0; k < 4; ++k) {
      if (k >= n) break;
      const double2 d = g.lim_d[s0 + k];
      const double t1 = gx * d.x + gy * d.y, txx = hxx * (d.x * d.x), txy = kxy * (d.x * d.y),
                   tyy = hyy * (d.y * d.y);
      const double out = t1 + ((txx + txy) + tyy);
      const double f = limiter_face_factor<LIMITER>(pv, ((t1 + txx) + txy) + tyy, lo, hi, tol);
      if (icmp::lt_nonneg(f, phi)) phi = f;
      o0 = k == 0 ? out : o0;
      o1 = k == 1 ? out : o1;
      o2 = k == 2 ? out : o2;
      o3 = k == 3 ? out : o3;
    }
    if (recon) {
      const double kept[4] = {o0, o1, o2, o3};
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (k < n) recon[4 * (size_t)g.lim_slot[s0 + k] + v] = pv + phi * kept[k];
    }
  } else {
    for (int s = s0; s < s1; ++s) {
      const double2 d = g.lim_d[s];
      const double inc = gx * d.x + gy * d.y + hxx * (d.x * d.x) + kxy * (d.x * d.y) + hyy * (d.y * d.y);
      const double f = limiter_face_factor<LIMITER>(pv, inc, lo, hi, tol);
      if (icmp::lt_nonneg(f, phi)) phi = f;
    }
    if (recon) {
      for (int s = s0; s < s1; ++s) {
        const double2 d = g.lim_d[s];
        double inc = gx * d.x + gy * d.y;
        inc += hxx * (d.x * d.x) + kxy * (d.x * d.y) + hyy * (d.y * d.y);
        recon[4 * (size_t)g.lim_slot[s] + v] = pv + phi * inc;
      }
    }
  }
  return phi;
}

// One thread per (cell, variable): the variables of a cell are independent
// given the plan, and four short threads leave room for the warps that hide
// the 64-cycle FP64 latency (the former thread per cell held 246 registers).
// Bound by FP64 issue.  RK3 step of the 181 x 181 mixed vortex (49,141 cells):
// 465 us per reconstruction with the plan recomputed in it, 142 us with the
// plan, 96 us now; the step 1,372, 532 and 385 us.
template <int LIMITER, bool FIELDS>
__global__ void __launch_bounds__(kBlock, MCFD_PAR_MIN_BLOCKS) k_reconstruct_parabolic(DevGeom g, const double* __restrict__ P,
                                                                  double* __restrict__ recon,
                                                                  double* __restrict__ grad_out,
                                                                  double* __restrict__ curv_out,
                                                                  double* __restrict__ fac_out) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int c = t >> 2, v = t & 3;
  if (c >= g.n_cells) return;
  const double pv = P[4 * (size_t)c + v];
  const int s0 = g.lim_ptr[c], s1 = g.lim_ptr[c + 1];
  double gx = 0.0, gy = 0.0, kxx = 0.0, kxy = 0.0, kyy = 0.0, phi, lo = pv, hi = pv;
  bool limited = true;
  if (g.n_parabolic > 0 && g.par_full[c]) {
    double b[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    for (int e = g.par_ptr[c], e1 = g.par_ptr[c + 1]; e < e1; ++e) {
      const double2* r = reinterpret_cast<const double2*>(g.par_rec + 6 * (size_t)e);
      const double2 r0 = r[0], r1 = r[1], r2 = r[2];
      const double q = P[4 * (size_t)(int)__double_as_longlong(r2.y) + v];
      const double diff = q - pv;
      if (icmp::lt(q, lo)) lo = q;
      if (icmp::lt(hi, q)) hi = q;
      b[0] += rhs_mul<0>(r0.x, diff);
      b[1] += rhs_mul<1>(r0.y, diff);
      b[2] += rhs_mul<2>(r1.x, diff);
      b[3] += rhs_mul<3>(r1.y, diff);
      b[4] += rhs_mul<4>(r2.x, diff);
    }
    const size_t C = g.n_cells;
    const double* f = g.par_fit + c;
#pragma unroll
    for (int i = 1; i < 5; ++i)
#pragma unroll
      for (int j = 0; j < i; ++j) b[i] = b[i] - f[(5 * i + j) * C] * b[j];
#pragma unroll
    for (int i = 4; i >= 0; --i) {
#pragma unroll
      for (int j = i + 1; j < 5; ++j) b[i] = b[i] - f[(5 * i + j) * C] * b[j];
      b[i] = div_rn_recip(b[i], f[(5 * i + i) * C], (unsigned long long)__double_as_longlong(f[(25 + i) * C]));
    }
    const double sc = f[30 * C], sc2 = f[31 * C];
    const unsigned long long x1 = (unsigned long long)__double_as_longlong(f[32 * C]),
                             x2 = (unsigned long long)__double_as_longlong(f[33 * C]);
    gx = div_rn_recip(b[0], sc, x1);
    gy = div_rn_recip(b[1], sc, x1);
    kxx = div_rn_recip(b[2], sc2, x2);
    kxy = div_rn_recip(b[3], sc2, x2);
    kyy = div_rn_recip(b[4], sc2, x2);
  } else {  // linear gradient and limiter (linear_cell, one variable): zero curvature
    for (int e = g.grad_ptr[c], e1 = g.grad_ptr[c + 1]; e < e1; ++e) {
      const double q = P[4 * (size_t)g.grad_nb[e] + v];
      const double d = q - pv;
      gx = gx + g.grad_cx[e] * d;
      gy = gy + g.grad_cy[e] * d;
      if (icmp::lt(q, lo)) lo = q;
      if (icmp::lt(hi, q)) hi = q;
    }
    limited = g.n_gradient > 0;
  }
  double* out = FIELDS ? nullptr : recon;
  if (!limited) {  // no gradient entries at all: zeros and ones (solver.py:2298-2302)
    phi = 1.0;
    if (!FIELDS)
      for (int s = s0; s < s1; ++s) recon[4 * (size_t)g.lim_slot[s] + v] = pv + 0.0;
  } else if (s1 - s0 <= 4) {
    phi = parabolic_faces<LIMITER, true>(g, out, v, pv, s0, s1, gx, gy, kxx, kxy, kyy, lo, hi);
  } else {
    phi = parabolic_faces<LIMITER, false>(g, out, v, pv, s0, s1, gx, gy, kxx, kxy, kyy, lo, hi);
  }
  if (FIELDS) {
    grad_out[8 * (size_t)c + 2 * v] = gx;
    grad_out[8 * (size_t)c + 2 * v + 1] = gy;
    fac_out[4 * (size_t)c + v] = phi;
    if (curv_out) {
      curv_out[12 * (size_t)c + 3 * v] = kxx;
      curv_out[12 * (size_t)c + 3 * v + 1] = kxy;
      curv_out[12 * (size_t)c + 3 * v + 2] = kyy;
    }
  }
}

inline int blocks_for(int n) { return (n + kBlock - 1) / kBlock; }

template <bool FIELDS>
cudaError_t launch_parabolic(const DevGeom& g, int limiter, const double* P, double* recon, double* grad, double* curv,
                             double* fac, cudaStream_t s) {
  if (g.n_cells == 0) return cudaSuccess;
  const int b = (int)((4LL * g.n_cells + kBlock - 1) / kBlock);
  count_launch();
  switch (limiter) {
    case 0: k_reconstruct_parabolic<0, FIELDS><<<b, kBlock, 0, s>>>(g, P, recon, grad, curv, fac); break;
    case 1: k_reconstruct_parabolic<1, FIELDS><<<b, kBlock, 0, s>>>(g, P, recon, grad, curv, fac); break;
    case 2: k_reconstruct_parabolic<2, FIELDS><<<b, kBlock, 0, s>>>(g, P, recon, grad, curv, fac); break;
    default: k_reconstruct_parabolic<3, FIELDS><<<b, kBlock, 0, s>>>(g, P, recon, grad, curv, fac); break;
  }
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_parabolic_plan(const DevGeom& g, double* fit, double* rec, int* full, cudaStream_t s) {
  if (g.n_cells == 0 || g.n_parabolic == 0) return cudaSuccess;
  count_launch();
  k_parabolic_plan<<<blocks_for(g.n_cells), kBlock, 0, s>>>(g, fit, rec, full);
  return cudaGetLastError();
}

cudaError_t launch_reconstruct_parabolic(const DevGeom& g, const mcfd_config& cfg, const double* P, double* recon,
                                         cudaStream_t s) {
  return launch_parabolic<false>(g, cfg.limiter, P, recon, nullptr, nullptr, nullptr, s);
}

cudaError_t launch_reconstruction_fields(const DevGeom& g, const mcfd_config& cfg, const double* P, double* grad,
                                         double* curv, double* fac, cudaStream_t s) {
  if (cfg.reconstruction == MCFD_RECON_MUSCL_PARABOLIC)
    return launch_parabolic<true>(g, cfg.limiter, P, nullptr, grad, curv, fac, s);
  if (g.n_cells == 0) return cudaSuccess;
  const int b = blocks_for(g.n_cells);
  count_launch();
  switch (cfg.limiter) {
    case 0: k_linear_fields<0><<<b, kBlock, 0, s>>>(g, P, grad, fac); break;
    case 1: k_linear_fields<1><<<b, kBlock, 0, s>>>(g, P, grad, fac); break;
    case 2: k_linear_fields<2><<<b, kBlock, 0, s>>>(g, P, grad, fac); break;
    default: k_linear_fields<3><<<b, kBlock, 0, s>>>(g, P, grad, fac); break;
  }
  return cudaGetLastError();
}

}  // namespace mcfd
