// osb_math.cuh -- device numerics of the residual path (characteristic LLF WENO/TENO flux,
// central-4 operators), templated on the arithmetic type T (double: FP64 path, float: FP32
// residual path).
//
// Everything is written in the local frame of the sweep direction: the conserved state of a
// point is (rho, m_n, m_t1[, m_t2], E) with m_n the momentum along the sweep.  For a Cartesian
// direction the eigensystem of physical_models/euler_eigensystem.py:53-166 with k = e_d is the
// k = e_0 system with the momentum components permuted (a cyclic permutation in 3D, a swap in
// 2D, which only flips the sign of one vorticity eigenvector); the characteristic flux is
// invariant under those relabelings, so one set of formulas serves every direction.
#pragma once
#include <cuda_runtime.h>
#include <math.h>

namespace osb {

enum { SCH_WENO5_JS = 1, SCH_WENO5_Z = 2, SCH_TENO5 = 3, SCH_TENO6 = 4, SCH_CENTRAL4 = 5 };
enum { AVG_SIMPLE = 0, AVG_ROE = 1 };

template <typename T> struct Lit;
template <> struct Lit<double> {
  static __device__ __forceinline__ double c(double x) { return x; }
};
template <> struct Lit<float> {
  static __device__ __forceinline__ float c(double x) { return (float)x; }
};
#define L_(x) Lit<T>::c(x)

struct SchemeParams {
  double gama;
  double teno_eps;   // TENO epsilon (reference value 1e-40)
  double teno_ct;    // TENO cut-off
  double sfc;        // shock_filter_control
  double eps32_rel;  // FP32 path: epsilon relative to the stencil's mean square
  double ig1;        // 1 / (gama - 1)
  // the same constants rounded to FP32 on the host (scheme_params): an FP32 kernel that
  // converted the doubles itself would run the conversions on the FP64 pipe, and under the
  // sweeps' register cap the compiler re-derives such values inside the loop instead of
  // keeping them in registers (measured: six FP64-pipe conversions per point in the FP32 y/z
  // sweeps, 34 % FP64-pipe activity)
  float gama_f, g1_f, ig1_f, teno_eps_f, teno_ct_f, sfc_f, eps32_rel_f;
};

__host__ __device__ inline SchemeParams scheme_params(double gama, double teno_eps, double teno_ct, double sfc,
                                                      double eps32_rel) {
  SchemeParams p;
  p.gama = gama;
  p.teno_eps = teno_eps;
  p.teno_ct = teno_ct;
  p.sfc = sfc;
  p.eps32_rel = eps32_rel;
  p.ig1 = 1.0 / (gama - 1.0);
  p.ig1_f = (float)p.ig1;
  p.gama_f = (float)gama;
  p.g1_f = (float)(gama - 1.0);
  p.teno_eps_f = (float)teno_eps;
  p.teno_ct_f = (float)teno_ct;
  p.sfc_f = (float)sfc;
  p.eps32_rel_f = (float)eps32_rel;
  return p;
}

// The constants in the arithmetic type of a kernel.
template <typename T>
struct SP;
template <>
struct SP<double> {
  double gama, g1, ig1, teno_eps, teno_ct, sfc, eps32_rel;
  float teno_ct_f;
  __device__ __forceinline__ explicit SP(const SchemeParams& p)
      : gama(p.gama), g1(p.gama - 1.0), ig1(p.ig1), teno_eps(p.teno_eps), teno_ct(p.teno_ct), sfc(p.sfc),
        eps32_rel(p.eps32_rel), teno_ct_f(p.teno_ct_f) {}
};
template <>
struct SP<float> {
  float gama, g1, ig1, teno_eps, teno_ct, sfc, eps32_rel;
  __device__ __forceinline__ explicit SP(const SchemeParams& p)
      : gama(p.gama_f), g1(p.g1_f), ig1(p.ig1_f), teno_eps(p.teno_eps_f), teno_ct(p.teno_ct_f), sfc(p.sfc_f),
        eps32_rel(p.eps32_rel_f) {}
};

// ---------------------------------------------------------------------------------------
// FP64 reconstructions.
//
// GB300 issues one FP64 warp instruction per 16.3 cycles and SM, against 4 FP32 ones per cycle: an
// FP64 kernel of this path costs what its FP64 instructions cost, and the FP32 / integer work next
// to them is free up to about 60 instructions for each.  So the FP64 reconstruction is written for
// the fewest FP64 instructions: everything runs on the four differences d_j of the stencil, the
// result is f0 plus a combination of them, and
//  * TENO's 0/1 weights are decided in FP32 wherever an error bound says that FP64 decides alike
//    (teno5_mask), then select one of eight rows of constants: 8 FP64 instructions instead of
//    about 120;
//  * WENO's weights, which need all 53 bits, are brought over one common denominator: one division
//    instead of four, 45 - 50 FP64 instructions instead of about 130.

// 1/x for a finite normal x by Newton's iteration from the hardware's 20-bit estimate (two steps:
// 2^-20 -> 2^-40 -> rounding), without the special-case branches of the IEEE division.  It gave the IEEE
// quotient for each of 2^30 random x from 1e-90 to 1e90.
__device__ __forceinline__ double rcp_newton(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  r = __fma_rn(r, __fma_rn(-x, r, 1.0), r);
  return __fma_rn(r, __fma_rn(-x, r, 1.0), r);
}
__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// 2^32 x truncated to FP32 with integer operations (relative error below 2^-23): zero below 2^-158,
// infinity from 2^96, so that the squares of differences from 1e-29 to 1e9 stay in FP32's range.
__device__ __forceinline__ float d2f_scaled(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const unsigned h = hi & 0x7fffffffu;
  unsigned b = __funnelshift_l(lo, hi, 3) - (864u << 23);
  b = h < (865u << 20) ? 0u : (h >= (1119u << 20) ? 0x7f800000u : b);
  return __uint_as_float(b | (hi & 0x80000000u));
}

// The TENO5 decision in FP64 (teno.py:419-477): bit r is set where stencil r is kept.
static __device__ __noinline__ unsigned teno5_mask_f64(double d1, double d2, double d3, double d4, double eps, double ct) {
  const double c0 = d3 - d2, s0 = d2 + d3, c1 = d4 - d3, s1 = c1 - 2.0 * d3, c2 = d2 - d1, s2 = c2 + 2.0 * d2;
  const double b0 = 0.25 * s0 * s0 + (13.0 / 12.0) * c0 * c0;
  const double b1 = 0.25 * s1 * s1 + (13.0 / 12.0) * c1 * c1;
  const double b2 = 0.25 * s2 * s2 + (13.0 / 12.0) * c2 * c2;
  const double tau = fabs(b0 - b2);
  const double t0 = 1.0 + tau / (eps + b0), t1 = 1.0 + tau / (eps + b1), t2 = 1.0 + tau / (eps + b2);
  const double a0 = t0 * t0 * t0 * t0 * t0 * t0, a1 = t1 * t1 * t1 * t1 * t1 * t1, a2 = t2 * t2 * t2 * t2 * t2 * t2;
  const double inv = 1.0 / (a0 + a1 + a2);
  return (a0 * inv < ct ? 0u : 1u) | (a1 * inv < ct ? 0u : 2u) | (a2 * inv < ct ? 0u : 4u);
}

// The TENO5 decision (stencils [-1,0,1], [0,1,2], [-2,-1,0]) from the FP64 differences d1..d4 of
// neighbouring values, in FP32 with an error bound.  eps32 is epsilon times 2^64 (d2f_scaled).
//
// Each indicator is a definite quadratic form of its stencil's two differences (condition number
// at most 19), so truncating the differences to FP32 leaves each with a relative error below
// 1.1e-5, whatever the scale of the other stencils.  With u_r = eps + beta_r and u_m the smallest, the
// cut-off compares x_r^6 with C_T sum x^6, x_r = (u_r + tau) u_m / ((u_m + tau) u_r) <= 1: relative
// error E <= 6.6e-5 F for x_r, F = (u_0 + u_2 + tau) / (u_m + tau), 12 E for the comparison.  These are
// first-order bounds, so they serve only while they are small: F above 500 (outer indicators that
// agree beside a vanishing third: tau may be FP32 rounding alone) goes to FP64, as does a comparison
// closer than 1e-3 F, or one that left FP32's range (infinity, NaN, or an indicator above 1e37, whose
// reciprocal would flush to zero).  At F = 500, E = 0.033: x_r^6 / sum x^6 is then within a factor of
// 1.033^6 / 0.967^6 = 1.49 < 1 + 1e-3 F of its FP64 value.  About one window in 6 000 goes to FP64 on random
// values; without the limit on F, 983 of 170 000 nearly tied windows called sure were decided wrongly.
__device__ __forceinline__ unsigned teno5_mask(double d1, double d2, double d3, double d4, double eps, float eps32,
                                               double ct, float ct32) {
  const float e1 = d2f_scaled(d1), e2 = d2f_scaled(d2), e3 = d2f_scaled(d3), e4 = d2f_scaled(d4);
  const float c0 = e3 - e2, s0 = e2 + e3, c1 = e4 - e3, s1 = c1 - 2.0f * e3, c2 = e2 - e1, s2 = c2 + 2.0f * e2;
  const float k = (float)(13.0 / 12.0);
  const float u0 = 0.25f * s0 * s0 + (k * c0 * c0 + eps32);
  const float u1 = 0.25f * s1 * s1 + (k * c1 * c1 + eps32);
  const float u2 = 0.25f * s2 * s2 + (k * c2 * c2 + eps32);
  const float tau = fabsf(u0 - u2);
  const float um = fminf(u0, fminf(u1, u2));
  const float it = rcp_approx(um + tau);
  float r0 = ((u0 + tau) * it) * (um * rcp_approx(u0));
  float r1 = ((u1 + tau) * it) * (um * rcp_approx(u1));
  float r2 = ((u2 + tau) * it) * (um * rcp_approx(u2));
  r0 = r0 * r0 * r0; r0 = r0 * r0;
  r1 = r1 * r1 * r1; r1 = r1 * r1;
  r2 = r2 * r2 * r2; r2 = r2 * r2;
  const float cs = ct32 * (r0 + r1 + r2);
  const float f = 1e-3f * ((u0 + u2 + tau) * it), g = cs * f;
  const float lo = cs - g, hi = cs + g;
  const bool k0 = r0 > hi, k1 = r1 > hi, k2 = r2 > hi;
  const bool sure = (k0 || r0 < lo) && (k1 || r1 < lo) && (k2 || r2 < lo) && f < 0.5f && fmaxf(u0, fmaxf(u1, u2)) < 1e37f;
  if (!sure) return teno5_mask_f64(d1, d2, d3, d4, eps, ct);
  return (k0 ? 1u : 0u) | (k1 ? 2u : 0u) | (k2 ? 4u : 0u);
}

// f0 + sum_j row[j] d_j is the TENO5 reconstruction with the stencils of a mask: with the kept
// weights (11/20, 4/10, 1/20) normalised to W_r, row = (-W2/3, W0/6 + 5 W2/6, W0/3 + 2 W1/3, -W1/6).
// No stencil kept (a cut-off above 1/3): 0/0, as the weights' own normalisation gives.
#define OSB_TENO5_ROW(a, b, c, s)   { -(c) / 3.0 / (s), ((a) / 6.0 + 5.0 * (c) / 6.0) / (s), ((a) / 3.0 + 2.0 * (b) / 3.0) / (s), -(b) / 6.0 / (s) }
static __device__ const double teno5_rows[8][4] = {
    {__builtin_nan(""), __builtin_nan(""), __builtin_nan(""), __builtin_nan("")},
    OSB_TENO5_ROW(1.0, 0.0, 0.0, 1.0),   OSB_TENO5_ROW(0.0, 1.0, 0.0, 1.0),   OSB_TENO5_ROW(11.0, 8.0, 0.0, 19.0),
    OSB_TENO5_ROW(0.0, 0.0, 1.0, 1.0),   OSB_TENO5_ROW(11.0, 0.0, 1.0, 12.0), OSB_TENO5_ROW(0.0, 8.0, 1.0, 9.0),
    OSB_TENO5_ROW(11.0, 8.0, 1.0, 20.0)};
#undef OSB_TENO5_ROW

// Blocks whose flux keeps the generated order of operations (projections, primitives, divisions and
// indicators) in both precisions: recon5_ieee says why these and what the others differ by.
template <int ND, int SCH>
__host__ __device__ constexpr bool generated_order() {
  return ND <= 2 && (SCH == SCH_TENO5 || SCH == SCH_TENO6);
}

// Fifth-order reconstruction in the generated order with IEEE divisions, FP64.  It serves
//   - values beyond the range of recon5_f64's common denominator,
//   - TENO5 on 1D and 2D blocks (generated_order; TENO6 keeps the order too).  Beside a front in exactly
//     uniform gas the outer indicators of a five-point window can tie while the middle one is zero to
//     rounding: tau is then the rounding of b0 - b2, and whether it is exactly zero decides if TENO5
//     keeps the outer stencils.  No order of the operations decides such a tie better than another: on
//     shear layers extruded to 3D, 9 steps, the generated order lies 3e-6 .. 3e-4 of the largest value
//     from plain IEEE arithmetic (median over 12 layers at three sizes), recon5_f64 5e-7 .. 6e-5; FP32 1e-3
//     and 1e-3.  1D and 2D blocks keep the order of the generated solver, so that their results are
//     the ones they always were; 3D blocks take recon5_f64 (a step of the 128^3 TENO5 vortex in the
//     generated order 68 ms, with it 17).
// WENO5-Z has such ties at zero-gradient ends: the mirrored window (x, y, y, y, x) has b0 = b2 and b1 = 0.  The
// differences make tau exactly zero there and the weights linear; the generated order does in 37 - 49 % of
// such windows and takes stencil [-1, 0, 1] alone in the others.
template <int SCH>
__device__ __forceinline__ double recon5_ieee(double fm2, double fm1, double f0, double fp1, double fp2, double eps,
                                              double ct) {
  if (SCH == SCH_TENO5) {
    const double s0 = fm1 - fp1, c0 = fm1 - 2.0 * f0 + fp1;
    const double s1 = 3.0 * f0 - 4.0 * fp1 + fp2, c1 = f0 - 2.0 * fp1 + fp2;
    const double s2 = fm2 - 4.0 * fm1 + 3.0 * f0, c2 = fm2 - 2.0 * fm1 + f0;
    const double b0 = 0.25 * s0 * s0 + (13.0 / 12.0) * c0 * c0;
    const double b1 = 0.25 * s1 * s1 + (13.0 / 12.0) * c1 * c1;
    const double b2 = 0.25 * s2 * s2 + (13.0 / 12.0) * c2 * c2;
    const double tau = fabs(b0 - b2);
    const double t0 = 1.0 + tau / (eps + b0), t1 = 1.0 + tau / (eps + b1), t2 = 1.0 + tau / (eps + b2);
    const double a0 = t0 * t0 * t0 * t0 * t0 * t0;
    const double a1 = t1 * t1 * t1 * t1 * t1 * t1;
    const double a2 = t2 * t2 * t2 * t2 * t2 * t2;
    const double inv = 1.0 / (a0 + a1 + a2);
    const double w0 = (11.0 / 20.0) * ((a0 * inv < ct) ? 0.0 : 1.0), w1 = (4.0 / 10.0) * ((a1 * inv < ct) ? 0.0 : 1.0),
                 w2 = (1.0 / 20.0) * ((a2 * inv < ct) ? 0.0 : 1.0);
    const double iw = 1.0 / (w0 + w1 + w2);
    const double e0 = -(1.0 / 6.0) * fm1 + (5.0 / 6.0) * f0 + (2.0 / 6.0) * fp1;
    const double e1 = (2.0 / 6.0) * f0 + (5.0 / 6.0) * fp1 - (1.0 / 6.0) * fp2;
    const double e2 = (2.0 / 6.0) * fm2 - (7.0 / 6.0) * fm1 + (11.0 / 6.0) * f0;
    return (w0 * e0 + w1 * e1 + w2 * e2) * iw;
  }
  const double c0 = f0 - 2.0 * fp1 + fp2, s0 = 3.0 * f0 - 4.0 * fp1 + fp2;
  const double c1 = fm1 - 2.0 * f0 + fp1, s1 = fm1 - fp1;
  const double c2 = fm2 - 2.0 * fm1 + f0, s2 = fm2 - 4.0 * fm1 + 3.0 * f0;
  const double b0 = (13.0 / 12.0) * c0 * c0 + 0.25 * s0 * s0;
  const double b1 = (13.0 / 12.0) * c1 * c1 + 0.25 * s1 * s1;
  const double b2 = (13.0 / 12.0) * c2 * c2 + 0.25 * s2 * s2;
  double a0, a1, a2;
  if (SCH == SCH_WENO5_Z) {
    const double tau = fabs(b0 - b2);
    const double r0 = tau / (eps + b0), r1 = tau / (eps + b1), r2 = tau / (eps + b2);
    a0 = 0.3 * (1.0 + r0 * r0);
    a1 = 0.6 * (1.0 + r1 * r1);
    a2 = 0.1 * (1.0 + r2 * r2);
  } else {
    a0 = 0.3 / ((eps + b0) * (eps + b0));
    a1 = 0.6 / ((eps + b1) * (eps + b1));
    a2 = 0.1 / ((eps + b2) * (eps + b2));
  }
  const double inv = 1.0 / (a0 + a1 + a2);
  const double e0 = (1.0 / 3.0) * f0 + (5.0 / 6.0) * fp1 - (1.0 / 6.0) * fp2;
  const double e1 = -(1.0 / 6.0) * fm1 + (5.0 / 6.0) * f0 + (1.0 / 3.0) * fp1;
  const double e2 = (1.0 / 3.0) * fm2 - (7.0 / 6.0) * fm1 + (11.0 / 6.0) * f0;
  return (a0 * inv) * e0 + (a1 * inv) * e1 + (a2 * inv) * e2;
}
template <int SCH>
static __device__ __noinline__ double recon5_wide(double fm2, double fm1, double f0, double fp1, double fp2, double eps) {
  return recon5_ieee<SCH>(fm2, fm1, f0, fp1, fp2, eps, 0.0);
}

// The epsilons of a scheme in the units of the reconstructed values: a caller that reconstructs
// s f instead of f passes s^2.
struct ReconEps {
  double eps;   // epsilon itself
  float eps32;  // times 2^64 (teno5_mask)
};
template <int SCH>
__device__ __forceinline__ ReconEps recon_eps(double teno_eps, double s2) {
  ReconEps e;
  if (SCH == SCH_TENO5) {
    e.eps = teno_eps * s2;
    e.eps32 = d2f_scaled(e.eps * 4294967296.0);
  } else {
    e.eps = SCH == SCH_WENO5_Z ? 1.0e-40 * s2 : 1.0e-6 * s2;
    e.eps32 = 0.f;
  }
  return e;
}

// Fifth-order reconstruction at the right face of f0, FP64 (see recon5 for the formulas).
template <int SCH>
__device__ __forceinline__ double recon5_f64(double fm2, double fm1, double f0, double fp1, double fp2,
                                             const ReconEps& e, double ct, float ct32) {
  const double d1 = fm1 - fm2, d2 = f0 - fm1, d3 = fp1 - f0, d4 = fp2 - fp1;
  if (SCH == SCH_TENO5) {
    const double* row = teno5_rows[teno5_mask(d1, d2, d3, d4, e.eps, e.eps32, ct, ct32)];
    return __fma_rn(__ldg(row + 1), d2, __fma_rn(__ldg(row + 2), d3, __fma_rn(__ldg(row), d1, __fma_rn(__ldg(row + 3), d4, f0))));
  }
  // four times the indicators plus epsilon, of [0,1,2], [-1,0,1] and [-2,-1,0]
  const double c0 = d4 - d3, s0 = __fma_rn(-2.0, d3, c0), c1 = d3 - d2, s1 = d2 + d3, c2 = d2 - d1, s2 = __fma_rn(2.0, d2, c2);
  const double e4 = 4.0 * e.eps, k = 13.0 / 3.0;
  const double u0 = __fma_rn(k * c0, c0, __fma_rn(s0, s0, e4));
  const double u1 = __fma_rn(k * c1, c1, __fma_rn(s1, s1, e4));
  const double u2 = __fma_rn(k * c2, c2, __fma_rn(s2, s2, e4));
  const double p01 = u0 * u1, p02 = u0 * u2, p12 = u1 * u2;
  double a0, a1, a2;  // the weights times (u0 u1 u2)^2, without the factors 3/10, 6/10, 1/10
  if (SCH == SCH_WENO5_Z) {
    const double tau = fabs(u0 - u2), P = p01 * u2, P2 = P * P;
    const double v0 = tau * p12, v1 = tau * p02, v2 = tau * p01;
    a0 = __fma_rn(v0, v0, P2);
    a1 = __fma_rn(v1, v1, P2);
    a2 = __fma_rn(v2, v2, P2);
  } else {
    a0 = p12 * p12;
    a1 = p02 * p02;
    a2 = p01 * p01;
  }
  const double D = __fma_rn(6.0, a1, __fma_rn(3.0, a0, a2));
  // 10 w_r (e_r - f0): e0 - f0 = (4 d3 - d4) / 6, e1 - f0 = (d2 + 2 d3) / 6, e2 - f0 = (5 d2 - 2 d1) / 6
  const double g0 = __fma_rn(2.0, d3, -0.5 * d4), g1 = __fma_rn(2.0, d3, d2),
               g2 = __fma_rn(5.0 / 6.0, d2, -(1.0 / 3.0) * d1);
  const double Nn = __fma_rn(a0, g0, __fma_rn(a1, g1, a2 * g2));
  // Nn, D and 1 / D stay inside FP64's range for indicators between 1e-47 and 1e43; beyond
  // (values above 1e21) the generated form takes over
  const int de = (__double2hiint(D) >> 20) & 0x7ff;
  if (de < 64 || de > 1903) return recon5_wide<SCH>(fm2, fm1, f0, fp1, fp2, e.eps);
  return __fma_rn(Nn, rcp_newton(D), f0);
}

// ---------------------------------------------------------------------------------------
// Fifth-order reconstruction at the right face of f2 from f0..f4 (offsets -2..+2).
//   WENO5-JS / WENO5-Z: weno.py:71-121 (ENO coefficients, optimal weights 3/10, 3/5, 1/10),
//     139-206 (Jiang-Shu smoothness), 290-376 (JS alpha = d/(1e-6+b)^2; Z alpha =
//     d(1+(|b0-b2|/(1e-40+b))^2)).
//   TENO5: teno.py:96-217, 419-477 (stencils [-1,0,1],[0,1,2],[-2,-1,0], weights 11/20, 4/10,
//     1/20, tau = |b0-b2|, alpha = (1+tau/(eps+b))^6, cut-off alpha/sum < C_T).
// In the FP32 path the epsilon of WENO-Z / TENO (1e-40, below the FP32 normal range) is
// replaced by eps32_rel * mean(f^2) + 1e-30, and TENO's alpha ratios are formed from
// t_r/t_max so that (1+tau/(eps+b))^6 cannot overflow.  The FP64 path takes recon5_f64.
template <typename T, int SCH>
__device__ __forceinline__ T recon5(T fm2, T fm1, T f0, T fp1, T fp2, const SP<T>& sp) {
  constexpr bool F32 = sizeof(T) == 4;
  if constexpr (!F32) {
    return recon5_f64<SCH>(fm2, fm1, f0, fp1, fp2, recon_eps<SCH>(sp.teno_eps, 1.0), sp.teno_ct, sp.teno_ct_f);
  }
  if (SCH == SCH_TENO5) {
    T s0 = fm1 - fp1, c0 = fm1 - L_(2.0) * f0 + fp1;
    T s1 = L_(3.0) * f0 - L_(4.0) * fp1 + fp2, c1 = f0 - L_(2.0) * fp1 + fp2;
    T s2 = fm2 - L_(4.0) * fm1 + L_(3.0) * f0, c2 = fm2 - L_(2.0) * fm1 + f0;
    T b0 = L_(0.25) * s0 * s0 + L_(13.0 / 12.0) * c0 * c0;
    T b1 = L_(0.25) * s1 * s1 + L_(13.0 / 12.0) * c1 * c1;
    T b2 = L_(0.25) * s2 * s2 + L_(13.0 / 12.0) * c2 * c2;
    T tau = fabs(b0 - b2);
    T eps = sp.eps32_rel * (fm2 * fm2 + fm1 * fm1 + f0 * f0 + fp1 * fp1 + fp2 * fp2) * L_(0.2) + L_(1e-30);
    T t0 = L_(1.0) + tau / (eps + b0), t1 = L_(1.0) + tau / (eps + b1), t2 = L_(1.0) + tau / (eps + b2);
    T tm = fmax(t0, fmax(t1, t2));
    T r0 = t0 / tm, r1 = t1 / tm, r2 = t2 / tm;
    r0 = r0 * r0 * r0; r0 = r0 * r0;
    r1 = r1 * r1 * r1; r1 = r1 * r1;
    r2 = r2 * r2 * r2; r2 = r2 * r2;
    // alpha_r / sum < C_T  <=>  alpha_r < C_T * sum (sum > 0)
    const T cs = sp.teno_ct * (r0 + r1 + r2);
    T d0 = (r0 < cs) ? L_(0.0) : L_(1.0);
    T d1 = (r1 < cs) ? L_(0.0) : L_(1.0);
    T d2 = (r2 < cs) ? L_(0.0) : L_(1.0);
    T w0 = L_(11.0 / 20.0) * d0, w1 = L_(4.0 / 10.0) * d1, w2 = L_(1.0 / 20.0) * d2;
    T iw = L_(1.0) / (w0 + w1 + w2);
    T e0 = -L_(1.0 / 6.0) * fm1 + L_(5.0 / 6.0) * f0 + L_(2.0 / 6.0) * fp1;
    T e1 = L_(2.0 / 6.0) * f0 + L_(5.0 / 6.0) * fp1 - L_(1.0 / 6.0) * fp2;
    T e2 = L_(2.0 / 6.0) * fm2 - L_(7.0 / 6.0) * fm1 + L_(11.0 / 6.0) * f0;
    return (w0 * e0 + w1 * e1 + w2 * e2) * iw;
  } else {
    T c0 = f0 - L_(2.0) * fp1 + fp2, s0 = L_(3.0) * f0 - L_(4.0) * fp1 + fp2;
    T c1 = fm1 - L_(2.0) * f0 + fp1, s1 = fm1 - fp1;
    T c2 = fm2 - L_(2.0) * fm1 + f0, s2 = fm2 - L_(4.0) * fm1 + L_(3.0) * f0;
    T b0 = L_(13.0 / 12.0) * c0 * c0 + L_(0.25) * s0 * s0;
    T b1 = L_(13.0 / 12.0) * c1 * c1 + L_(0.25) * s1 * s1;
    T b2 = L_(13.0 / 12.0) * c2 * c2 + L_(0.25) * s2 * s2;
    T a0, a1, a2;
    if (SCH == SCH_WENO5_Z) {
      T eps = sp.eps32_rel * (fm2 * fm2 + fm1 * fm1 + f0 * f0 + fp1 * fp1 + fp2 * fp2) * L_(0.2) + L_(1e-30);
      T tau = fabs(b0 - b2);
      T r0 = tau / (eps + b0), r1 = tau / (eps + b1), r2 = tau / (eps + b2);
      a0 = L_(0.3) * (L_(1.0) + r0 * r0);
      a1 = L_(0.6) * (L_(1.0) + r1 * r1);
      a2 = L_(0.1) * (L_(1.0) + r2 * r2);
    } else {
      T eps = L_(1.0e-6);
      a0 = L_(0.3) / ((eps + b0) * (eps + b0));
      a1 = L_(0.6) / ((eps + b1) * (eps + b1));
      a2 = L_(0.1) / ((eps + b2) * (eps + b2));
    }
    T inv = L_(1.0) / (a0 + a1 + a2);
    T e0 = L_(1.0 / 3.0) * f0 + L_(5.0 / 6.0) * fp1 - L_(1.0 / 6.0) * fp2;
    T e1 = -L_(1.0 / 6.0) * fm1 + L_(5.0 / 6.0) * f0 + L_(1.0 / 3.0) * fp1;
    T e2 = L_(1.0 / 3.0) * fm2 - L_(7.0 / 6.0) * fm1 + L_(11.0 / 6.0) * f0;
    return (a0 * inv) * e0 + (a1 * inv) * e1 + (a2 * inv) * e2;
  }
}

// Sixth-order TENO at the interface i+1/2 from six points f0..f5 = i-2..i+3 (teno.py:59-194 for
// sides +1 / -1, 220-240 tau_6 = |b3 - (b0 + b2 - 4 b1)/6|, 419-477 cut-off and weights with
// optimal weights 231/500, 3/10, 27/500, 23/125).  Side +1 reconstructs the positive split
// flux, side -1 the negative one.  The reference's side +1 fourth smoothness indicator has its
// 781/720 term unsquared (teno.py:160-161, squared on side -1), and so does this: its generated
// solvers compute it that way.  The FP32 path uses the rescaled epsilon of recon5 and forms
// the cut-off from t_r / max|t|.
template <typename T, int SIDE>
__device__ __forceinline__ T recon6(T fm2, T fm1, T f0, T fp1, T fp2, T fp3, const SP<T>& sp) {
  constexpr bool F32 = sizeof(T) == 4;
  T b0, b1, b2, b3, e0, e1, e2, e3;
  if (SIDE > 0) {
    T s0 = fm1 - fp1, c0 = fm1 - L_(2.0) * f0 + fp1;
    T s1 = L_(3.0) * f0 - L_(4.0) * fp1 + fp2, c1 = f0 - L_(2.0) * fp1 + fp2;
    T s2 = fm2 - L_(4.0) * fm1 + L_(3.0) * f0, c2 = fm2 - L_(2.0) * fm1 + f0;
    b0 = L_(0.25) * s0 * s0 + L_(13.0 / 12.0) * c0 * c0;
    b1 = L_(0.25) * s1 * s1 + L_(13.0 / 12.0) * c1 * c1;
    b2 = L_(0.25) * s2 * s2 + L_(13.0 / 12.0) * c2 * c2;
    T u1 = -L_(11.0) * f0 + L_(18.0) * fp1 - L_(9.0) * fp2 + L_(2.0) * fp3;
    T u2 = L_(2.0) * f0 - L_(5.0) * fp1 + L_(4.0) * fp2 - fp3;
    T u3 = -f0 + L_(3.0) * fp1 - L_(3.0) * fp2 + fp3;
    b3 = L_(1.0 / 36.0) * u1 * u1 + L_(13.0 / 12.0) * u2 * u2 + L_(781.0 / 720.0) * u3;
    e0 = -L_(1.0 / 6.0) * fm1 + L_(5.0 / 6.0) * f0 + L_(2.0 / 6.0) * fp1;
    e1 = L_(2.0 / 6.0) * f0 + L_(5.0 / 6.0) * fp1 - L_(1.0 / 6.0) * fp2;
    e2 = L_(2.0 / 6.0) * fm2 - L_(7.0 / 6.0) * fm1 + L_(11.0 / 6.0) * f0;
    e3 = L_(3.0 / 12.0) * f0 + L_(13.0 / 12.0) * fp1 - L_(5.0 / 12.0) * fp2 + L_(1.0 / 12.0) * fp3;
  } else {
    T s0 = f0 - fp2, c0 = f0 - L_(2.0) * fp1 + fp2;
    T s1 = fm1 - L_(4.0) * f0 + L_(3.0) * fp1, c1 = fm1 - L_(2.0) * f0 + fp1;
    T s2 = L_(3.0) * fp1 - L_(4.0) * fp2 + fp3, c2 = fp1 - L_(2.0) * fp2 + fp3;
    b0 = L_(0.25) * s0 * s0 + L_(13.0 / 12.0) * c0 * c0;
    b1 = L_(0.25) * s1 * s1 + L_(13.0 / 12.0) * c1 * c1;
    b2 = L_(0.25) * s2 * s2 + L_(13.0 / 12.0) * c2 * c2;
    T u1 = -L_(2.0) * fm2 + L_(9.0) * fm1 - L_(18.0) * f0 + L_(11.0) * fp1;
    T u2 = -fm2 + L_(4.0) * fm1 - L_(5.0) * f0 + L_(2.0) * fp1;
    T u3 = -fm2 + L_(3.0) * fm1 - L_(3.0) * f0 + fp1;
    b3 = L_(1.0 / 36.0) * u1 * u1 + L_(13.0 / 12.0) * u2 * u2 + L_(781.0 / 720.0) * u3 * u3;
    e0 = L_(2.0 / 6.0) * f0 + L_(5.0 / 6.0) * fp1 - L_(1.0 / 6.0) * fp2;
    e1 = -L_(1.0 / 6.0) * fm1 + L_(5.0 / 6.0) * f0 + L_(2.0 / 6.0) * fp1;
    e2 = L_(11.0 / 6.0) * fp1 - L_(7.0 / 6.0) * fp2 + L_(1.0 / 3.0) * fp3;
    e3 = L_(1.0 / 12.0) * fm2 - L_(5.0 / 12.0) * fm1 + L_(13.0 / 12.0) * f0 + L_(3.0 / 12.0) * fp1;
  }
  const T tau = fabs(b3 - L_(1.0 / 6.0) * (b0 + b2 - L_(4.0) * b1));
  T a0, a1, a2, a3;
  if (F32) {
    T eps = sp.eps32_rel * (fm2 * fm2 + fm1 * fm1 + f0 * f0 + fp1 * fp1 + fp2 * fp2 + fp3 * fp3) * L_(1.0 / 6.0) +
            L_(1e-30);
    T t0 = L_(1.0) + tau / (eps + b0), t1 = L_(1.0) + tau / (eps + b1), t2 = L_(1.0) + tau / (eps + b2),
      t3 = L_(1.0) + tau / (eps + b3);
    T im = L_(1.0) / fmax(fmax(fabs(t0), fabs(t1)), fmax(fabs(t2), fabs(t3)));
    t0 *= im; t1 *= im; t2 *= im; t3 *= im;
    a0 = t0 * t0 * t0; a0 = a0 * a0;
    a1 = t1 * t1 * t1; a1 = a1 * a1;
    a2 = t2 * t2 * t2; a2 = a2 * a2;
    a3 = t3 * t3 * t3; a3 = a3 * a3;
  } else {
    const T eps = sp.teno_eps;
    T t0 = L_(1.0) + tau / (eps + b0), t1 = L_(1.0) + tau / (eps + b1), t2 = L_(1.0) + tau / (eps + b2),
      t3 = L_(1.0) + tau / (eps + b3);
    t0 = t0 * t0; t1 = t1 * t1; t2 = t2 * t2; t3 = t3 * t3;
    a0 = t0 * t0 * t0;
    a1 = t1 * t1 * t1;
    a2 = t2 * t2 * t2;
    a3 = t3 * t3 * t3;
  }
  const T inv = L_(1.0) / (a0 + a1 + a2 + a3);
  const T ct = sp.teno_ct;
  const T w0 = (a0 * inv < ct) ? L_(0.0) : L_(231.0 / 500.0);
  const T w1 = (a1 * inv < ct) ? L_(0.0) : L_(3.0 / 10.0);
  const T w2 = (a2 * inv < ct) ? L_(0.0) : L_(27.0 / 500.0);
  const T w3 = (a3 * inv < ct) ? L_(0.0) : L_(23.0 / 125.0);
  return (w0 * e0 + w1 * e1 + w2 * e2 + w3 * e3) * (L_(1.0) / (w0 + w1 + w2 + w3));
}

// Reconstruction of one characteristic wave at i+1/2 from the positive and negative split
// fluxes at points i-2..i+3 (GEN: FP64 in the generated order).
template <typename T, int SCH, bool GEN = false>
__device__ __forceinline__ T recon_wave(const T (&fp)[6], const T (&fm)[6], const SP<T>& sp) {
  if constexpr (SCH == SCH_TENO6) {
    return recon6<T, 1>(fp[0], fp[1], fp[2], fp[3], fp[4], fp[5], sp) +
           recon6<T, -1>(fm[0], fm[1], fm[2], fm[3], fm[4], fm[5], sp);
  } else if constexpr (GEN && sizeof(T) == 8) {
    const double eps = recon_eps<SCH>(sp.teno_eps, 1.0).eps;
    return recon5_ieee<SCH>(fp[0], fp[1], fp[2], fp[3], fp[4], eps, sp.teno_ct) +
           recon5_ieee<SCH>(fm[5], fm[4], fm[3], fm[2], fm[1], eps, sp.teno_ct);
  } else {
    return recon5<T, SCH>(fp[0], fp[1], fp[2], fp[3], fp[4], sp) +
           recon5<T, SCH>(fm[5], fm[4], fm[3], fm[2], fm[1], sp);
  }
}

// Point data carried through a sweep: conserved state in the local frame plus primitives.
template <typename T, int ND>
struct Pt {
  T q[ND + 2];  // rho, m_n, m_t.., E
  T u[ND];      // u_n, u_t..
  T p, a;
};

// GEN: the sweep keeps the generated order (generated_order).
template <typename T, int ND, bool GEN = false>
__device__ __forceinline__ void make_pt(Pt<T, ND>& s, T gm) {
  T rho = s.q[0];
  T ir = L_(1.0) / rho;
  T ke = L_(0.0);
#pragma unroll
  for (int i = 0; i < ND; ++i) {
    s.u[i] = s.q[1 + i] * ir;
    ke += s.u[i] * s.u[i];
  }
  s.p = (gm - L_(1.0)) * (s.q[ND + 1] - L_(0.5) * rho * ke);
  s.a = sqrt(gm * s.p * ir);
}

// FP32 2D: the kinetic energy as a sum of two rounded squares, which does not depend on the order of
// the components: the persistent stage forms a point's primitives once for both directions, the
// sweeps in each direction's own frame, and they agree bit for bit.
template <typename T, int ND, bool GEN = false>
__device__ __forceinline__ void make_pt(Pt<float, 2>& s, float gm) {
  if constexpr (GEN) {
    const float rho = s.q[0], ir = 1.0f / rho;
    float ke = 0.0f;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      s.u[i] = s.q[1 + i] * ir;
      ke += s.u[i] * s.u[i];
    }
    s.p = (gm - 1.0f) * (s.q[3] - 0.5f * rho * ke);
    s.a = sqrtf(gm * s.p * ir);
    return;
  }
  const float ir = 1.0f / s.q[0];
  s.u[0] = __fmul_rn(s.q[1], ir);
  s.u[1] = __fmul_rn(s.q[2], ir);
  const float ke = __fadd_rn(__fmul_rn(s.u[0], s.u[0]), __fmul_rn(s.u[1], s.u[1]));
  s.p = __fmul_rn(gm - 1.0f, __fmaf_rn(__fmul_rn(-0.5f, s.q[0]), ke, s.q[3]));
  s.a = sqrtf(__fmul_rn(__fmul_rn(gm, s.p), ir));
}

// FP64: the square root of the density and the total enthalpy that the Roe average takes from
// either side of an interface are formed once per point (a point is a side of two interfaces).
template <int ND>
struct Pt<double, ND> {
  double q[ND + 2], u[ND];
  double p, a, s, H;  // s = sqrt(rho), H = (E + p) / rho
};
template <typename T, int ND, bool GEN = false>
__device__ __forceinline__ void make_pt(Pt<double, ND>& s, double gm) {
  if constexpr (ND <= 2) {  // the generated order (recon5_ieee)
    const double rho = s.q[0], ir = 1.0 / rho;
    double ke = 0.0;
#pragma unroll
    for (int i = 0; i < ND; ++i) {
      s.u[i] = s.q[1 + i] * ir;
      ke += s.u[i] * s.u[i];
    }
    s.p = (gm - 1.0) * (s.q[ND + 1] - 0.5 * rho * ke);
    s.a = sqrt(gm * s.p * ir);
    s.s = sqrt(rho);
    s.H = (s.q[ND + 1] + s.p) * ir;
    return;
  }
  const double ir = rcp_newton(s.q[0]);
  double ke2 = 0.0;
#pragma unroll
  for (int i = 0; i < ND; ++i) {
    s.u[i] = s.q[1 + i] * ir;
    ke2 += s.q[1 + i] * s.u[i];
  }
  s.p = (gm - 1.0) * (s.q[ND + 1] - 0.5 * ke2);
  s.a = sqrt(gm * s.p * ir);
  s.s = sqrt(s.q[0]);
  s.H = (s.q[ND + 1] + s.p) * ir;
}

// FP64 averaged state of an interface (averaging.py:31-124): velocity, sound speed and its
// reciprocal, the average density squared, |u|^2.
template <int ND, int AVG>
__device__ __forceinline__ void face_average_f64(const Pt<double, ND>& L, const Pt<double, ND>& R, double g1,
                                                 double (&u)[ND], double& a, double& ia, double& rho2, double& ke) {
  ke = 0.0;
  if (AVG == AVG_ROE) {
    const double inv = rcp_newton(L.s + R.s), wl = L.s * inv, wr = R.s * inv;
#pragma unroll
    for (int i = 0; i < ND; ++i) {
      u[i] = wl * L.u[i] + wr * R.u[i];
      ke += u[i] * u[i];
    }
    const double a2 = g1 * (wl * L.H + wr * R.H - 0.5 * ke);
    ia = rsqrt(a2);
    a = a2 * ia;
    rho2 = L.q[0] * R.q[0];
  } else {
#pragma unroll
    for (int i = 0; i < ND; ++i) {
      u[i] = 0.5 * (L.u[i] + R.u[i]);
      ke += u[i] * u[i];
    }
    a = 0.5 * (L.a + R.a);
    ia = rcp_newton(a);
    const double rho = 0.5 * (L.q[0] + R.q[0]);
    rho2 = rho * rho;
  }
}

// FP64 characteristic LLF flux at the interface between w[2] and w[3] (the FP32 form and the
// citations: char_flux), arranged for the fewest FP64 instructions.  With the averaged state u, a,
// a point's projections are
//   P = E - u.m + |u|^2/2 rho,  D = m_n - u_n rho,
//   entropy wave   e  = rho - (gama - 1) / a^2 P,
//   vorticity      m_t2 - u_t2 rho  and  u_t1 rho - m_t1       (the rows times the average density)
//   acoustic       (gama - 1) / a P +- D                       (the rows over their common factor)
// and the projected flux of a point is its own u_n times that, plus (gama - 1) / a p (u_n' - u_n) +- p in
// the acoustic rows (the pressure then reaches the momentum flux without a rounded factor) and
// -(gama - 1) / a^2 p (u_n' - u_n) in the entropy row.  A
// row's constant factor commutes with the reconstruction (its epsilon is scaled instead, ReconEps),
// so neither it nor the 1/2 of the flux splitting is applied to the twelve values of a wave, and
// 1D, 2D and 3D share the form: their rows differ by that factor alone.  (generated_order: not here.)
//
// One interface of a 3D TENO5 block takes about 360 FP64 instructions here, against the 2 300 that
// the generated order costs: a step of the 128^3 TENO5 vortex took 63.4 ms before and 19.2 ms with
// it (6.8 of them in the central and update kernels), the 457 x 255 WENO5-Z shock reflection 2.21
// and 1.12 ms, at the same error against plain 64-bit arithmetic (2e-16; TENO5 decides alike).
// A register window as the window that char_flux_f64 reads.
template <int ND>
struct WindowF64 {
  const Pt<double, ND> (&w)[6];
  __device__ __forceinline__ const Pt<double, ND>& side(int m) const { return w[m]; }
  __device__ __forceinline__ double q(int m, int v) const { return w[m].q[v]; }
  __device__ __forceinline__ double un(int m) const { return w[m].u[0]; }
  __device__ __forceinline__ double p(int m) const { return w[m].p; }
};

// A(m) gives point m of the window: the six of a register window, or of a tile in shared memory.
template <int ND, int SCH, int AVG, typename Acc>
__device__ __forceinline__ void char_flux_f64(const Acc& A, const SP<double>& sp, double (&fh)[ND + 2]) {
  constexpr int NV = ND + 2, E = ND + 1;
  const double g1 = sp.g1;
  const Pt<double, ND> L = A.side(2), R = A.side(3);
  double u[ND], a, ia, rho2, ke;
  face_average_f64<ND, AVG>(L, R, g1, u, a, ia, rho2, ke);
  const double hk = 0.5 * ke, gi = g1 * ia, g = gi * ia;
  const double lam_u = sp.sfc * fmax(fabs(L.u[0]), fabs(R.u[0]));
  const double lam_p = sp.sfc * fmax(fabs(L.u[0] + L.a), fabs(R.u[0] + R.a));
  const double lam_m = sp.sfc * fmax(fabs(L.u[0] - L.a), fabs(R.u[0] - R.a));
  double P[6], D[6], W[6];
#pragma unroll
  for (int m = 0; m < 6; ++m) {
    double x = A.q(m, E);
#pragma unroll
    for (int i = 0; i < ND; ++i) x = __fma_rn(-u[i], A.q(m, 1 + i), x);
    P[m] = __fma_rn(hk, A.q(m, 0), x);
    D[m] = __fma_rn(-u[0], A.q(m, 0), A.q(m, 1));
    W[m] = A.p(m) * (A.un(m) - u[0]);
  }
  // reconstruction of one wave from its split fluxes, twice a scale times the generated ones: s2 is
  // that factor squared; TENO6, whose side +1 indicator is not homogeneous, takes them unscaled
  auto wave = [&](const double (&fp)[6], const double (&fm)[6], double s2) -> double {
    if constexpr (SCH == SCH_TENO6) {
      const double sc = sqrt(s2), isc = rcp_newton(sc);
      double x[6], y[6];
#pragma unroll
      for (int m = 0; m < 6; ++m) {
        x[m] = fp[m] * isc;
        y[m] = fm[m] * isc;
      }
      return sc * (recon6<double, 1>(x[0], x[1], x[2], x[3], x[4], x[5], sp) +
                   recon6<double, -1>(y[0], y[1], y[2], y[3], y[4], y[5], sp));
    } else {
      const ReconEps e = recon_eps<SCH>(sp.teno_eps, s2);
      return recon5_f64<SCH>(fp[0], fp[1], fp[2], fp[3], fp[4], e, sp.teno_ct, sp.teno_ct_f) +
             recon5_f64<SCH>(fm[5], fm[4], fm[3], fm[2], fm[1], e, sp.teno_ct, sp.teno_ct_f);
    }
  };
  double fp[6], fm[6];
  // entropy wave
#pragma unroll
  for (int m = 0; m < 6; ++m) {
    const double c = __fma_rn(-g, P[m], A.q(m, 0)), t = g * W[m];
    fp[m] = __fma_rn(A.un(m) + lam_u, c, -t);
    fm[m] = __fma_rn(A.un(m) - lam_u, c, -t);
  }
  const double r0 = 0.5 * wave(fp, fm, 4.0);
  // vorticity waves: t1 along +t2, t2 along -t1 (3D); 2D has the second alone
  double t1 = 0.0, t2 = 0.0;
  if constexpr (ND == 3) {
#pragma unroll
    for (int m = 0; m < 6; ++m) {
      const double c = __fma_rn(-u[ND - 1], A.q(m, 0), A.q(m, ND));
      fp[m] = (A.un(m) + lam_u) * c;
      fm[m] = (A.un(m) - lam_u) * c;
    }
    t1 = 0.5 * wave(fp, fm, 4.0 * rho2);
  }
  if constexpr (ND >= 2) {
#pragma unroll
    for (int m = 0; m < 6; ++m) {
      const double c = __fma_rn(u[1], A.q(m, 0), -A.q(m, 2));
      fp[m] = (A.un(m) + lam_u) * c;
      fm[m] = (A.un(m) - lam_u) * c;
    }
    t2 = 0.5 * wave(fp, fm, 4.0 * rho2);
  }
  // acoustic waves
  const double s2a = ND == 1 ? 16.0 * a * a : 8.0 * rho2;
#pragma unroll
  for (int m = 0; m < 6; ++m) {
    const double c = __fma_rn(gi, P[m], D[m]);
    const double f = __fma_rn(A.un(m), c, __fma_rn(gi, W[m], A.p(m)));
    fp[m] = __fma_rn(lam_p, c, f);
    fm[m] = __fma_rn(-lam_p, c, f);
  }
  const double rp = wave(fp, fm, s2a);
#pragma unroll
  for (int m = 0; m < 6; ++m) {
    const double c = __fma_rn(gi, P[m], -D[m]);
    const double f = __fma_rn(A.un(m), c, __fma_rn(gi, W[m], -A.p(m)));
    fp[m] = __fma_rn(lam_m, c, f);
    fm[m] = __fma_rn(-lam_m, c, f);
  }
  const double rm = wave(fp, fm, s2a);
  // back to physical space
  const double S = 0.25 * (rp + rm), B = 0.25 * (rp - rm), F0 = __fma_rn(ia, S, r0);
  fh[0] = F0;
  fh[1] = __fma_rn(u[0], F0, B);
  double e = __fma_rn(hk, F0, __fma_rn(a * sp.ig1, S, u[0] * B));
  if constexpr (ND >= 2) {
    fh[2] = __fma_rn(u[1], F0, -t2);
    e = __fma_rn(-u[1], t2, e);
  }
  if constexpr (ND == 3) {
    fh[ND] = __fma_rn(u[ND - 1], F0, t1);
    e = __fma_rn(u[ND - 1], t1, e);
  }
  fh[NV - 1] = e;
}

// ---------------------------------------------------------------------------------------
// FP32 characteristic flux on packed pairs.
//
// In scalar form the FP32 sweeps were bound by instruction issue (81-83 % of the issue slots, the FMA pipe
// 65-68 % busy).  sm_103a's packed FP32 instructions (fma / mul / add on a float2) do two lanes' work in
// one issue slot at the same FMA-pipe time: 946 instructions per interface instead of 1 530, issue 61 %, FMA
// pipe 65 %, with 12 warps per SM the latency of a reconstruction's chain now counts.  The reconstruction
// runs on pairs that share every coefficient: the two acoustic waves, the two vorticity waves (2D: the
// entropy and the vorticity wave), and the two sides of the 3D entropy wave.
__device__ __forceinline__ float2 f2(float x, float y) { return make_float2(x, y); }
__device__ __forceinline__ float2 f2(float x) { return make_float2(x, x); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, f2(-1.f), a); }
__device__ __forceinline__ float2 rcp2(float2 a) { return f2(rcp_approx(a.x), rcp_approx(a.y)); }
__device__ __forceinline__ float2 abs2(float2 a) { return f2(fabsf(a.x), fabsf(a.y)); }

// recon5 (FP32 form: see its epsilon) of two waves at once, on the differences of the stencil values.
// s2: the square of the waves' scale (ReconEps), which the absolute epsilon of WENO5-JS takes.  The floor
// under every epsilon, 4e-36, only keeps a wave without differences off 0/0 (FP32 still holds its
// reciprocal): these waves carry the density, and at 4e-30 it swamped the indicators of a thin gas
// (below about 1e-13).
template <int SCH>
__device__ __forceinline__ float2 recon5_x2(float2 fm2, float2 fm1, float2 f0, float2 fp1, float2 fp2, float eps_rel,
                                            float ct, float2 s2) {
  const float2 d1 = sub2(fm1, fm2), d2 = sub2(f0, fm1), d3 = sub2(fp1, f0), d4 = sub2(fp2, fp1);
  const float2 c0 = sub2(d4, d3), s0 = fma2(f2(-2.f), d3, c0);  // [0, 1, 2]
  const float2 c1 = sub2(d3, d2), s1 = add2(d2, d3);            // [-1, 0, 1]
  const float2 c2 = sub2(d2, d1), s2_ = fma2(f2(2.f), d2, c2);  // [-2, -1, 0]
  // four times epsilon: relative to the stencil's mean square, or WENO5-JS's constant
  float2 e4;
  if (SCH == SCH_WENO5_JS) {
    e4 = f2(4.0e-6f * s2.x + 4e-36f, 4.0e-6f * s2.y + 4e-36f);  // a constant where s2 is one
  } else {
    const float2 ss = fma2(fp2, fp2, fma2(fp1, fp1, fma2(f0, f0, fma2(fm1, fm1, mul2(fm2, fm2)))));
    e4 = fma2(f2(0.8f * eps_rel), ss, f2(4e-36f));
  }
  const float2 k = f2((float)(13.0 / 3.0));
  const float2 u0 = fma2(mul2(k, c0), c0, fma2(s0, s0, e4));
  const float2 u1 = fma2(mul2(k, c1), c1, fma2(s1, s1, e4));
  const float2 u2 = fma2(mul2(k, c2), c2, fma2(s2_, s2_, e4));
  if (SCH == SCH_TENO5) {
    const float2 tau = abs2(sub2(u1, u2));
    float2 x0 = fma2(tau, rcp2(u0), f2(1.f)), x1 = fma2(tau, rcp2(u1), f2(1.f)), x2 = fma2(tau, rcp2(u2), f2(1.f));
    const float2 im = f2(rcp_approx(fmaxf(x0.x, fmaxf(x1.x, x2.x))), rcp_approx(fmaxf(x0.y, fmaxf(x1.y, x2.y))));
    x0 = mul2(x0, im);
    x1 = mul2(x1, im);
    x2 = mul2(x2, im);
    x0 = mul2(mul2(x0, x0), x0); x0 = mul2(x0, x0);
    x1 = mul2(mul2(x1, x1), x1); x1 = mul2(x1, x1);
    x2 = mul2(mul2(x2, x2), x2); x2 = mul2(x2, x2);
    const float2 cs = mul2(f2(ct), add2(add2(x0, x1), x2));
    const float2 m0 = f2(x0.x < cs.x ? 0.f : 1.f, x0.y < cs.y ? 0.f : 1.f);
    const float2 m1 = f2(x1.x < cs.x ? 0.f : 1.f, x1.y < cs.y ? 0.f : 1.f);
    const float2 m2 = f2(x2.x < cs.x ? 0.f : 1.f, x2.y < cs.y ? 0.f : 1.f);
    // weights times (e_r - f0): e0 - f0 = (4 d3 - d4) / 6, e1 - f0 = (d2 + 2 d3) / 6, e2 - f0 = (5 d2 - 2 d1) / 6
    const float2 g0 = fma2(f2((float)(0.4 * 4.0 / 6.0)), d3, mul2(f2((float)(-0.4 / 6.0)), d4));
    const float2 g1 = fma2(f2((float)(0.55 / 3.0)), d3, mul2(f2((float)(0.55 / 6.0)), d2));
    const float2 g2 = fma2(f2((float)(0.05 * 5.0 / 6.0)), d2, mul2(f2((float)(-0.05 / 3.0)), d1));
    const float2 Dn = fma2(f2(0.4f), m0, fma2(f2(0.55f), m1, mul2(f2(0.05f), m2)));
    return fma2(fma2(m0, g0, fma2(m1, g1, mul2(m2, g2))), rcp2(Dn), f0);
  }
  float2 a0, a1, a2;  // the weights without the factors 3/10, 6/10, 1/10
  if (SCH == SCH_WENO5_Z) {
    const float2 tau = sub2(u0, u2);  // squared below
    const float2 r0 = mul2(tau, rcp2(u0)), r1 = mul2(tau, rcp2(u1)), r2 = mul2(tau, rcp2(u2));
    a0 = fma2(r0, r0, f2(1.f));
    a1 = fma2(r1, r1, f2(1.f));
    a2 = fma2(r2, r2, f2(1.f));
  } else {
    const float2 r0 = rcp2(u0), r1 = rcp2(u1), r2 = rcp2(u2);
    const float2 im = f2(rcp_approx(fmaxf(r0.x, fmaxf(r1.x, r2.x))), rcp_approx(fmaxf(r0.y, fmaxf(r1.y, r2.y))));
    a0 = mul2(r0, im); a0 = mul2(a0, a0);
    a1 = mul2(r1, im); a1 = mul2(a1, a1);
    a2 = mul2(r2, im); a2 = mul2(a2, a2);
  }
  // ten times the weights times (e_r - f0)
  const float2 g0 = fma2(f2(2.f), d3, mul2(f2(-0.5f), d4));
  const float2 g1 = fma2(f2(2.f), d3, d2);
  const float2 g2 = fma2(f2((float)(5.0 / 6.0)), d2, mul2(f2((float)(-1.0 / 3.0)), d1));
  const float2 Dn = fma2(f2(6.f), a1, fma2(f2(3.f), a0, a2));
  return fma2(fma2(a0, g0, fma2(a1, g1, mul2(a2, g2))), rcp2(Dn), f0);
}

// FP32 characteristic LLF flux of a 2D / 3D interface in the factored form of char_flux_f64 (waves
// scaled by a constant factor, projected flux in closed form) on packed pairs of waves.  Products
// that feed sums are written as explicit multiply-adds: the sweeps and the persistent stage inline
// this into different code and still give the same bits.
template <int ND, int SCH, int AVG>
__device__ __forceinline__ void char_flux_f32(const Pt<float, ND> (&w)[6], const SP<float>& sp, float (&fh)[ND + 2]) {
  constexpr int NV = ND + 2, E = ND + 1;
  const float g1 = sp.g1;
  const Pt<float, ND>& L = w[2];
  const Pt<float, ND>& R = w[3];
  float u[ND], a, ia, rho2, ke = 0.f;
  if (AVG == AVG_ROE) {
    const float iL = rsqrtf(L.q[0]), iR = rsqrtf(R.q[0]), sL = L.q[0] * iL, sR = R.q[0] * iR;
    const float inv = rcp_approx(sL + sR), wl = sL * inv, wr = sR * inv;
#pragma unroll
    for (int i = 0; i < ND; ++i) {
      u[i] = __fmaf_rn(wl, L.u[i], __fmul_rn(wr, R.u[i]));
      ke = __fmaf_rn(u[i], u[i], ke);
    }
    const float H = __fmul_rn(__fmaf_rn(L.q[E] + L.p, iL, __fmul_rn(R.q[E] + R.p, iR)), inv);
    const float a2 = __fmul_rn(g1, __fmaf_rn(-0.5f, ke, H));
    a = a2 * rsqrtf(a2);
    rho2 = L.q[0] * R.q[0];
  } else {
#pragma unroll
    for (int i = 0; i < ND; ++i) {
      u[i] = 0.5f * (L.u[i] + R.u[i]);
      ke = __fmaf_rn(u[i], u[i], ke);
    }
    a = 0.5f * (L.a + R.a);
    const float rho = 0.5f * (L.q[0] + R.q[0]);
    rho2 = rho * rho;
  }
  ia = rcp_approx(a);
  const float hk = 0.5f * ke, gi = g1 * ia, g = gi * ia;
  const float lam_u = sp.sfc * fmaxf(fabsf(L.u[0]), fabsf(R.u[0]));
  const float lam_p = sp.sfc * fmaxf(fabsf(L.u[0] + L.a), fabsf(R.u[0] + R.a));
  const float lam_m = sp.sfc * fmaxf(fabsf(L.u[0] - L.a), fabsf(R.u[0] - R.a));
  float P[6], W[6], up[6], um[6];
#pragma unroll
  for (int m = 0; m < 6; ++m) {
    float x = w[m].q[E];
#pragma unroll
    for (int i = 0; i < ND; ++i) x = __fmaf_rn(-u[i], w[m].q[1 + i], x);
    P[m] = __fmaf_rn(hk, w[m].q[0], x);
    W[m] = __fmul_rn(w[m].p, w[m].u[0] - u[0]);
    up[m] = w[m].u[0] + lam_u;
    um[m] = w[m].u[0] - lam_u;
  }
  auto sides = [&](const float2 (&fp)[6], const float2 (&fm)[6], float2 s2) -> float2 {
    return add2(recon5_x2<SCH>(fp[0], fp[1], fp[2], fp[3], fp[4], sp.eps32_rel, sp.teno_ct, s2),
                recon5_x2<SCH>(fm[5], fm[4], fm[3], fm[2], fm[1], sp.eps32_rel, sp.teno_ct, s2));
  };
  float2 fp[6], fm[6];
  float r0, t1 = 0.f, t2;
  if constexpr (ND == 3) {
    // entropy wave: its + side and its mirrored - side are the pair
    float p[6], q[6];
#pragma unroll
    for (int m = 0; m < 6; ++m) {
      const float c = __fmaf_rn(-g, P[m], w[m].q[0]), t = __fmul_rn(g, W[m]);
      p[m] = __fmaf_rn(up[m], c, -t);
      q[m] = __fmaf_rn(um[m], c, -t);
    }
    const float2 r = recon5_x2<SCH>(f2(p[0], q[5]), f2(p[1], q[4]), f2(p[2], q[3]), f2(p[3], q[2]), f2(p[4], q[1]),
                                    sp.eps32_rel, sp.teno_ct, f2(4.f));
    r0 = 0.5f * (r.x + r.y);
    const float2 cu = f2(-u[ND - 1], u[1]);
#pragma unroll
    for (int m = 0; m < 6; ++m) {
      const float2 c = fma2(cu, f2(w[m].q[0]), f2(w[m].q[ND], -w[m].q[2]));
      fp[m] = mul2(f2(up[m]), c);
      fm[m] = mul2(f2(um[m]), c);
    }
    const float2 v = sides(fp, fm, f2(4.f * rho2));
    t1 = 0.5f * v.x;
    t2 = 0.5f * v.y;
  } else {
    const float2 cu = f2(-g, u[1]);
#pragma unroll
    for (int m = 0; m < 6; ++m) {
      const float2 c = fma2(cu, f2(P[m], w[m].q[0]), f2(w[m].q[0], -w[m].q[2]));
      const float2 t = f2(__fmul_rn(-g, W[m]), 0.f);
      fp[m] = fma2(f2(up[m]), c, t);
      fm[m] = fma2(f2(um[m]), c, t);
    }
    const float2 v = sides(fp, fm, f2(4.f, 4.f * rho2));
    r0 = 0.5f * v.x;
    t2 = 0.5f * v.y;
  }
  // acoustic waves u + a, u - a
  const float2 lp = f2(lam_p, lam_m), lm = f2(-lam_p, -lam_m);
#pragma unroll
  for (int m = 0; m < 6; ++m) {
    const float D = __fmaf_rn(-u[0], w[m].q[0], w[m].q[1]);
    const float2 c = f2(__fmaf_rn(gi, P[m], D), __fmaf_rn(gi, P[m], -D));
    const float2 f = fma2(f2(w[m].u[0]), c, f2(__fmaf_rn(gi, W[m], w[m].p), __fmaf_rn(gi, W[m], -w[m].p)));
    fp[m] = fma2(lp, c, f);
    fm[m] = fma2(lm, c, f);
  }
  const float2 r = sides(fp, fm, f2(8.f * rho2));
  const float S = __fmul_rn(0.25f, r.x + r.y), B = __fmul_rn(0.25f, r.x - r.y), F0 = __fmaf_rn(ia, S, r0);
  fh[0] = F0;
  fh[1] = __fmaf_rn(u[0], F0, B);
  fh[2] = __fmaf_rn(u[1], F0, -t2);
  float e = __fmaf_rn(hk, F0, __fmaf_rn(__fmul_rn(a, sp.ig1), S, __fmul_rn(u[0], B)));
  e = __fmaf_rn(-u[1], t2, e);
  if constexpr (ND == 3) {
    fh[ND] = __fmaf_rn(u[ND - 1], F0, t1);
    e = __fmaf_rn(u[ND - 1], t1, e);
  }
  fh[NV - 1] = e;
}

// Averaged state of a 1D interface (averaging.py:31-124) in the generated order.
template <typename T, int AVG>
struct Face1D {
  T u, a, H, iden, ia;
  __device__ __forceinline__ Face1D(const Pt<T, 1>& L, const Pt<T, 1>& R, const SP<T>& sp) {
    if (AVG == AVG_ROE) {
      T sL = sqrt(L.q[0]), sR = sqrt(R.q[0]);
      T inv = L_(1.0) / (sL + sR);
      u = (sL * L.u[0] + sR * R.u[0]) * inv;
      T ke = L_(0.0) + u * u;
      T h = ((L.q[2] + L.p) / sL + (R.q[2] + R.p) / sR) * inv;
      a = sqrt(sp.g1 * (h - L_(0.5) * ke));
    } else {
      u = L_(0.5) * (L.u[0] + R.u[0]);
      a = L_(0.5) * (L.a + R.a);
    }
    H = a * a / sp.g1 + L_(0.5) * u * u;
    const T den = L_(2.0) * H - u * u;
    iden = L_(1.0) / den;
    ia = L_(1.0) / a;
  }
};

// Reconstructed wave k of a 1D interface, 1D system of euler_eigensystem.py:85-99, H = a^2/(gama-1) +
// u^2/2, waves (u-a, u, u+a), LLF speeds over points i, i+1 (shock_capturing.py:1000-1028).
template <typename T, int SCH, int AVG>
__device__ __forceinline__ T wave_1d(int k, const Pt<T, 1> (&w)[6], const SP<T>& sp, const Face1D<T, AVG>& fc) {
  const Pt<T, 1>& L = w[2];
  const Pt<T, 1>& R = w[3];
  const T u0 = fc.u, a = fc.a, H = fc.H, iden = fc.iden, ia = fc.ia;
  T l0, l1, l2, lam;
  if (k == 0) {
    l0 = u0 * (L_(2.0) * H + a * u0 - u0 * u0) * L_(0.5) * ia * iden;
    l1 = (-H - a * u0 + L_(0.5) * u0 * u0) * ia * iden;
    l2 = iden;
    lam = sp.sfc * fmax(fabs(L.u[0] - L.a), fabs(R.u[0] - R.a));
  } else if (k == 1) {
    l0 = L_(2.0) * (H - u0 * u0) * iden;
    l1 = L_(2.0) * u0 * iden;
    l2 = -L_(2.0) * iden;
    lam = sp.sfc * fmax(fabs(L.u[0]), fabs(R.u[0]));
  } else {
    l0 = u0 * (-L_(2.0) * H + a * u0 + u0 * u0) * L_(0.5) * ia * iden;
    l1 = (H - a * u0 - L_(0.5) * u0 * u0) * ia * iden;
    l2 = iden;
    lam = sp.sfc * fmax(fabs(L.u[0] + L.a), fabs(R.u[0] + R.a));
  }
  T fp[6], fm[6];
#pragma unroll
  for (int m = 0; m < 6; ++m) {
    const T F0 = w[m].q[1];
    const T F1 = w[m].u[0] * w[m].q[1] + w[m].p;
    const T F2 = w[m].u[0] * (w[m].q[2] + w[m].p);
    T cs = l0 * w[m].q[0] + l1 * w[m].q[1] + l2 * w[m].q[2];
    T cf = l0 * F0 + l1 * F1 + l2 * F2;
    fp[m] = L_(0.5) * (cf + lam * cs);
    fm[m] = L_(0.5) * (cf - lam * cs);
  }
  return recon_wave<T, SCH, true>(fp, fm, sp);
}

template <typename T>
__device__ __forceinline__ void flux_1d(const T (&rec)[3], T u0, T a, T H, T (&fh)[3]) {
  fh[0] = rec[0] + rec[1] + rec[2];
  fh[1] = (u0 - a) * rec[0] + u0 * rec[1] + (u0 + a) * rec[2];
  fh[2] = (H - u0 * a) * rec[0] + L_(0.5) * u0 * u0 * rec[1] + (H + u0 * a) * rec[2];
}

// Characteristic LLF flux at the interface between w[2] and w[3] of a 6-point window
// (offsets -2..+3), local frame.  Restates shock_capturing.py:786-891 and 979-1028 with the
// eigensystems of euler_eigensystem.py for k = e_0.
template <typename T, int ND, int SCH, int AVG>
__device__ __forceinline__ void char_flux(const Pt<T, ND> (&w)[6], const SP<T>& sp, T (&fh)[ND + 2]) {
  if constexpr (sizeof(T) == 8 && !generated_order<ND, SCH>()) {
    char_flux_f64<ND, SCH, AVG>(WindowF64<ND>{w}, sp, fh);
    return;
  } else if constexpr (sizeof(T) == 4 && ND >= 2 && SCH != SCH_TENO6 && !generated_order<ND, SCH>()) {
    char_flux_f32<ND, SCH, AVG>(w, sp, fh);
    return;
  }
  if constexpr (ND == 1) {
    const Face1D<T, AVG> fc(w[2], w[3], sp);
    T rec[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) rec[k] = wave_1d<T, SCH, AVG>(k, w, sp, fc);
    flux_1d(rec, fc.u, fc.a, fc.H, fh);
    return;
  }
  constexpr int NV = ND + 2;
  const T g1 = sp.g1;
  const Pt<T, ND>& L = w[2];
  const Pt<T, ND>& R = w[3];
  // ---- averaged state (averaging.py:31-124)
  T rho, u[ND], a;
  if (AVG == AVG_ROE) {
    T sL = sqrt(L.q[0]), sR = sqrt(R.q[0]);
    rho = sqrt(L.q[0] * R.q[0]);
    T inv = L_(1.0) / (sL + sR);
    T ke = L_(0.0);
#pragma unroll
    for (int i = 0; i < ND; ++i) {
      u[i] = (sL * L.u[i] + sR * R.u[i]) * inv;
      ke += u[i] * u[i];
    }
    T H = ((L.q[NV - 1] + L.p) / sL + (R.q[NV - 1] + R.p) / sR) * inv;
    a = sqrt(g1 * (H - L_(0.5) * ke));
  } else {
    rho = L_(0.5) * (L.q[0] + R.q[0]);
#pragma unroll
    for (int i = 0; i < ND; ++i) u[i] = L_(0.5) * (L.u[i] + R.u[i]);
    a = L_(0.5) * (L.a + R.a);
  }
  // ---- LLF wave speeds over points i, i+1 (shock_capturing.py:1000-1028)
  const T sfc = sp.sfc;
  T lam_u = sfc * fmax(fabs(L.u[0]), fabs(R.u[0]));
  T lam_p = sfc * fmax(fabs(L.u[0] + L.a), fabs(R.u[0] + R.a));
  T lam_m = sfc * fmax(fabs(L.u[0] - L.a), fabs(R.u[0] - R.a));

  T rec[NV];
  // ---- 2D / 3D with k = e_0: waves 0..ND-1 move with u_n, ND with u_n + a, ND+1 with u_n - a
  const T ia = L_(1.0) / a, ia2 = ia * ia, irho = L_(1.0) / rho;
  T ke = L_(0.0);
#pragma unroll
  for (int i = 0; i < ND; ++i) ke += u[i] * u[i];
  const T phi = g1 * L_(0.5) * ke;
  const T bta = ia * irho * L_(0.70710678118654752440);   // 1/(rho a sqrt 2)
  const T alf = rho * ia * L_(0.70710678118654752440);    // rho/(a sqrt 2)
  // projections L*v of a conserved-like vector v (rows of LEV, euler_eigensystem.py):
  //   S = phi*v0 - g1*(u.vm) + g1*vE ; D = v_n - u_n v0
  //   row0 = v0 - S/a^2, row_{1..ND-1} = vorticity rows, row ND = bta(S + a D), row ND+1 = bta(S - a D)
  T fp[NV][6], fmn[NV][6];
#pragma unroll
  for (int m = 0; m < 6; ++m) {
    const Pt<T, ND>& s = w[m];
    T Fv[NV];
    Fv[0] = s.q[1];
    Fv[1] = s.u[0] * s.q[1] + s.p;
#pragma unroll
    for (int i = 1; i < ND; ++i) Fv[1 + i] = s.u[0] * s.q[1 + i];
    Fv[NV - 1] = s.u[0] * (s.q[NV - 1] + s.p);
    T cs[NV], cf[NV];
    // FP32 path: the flux is F = u_n q + p (0, 1, 0.., u_n), so L.F = u_n (L.q) + p (L e_1 + u_n L e_E)
    // with the two LEV columns in closed form; the FP64 path projects F itself (the reference's
    // operation order).
    constexpr int NPASS = sizeof(T) == 4 ? 1 : 2;
#pragma unroll
    for (int pass = 0; pass < NPASS; ++pass) {
      const T* v = pass == 0 ? s.q : Fv;
      T* o = pass == 0 ? cs : cf;
      T um = L_(0.0);
#pragma unroll
      for (int i = 0; i < ND; ++i) um += u[i] * v[1 + i];
      T S = phi * v[0] - g1 * um + g1 * v[NV - 1];
      T D = v[1] - u[0] * v[0];
      o[0] = v[0] - S * ia2;
      if (ND == 2) {
        o[1] = (u[1] * v[0] - v[2]) * irho;
      } else {
        o[1] = (v[3] - u[2] * v[0]) * irho;
        o[2] = (u[1] * v[0] - v[2]) * irho;
      }
      o[ND] = bta * (S + a * D);
      o[ND + 1] = bta * (S - a * D);
    }
    if (NPASS == 1) {
      const T un = s.u[0], du = un - u[0];
      const T pb = s.p * bta, gd = g1 * du;
      cf[0] = un * cs[0] - s.p * g1 * ia2 * du;
#pragma unroll
      for (int k = 1; k < ND; ++k) cf[k] = un * cs[k];
      cf[ND] = un * cs[ND] + pb * (a + gd);
      cf[ND + 1] = un * cs[ND + 1] + pb * (gd - a);
    }
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      const T lk = (k < ND) ? lam_u : (k == ND ? lam_p : lam_m);
      fp[k][m] = L_(0.5) * (cf[k] + lk * cs[k]);
      fmn[k][m] = L_(0.5) * (cf[k] - lk * cs[k]);
    }
  }
#pragma unroll
  for (int k = 0; k < NV; ++k) rec[k] = recon_wave<T, SCH, true>(fp[k], fmn[k], sp);
  // back to physical space with the REV columns (k = e_0)
  const T rp = rec[ND] + rec[ND + 1], rm = rec[ND] - rec[ND + 1];
  const T F0 = rec[0] + alf * rp;
  fh[0] = F0;
  fh[1] = u[0] * F0 + alf * a * rm;
  const T h0 = (phi + a * a) / g1;
  if (ND == 2) {
    fh[2] = u[1] * F0 - rho * rec[1];
    fh[3] = phi / g1 * rec[0] - rho * u[1] * rec[1] + alf * h0 * rp + alf * u[0] * a * rm;
  } else {
    fh[2] = u[1] * F0 - rho * rec[2];
    fh[3] = u[2] * F0 + rho * rec[1];
    fh[4] = phi / g1 * rec[0] + rho * u[2] * rec[1] - rho * u[1] * rec[2] + alf * h0 * rp + alf * u[0] * a * rm;
  }
}

// HLLC-LM flux at the interface between w[2] and w[3] of a 6-point window (offsets -2..+3),
// Cartesian local frame (HLLCWeno with flux_type 'HLLC-LM', shock_capturing.py:1031-1256):
// the averaged state and eigensystem as char_flux; the characteristic projections CS = L q of
// the six points; per wave the scheme's fifth-order reconstruction from the left (points
// i-2..i+2) and from the right (i+3..i-1, mirrored); back to physical left and right states with
// the REV columns; then u, p, a of each side, the outer wave speeds sL = min(u_av - a_av,
// uL - aL), sR = max(u_av + a_av, uR + aR), the contact speed s*, both outer speeds scaled by
// phi = sin(pi/2 min(1, 10 M)) with M = max |u/a| of the two sides (the low-Mach correction),
// and the flux in the generated central-plus-dissipation form.  The generated right-state
// energy term divides pR by (sL - uR) rho_R, not (sR - uR) rho_R; this follows it.
template <typename T>
__device__ __forceinline__ T lm_sin(T x);
template <>
__device__ __forceinline__ double lm_sin<double>(double x) { return sin(x); }
template <>
__device__ __forceinline__ float lm_sin<float>(float x) { return sinf(x); }

template <typename T, int ND, int SCH, int AVG>
__device__ __forceinline__ void hllc_flux(const Pt<T, ND> (&w)[6], const SP<T>& sp, T (&fh)[ND + 2]) {
  constexpr int NV = ND + 2;
  const T g1 = sp.g1;
  const Pt<T, ND>& L = w[2];
  const Pt<T, ND>& R = w[3];
  T rho, u[ND], a;
  if (AVG == AVG_ROE) {
    T sL = sqrt(L.q[0]), sR = sqrt(R.q[0]);
    rho = sqrt(L.q[0] * R.q[0]);
    T inv = L_(1.0) / (sL + sR);
    T ke = L_(0.0);
#pragma unroll
    for (int i = 0; i < ND; ++i) {
      u[i] = (sL * L.u[i] + sR * R.u[i]) * inv;
      ke += u[i] * u[i];
    }
    T H = ((L.q[NV - 1] + L.p) / sL + (R.q[NV - 1] + R.p) / sR) * inv;
    a = sqrt(g1 * (H - L_(0.5) * ke));
  } else {
    rho = L_(0.5) * (L.q[0] + R.q[0]);
#pragma unroll
    for (int i = 0; i < ND; ++i) u[i] = L_(0.5) * (L.u[i] + R.u[i]);
    a = L_(0.5) * (L.a + R.a);
  }
  const T ia = L_(1.0) / a, ia2 = ia * ia, irho = L_(1.0) / rho;
  T ke = L_(0.0);
#pragma unroll
  for (int i = 0; i < ND; ++i) ke += u[i] * u[i];
  const T phi = g1 * L_(0.5) * ke;
  const T bta = ia * irho * L_(0.70710678118654752440);
  const T alf = rho * ia * L_(0.70710678118654752440);
  T cs[NV][6];
#pragma unroll
  for (int m = 0; m < 6; ++m) {
    const T* v = w[m].q;
    T um = L_(0.0);
#pragma unroll
    for (int i = 0; i < ND; ++i) um += u[i] * v[1 + i];
    T S = phi * v[0] - g1 * um + g1 * v[NV - 1];
    T D = v[1] - u[0] * v[0];
    cs[0][m] = v[0] - S * ia2;
    if (ND == 2) {
      cs[1][m] = (u[1] * v[0] - v[2]) * irho;
    } else {
      cs[1][m] = (v[3] - u[2] * v[0]) * irho;
      cs[2][m] = (u[1] * v[0] - v[2]) * irho;
    }
    cs[ND][m] = bta * (S + a * D);
    cs[ND + 1][m] = bta * (S - a * D);
  }
  T rl[NV], rr[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    if constexpr (sizeof(T) == 8 && generated_order<ND, SCH>()) {
      rl[k] = recon5_ieee<SCH>(cs[k][0], cs[k][1], cs[k][2], cs[k][3], cs[k][4], sp.teno_eps, sp.teno_ct);
      rr[k] = recon5_ieee<SCH>(cs[k][5], cs[k][4], cs[k][3], cs[k][2], cs[k][1], sp.teno_eps, sp.teno_ct);
    } else {
      rl[k] = recon5<T, SCH>(cs[k][0], cs[k][1], cs[k][2], cs[k][3], cs[k][4], sp);
      rr[k] = recon5<T, SCH>(cs[k][5], cs[k][4], cs[k][3], cs[k][2], cs[k][1], sp);
    }
  }
  // REV columns (k = e_0): characteristic -> conserved, both sides
  T qL[NV], qR[NV];
  const T h0 = (phi + a * a) / g1;
  auto rev = [&](const T (&c)[NV], T (&o)[NV]) {
    const T rp = c[ND] + c[ND + 1], rm = c[ND] - c[ND + 1];
    const T F0 = c[0] + alf * rp;
    o[0] = F0;
    o[1] = u[0] * F0 + alf * a * rm;
    if (ND == 2) {
      o[2] = u[1] * F0 - rho * c[1];
      o[3] = phi / g1 * c[0] - rho * u[1] * c[1] + alf * h0 * rp + alf * u[0] * a * rm;
    } else {
      o[2] = u[1] * F0 - rho * c[2];
      o[3] = u[2] * F0 + rho * c[1];
      o[4] = phi / g1 * c[0] + rho * u[2] * c[1] - rho * u[1] * c[2] + alf * h0 * rp + alf * u[0] * a * rm;
    }
  };
  rev(rl, qL);
  rev(rr, qR);
  const T gm = sp.gama;
  const T irL = L_(1.0) / qL[0], irR = L_(1.0) / qR[0];
  T uL[ND], uR[ND], kL = L_(0.0), kR = L_(0.0);
#pragma unroll
  for (int i = 0; i < ND; ++i) {
    uL[i] = irL * qL[1 + i];
    uR[i] = irR * qR[1 + i];
    kL += uL[i] * uL[i];
    kR += uR[i] * uR[i];
  }
  const T EL = qL[NV - 1], ER = qR[NV - 1];
  const T pL = (-L_(0.5) * kL * qL[0] + EL) * g1, pR = (-L_(0.5) * kR * qR[0] + ER) * g1;
  const T aL = sqrt(gm * irL * pL), aR = sqrt(gm * irR * pR);
  const T un = u[0], uLn = uL[0], uRn = uR[0];
  T sL = fmin(-a + un, -aL + uLn), sR = fmax(a + un, aR + uRn);
  const T ss = (-pL + (-uLn + sL) * qL[0] * uLn - (-uRn + sR) * qR[0] * uRn + pR) /
               ((-uLn + sL) * qL[0] - (-uRn + sR) * qR[0]);
  const T M = fmax(fabs(uLn / aL), fabs(uRn / aR));
  const T lm = lm_sin<T>(L_(0.5) * L_(3.14159265358979323846) * fmin(L_(1.0), L_(10.0) * M));
  sL = lm * sL;
  sR = lm * sR;
  const T mL = (-uLn + sL) * qL[0] / (-ss + sL), mR = (-uRn + sR) * qR[0] / (-ss + sR);
  const T as = fabs(ss);
  if (sL >= L_(0.0)) {
    fh[0] = qL[1];
#pragma unroll
    for (int i = 0; i < ND; ++i) fh[1 + i] = i == 0 ? qL[1] * uLn + pL : qL[1 + i] * uLn;
    fh[NV - 1] = (pL + EL) * uLn;
  } else if (sR <= L_(0.0)) {
    fh[0] = qR[1];
#pragma unroll
    for (int i = 0; i < ND; ++i) fh[1 + i] = i == 0 ? qR[1] * uRn + pR : qR[1 + i] * uRn;
    fh[NV - 1] = (pR + ER) * uRn;
  } else {
    const T hf = L_(0.5);
    fh[0] = hf * qL[1] + hf * qR[1] + hf * (-qL[0] + mL) * sL + hf * (-qR[0] + mR) * sR + hf * (mL - mR) * as;
#pragma unroll
    for (int i = 0; i < ND; ++i) {
      if (i == 0) {
        const T xL = (-uLn + sL) * qL[0] * ss / (-ss + sL), xR = (-uRn + sR) * qR[0] * ss / (-ss + sR);
        fh[1] = hf * pL + hf * pR + hf * (-qL[1] + xL) * sL + hf * (-qR[1] + xR) * sR + hf * (xL - xR) * as +
                hf * qL[1] * uLn + hf * qR[1] * uRn;
      } else {
        const T xL = (-uLn + sL) * qL[0] * uL[i] / (-ss + sL), xR = (-uRn + sR) * qR[0] * uR[i] / (-ss + sR);
        fh[1 + i] = hf * (-qL[1 + i] + xL) * sL + hf * (-qR[1 + i] + xR) * sR + hf * (xL - xR) * as +
                    hf * qL[1 + i] * uLn + hf * qR[1 + i] * uRn;
      }
    }
    const T eL = (-uLn + sL) * ((-uLn + ss) * (pL / ((-uLn + sL) * qL[0]) + ss) + irL * EL) * qL[0] / (-ss + sL);
    const T eR = (-uRn + sR) * ((-uRn + ss) * (pR / ((-uRn + sL) * qR[0]) + ss) + irR * ER) * qR[0] / (-ss + sR);
    fh[NV - 1] = hf * (-EL + eL) * sL + hf * (-ER + eR) * sR + hf * (eL - eR) * as + hf * (pL + EL) * uLn +
                 hf * (pR + ER) * uRn;
  }
}

// Interface flux of a Cartesian sweep: characteristic LLF (FLX 0) or HLLC-LM (FLX 1).
template <typename T, int ND, int SCH, int AVG, int FLX>
__device__ __forceinline__ void cart_flux(const Pt<T, ND> (&w)[6], const SP<T>& sp, T (&fh)[ND + 2]) {
  if constexpr (FLX == 1) {
    hllc_flux<T, ND, SCH, AVG>(w, sp, fh);
  } else {
    char_flux<T, ND, SCH, AVG>(w, sp, fh);
  }
}

// ---------------------------------------------------------------------------------------
// Curvilinear sweeps work in the global frame.  A point carries its conserved state and
// primitives plus the metric row of the sweep direction d, k_i = D_di = d xi_d / d x_i, and
// det J.
template <typename T, int ND>
struct PtC {
  T q[ND + 2];  // rho, rho u_0.., E (global frame)
  T u[ND];
  T p, a;
  T k[ND];      // D_d0 .. D_d(ND-1)
  T J;          // det(d x / d xi)
};

template <typename T, int ND, bool GEN = false>
__device__ __forceinline__ void make_pt(PtC<T, ND>& s, T gm) {
  T rho = s.q[0];
  T ir = L_(1.0) / rho;
  T ke = L_(0.0);
#pragma unroll
  for (int i = 0; i < ND; ++i) {
    s.u[i] = s.q[1 + i] * ir;
    ke += s.u[i] * s.u[i];
  }
  s.p = (gm - L_(1.0)) * (s.q[ND + 1] - L_(0.5) * rho * ke);
  s.a = sqrt(gm * s.p * ir);
}

// Characteristic LLF flux of the curvilinear form at the interface between w[2] and w[3]:
// contravariant flux F = J [rho U, rho u_i U + p D_di, (E + p) U] with U = D_d . u
// (the conservative metric form of the reference's curvilinear Euler equations,
// equation_types/metric.py with the generated "LFWeno_reconstruction" kernels), eigensystem of
// euler_eigensystem.py:100-165 for the unit direction k = avg(D_d) / |avg(D_d)|, LLF speeds
// from the pointwise J (U +- a |D_d|) over points i, i+1.  The eigenvector matrices are
// applied in factored form: with S = phi v0 - g1 (u . v_m) + g1 v_E, E = v0 - S/a^2,
// w = (v_m - u v0)/rho and Dn = k . v_m - (k . u) v0 the rows of LEV are
//   2D: E, k1 w0 - k0 w1, bta (S + a Dn), bta (S - a Dn)
//   3D: k_i E + (w x k)_i (i = 0..2), bta (S + a Dn), bta (S - a Dn)
// and REV is applied column-wise (see the back-projection below).
template <typename T, int ND, int SCH, int AVG>
__device__ __forceinline__ void char_flux_curv(const PtC<T, ND> (&w)[6], const SP<T>& sp, T (&fh)[ND + 2]) {
  static_assert(ND == 2 || ND == 3, "curvilinear sweeps are 2D or 3D");
  constexpr int NV = ND + 2;
  const T g1 = sp.g1;
  const PtC<T, ND>& L = w[2];
  const PtC<T, ND>& R = w[3];
  T rho, u[ND], a;
  if (AVG == AVG_ROE) {
    T sL = sqrt(L.q[0]), sR = sqrt(R.q[0]);
    rho = sqrt(L.q[0] * R.q[0]);
    T inv = L_(1.0) / (sL + sR);
    T ke = L_(0.0);
#pragma unroll
    for (int i = 0; i < ND; ++i) {
      u[i] = (sL * L.u[i] + sR * R.u[i]) * inv;
      ke += u[i] * u[i];
    }
    T H = ((L.q[NV - 1] + L.p) / sL + (R.q[NV - 1] + R.p) / sR) * inv;
    a = sqrt(g1 * (H - L_(0.5) * ke));
  } else {
    rho = L_(0.5) * (L.q[0] + R.q[0]);
#pragma unroll
    for (int i = 0; i < ND; ++i) u[i] = L_(0.5) * (L.u[i] + R.u[i]);
    a = L_(0.5) * (L.a + R.a);
  }
  // unit direction of the averaged metric row
  T k[ND];
  {
    T kn = L_(0.0);
#pragma unroll
    for (int i = 0; i < ND; ++i) {
      k[i] = L_(0.5) * (L.k[i] + R.k[i]);
      kn += k[i] * k[i];
    }
    kn = L_(1.0) / sqrt(kn);
#pragma unroll
    for (int i = 0; i < ND; ++i) k[i] *= kn;
  }
  // LLF speeds: J U and J U +- a |J D_d| at i and i+1
  const T sfc = sp.sfc;
  T lam_u, lam_p, lam_m;
  {
    T UL = L_(0.0), UR = L_(0.0), mL = L_(0.0), mR = L_(0.0);
#pragma unroll
    for (int i = 0; i < ND; ++i) {
      T kl = L.J * L.k[i], kr = R.J * R.k[i];
      UL += kl * L.u[i];
      UR += kr * R.u[i];
      mL += kl * kl;
      mR += kr * kr;
    }
    mL = sqrt(mL);
    mR = sqrt(mR);
    lam_u = sfc * fmax(fabs(UL), fabs(UR));
    lam_p = sfc * fmax(fabs(UL + L.a * mL), fabs(UR + R.a * mR));
    lam_m = sfc * fmax(fabs(UL - L.a * mL), fabs(UR - R.a * mR));
  }
  const T ia = L_(1.0) / a, ia2 = ia * ia, irho = L_(1.0) / rho;
  T ke = L_(0.0), th = L_(0.0);
#pragma unroll
  for (int i = 0; i < ND; ++i) {
    ke += u[i] * u[i];
    th += k[i] * u[i];
  }
  const T phi = g1 * L_(0.5) * ke;
  const T bta = ia * irho * L_(0.70710678118654752440);
  const T alf = rho * ia * L_(0.70710678118654752440);
  T fp[NV][6], fmn[NV][6];
#pragma unroll
  for (int m = 0; m < 6; ++m) {
    const PtC<T, ND>& s = w[m];
    T U = L_(0.0);
#pragma unroll
    for (int i = 0; i < ND; ++i) U += s.k[i] * s.u[i];
    T Fv[NV];
    Fv[0] = s.J * (s.q[0] * U);
#pragma unroll
    for (int i = 0; i < ND; ++i) Fv[1 + i] = s.J * (s.q[1 + i] * U + s.p * s.k[i]);
    Fv[NV - 1] = s.J * ((s.q[NV - 1] + s.p) * U);
    T cs[NV], cf[NV];
#pragma unroll
    for (int pass = 0; pass < 2; ++pass) {
      const T* v = pass == 0 ? s.q : Fv;
      T* o = pass == 0 ? cs : cf;
      T um = L_(0.0), kv = L_(0.0);
#pragma unroll
      for (int i = 0; i < ND; ++i) {
        um += u[i] * v[1 + i];
        kv += k[i] * v[1 + i];
      }
      T S = phi * v[0] - g1 * um + g1 * v[NV - 1];
      T E = v[0] - S * ia2;
      T Dn = kv - th * v[0];
      T wv[ND];
#pragma unroll
      for (int i = 0; i < ND; ++i) wv[i] = (v[1 + i] - u[i] * v[0]) * irho;
      if (ND == 2) {
        o[0] = E;
        o[1] = k[1] * wv[0] - k[0] * wv[1];
      } else {
        o[0] = k[0] * E + (wv[1] * k[2] - wv[2] * k[1]);
        o[1] = k[1] * E + (wv[2] * k[0] - wv[0] * k[2]);
        o[2] = k[2] * E + (wv[0] * k[1] - wv[1] * k[0]);
      }
      o[ND] = bta * (S + a * Dn);
      o[ND + 1] = bta * (S - a * Dn);
    }
#pragma unroll
    for (int c = 0; c < NV; ++c) {
      const T lk = (c < ND) ? lam_u : (c == ND ? lam_p : lam_m);
      fp[c][m] = L_(0.5) * (cf[c] + lk * cs[c]);
      fmn[c][m] = L_(0.5) * (cf[c] - lk * cs[c]);
    }
  }
  T rec[NV];
  if constexpr (sizeof(T) == 4 && (SCH == SCH_WENO5_JS || SCH == SCH_WENO5_Z)) {
    // the waves in pairs (recon5_x2): 0 and 1, the acoustic ones, and in 3D the two sides of wave 2.
    // TENO5 keeps the scalar form: on a curvilinear mesh its cut-off decides on differences that
    // the metric's variation leaves near FP32's rounding, and the pairs' other roundings decide some
    // of them differently (4e-5 instead of 7e-6 from the FP64 path on a 4-block case with 8 points
    // per mesh wavelength; 2.24 against 2.51 ms of its y sweeps at full size).
    const float2 one = f2(1.f);
#pragma unroll
    for (int c = 0; c < NV; c += ND == 3 && c == 0 ? 3 : 2) {
      float2 x[6], y[6];
#pragma unroll
      for (int m = 0; m < 6; ++m) {
        x[m] = f2(fp[c][m], fp[c + 1][m]);
        y[m] = f2(fmn[c][m], fmn[c + 1][m]);
      }
      const float2 r = add2(recon5_x2<SCH>(x[0], x[1], x[2], x[3], x[4], sp.eps32_rel, sp.teno_ct, one),
                            recon5_x2<SCH>(y[5], y[4], y[3], y[2], y[1], sp.eps32_rel, sp.teno_ct, one));
      rec[c] = r.x;
      rec[c + 1] = r.y;
    }
    if constexpr (ND == 3) {
      const float2 r = recon5_x2<SCH>(f2(fp[2][0], fmn[2][5]), f2(fp[2][1], fmn[2][4]), f2(fp[2][2], fmn[2][3]),
                                      f2(fp[2][3], fmn[2][2]), f2(fp[2][4], fmn[2][1]), sp.eps32_rel, sp.teno_ct, one);
      rec[2] = r.x + r.y;
    }
  } else {
#pragma unroll
    for (int c = 0; c < NV; ++c) rec[c] = recon_wave<T, SCH, generated_order<ND, SCH>()>(fp[c], fmn[c], sp);
  }
  // REV: 2D columns (1, u, phi/g1), rho (0, t, t.u) with t = (k1, -k0), and the acoustic
  // pair alf (1, u +- a k, h0 +- a th); 3D vorticity columns give u (k.r) + rho (k x r) and
  // phi/g1 (k.r) + rho (u x k).r.
  const T rp = rec[ND] + rec[ND + 1], rm = rec[ND] - rec[ND + 1];
  const T h0 = (phi + a * a) / g1;
  if (ND == 2) {
    const T t0 = k[1], t1 = -k[0];
    const T F0 = rec[0] + alf * rp;
    fh[0] = F0;
    fh[1] = u[0] * F0 + alf * a * k[0] * rm + rho * rec[1] * t0;
    fh[2] = u[1] * F0 + alf * a * k[ND - 1] * rm + rho * rec[1] * t1;
    fh[NV - 1] = phi / g1 * rec[0] + rho * (t0 * u[0] + t1 * u[1]) * rec[1] + alf * h0 * rp + alf * a * th * rm;
  } else {
    const T kr = k[0] * rec[0] + k[1] * rec[1] + k[ND - 1] * rec[2];
    const T c0 = k[1] * rec[2] - k[ND - 1] * rec[1];
    const T c1 = k[ND - 1] * rec[0] - k[0] * rec[2];
    const T c2 = k[0] * rec[1] - k[1] * rec[0];
    const T F0 = kr + alf * rp;
    fh[0] = F0;
    fh[1] = u[0] * F0 + rho * c0 + alf * a * k[0] * rm;
    fh[2] = u[1] * F0 + rho * c1 + alf * a * k[1] * rm;
    fh[3] = u[ND - 1] * F0 + rho * c2 + alf * a * k[ND - 1] * rm;
    const T x0 = u[1] * k[ND - 1] - u[ND - 1] * k[1];
    const T x1 = u[ND - 1] * k[0] - u[0] * k[ND - 1];
    const T x2 = u[0] * k[1] - u[1] * k[0];
    fh[NV - 1] = phi / g1 * kr + rho * (x0 * rec[0] + x1 * rec[1] + x2 * rec[2]) + alf * (h0 * rp + a * th * rm);
  }
}

// Central 4th-order first / second derivative weights (scheme.py:83-87), applied to
// differences of the stencil values: the weights of either rule sum to zero, and in this form
// they stay exactly consistent after rounding (a constant field gives exactly zero).  In the
// weighted-sum form the FP32 roundings of 1/12 and 4/3 leave the second-derivative weights
// summing to 7.5e-8, which 1/Delta^2 turns into a systematic source of 7.5e-8 f / Delta^2 (on a
// wall-normal Delta of 2/256 with T ~ 1, 1.2e-3 per point in the Laplacian of T).  The differences
// of neighbouring values are exact when they lie within a factor of two of each other.
template <typename T>
__device__ __forceinline__ T d1w(T fm2, T fm1, T fp1, T fp2) {
  return L_(1.0 / 12.0) * (fm2 - fp2) + L_(2.0 / 3.0) * (fp1 - fm1);
}
template <typename T>
__device__ __forceinline__ T d2w(T fm2, T fm1, T f0, T fp1, T fp2) {
  return L_(4.0 / 3.0) * ((fm1 - f0) + (fp1 - f0)) - L_(1.0 / 12.0) * ((fm2 - f0) + (fp2 - f0));
}

}  // namespace osb
