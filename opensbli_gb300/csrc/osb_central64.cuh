// osb_central64.cuh -- FP64 central 4th-order kernel: skew-symmetric (Feiereisen) convective terms
// and/or viscous stress and heat flux of a 3D block without wall faces (the terms and their
// sources in the generated solver: k_central3d).
//
// Bound by the FP64 pipe (16.3 cycles per warp instruction and SM), so it is arranged for the
// fewest FP64 instructions per point, about 290 (viscous terms with the Sutherland law) and 390
// (Feiereisen with constant viscosity) against 615 and 1 030 of k_central3d in FP64:
//  * the mixed second derivatives enter the momentum equations only as the derivative along i of
//    the other two directions' D_j u_j, so those sums are formed once per point -- in shared memory
//    for x and y, in registers along z -- instead of six 4x4-point stencils;
//  * E / rho, 2 p and p + E / 2 are staged, so no division is repeated for the twelve neighbours of
//    a point, and reciprocals are Newton's (rcp_newton);
//  * the energy equation takes u_i times the momentum contributions already formed, and the
//    dissipation the symmetric half of tau : grad u;
//  * a column of 32 x 8 points stages 1.7 points per computed one (2.25 with 32 x 4).
#pragma once
#include "osb_kernels.cuh"

namespace osb {

constexpr int C64Y = 8, C64SY = C64Y + 2 * CH, C64PL = CSX * C64SY, C64T = CX * C64Y;
constexpr int C64PP = (C64PL + C64T - 1) / C64T;  // staged points per thread and plane

// Staged fields: velocity; VISC: temperature (and viscosity unless constant); CONV: momentum, 2 p,
// E / rho and p + E / 2.
template <int CONV, int VISC>
struct C64Fields {
  static constexpr int U = 0, TT = 3, MU = 4;
  static constexpr int M = 3 + (VISC ? (VISC == 1 ? 2 : 1) : 0), P2 = M + 3, EE = M + 4, HH = M + 5;
  static constexpr int N = CONV ? M + 6 : M;
};
template <int CONV, int VISC>
constexpr size_t c64_smem() {
  return sizeof(double) * ((size_t)C64Fields<CONV, VISC>::N * CRING * C64PL + (VISC ? CSX * C64Y + CX * C64SY : 0));
}

template <int CONV, int VISC>
__global__ void __launch_bounds__(C64T, CONV ? 1 : 2) k_central_f64(BlockK b, CentralParams cp, int first, int czc) {
  using Fd = C64Fields<CONV, VISC>;
  constexpr int FS = CRING * C64PL;
  extern __shared__ __align__(16) unsigned char osb_smem[];
  double* sm = reinterpret_cast<double*>(osb_smem);
  double* Sx = sm + Fd::N * FS;       // [C64Y][CSX]: D_y u_y + D_z u_z of the current plane
  double* Sy = Sx + CSX * C64Y;       // [C64SY][CX]: D_x u_x + D_z u_z
  const int tx = threadIdx.x % CX, ty = threadIdx.x / CX;
  const int x0 = blockIdx.x * CX, y0 = blockIdx.y * C64Y;
  const int zb = blockIdx.z * czc, ze = min(b.n[2], zb + czc);
  const double g1 = cp.gama - 1.0;
  double qv[C64PP][5];
  auto load_plane = [&](int gz) {
#pragma unroll
    for (int u = 0; u < C64PP; ++u) {
      const int idx = threadIdx.x + u * C64T;
      const int gx = x0 - CH + idx % CSX, gy = y0 - CH + idx / CSX;
      if (idx < C64PL && gx <= b.n[0] + CH && gy <= b.n[1] + CH) {
        const int id = lin(b, gx, gy, gz);
#pragma unroll
        for (int v = 0; v < 5; ++v) qv[u][v] = __ldg(b.q[v] + id);
      }
    }
  };
  auto store_plane = [&](int slot) {
#pragma unroll
    for (int u = 0; u < C64PP; ++u) {
      const int idx = threadIdx.x + u * C64T;
      const int gx = x0 - CH + idx % CSX, gy = y0 - CH + idx / CSX;
      if (!(idx < C64PL && gx <= b.n[0] + CH && gy <= b.n[1] + CH)) continue;
      double* at = sm + slot * C64PL + idx;
      const double rho = qv[u][0], m0 = qv[u][1], m1 = qv[u][2], m2 = qv[u][3], E = qv[u][4];
      const double ir = rcp_newton(rho);
      const double u0 = m0 * ir, u1 = m1 * ir, u2 = m2 * ir;
      const double p = g1 * (E - 0.5 * (m0 * u0 + m1 * u1 + m2 * u2));
      at[(Fd::U + 0) * FS] = u0;
      at[(Fd::U + 1) * FS] = u1;
      at[(Fd::U + 2) * FS] = u2;
      if (VISC) {
        const double Tt = (cp.M2 * cp.gama) * p * ir;
        at[Fd::TT * FS] = Tt;
        if (VISC == 1)
          at[Fd::MU * FS] = cp.mu_pow > 0.0 ? pow(Tt, cp.mu_pow) : 1.4042 * Tt * sqrt(Tt) * rcp_newton(0.40417 + Tt);
      }
      if (CONV) {
        at[(Fd::M + 0) * FS] = m0;
        at[(Fd::M + 1) * FS] = m1;
        at[(Fd::M + 2) * FS] = m2;
        at[Fd::P2 * FS] = 2.0 * p;
        at[Fd::EE * FS] = E * ir;
        at[Fd::HH * FS] = __fma_rn(0.5, E, p);
      }
    }
  };
  auto slot_of = [](int gz) { return (gz + 2 * CRING) % CRING; };
  // first derivative of differences t1 = f(+1) - f(-1), t2 = f(+2) - f(-2) along j; second
  // derivative with each neighbour's difference from the centre (exactly zero on a constant)
  const double a8[3] = {(2.0 / 3.0) * cp.invd[0], (2.0 / 3.0) * cp.invd[1], (2.0 / 3.0) * cp.invd[2]};
  const double a1[3] = {(1.0 / 12.0) * cp.invd[0], (1.0 / 12.0) * cp.invd[1], (1.0 / 12.0) * cp.invd[2]};
  const double b4[3] = {(4.0 / 3.0) * cp.inv2d[0], (4.0 / 3.0) * cp.inv2d[1], (4.0 / 3.0) * cp.inv2d[2]};
  const double b1[3] = {(1.0 / 12.0) * cp.inv2d[0], (1.0 / 12.0) * cp.inv2d[1], (1.0 / 12.0) * cp.inv2d[2]};
  auto d1 = [&](int j, double fm2, double fm1, double fp1, double fp2) -> double {
    return __fma_rn(a8[j], fp1 - fm1, -(a1[j] * (fp2 - fm2)));
  };
  auto d2 = [&](int j, double fm2, double fm1, double f0, double fp1, double fp2) -> double {
    return __fma_rn(b4[j], (fm1 - f0) + (fp1 - f0), -(b1[j] * ((fm2 - f0) + (fp2 - f0))));
  };
  const int gx = x0 + tx, gy = y0 + ty;
  const bool active = gx < b.n[0] && gy < b.n[1];
  const int own = (ty + CH) * CSX + (tx + CH);
  int pb[2 * CH + 1] = {0};  // ring bases of planes gz-2 .. gz+2
  // in-plane derivative of a field at staged point `at` of plane pb[k]
  auto dp = [&](int f, int j, int k, int at) -> double {
    const double* s = sm + f * FS + pb[k] + at;
    const int o = j == 0 ? 1 : CSX;
    return d1(j, s[-2 * o], s[-o], s[o], s[2 * o]);
  };
  // z derivative at the current plane
  auto dz = [&](int f, int at) -> double {
    const double* s = sm + f * FS + at;
    return d1(2, s[pb[0]], s[pb[1]], s[pb[3]], s[pb[4]]);
  };
  for (int gz = zb - CH; gz < zb + CH; ++gz) {
    load_plane(gz);
    store_plane(slot_of(gz));
  }
  load_plane(zb + CH);
  // this column's D_x u_x and D_y u_y of planes gz .. gz+2, and their sum of planes gz-2 .. gz+2
  double d00[3], d11[3], sz[5];
  if (VISC) {
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      pb[k] = slot_of(zb - CH + k) * C64PL;
      const double x = dp(Fd::U + 0, 0, k, own), y = dp(Fd::U + 1, 1, k, own);
      sz[k + 1] = x + y;
      if (k >= 2) {
        d00[k - 1] = x;
        d11[k - 1] = y;
      }
    }
  }
  for (int gz = zb; gz < ze; ++gz) {
    store_plane(slot_of(gz + CH));
    __syncthreads();
    if (gz + CH + 1 < ze + CH) load_plane(gz + CH + 1);
#pragma unroll
    for (int k = 0; k <= 2 * CH; ++k) pb[k] = slot_of(gz + k - CH) * C64PL;
    double du[3][3];
    if (VISC) {
#pragma unroll
      for (int k = 0; k < 4; ++k) sz[k] = sz[k + 1];
      d00[0] = d00[1]; d00[1] = d00[2];
      d11[0] = d11[1]; d11[1] = d11[2];
      d00[2] = dp(Fd::U + 0, 0, 4, own);
      d11[2] = dp(Fd::U + 1, 1, 4, own);
      sz[4] = d00[2] + d11[2];
      du[0][0] = d00[0];
      du[1][1] = d11[0];
      du[2][2] = dz(Fd::U + 2, own);
      Sx[ty * CSX + tx + CH] = du[1][1] + du[2][2];
      Sy[(ty + CH) * CX + tx] = du[0][0] + du[2][2];
      // the halo of those sums: rows 0, 1, 10, 11 of Sy by warps 0..3, columns 0, 1, 34, 35 of Sx by warp 4
      if (ty < 4) {
        const int r = ty < 2 ? ty : ty + C64Y;
        const int at = r * CSX + tx + CH;
        Sy[r * CX + tx] = dp(Fd::U + 0, 0, 2, at) + dz(Fd::U + 2, at);
      } else if (ty == 4) {
        const int r = tx >> 2, c = (tx & 3) < 2 ? (tx & 3) : CX + (tx & 3);
        const int at = (r + CH) * CSX + c;
        Sx[r * CSX + c] = dp(Fd::U + 1, 1, 2, at) + dz(Fd::U + 2, at);
      }
      __syncthreads();
    }
    if (active) {
      const int gid = lin(b, gx, gy, gz);
      double R0[5];
      if (!first) {
#pragma unroll
        for (int v = CONV ? 0 : 1; v < 5; ++v) R0[v] = b.R[v][gid];
      }
      const double* c = sm + pb[2] + own;
      // stencil values along j: f(m) at m = -2 .. 2
      auto F = [&](int f, int j, int m) -> double {
        return j == 2 ? sm[f * FS + pb[m + CH] + own] : c[f * FS + m * (j == 0 ? 1 : CSX)];
      };
      double racc[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
      if (!VISC) du[0][0] = d1(0, F(0, 0, -2), F(0, 0, -1), F(0, 0, 1), F(0, 0, 2));
      if (!VISC) du[1][1] = d1(1, F(1, 1, -2), F(1, 1, -1), F(1, 1, 1), F(1, 1, 2));
      if (!VISC) du[2][2] = d1(2, F(2, 2, -2), F(2, 2, -1), F(2, 2, 1), F(2, 2, 2));
      const double uc[3] = {c[0], c[FS], c[2 * FS]};
      double lap[3] = {0.0, 0.0, 0.0}, dT[3], dmu[3], lapT = 0.0;
      double divm = 0.0, cm[3] = {0.0, 0.0, 0.0}, ce = 0.0;
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        double u[3][5];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
#pragma unroll
          for (int m = 0; m < 5; ++m) u[i][m] = m == 2 ? uc[i] : F(Fd::U + i, j, m - 2);
          if (i != j) du[i][j] = d1(j, u[i][0], u[i][1], u[i][3], u[i][4]);
          if (VISC) {
            const double s = d2(j, u[i][0], u[i][1], u[i][2], u[i][3], u[i][4]);
            lap[i] = i == j ? __fma_rn(4.0 / 3.0, s, lap[i]) : lap[i] + s;
          }
        }
        if (VISC) {
          const double t[5] = {F(Fd::TT, j, -2), F(Fd::TT, j, -1), c[Fd::TT * FS], F(Fd::TT, j, 1), F(Fd::TT, j, 2)};
          lapT += d2(j, t[0], t[1], t[2], t[3], t[4]);
          if (VISC == 1) {
            dT[j] = d1(j, t[0], t[1], t[3], t[4]);
            dmu[j] = d1(j, F(Fd::MU, j, -2), F(Fd::MU, j, -1), F(Fd::MU, j, 1), F(Fd::MU, j, 2));
          }
        }
        if (CONV) {
          // R_rho -= D_j m_j ; R_m_i -= 1/2 [D_j(m_i u_j + 2 p delta_ij) + u_i D_j m_j + m_j D_j u_i]
          // R_E -= D_j((p + E/2) u_j) + 1/2 [m_j D_j(E/rho) + (E/rho) D_j m_j]
          double mm[3][4], hh[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int m = k < 2 ? k - 2 : k - 1;
            const double uj = u[j][m + 2];
#pragma unroll
            for (int i = 0; i < 3; ++i) mm[i][k] = F(Fd::M + i, j, m);
            hh[k] = F(Fd::HH, j, m) * uj;
          }
          divm += d1(j, mm[j][0], mm[j][1], mm[j][2], mm[j][3]);
          const double mj = c[(Fd::M + j) * FS];
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            double pr[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const int m = k < 2 ? k - 2 : k - 1;
              pr[k] = i == j ? __fma_rn(mm[i][k], u[j][m + 2], F(Fd::P2, j, m)) : mm[i][k] * u[j][m + 2];
            }
            cm[i] += __fma_rn(mj, du[i][j], d1(j, pr[0], pr[1], pr[2], pr[3]));
          }
          const double dE = d1(j, F(Fd::EE, j, -2), F(Fd::EE, j, -1), F(Fd::EE, j, 1), F(Fd::EE, j, 2));
          ce += __fma_rn(0.5 * mj, dE, d1(j, hh[0], hh[1], hh[2], hh[3]));
        }
      }
      if (CONV) {
        racc[0] = -divm;
#pragma unroll
        for (int i = 0; i < 3; ++i) racc[1 + i] = -0.5 * __fma_rn(uc[i], divm, cm[i]);
        racc[4] = -__fma_rn(0.5 * divm, c[Fd::EE * FS], ce);
      }
      if (VISC) {
        const double* px = Sx + ty * CSX + tx + CH;
        const double* py = Sy + (ty + CH) * CX + tx;
        lap[0] = __fma_rn(1.0 / 3.0, d1(0, px[-2], px[-1], px[1], px[2]), lap[0]);
        lap[1] = __fma_rn(1.0 / 3.0, d1(1, py[-2 * CX], py[-CX], py[CX], py[2 * CX]), lap[1]);
        lap[2] = __fma_rn(1.0 / 3.0, d1(2, sz[0], sz[1], sz[3], sz[4]), lap[2]);
        const double mu = VISC == 1 ? c[Fd::MU * FS] : cp.mu_c;
        const double div3 = (2.0 / 3.0) * (du[0][0] + du[1][1] + du[2][2]);
        const double t01 = du[0][1] + du[1][0], t02 = du[0][2] + du[2][0], t12 = du[1][2] + du[2][1];
        const double t0 = __fma_rn(2.0, du[0][0], -div3), t1 = __fma_rn(2.0, du[1][1], -div3),
                     t2 = __fma_rn(2.0, du[2][2], -div3);
        double m[3] = {mu * lap[0], mu * lap[1], mu * lap[2]};
        if (VISC == 1) {
          m[0] += t0 * dmu[0] + t01 * dmu[1] + t02 * dmu[2];
          m[1] += t01 * dmu[0] + t1 * dmu[1] + t12 * dmu[2];
          m[2] += t02 * dmu[0] + t12 * dmu[1] + t2 * dmu[2];
        }
        const double phi = t0 * du[0][0] + t1 * du[1][1] + t2 * du[2][2] + t01 * t01 + t02 * t02 + t12 * t12;
        const double e = mu * phi + uc[0] * m[0] + uc[1] * m[1] + uc[2] * m[2];
        double h = mu * lapT;
        if (VISC == 1) h += dT[0] * dmu[0] + dT[1] * dmu[1] + dT[2] * dmu[2];
#pragma unroll
        for (int i = 0; i < 3; ++i) racc[1 + i] = __fma_rn(m[i], cp.invRe, racc[1 + i]);
        racc[4] += e * cp.invRe + h * cp.kheat;
        if (cp.forced) {
          double w = 0.0;
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            racc[1 + i] -= cp.force[i];
            w += cp.force[i] * uc[i];
          }
          racc[4] -= w;
        }
      }
#pragma unroll
      for (int v = CONV ? 0 : 1; v < 5; ++v) b.R[v][gid] = first ? racc[v] : R0[v] + racc[v];
    }
    __syncthreads();  // the next iteration overwrites plane gz-2 and the sums
  }
}

}  // namespace osb
