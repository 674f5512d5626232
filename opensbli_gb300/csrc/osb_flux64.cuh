// osb_flux64.cuh -- FP64 characteristic sweep along one direction, one interface per thread.
//
// A CTA stages the points of a tile (their state in the direction's frame and their primitives,
// formed once per point) in shared memory, computes the tile's 512 interfaces in two rounds of 256
// threads, and updates the residual of the points between them.  Along x a tile is 64 interfaces of 8
// rows, along y and z 16 interfaces of 32 lines (the lines numbered across rows, as in
// k_flux_sweep), so its loads and stores run along x either way; a line's points are cut evenly.
//
// The FP64 pipe is the bound (16.3 cycles per warp instruction and SM), but a result takes several
// times that, so warps are what keeps it busy: the window of six points stays in shared memory
// (read again by every wave, 140 loads of 64 bits per interface against 5 800 cycles of
// arithmetic), which leaves 16 warps per SM where a window in registers (255 of them) left 8, and
// gives small blocks a thread per interface instead of one per line segment.
#pragma once
#include "osb_kernels.cuh"

namespace osb {

constexpr int F64T = 256, F64I = 512;  // threads, interfaces per tile
template <int D>
struct F64Tile {
  static constexpr int NI = D == 0 ? 64 : 16;  // interfaces along D
  static constexpr int NC = F64I / NI;         // lines
  static constexpr int NP = NI + 5;            // staged points along D
};
template <int ND, int D, int AVG>
struct F64Fields {
  // state, u_n, p, tangential velocities, a; Roe: sqrt(rho), H
  static constexpr int NV = ND + 2, UN = NV, P = NV + 1, UT = NV + 2, A = NV + 1 + ND;
  static constexpr int S = A + 1, H = A + 2, N = A + 1 + (AVG == AVG_ROE ? 2 : 0);
  static constexpr int PL = F64Tile<D>::NP * F64Tile<D>::NC;
  static constexpr size_t bytes = sizeof(double) * ((size_t)N * PL + (size_t)NV * F64I);
};

// Window of an interface in the staged tile; volatile: read where it is used, not held in registers.
template <int ND, int D, int AVG>
struct TileF64 {
  using Fd = F64Fields<ND, D, AVG>;
  static constexpr int ST = D == 0 ? 1 : F64Tile<D>::NC;  // step along D
  const volatile double* s;
  __device__ __forceinline__ double f(int m, int v) const { return s[v * Fd::PL + m * ST]; }
  __device__ __forceinline__ double q(int m, int v) const { return f(m, v); }
  __device__ __forceinline__ double un(int m) const { return f(m, Fd::UN); }
  __device__ __forceinline__ double p(int m) const { return f(m, Fd::P); }
  __device__ __forceinline__ Pt<double, ND> side(int m) const {
    Pt<double, ND> w;
    w.q[0] = f(m, 0);
    w.u[0] = f(m, Fd::UN);
#pragma unroll
    for (int i = 1; i < ND; ++i) w.u[i] = f(m, Fd::UT + i - 1);
    w.a = f(m, Fd::A);
    if (AVG == AVG_ROE) {
      w.s = f(m, Fd::S);
      w.H = f(m, Fd::H);
    }
    return w;
  }
  __device__ __forceinline__ Pt<double, ND> point(int m) const {
    Pt<double, ND> w;
#pragma unroll
    for (int v = 0; v < ND + 2; ++v) w.q[v] = f(m, v);
    w.u[0] = f(m, Fd::UN);
#pragma unroll
    for (int i = 1; i < ND; ++i) w.u[i] = f(m, Fd::UT + i - 1);
    w.p = f(m, Fd::P);
    w.a = f(m, Fd::A);
    return w;
  }
};

// Sweep of `pts` points per line part, blockIdx.y parts; `first` writes the residual, else adds to it.
template <int ND, int D, int SCH, int AVG>
__global__ void __launch_bounds__(F64T, generated_order<ND, SCH>() ? 1 : 2) k_flux_tile(BlockK b, SchemeParams spd, int pts, int first) {
  constexpr int NV = ND + 2;
  using Tl = F64Tile<D>;
  using Fd = F64Fields<ND, D, AVG>;
  const SP<double> sp(spd);
  extern __shared__ __align__(16) unsigned char osb_smem[];
  double* sm = reinterpret_cast<double*>(osb_smem);
  double* fl = sm + Fd::N * Fd::PL;  // [NV][interface]
  const int N = b.n[D], s = b.st[D];
  const int i0 = blockIdx.y * pts, np = min(pts, N - i0);  // points i0 .. i0 + np - 1, interfaces 0 .. np
  if (np <= 0) return;
  // line c of the tile: linear index of its point 0 along D; lines past the end repeat the last
  const int lines = (D == 0 ? 1 : b.n[0]) * (ND == 3 ? (D == 2 ? b.n[1] : D == 1 ? b.n[2] : b.n[1] * b.n[2]) : (D == 0 ? b.n[1] : 1));
  const int l0 = blockIdx.x * Tl::NC;
  auto line_base = [&](int c) -> int {
    const int l = min(l0 + c, lines - 1);
    if (D == 0) return lin(b, 0, ND == 3 ? l % b.n[1] : l, ND == 3 ? l / b.n[1] : 0);
    const int o = ND == 3 ? l / b.n[0] : 0, x = l - o * b.n[0];
    return lin(b, x, ND == 3 && D == 2 ? o : 0, ND == 3 && D == 1 ? o : 0);
  };
  // staged point k of line c sits at c * NP + k (x) or k * NC + c
  for (int u = threadIdx.x; u < (np + 6) * Tl::NC; u += F64T) {
    const int k = D == 0 ? u % (np + 6) : u / Tl::NC, c = D == 0 ? u / (np + 6) : u % Tl::NC;
    const int id = line_base(c) + (i0 - 3 + k) * s;
    Pt<double, ND> w;
#pragma unroll
    for (int lv = 0; lv < NV; ++lv) w.q[lv] = __ldg(b.q[gvar_fwd<ND, D>(lv)] + id);
    make_pt<double, ND>(w, sp.gama);
    double* at = sm + (D == 0 ? c * Tl::NP + k : k * Tl::NC + c);
#pragma unroll
    for (int lv = 0; lv < NV; ++lv) at[lv * Fd::PL] = w.q[lv];
    at[Fd::UN * Fd::PL] = w.u[0];
    at[Fd::P * Fd::PL] = w.p;
#pragma unroll
    for (int i = 1; i < ND; ++i) at[(Fd::UT + i - 1) * Fd::PL] = w.u[i];
    at[Fd::A * Fd::PL] = w.a;
    if (AVG == AVG_ROE) {
      at[Fd::S * Fd::PL] = w.s;
      at[Fd::H * Fd::PL] = w.H;
    }
  }
  __syncthreads();
  for (int u = threadIdx.x; u < (np + 1) * Tl::NC; u += F64T) {
    const int i = D == 0 ? u % (np + 1) : u / Tl::NC, c = D == 0 ? u / (np + 1) : u % Tl::NC;  // left face of point i
    double fh[NV];
    const TileF64<ND, D, AVG> win{sm + (D == 0 ? c * Tl::NP + i : i * Tl::NC + c)};
    if constexpr (generated_order<ND, SCH>()) {
      Pt<double, ND> w[6];
#pragma unroll
      for (int m = 0; m < 6; ++m) w[m] = win.point(m);
      char_flux<double, ND, SCH, AVG>(w, sp, fh);
    } else {
      char_flux_f64<ND, SCH, AVG>(win, sp, fh);
    }
    double* at = fl + (D == 0 ? c * Tl::NI + i : i * Tl::NC + c);
#pragma unroll
    for (int lv = 0; lv < NV; ++lv) at[lv * F64I] = fh[lv];
  }
  __syncthreads();
  for (int u = threadIdx.x; u < np * Tl::NC; u += F64T) {
    const int i = D == 0 ? u % np : u / Tl::NC, c = D == 0 ? u / np : u % Tl::NC;
    if (l0 + c >= lines) continue;
    const int id = line_base(c) + (i0 + i) * s;
    const double* at = fl + (D == 0 ? c * Tl::NI + i : i * Tl::NC + c);
    double sc = b.invd[D];
    // stretched y grid: -(F_j+1/2 - F_j-1/2) / Delta_1 * D11_j (the generated residual's order)
    if (D == 1)
      if (b.ys[0]) sc *= b.ys[0][i0 + i];
#pragma unroll
    for (int lv = 0; lv < NV; ++lv)
      acc_flux(b, gvar_fwd<ND, D>(lv), id, at[lv * F64I + (D == 0 ? 1 : Tl::NC)], at[lv * F64I], sc, first);
  }
}

}  // namespace osb
