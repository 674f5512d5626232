// osb_resident.cu -- whole calls of osb_step on small 1D blocks in one launch.
//
// A 1D block of a few thousand points (the Sod shock tube: 400) is far too small to fill a GPU;
// per-stage launches (flux, update, boundaries) leave it bound by launch latency.  Here one cluster
// of up to 16 CTAs holds a block's state, RK register and interface fluxes in shared memory and runs
// every stage of every requested step itself: boundary treatment, the primitives of every point,
// the characteristic flux of every interface (one thread per interface, the same char_flux as the
// sweeps), the residual and the RK update (rk_LS.py:204-215 / rk_sbli.py:138-154).  A CTA owns a
// run of points; after an update it writes its outer three points into its neighbours' shared
// memory, and one cluster barrier ends the stage.  One cluster per block: blocks of one context
// advance independently (no interfaces).  Both precisions; FP32 blocks of a few hundred points, and
// contexts with more of them than the chip has room for clusters, take one CTA each (k_resident_cta).
//
// FP64 is bound by the FP64 pipe (one warp instruction per 16 cycles and SM), so the points go to as
// many SMs as still get a full warp of interfaces: one CTA took 61 us a stage for 400 points (100 us
// before the flux was rewritten), see launch_resident for the split and the time now.
#include <cooperative_groups.h>

#include <algorithm>
#include <vector>

#include "osb_internal.h"

// compiled once per residual precision (OSB_RESIDENT_T), the FP32 one with fast-math intrinsics
// like the other FP32-residual kernels
#ifndef OSB_RESIDENT_T
#define OSB_RESIDENT_T double
#define OSB_RESIDENT_NAME resident_f64
#endif

namespace cg = cooperative_groups;

namespace osb {
namespace {

constexpr int RT = 256;        // most threads per CTA
constexpr int RH = 3;          // stencil reach of the flux difference
constexpr int RC = 16;         // most CTAs per cluster (8 where 16 are not to be had)
constexpr size_t SMEM_MAX = 227 * 1024;  // shared memory of a CTA

struct RkCoef {
  int kind, nst;
  double A[8], B[8];
};

struct Resident1D {
  BlockK k;
  int bc[2], depth[2];
};

// Shared memory of a CTA that owns up to `most` points.
template <typename T>
struct RLayout {
  double *q, *o;       // [3][most]: state and register
  double* halo;        // [2 parities][2 sides][RH points][3]: the neighbours' outer points
  T *F;                // [3][most + 1]: flux at the left face of point i (FP64: its three reconstructed waves)
  T *V;                // FP64: [3][most + 1]: averaged u, a, 1 / a (or H) of the face
  T* P;                // [8][most + 2 RH]: rho, m, E, u, p, a (, sqrt(rho), H in FP64) from point -RH
  __device__ RLayout(unsigned char* sm, int most) {
    q = reinterpret_cast<double*>(sm);
    o = q + 3 * most;
    halo = o + 3 * most;
    F = reinterpret_cast<T*>(halo + 2 * 2 * RH * 3);
    V = F + 3 * (most + 1);
    P = V + (sizeof(T) == 8 ? 3 * (most + 1) : 0);
  }
  static size_t bytes(int most) {
    return sizeof(double) * (6 * (size_t)most + 2 * 2 * RH * 3) + sizeof(T) * ((sizeof(T) == 8 ? 6 : 3) * (size_t)(most + 1) + 8 * (size_t)(most + 2 * RH));
  }
};

// Halo value m = 1 .. depth of variable array f beyond the end point f[0] on one side of a block
// (s: inward step), zero-gradient and extrapolation as k_zero_grad / k_extrap; e0: the end point's
// value after the boundary treatment.
__device__ __forceinline__ double end_point(int kind, const double* f, int s) {
  return kind == OSB_BC_EXTRAP1 ? f[0] : f[s];
}
__device__ __forceinline__ double halo_point(int kind, const double* f, int s, int m) {
  if (kind == OSB_BC_ZERO_GRAD) return f[m * s];
  if (kind == OSB_BC_EXTRAP0) return f[s];
  double a = f[s], b = f[0];
  for (int i = 0; i < m; ++i) {
    const double c = -a + 2.0 * b;
    a = b;
    b = c;
  }
  return b;
}

template <typename T>
__device__ __forceinline__ T to_t(double x) {
  if constexpr (sizeof(T) == 8) return x;
  else return d2f_rn(x);
}

// Primitives of a point (make_pt) to and from its column of the staged arrays.
template <typename T, int AVG>
__device__ __forceinline__ void put_prims(T* P, int stride, const Pt<T, 1>& w) {
  P[3 * stride] = w.u[0];
  P[4 * stride] = w.p;
  P[5 * stride] = w.a;
  if constexpr (sizeof(T) == 8 && AVG == AVG_ROE) {
    P[6 * stride] = w.s;
    P[7 * stride] = w.H;
  }
}
template <typename T, int AVG>
__device__ __forceinline__ void get_prims(const T* P, int stride, Pt<T, 1>& w) {
  w.u[0] = P[3 * stride];
  w.p = P[4 * stride];
  w.a = P[5 * stride];
  if constexpr (sizeof(T) == 8 && AVG == AVG_ROE) {
    w.s = P[6 * stride];
    w.H = P[7 * stride];
  }
}

// FP64: the interfaces of a CTA are few (a warp of them), and an FP64 instruction's result takes
// several times the 16 cycles of its issue, so one warp leaves the pipe mostly waiting.  Each
// wave of an interface goes to its own warp, and the point's own thread turns the waves of its two
// faces into fluxes.  WENO takes char_flux_f64's rows for one dimension, k = 0 entropy, 1 u + a, 2 u - a
// (the 400-point shock tube's 50 steps: 0.46 ms, and 0.65 ms with wave_1d's divisions), TENO wave_1d.
template <int SCH>
__device__ __forceinline__ double wave_1d_f64(int k, const Pt<double, 1> (&w)[6], const SP<double>& sp, double u, double a,
                                          double ia, double ke) {
  const Pt<double, 1>& L = w[2];
  const Pt<double, 1>& R = w[3];
  const double hk = 0.5 * ke, gi = sp.g1 * ia, g = gi * ia;
  const double sg = k == 0 ? 0.0 : (k == 1 ? 1.0 : -1.0);
  const double lam = sp.sfc * fmax(fabs(__fma_rn(sg, L.a, L.u[0])), fabs(__fma_rn(sg, R.a, R.u[0])));
  const double cp = k == 0 ? -g : gi;  // c = cp P + rho (entropy) or + sg D
  double fp[6], fm[6];
#pragma unroll
  for (int m = 0; m < 6; ++m) {
    const double P = __fma_rn(hk, w[m].q[0], __fma_rn(-u, w[m].q[1], w[m].q[2]));
    const double D = k == 0 ? w[m].q[0] : sg * __fma_rn(-u, w[m].q[0], w[m].q[1]);
    const double W = w[m].p * (w[m].u[0] - u);
    const double c = __fma_rn(cp, P, D), t = __fma_rn(cp, W, sg * w[m].p);
    fp[m] = __fma_rn(w[m].u[0] + lam, c, t);
    fm[m] = __fma_rn(w[m].u[0] - lam, c, t);
  }
  const double s2 = k == 0 ? 4.0 : 16.0 * a * a;
  const ReconEps e = recon_eps<SCH>(sp.teno_eps, s2);
  return recon5_f64<SCH>(fp[0], fp[1], fp[2], fp[3], fp[4], e, sp.teno_ct, sp.teno_ct_f) +
         recon5_f64<SCH>(fm[5], fm[4], fm[3], fm[2], fm[1], e, sp.teno_ct, sp.teno_ct_f);
}

// T = double: the FP64 path.  T = float: the FP32-residual path -- the state and RK register
// stay FP64 in shared memory; the fluxes come from the FP32 copy of the state, the residual is the
// compensated (float-float) flux difference and the update takes dt x residual rounded once to FP32
// (dt_residual) and applies it with FP64 FMAs, as the fused RK epilogue of the per-block path does.
template <typename T, int SCH, int AVG>
__global__ void __launch_bounds__(RT) k_resident_1d(const Resident1D* __restrict__ blocks, SchemeParams spd, RkCoef rk,
                                                    double dt, int nsteps, int most, unsigned long long* bad) {
  constexpr bool F32 = sizeof(T) == 4;
  cg::cluster_group cl = cg::this_cluster();
  const int cs = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const Resident1D& r = blocks[blockIdx.x / cs];
  const SP<T> sp(spd);
  extern __shared__ __align__(16) unsigned char osb_smem[];
  const RLayout<T> L(osb_smem, most);
  const int N = r.k.n[0], off = r.k.off0;
  // a block too small for the launch's cluster leaves the last CTAs without points: at least 2 RH each
  const int C = min(cs, N / (2 * RH));
  if (rank >= C) {
    cl.sync();
    for (long s = 0; s < (long)nsteps * rk.nst; ++s) cl.sync();
    return;
  }
  const int g0 = (int)((long)rank * N / C), n = (int)((long)(rank + 1) * N / C) - g0;  // points g0 .. g0 + n - 1
  const bool per = r.bc[0] == OSB_BC_PERIODIC;
  // neighbours across the left and right end; none at a block's non-periodic end
  const bool end[2] = {rank == 0, rank == C - 1};
  const int peer[2] = {rank > 0 ? rank - 1 : C - 1, rank < C - 1 ? rank + 1 : 0};
  const bool linked[2] = {!end[0] || per, !end[1] || per};
  // halo points that an exchange fills (a periodic face fills the other side's); those beyond the depth of
  // a block's end keep the caller's values
  const int fill[2] = {end[0] ? r.depth[per ? 1 : 0] : RH, end[1] ? r.depth[per ? 0 : 1] : RH};
  auto hal = [&](int parity, int side, int m, int v) { return ((parity * 2 + side) * RH + m) * 3 + v; };
  // halo point m = 0 .. RH - 1 counted outwards from the end
  for (int u = threadIdx.x; u < 3 * n; u += blockDim.x) {
    const int v = u / n, i = u - v * n;
    L.q[v * most + i] = r.k.q[v][off + g0 + i];
    L.o[v * most + i] = r.k.rk[v][off + g0 + i];
  }
  for (int u = threadIdx.x; u < 2 * RH * 3; u += blockDim.x) {
    const int side = u / (RH * 3), m = (u / 3) % RH, v = u % 3;
    if (linked[side]) {
      int g = side == 0 ? g0 - 1 - m : g0 + n + m;
      g = g < 0 ? g + N : (g >= N ? g - N : g);
      L.halo[hal(0, side, m, v)] = r.k.q[v][off + g];
    }
  }
  double* const ph[2] = {cl.map_shared_rank(L.halo, peer[0]), cl.map_shared_rank(L.halo, peer[1])};
  cl.sync();  // every CTA of the cluster runs before one writes to another
  const double invd = r.k.invd[0];
  const float invd_f = (float)invd;
  const float dt_h = (float)dt, dt_l = (float)(dt - (double)dt_h);
  const T gm = sp.gama;
  const int PS = most + 2 * RH;
  int parity = 0;
  for (int step = 0; step < nsteps; ++step) {
    // SBLI RK3 saves the state at the start of the step (a point's own thread, as everywhere below)
    if (rk.kind == 1)
      for (int i = threadIdx.x; i < n; i += blockDim.x)
#pragma unroll
        for (int v = 0; v < 3; ++v) L.o[v * most + i] = L.q[v * most + i];
    for (int s = 0; s < rk.nst; ++s) {
      // boundary treatment and primitives of points -RH .. n + RH - 1
      for (int k = threadIdx.x; k < n + 2 * RH; k += blockDim.x) {
        const int i = k < n ? k : (k < n + RH ? -1 - (k - n) : n + (k - n - RH));
        Pt<T, 1> w;
#pragma unroll
        for (int v = 0; v < 3; ++v) {
          const double* f = L.q + v * most;
          double x;
          if (-i > fill[0] || i - n >= fill[1]) x = r.k.q[v][off + g0 + i];
          else if (i < 0) x = linked[0] ? L.halo[hal(parity, 0, -1 - i, v)] : halo_point(r.bc[0], f, 1, -i);
          else if (i >= n) x = linked[1] ? L.halo[hal(parity, 1, i - n, v)] : halo_point(r.bc[1], f + n - 1, -1, i - n + 1);
          else if (i == 0 && !linked[0]) L.q[v * most] = x = end_point(r.bc[0], f, 1);
          else if (i == n - 1 && !linked[1]) L.q[v * most + i] = x = end_point(r.bc[1], f + i, -1);
          else x = f[i];
          w.q[v] = to_t<T>(x);
        }
        make_pt<T, 1>(w, gm);
        T* P = L.P + i + RH;
#pragma unroll
        for (int v = 0; v < 3; ++v) P[v * PS] = w.q[v];
        put_prims<T, AVG>(P, PS, w);
      }
      __syncthreads();
      const int W = (n + 32) / 32 * 32;  // n + 1 faces, whole warps
      for (int k = threadIdx.x; k < (F32 ? n + 1 : 3 * W); k += blockDim.x) {
        const int wave = F32 ? 0 : k / W, i = k - wave * W;  // left face of point i
        if (i > n) continue;
        Pt<T, 1> w[6];
#pragma unroll
        for (int m = 0; m < 6; ++m) {
          const T* P = L.P + i + m;
#pragma unroll
          for (int v = 0; v < 3; ++v) w[m].q[v] = P[v * PS];
          get_prims<T, AVG>(P, PS, w[m]);
        }
        if constexpr (!F32) {
          double u, a, x;  // x: 1 / a, or H in the generated order
          if constexpr (generated_order<1, SCH>()) {
            const Face1D<T, AVG> fc(w[2], w[3], sp);
            L.F[wave * (most + 1) + i] = wave_1d<T, SCH, AVG>(wave, w, sp, fc);
            u = fc.u, a = fc.a, x = fc.H;
          } else {
            double uu[1], rho2, ke;
            face_average_f64<1, AVG>(w[2], w[3], sp.g1, uu, a, x, rho2, ke);
            u = uu[0];
            L.F[wave * (most + 1) + i] = wave_1d_f64<SCH>(wave, w, sp, u, a, x, ke);
          }
          if (wave == 0) {
            L.V[i] = u;
            L.V[most + 1 + i] = a;
            L.V[2 * (most + 1) + i] = x;
          }
          continue;
        }
        T fh[3];
        char_flux<T, 1, SCH, AVG>(w, sp, fh);
#pragma unroll
        for (int v = 0; v < 3; ++v) L.F[v * (most + 1) + i] = fh[v];
      }
      __syncthreads();
      const double A = rk.A[s], B = rk.B[s];
      const bool a_zero = rk.kind == 0 && A == 0.0;
      for (int i = threadIdx.x; i < n; i += blockDim.x) {
        T face[2][3];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const T* F = L.F + i + e;
          if constexpr (F32) {
#pragma unroll
            for (int v = 0; v < 3; ++v) face[e][v] = F[v * (most + 1)];
          } else {
            const double* V = L.V + i + e;
            const double rec[3] = {F[0], F[most + 1], F[2 * (most + 1)]}, u = V[0], a = V[most + 1], x = V[2 * (most + 1)];
            if constexpr (generated_order<1, SCH>()) {
              flux_1d(rec, u, a, x, face[e]);
            } else {
              const double S = 0.25 * (rec[1] + rec[2]), Bm = 0.25 * (rec[1] - rec[2]), F0 = __fma_rn(x, S, 0.5 * rec[0]);
              face[e][0] = F0;
              face[e][1] = __fma_rn(u, F0, Bm);
              face[e][2] = __fma_rn(0.5 * (u * u), F0, __fma_rn(a * sp.ig1, S, u * Bm));
            }
          }
        }
#pragma unroll
        for (int v = 0; v < 3; ++v) {
          const T fl = face[0][v], fr = face[1][v];
          double ov = L.o[v * most + i], qv = L.q[v * most + i];
          if constexpr (F32) {
            float p, pe;
            ff_flux_diff(fr, fl, invd_f, p, pe);
            const float hh = __fadd_rn(p, pe);
            const float ll = __fsub_rn(pe, __fsub_rn(hh, p));
            const double x = dt_residual(hh, ll, dt_h, dt_l);  // as rk_point
            if (rk.kind == 0) {
              ov = a_zero ? x : __fma_rn(A, ov, x);
              qv = __fma_rn(B, ov, qv);
            } else {
              qv = __fma_rn(A, x, ov);
              ov = __fma_rn(B, x, ov);
            }
          } else {
            const double r0 = -(fr - fl) * invd;
            if (rk.kind == 0) {
              ov = A * ov + dt * r0;
              qv = B * ov + qv;
            } else {
              qv = A * dt * r0 + ov;
              ov = B * dt * r0 + ov;
            }
          }
          L.o[v * most + i] = ov;
          L.q[v * most + i] = qv;
          // the outer points go to the neighbours' halos of the next stage: the other parity, since a
          // neighbour may still read this stage's
          if (i < RH && linked[0]) ph[0][hal(parity ^ 1, 1, i, v)] = qv;
          if (i >= n - RH && linked[1]) ph[1][hal(parity ^ 1, 0, n - 1 - i, v)] = qv;
        }
      }
      if (cs == 1) __syncthreads();
      else cl.sync();  // also this CTA's barrier; after the last one nobody writes to a neighbour any more
      parity ^= 1;
    }
  }
  // the state, the register and the halos a caller observes after the call
  unsigned long long nb = 0;
  for (int u = threadIdx.x; u < 3 * n; u += blockDim.x) {
    const int v = u / n, i = u - v * n, g = g0 + i;
    double x = L.q[v * most + i];
    if (i == 0 && !linked[0]) x = end_point(r.bc[0], L.q + v * most, 1);
    if (i == n - 1 && !linked[1]) x = end_point(r.bc[1], L.q + v * most + i, -1);
    double* q = r.k.q[v] + off;
    q[g] = x;
    r.k.rk[v][off + g] = L.o[v * most + i];
    if (per) {
      if (g < r.depth[0]) q[N + g] = x;
      if (g >= N - r.depth[1]) q[g - N] = x;
    }
    if (!isfinite(x)) ++nb;
  }
  for (int side = 0; side < 2; ++side)
    if (!linked[side])
      for (int u = threadIdx.x; u < 3 * r.depth[side]; u += blockDim.x) {
        const int v = u % 3, m = 1 + u / 3, e = side == 0 ? 0 : n - 1;
        r.k.q[v][off + g0 + e + (side == 0 ? -m : m)] = halo_point(r.bc[side], L.q + v * most + e, side == 0 ? 1 : -1, m);
      }
  if (nb) atomicAdd(bad, nb);
}

#ifdef OSB_RESIDENT_F32
// Boundary treatment of one 1D block held in shared memory (x fastest, halo h): periodic,
// zero-gradient and extrapolation as k_periodic / k_zero_grad / k_extrap; side 0 then side 1.
__device__ void bc_1d(double* q, int E, int h, int N, const Resident1D& r) {
  const int t = threadIdx.x;
  if (r.bc[0] == OSB_BC_PERIODIC) {
    // both sides in one pass (they read the interior only): [0, d) -> [N, N+d), [N-d, N) -> [-d, 0)
    const int d0 = r.depth[0], d1 = r.depth[1];
    for (int u = t; u < 3 * (d0 + d1); u += blockDim.x) {
      const int v = u / (d0 + d1), m = u % (d0 + d1);
      double* f = q + v * E + h;
      if (m < d0) f[N + m] = f[m];
      else f[-d1 + (m - d0)] = f[N - d1 + (m - d0)];
    }
    return;
  }
  if (t < 6) {
    const int side = t / 3, v = t % 3;
    double* f = q + v * E + h;
    const int kind = r.bc[side], depth = r.depth[side];
    const int id = side == 0 ? 0 : N - 1;
    const int s = side == 0 ? 1 : -1;  // inward step
    if (kind == OSB_BC_ZERO_GRAD) {
      f[id] = f[id + s];
      for (int m = 1; m <= depth; ++m) f[id - m * s] = f[id + m * s];
    } else if (kind == OSB_BC_EXTRAP0) {
      f[id] = f[id + s];
      for (int m = 1; m <= depth; ++m) f[id - m * s] = f[id + s];
    } else if (kind == OSB_BC_EXTRAP1) {
      for (int m = 1; m <= depth; ++m) f[id - m * s] = -f[id - (m - 2) * s] + 2.0 * f[id - (m - 1) * s];
    }
  }
}

// FP32 blocks that one CTA runs alone, halos and an FP32 copy of the state in its shared memory: every
// interface forms its six points' primitives itself, which costs less than staging them where the
// chain of a stage counts and not the arithmetic (see launch_resident for both sides' times).
template <int SCH, int AVG>
__global__ void __launch_bounds__(RT) k_resident_cta(const Resident1D* __restrict__ blocks, SchemeParams spd, RkCoef rk,
                                                     double dt, int nsteps, unsigned long long* bad) {
  const Resident1D r = blocks[blockIdx.x];
  const BlockK& b = r.k;
  const SP<float> sp(spd);
  extern __shared__ __align__(16) unsigned char osb_smem[];
  const int N = b.n[0], h = b.off0, E = b.alloc;
  double* q = reinterpret_cast<double*>(osb_smem);   // [3][E]
  double* o = q + 3 * E;                              // [3][E]
  float* F = reinterpret_cast<float*>(o + 3 * E);     // [3][E]: flux at the right face of point i
  float* qf = F + 3 * E;                              // [3][E]: FP32 copy of the state
  for (int u = threadIdx.x; u < 3 * E; u += blockDim.x) {
    q[u] = b.q[u / E][u % E];
    o[u] = b.rk[u / E][u % E];
    qf[u] = d2f_rn(q[u]);
  }
  const float invd_f = (float)b.invd[0];
  const float dt_h = (float)dt, dt_l = (float)(dt - (double)dt_h);
  for (int step = 0; step < nsteps; ++step) {
    __syncthreads();     // the previous stage's update is complete
    if (rk.kind == 1) {  // SBLI RK3 saves the state at the start of the step
      for (int u = threadIdx.x; u < 3 * N; u += blockDim.x) o[(u / N) * E + h + u % N] = q[(u / N) * E + h + u % N];
    }
    for (int s = 0; s < rk.nst; ++s) {
      __syncthreads();
      bc_1d(q, E, h, N, r);
      __syncthreads();
      // the boundary treatment changed the halos and at most the end points: refresh their copy
      for (int u = threadIdx.x; u < 3 * 2 * (h + 2); u += blockDim.x) {
        const int v = u / (2 * (h + 2)), m = u % (2 * (h + 2));
        const int i = m < h + 2 ? m - h : N - 2 + (m - (h + 2));
        qf[v * E + h + i] = d2f_rn(q[v * E + h + i]);
      }
      __syncthreads();
      for (int i = (int)threadIdx.x - 1; i < N; i += blockDim.x) {
        Pt<float, 1> w[6];
#pragma unroll
        for (int m = 0; m < 6; ++m) {
#pragma unroll
          for (int v = 0; v < 3; ++v) w[m].q[v] = qf[v * E + h + i - 2 + m];
          make_pt<float, 1>(w[m], sp.gama);
        }
        float fh[3];
        char_flux<float, 1, SCH, AVG>(w, sp, fh);
#pragma unroll
        for (int v = 0; v < 3; ++v) F[v * E + h + i] = fh[v];
      }
      __syncthreads();
      const double A = rk.A[s], B = rk.B[s];
      const bool a_zero = rk.kind == 0 && A == 0.0;
      for (int i = threadIdx.x; i < N; i += blockDim.x) {
#pragma unroll
        for (int v = 0; v < 3; ++v) {
          const int id = v * E + h + i;
          double ov = o[id], qv = q[id];
          float p, pe;
          ff_flux_diff(F[id], F[id - 1], invd_f, p, pe);
          const float hh = __fadd_rn(p, pe);
          const float ll = __fsub_rn(pe, __fsub_rn(hh, p));
          const double x = dt_residual(hh, ll, dt_h, dt_l);  // as rk_point
          if (rk.kind == 0) {
            ov = a_zero ? x : __fma_rn(A, ov, x);
            qv = __fma_rn(B, ov, qv);
          } else {
            qv = __fma_rn(A, x, ov);
            ov = __fma_rn(B, x, ov);
          }
          qf[id] = d2f_rn(qv);
          o[id] = ov;
          q[id] = qv;
        }
      }
    }
  }
  __syncthreads();
  bc_1d(q, E, h, N, r);  // the halos a caller observes after the call
  __syncthreads();
  unsigned long long nb = 0;
  for (int u = threadIdx.x; u < 3 * E; u += blockDim.x) {
    b.q[u / E][u % E] = q[u];
    b.rk[u / E][u % E] = o[u];
    const int i = u % E - h;
    if (i >= 0 && i < N && !isfinite(q[u])) ++nb;
  }
  if (nb) atomicAdd(bad, nb);
}
#endif

// Points are split over the smallest power of two of CTAs that leaves each a warp of interfaces
// (31 points), up to the largest cluster the GPU grants: below a warp an FP64 instruction costs the
// same.  400 points: 16 CTAs of 25.  FP32: 125 points, four warps, which take as long as one (400
// points, 20 steps: 4 CTAs 0.17 ms, 2 0.20).  One CTA alone is no cluster: a plain launch and CTA barriers.  Contexts of many blocks take smaller clusters, enough to fill
// the SMs: no fewer than two CTAs where a block has more than 31 points, and no larger shares than a
// CTA's shared memory holds (FP64: 160 bytes a point, 1 448 points).
template <typename T, int SCH, int AVG>
int launch_resident(osb_ctx* c, const Resident1D* dev, int nblocks, int maxN, double dt, int nsteps) {
  const Block& f = c->blocks[0];
  SchemeParams sp = scheme_params(f.d.gama, f.d.eps, f.d.teno_ct, f.d.shock_filter_control, 1e-12);
  RkCoef rk{};
  rk.kind = c->rk_kind == OSB_RK_LOW_STORAGE ? 0 : 1;
  rk.nst = c->nst;
  for (int s = 0; s < c->nst; ++s) {
    rk.A[s] = c->A[s];
    rk.B[s] = c->B[s];
  }
  auto points = [&](int C) { return (maxN + C - 1) / C; };
  int C = 1;
  while (C < RC && points(C) > (sizeof(T) == 8 ? 31 : 125)) C *= 2;
  auto fits = [&](int C) { return RLayout<T>::bytes(points(C)) <= SMEM_MAX; };
  while (C > 2 && (long)nblocks * (C / 2) >= 2L * c->sm_count && fits(C / 2)) C /= 2;
  auto kern = k_resident_1d<T, SCH, AVG>;
  if (C > 8) OSB_CK(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  cfg.attrs = &at;
  cfg.stream = c->stream;
  int most = 0, granted = 0;  // points of the largest share; clusters of this shape that run at once
  for (;; C /= 2) {
    most = std::max(points(C), 4 * RH);  // a smaller block's share: below 2 (2 RH) points each
    const size_t smem = RLayout<T>::bytes(most);
    if (smem > 48 * 1024) OSB_CK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    cfg.numAttrs = C > 1 ? 1 : 0;
    at.val.clusterDim.x = (unsigned)C;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)(nblocks * C));
    const int W = (most + 32) / 32 * 32;
    cfg.blockDim = dim3((unsigned)std::min(RT, sizeof(T) == 8 ? 3 * W : (most + 2 * RH + 31) / 32 * 32));
    cfg.dynamicSmemBytes = smem;
    granted = nblocks;
    if (C <= 8 && (sizeof(T) == 8 || (long)nblocks * C <= 2L * c->sm_count)) break;
    if (cudaOccupancyMaxActiveClusters(&granted, kern, &cfg) == cudaSuccess && granted > 0) break;
    cudaGetLastError();
    granted = 0;
    if (C <= 8) break;  // a portable cluster size
  }
#ifdef OSB_RESIDENT_F32
  // One CTA per block (k_resident_cta) or the cluster, 20 steps, CTA and cluster:
  //  - up to 244 points (two CTAs of the cluster) the CTA's chain is the shorter one: 6 points 0.113 and 0.138 ms,
  //    100 points 0.118 and 0.133, 200 points 0.143 and 0.157; 255 points 0.146 and 0.125, but from half as many
  //    blocks as SMs on the CTA again (100 blocks 0.151 and 0.173);
  //  - many larger blocks, of similar sizes, whose clusters do not all run at once: 300 points x 256 0.296 and
  //    0.463, 400 x 150 0.249 and 0.382, 600 x 130 0.323 and 0.450, 1000 x 220 0.644 and 0.760; where they do,
  //    the cluster: 600 x 100 0.313 and 0.231, 300 x 220 0.297 and 0.245; a few blocks too (1500 x 40 0.613 and
  //    0.406).  The CTA has to leave room for a second one on its SM (2 000 points x 304 1.61 and 1.41).
  // The CTA has a thread per interface, and 64 at least while the blocks leave SMs with room (6 points: 32
  // threads 0.122, 64 0.113; 1 500 blocks 0.193 and 0.309).
  long alloc = 0, sum = 0;
  for (const auto& bl : c->blocks) {
    alloc = std::max(alloc, bl.k.alloc);
    sum += bl.k.n[0];
  }
  const size_t cta_smem = (size_t)3 * alloc * (2 * sizeof(double) + 2 * sizeof(float));
  const bool waves = granted < nblocks && 5 * nblocks >= 3 * c->sm_count && 2 * sum > (long)maxN * nblocks &&
                     2 * (cta_smem + 1024) <= 228 * 1024;
  if (maxN <= 244 || (maxN <= 255 && 2 * nblocks >= c->sm_count) || waves) {
    auto cta = k_resident_cta<SCH, AVG>;
    if (cta_smem > 48 * 1024)
      OSB_CK(cudaFuncSetAttribute(cta, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cta_smem));
    const int threads = std::max(nblocks <= 2 * c->sm_count ? 64 : 32, std::min(RT, (maxN + 32) / 32 * 32));
    timing_begin(c, FAM_PERSISTENT);
    cta<<<nblocks, threads, cta_smem, c->stream>>>(dev, sp, rk, dt, nsteps, c->bad);
    timing_end(c);
    c->launches++;
    OSB_CK(cudaGetLastError());
    return OSB_OK;
  }
#endif
  timing_begin(c, FAM_PERSISTENT);
  OSB_CK(cudaLaunchKernelEx(&cfg, kern, dev, sp, rk, dt, nsteps, most, c->bad));
  timing_end(c);
  c->launches++;
  return OSB_OK;
}

}  // namespace

#ifndef OSB_RESIDENT_F32
// Largest allocated 1D extent (interior + 2 x 5 halo) of the resident path.
constexpr int RESIDENT_MAX_E = 3000;

bool resident_eligible(const osb_ctx* c) {
  if (c->blocks.empty() || c->sched.mode == OSB_SCHED_PER_BLOCK) return false;
  if (c->nst > 8) return false;
  const osb_block_desc& f = c->blocks[0].d;
  for (const auto& bl : c->blocks) {
    const osb_block_desc& d = bl.d;
    if (d.ndim != 1 || d.scheme == OSB_SCHEME_CENTRAL4 || d.viscous != OSB_VISC_NONE || d.metric[9]) return false;
    if (d.scheme != f.scheme || d.averaging != f.averaging) return false;
    if (bl.k.alloc > RESIDENT_MAX_E) return false;
    for (int s = 0; s < 2; ++s)
      if (d.bc[0][s] == OSB_BC_INTERFACE || d.bc[0][s] == OSB_BC_SYMMETRY || d.bc[0][s] == OSB_BC_DIRICHLET ||
          d.bc[0][s] == OSB_BC_PRESSURE_OUTLET)
        return false;
    if (d.flux_type != OSB_FLUX_LLF) return false;
    if ((d.bc[0][0] == OSB_BC_PERIODIC) != (d.bc[0][1] == OSB_BC_PERIODIC)) return false;
  }
  return true;
}

int resident_step(osb_ctx* c, double dt, int nsteps) {
  return c->prec == OSB_PREC_FP32_RESIDUAL ? resident_f32(c, dt, nsteps) : resident_f64(c, dt, nsteps);
}
#endif

int OSB_RESIDENT_NAME(osb_ctx* c, double dt, int nsteps) {
  if (nsteps <= 0) return OSB_OK;
  const int nb = (int)c->blocks.size();
  if (!c->resident || c->resident_n != nb) {
    if (c->resident) cudaFree(c->resident);
    c->resident = nullptr;
    OSB_CK(cudaMalloc(&c->resident, sizeof(Resident1D) * nb));
    c->resident_n = nb;
  }
  std::vector<Resident1D> host(nb);
  int maxN = 0;
  for (int i = 0; i < nb; ++i) {
    const Block& bl = c->blocks[i];
    host[i].k = bl.k;
    for (int s = 0; s < 2; ++s) {
      host[i].bc[s] = bl.d.bc[0][s];
      host[i].depth[s] = bl.d.bc_depth[0][s] > 0 ? bl.d.bc_depth[0][s] : 4;
    }
    maxN = std::max(maxN, bl.k.n[0]);
  }
  OSB_CK(cudaMemcpyAsync(c->resident, host.data(), sizeof(Resident1D) * nb, cudaMemcpyHostToDevice, c->stream));
  const Resident1D* dev = reinterpret_cast<const Resident1D*>(c->resident);
  const int sch = c->blocks[0].d.scheme, avg = c->blocks[0].d.averaging;
  if (avg == OSB_AVG_ROE) {
    if (sch == OSB_SCHEME_WENO5_JS) return launch_resident<OSB_RESIDENT_T, SCH_WENO5_JS, AVG_ROE>(c, dev, nb, maxN, dt, nsteps);
    if (sch == OSB_SCHEME_WENO5_Z) return launch_resident<OSB_RESIDENT_T, SCH_WENO5_Z, AVG_ROE>(c, dev, nb, maxN, dt, nsteps);
    if (sch == OSB_SCHEME_TENO5) return launch_resident<OSB_RESIDENT_T, SCH_TENO5, AVG_ROE>(c, dev, nb, maxN, dt, nsteps);
    if (sch == OSB_SCHEME_TENO6) return launch_resident<OSB_RESIDENT_T, SCH_TENO6, AVG_ROE>(c, dev, nb, maxN, dt, nsteps);
  } else {
    if (sch == OSB_SCHEME_WENO5_JS) return launch_resident<OSB_RESIDENT_T, SCH_WENO5_JS, AVG_SIMPLE>(c, dev, nb, maxN, dt, nsteps);
    if (sch == OSB_SCHEME_WENO5_Z) return launch_resident<OSB_RESIDENT_T, SCH_WENO5_Z, AVG_SIMPLE>(c, dev, nb, maxN, dt, nsteps);
    if (sch == OSB_SCHEME_TENO5) return launch_resident<OSB_RESIDENT_T, SCH_TENO5, AVG_SIMPLE>(c, dev, nb, maxN, dt, nsteps);
    if (sch == OSB_SCHEME_TENO6) return launch_resident<OSB_RESIDENT_T, SCH_TENO6, AVG_SIMPLE>(c, dev, nb, maxN, dt, nsteps);
  }
  return fail(OSB_ENOTSUP, "scheme %d not available in the resident 1D path", sch);
}

}  // namespace osb
