// osb_central_tile.cuh -- central 4th-order terms of a 3D block without wall faces, both precisions:
//   CONV: central convective terms, 1 = skew-symmetric (Feiereisen) form, split_forms.py:111-145
//         as generated for the low-Mach TGV ("Convective terms" kernel); 2 = Kennedy-Gruber-
//         Pirozzoli form, split_forms.py:178-236 as generated for the Central4-WENO5 benchmark;
//         0 = none.
//   VISC: viscous stress and heat flux (StoreSome "Viscous terms" kernel), mu from the modified
//         Sutherland or a power law (VISC == 1) or constant (VISC == 2); 0 = none.
//   FUSE (FP32): the RK update of the point, whose residual is complete here.
//   WRAP: every face of the block is periodic, and the staged halo points are read at their images
//         inside the block: osb_step of a central-scheme block then exchanges no halos between
//         stages (8 us of the 30 that a stage of a 64^3 block took).
//
// A CTA owns a 32 x 8 column of points and streams it through czc planes of z (a launch argument,
// chosen on the host so the CTAs fill whole waves): the planes z-2 .. z+2 around the current one sit
// in a 5-plane ring of primitives in shared memory (halo 2 in x and y), the raw state of plane z+3
// is loaded into registers while plane z is computed, then converted into the slot plane z-2 vacates.
//
// FP64 is bound by the FP64 pipe (16.3 cycles per warp instruction and SM) and FP32 by instruction
// issue, so the terms are arranged for the fewest operations:
//  * the mixed second derivatives enter the momentum equations only as the derivative along i of
//    the other two directions' D_j u_j, so those sums are formed once per point -- in shared memory
//    for x and y, in registers along z -- instead of six 4x4-point stencils;
//  * E / rho (Feiereisen) or H = (E + p) / rho (KGP) is staged, so no division is repeated for the
//    twelve neighbours of a point;
//  * KGP: D_j(u_i m_j) + rho D_j(u_i u_j) is one derivative of u_i (m_j + rho_0 u_j);
//  * the energy equation takes u_i times the momentum contributions already formed, and the
//    dissipation the symmetric half of tau : grad u;
//  * a column of 32 x 8 points stages 1.7 points per computed one (2.25 with 32 x 4).
// FP64: about 290 FP64 instructions per point (viscous terms, Sutherland law) and 390 (Feiereisen,
// constant viscosity), 615 and 1 030 before: 128^3 viscous 2.16 -> 1.38 ms, 64^3 Feiereisen 0.45 ->
// 0.23 ms per launch.
//
// FP32, FUSE: half of the bytes are the update's (FP64 state and register), loaded at the start of a
// plane's arithmetic; through shared memory a plane ahead (cp.async) they gained nothing (viscous) or
// lost 20 % (KGP: one more CTA's worth of shared memory).  256^3 viscous + update 0.92 -> 0.82 ms per
// stage (240 bytes per point, 4.9 TB/s), 131 x 97 x 110 0.109 -> 0.096, 64^3 Feiereisen + update 27 ->
// 22 us, KGP 128^3 0.168 -> 0.134 ms.
//
// BULK (FP32 state only): the raw planes come in through the bulk-copy (TMA) engine instead --
// one cp.async.bulk per staged row and variable into a two-slot raw buffer in shared memory,
// completion counted on an mbarrier per slot, two planes ahead of the computed one.  The OPS
// row pitch (n + 10 elements) is not a multiple of 16 bytes, which a tiled tensor map needs,
// so each row copy starts at the 16-byte boundary at or below the row's first staged element
// and moves CRW elements; the lead (0..3 elements) is recomputed by the reading thread.
#pragma once
#include "osb_kernels.cuh"

namespace osb {

constexpr int CTY = 8, CTSY = CTY + 2 * CH, CTPL = CSX * CTSY, CTT = CX * CTY;
constexpr int CTPP = (CTPL + CTT - 1) / CTT;   // staged points per thread and plane
constexpr int CTRAW = 2 * 5 * CTSY * CRW;      // floats of the two raw plane slots (BULK)

// Staged fields: velocity; VISC: temperature (and viscosity unless constant); CONV: momentum, then
// Feiereisen E / rho, p + E / 2 and 2 p, or KGP H, rho and p (p itself also with viscous terms: rho T
// would round a uniform pressure differently at every density).  FP32: two CTAs' rings fit an SM.
template <int CONV, int VISC>
struct CtFields {
  static constexpr int U = 0, TT = 3, MU = 4;
  static constexpr int M = 3 + (VISC ? (VISC == 1 ? 2 : 1) : 0), EE = M + 3, HH = M + 4, P = M + 5;
  static constexpr int N = CONV ? M + 6 : M;
};
template <typename T, int CONV, int VISC, bool BULK>
constexpr size_t ct_smem() {
  return sizeof(T) * ((size_t)CtFields<CONV, VISC>::N * CRING * CTPL + (VISC ? CSX * CTY + CX * CTSY : 0)) +
         (BULK ? CTRAW * sizeof(float) + 2 * sizeof(unsigned long long) : 0);
}
// CTAs per SM that the register allocation has to leave room for: what shared memory admits, at
// most two (the update's FP64 values spill at the 80 registers of three).
template <typename T, int CONV, int VISC, bool BULK>
constexpr int ct_ctas() {
  return (228 * 1024) / (ct_smem<T, CONV, VISC, BULK>() + 1024) >= 2 ? 2 : 1;
}

template <typename T>
__device__ __forceinline__ T recip(T x) {
  if constexpr (sizeof(T) == 8) return rcp_newton(x);
  else return T(1) / x;
}
template <typename T>
__device__ __forceinline__ T fmat(T a, T b, T c) {
  if constexpr (sizeof(T) == 8) return __fma_rn(a, b, c);
  else return __fmaf_rn(a, b, c);
}

template <typename T, int CONV, int VISC, bool FUSE, bool BULK, bool WRAP>
__global__ void __launch_bounds__(CTT, ct_ctas<T, CONV, VISC, BULK>())
    k_central(BlockK b, CentralParams cp, int first, int czc, RkFuse rf) {
  static_assert(!BULK || (sizeof(T) == 4 && !WRAP), "bulk staging: FP32 state, rows as they lie");
  using Fd = CtFields<CONV, VISC>;
  constexpr int FS = CRING * CTPL;
  constexpr int V0 = CONV ? 0 : 1;  // first variable with a contribution
  extern __shared__ __align__(16) unsigned char osb_smem[];
  // BULK: the raw plane slots (rows 16-byte aligned), one mbarrier per slot, then the ring
  float* raw = reinterpret_cast<float*>(osb_smem);
  unsigned long long* bar = reinterpret_cast<unsigned long long*>(raw + CTRAW);
  T* sm = reinterpret_cast<T*>(osb_smem + (BULK ? CTRAW * sizeof(float) + 2 * sizeof(unsigned long long) : 0));
  T* Sx = sm + Fd::N * FS;       // [CTY][CSX]: D_y u_y + D_z u_z of the current plane
  T* Sy = Sx + CSX * CTY;        // [CTSY][CX]: D_x u_x + D_z u_z
  const int tx = threadIdx.x % CX, ty = threadIdx.x / CX;
  const int x0 = blockIdx.x * CX, y0 = blockIdx.y * CTY;
  const int zb = blockIdx.z * czc, ze = min(b.n[2], zb + czc);
  const T gm = cpar<T>(cp.gama, cp.gama_f), g1 = gm - L_(1.0);
  const T M2g = cpar<T>(cp.M2, cp.M2_f) * gm;
  const T mu_pw = cpar<T>(cp.mu_pow, cp.mu_pow_f);
  T qv[CTPP][5];
  // WRAP: the staged points' images in x and y, the same for every plane
  int image[CTPP];
  if constexpr (WRAP) {
#pragma unroll
    for (int u = 0; u < CTPP; ++u) {
      const int idx = threadIdx.x + u * CTT;
      const int gx = x0 - CH + idx % CSX, gy = y0 - CH + idx / CSX;
      image[u] = lin(b, gx < 0 ? gx + b.n[0] : (gx >= b.n[0] ? gx - b.n[0] : gx),
                     gy < 0 ? gy + b.n[1] : (gy >= b.n[1] ? gy - b.n[1] : gy), 0);
    }
  }
  auto load_plane = [&](int gz) {
    const int wz = gz < 0 ? gz + b.n[2] : (gz >= b.n[2] ? gz - b.n[2] : gz);
#pragma unroll
    for (int u = 0; u < CTPP; ++u) {
      const int idx = threadIdx.x + u * CTT;
      const int gx = x0 - CH + idx % CSX, gy = y0 - CH + idx / CSX;
      if (idx < CTPL && gx <= b.n[0] + CH && gy <= b.n[1] + CH) {
        const int id = WRAP ? image[u] + wz * b.st[2] : lin(b, gx, gy, gz);
#pragma unroll
        for (int v = 0; v < 5; ++v) qv[u][v] = ld_q<T>(b, v, id);
      }
    }
  };
  auto store_plane = [&](int slot) {
#pragma unroll
    for (int u = 0; u < CTPP; ++u) {
      const int idx = threadIdx.x + u * CTT;
      const int gx = x0 - CH + idx % CSX, gy = y0 - CH + idx / CSX;
      if (!(idx < CTPL && gx <= b.n[0] + CH && gy <= b.n[1] + CH)) continue;
      T* at = sm + slot * CTPL + idx;
      const T rho = qv[u][0], m0 = qv[u][1], m1 = qv[u][2], m2 = qv[u][3], E = qv[u][4];
      const T ir = recip(rho);
      const T u0 = m0 * ir, u1 = m1 * ir, u2 = m2 * ir;
      const T p = g1 * (E - L_(0.5) * (m0 * u0 + m1 * u1 + m2 * u2));
      at[(Fd::U + 0) * FS] = u0;
      at[(Fd::U + 1) * FS] = u1;
      at[(Fd::U + 2) * FS] = u2;
      if (VISC) {
        const T Tt = M2g * p * ir;
        at[Fd::TT * FS] = Tt;
        if (VISC == 1)
          at[Fd::MU * FS] = mu_pw > L_(0.0) ? pow(Tt, mu_pw) : L_(1.4042) * Tt * sqrt(Tt) * recip(L_(0.40417) + Tt);
      }
      if (CONV) {
        at[(Fd::M + 0) * FS] = m0;
        at[(Fd::M + 1) * FS] = m1;
        at[(Fd::M + 2) * FS] = m2;
        at[Fd::P * FS] = CONV == 1 ? L_(2.0) * p : p;
        at[Fd::EE * FS] = CONV == 1 ? E * ir : (E + p) * ir;
        at[Fd::HH * FS] = CONV == 1 ? fmat(L_(0.5), E, p) : rho;
      }
    }
  };
  auto slot_of = [](int gz) { return (gz + 2 * CRING) % CRING; };
  // BULK: plane gz goes to raw slot (gz - zb + CH) & 1 and completes that slot's phase of
  // parity ((gz - zb + CH) >> 1) & 1; rows past y = n1 + CH are not copied.  A wait that runs
  // out marks the CTA broken (uniformly, through the next barrier): it issues no further copies,
  // counts the event in *rf.stall, and before returning waits (bounded) for the copies it issued.
  const int nrow = min(CTSY, b.n[1] + 2 * CH + 1 - y0);
  bool broken = false;
  unsigned pend = 0, ppar = 0;  // raw slots with a copy in flight no wait has seen complete, its parity
  auto rslot = [&](int gz) { return (gz - zb + CH) & 1; };
  auto rpar = [&](int gz) { return (unsigned)((gz - zb + CH) >> 1) & 1u; };
  // The copies of a plane are spread over lanes 0..7 of every warp (one warp issuing all of them
  // measured 10 % slower); thread 0 arms the slot's next phase (arrive + expected bytes) as soon
  // as its wait saw the previous one complete, so the copies need no extra barrier.
  const unsigned plane_bytes = (unsigned)(nrow * 5 * CRW * 4);
  auto issue = [&](int gz) {  // the bookkeeping is uniform
    if (!BULK || broken || gz > ze + CH - 1) return;
    const int s = rslot(gz);
    pend |= 1u << s;
    ppar = (ppar & ~(1u << s)) | (rpar(gz) << s);
    const int lane = threadIdx.x & 31;
    if (lane >= 8) return;
    fence_async_smem();
    for (int c = (threadIdx.x >> 5) * 8 + lane; c < 5 * nrow; c += CTY * 8) {
      const int v = c / nrow, r = c - v * nrow;
      const float* src = b.qf[v] + lin(b, x0 - CH, y0 - CH + r, gz);
      const float* al = reinterpret_cast<const float*>(reinterpret_cast<size_t>(src) & ~(size_t)15);
      bulk_copy_g2s(raw + ((s * 5 + v) * CTSY + r) * CRW, al, CRW * 4, &bar[s]);
    }
  };
  // the 16-byte phase (0..3 elements) of each variable's array, two bits per variable: a row
  // copy's lead is that phase plus the row's linear index, mod 4
  unsigned phase = 0;
  if constexpr (BULK) {
#pragma unroll
    for (int v = 0; v < 5; ++v) phase |= (unsigned)((reinterpret_cast<size_t>(b.qf[v]) >> 2) & 3) << (2 * v);
  }
  // raw plane gz from its slot into the registers of the staged points (waits for the copy)
  auto fetch_plane = [&](int gz) -> int {
    const int s = rslot(gz);
    int late = 0;
    if (!broken) {
      late = mbar_wait_bounded(&bar[s], rpar(gz)) ? 0 : 1;
      if (!late) pend &= ~(1u << s);
      if (!late && threadIdx.x == 0 && gz + 2 <= ze + CH - 1) mbar_arrive_expect(&bar[s], plane_bytes);
    }
#pragma unroll
    for (int u = 0; u < CTPP; ++u) {
      const int idx = threadIdx.x + u * CTT;
      const int ry = idx / CSX, cx = idx % CSX;
      if (idx < CTPL && x0 - CH + cx <= b.n[0] + CH && y0 - CH + ry <= b.n[1] + CH) {
        const unsigned rl = (unsigned)lin(b, x0 - CH, y0 - CH + ry, gz);
        const float* rrow = raw + (s * 5 * CTSY + ry) * CRW + cx;
#pragma unroll
        for (int v = 0; v < 5; ++v) qv[u][v] = rrow[v * CTSY * CRW + (int)(((phase >> (2 * v)) + rl) & 3u)];
      }
    }
    return late;
  };
  // the barrier after a staged plane; BULK: also makes `broken` uniform
  auto plane_barrier = [&](int late) {
    if constexpr (BULK) {
      const bool was = broken;
      broken = __syncthreads_or(late) != 0 || was;
      if (broken && !was && threadIdx.x == 0) atomicAdd(rf.stall, 1ull);
    } else {
      __syncthreads();
    }
  };
  // first derivative from the neighbours at -2, -1, 1, 2 along j; second derivative from each
  // neighbour's difference from the centre (exactly zero on a constant: d2w)
  T a8[3], a1[3], b4[3], b1[3];
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const T id = cpar<T>(cp.invd[j], cp.invd_f[j]), jd = cpar<T>(cp.inv2d[j], cp.inv2d_f[j]);
    a8[j] = L_(2.0 / 3.0) * id;
    a1[j] = L_(1.0 / 12.0) * id;
    b4[j] = L_(4.0 / 3.0) * jd;
    b1[j] = L_(1.0 / 12.0) * jd;
  }
  auto d1 = [&](int j, T fm2, T fm1, T fp1, T fp2) -> T { return fmat(a8[j], fp1 - fm1, -(a1[j] * (fp2 - fm2))); };
  auto d2 = [&](int j, T fm2, T fm1, T f0, T fp1, T fp2) -> T {
    return fmat(b4[j], (fm1 - f0) + (fp1 - f0), -(b1[j] * ((fm2 - f0) + (fp2 - f0))));
  };
  const int gx = x0 + tx, gy = y0 + ty;
  const bool active = gx < b.n[0] && gy < b.n[1];
  const int own = (ty + CH) * CSX + (tx + CH);
  int pb[2 * CH + 1] = {0};  // ring bases of planes gz-2 .. gz+2
  // in-plane derivative of a field at staged point `at` of plane pb[k]
  auto dp = [&](int f, int j, int k, int at) -> T {
    const T* s = sm + f * FS + pb[k] + at;
    const int o = j == 0 ? 1 : CSX;
    return d1(j, s[-2 * o], s[-o], s[o], s[2 * o]);
  };
  // z derivative at the current plane
  auto dz = [&](int f, int at) -> T {
    const T* s = sm + f * FS + at;
    return d1(2, s[pb[0]], s[pb[1]], s[pb[3]], s[pb[4]]);
  };
  if constexpr (BULK) {
    if (threadIdx.x == 0) {
      mbar_init(&bar[0], 1);
      mbar_init(&bar[1], 1);
      mbar_init_fence();
      mbar_arrive_expect(&bar[0], plane_bytes);  // planes zb-2 and zb-1
      mbar_arrive_expect(&bar[1], plane_bytes);
    }
    __syncthreads();
    issue(zb - CH);
    issue(zb - CH + 1);
    // prologue: planes zb-2 .. zb+1 into the ring, each slot refilled two planes ahead
    for (int gz = zb - CH; gz < zb + CH; ++gz) {
      const int late = fetch_plane(gz);
      store_plane(slot_of(gz));
      plane_barrier(late);
      issue(gz + 2);
    }
  } else {
    // prologue: planes zb-2 .. zb+1 into the ring, plane zb+2 into registers
    for (int gz = zb - CH; gz < zb + CH; ++gz) {
      load_plane(gz);
      store_plane(slot_of(gz));
    }
    load_plane(zb + CH);
  }
  // this column's D_x u_x and D_y u_y of planes gz .. gz+2, and their sum of planes gz-2 .. gz+2
  T d00[3], d11[3], sz[5];
  if (VISC) {
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      pb[k] = slot_of(zb - CH + k) * CTPL;
      const T x = dp(Fd::U + 0, 0, k, own), y = dp(Fd::U + 1, 1, k, own);
      sz[k + 1] = x + y;
      if (k >= 2) {
        d00[k - 1] = x;
        d11[k - 1] = y;
      }
    }
  }
  for (int gz = zb; gz < ze; ++gz) {
    if constexpr (BULK) {
      const int late = fetch_plane(gz + CH);  // copied during iteration gz - 2
      store_plane(slot_of(gz + CH));
      plane_barrier(late);
      issue(gz + CH + 2);
    } else {
      store_plane(slot_of(gz + CH));  // plane gz+2, loaded during the previous iteration
      __syncthreads();
      if (gz + CH + 1 < ze + CH) load_plane(gz + CH + 1);
    }
#pragma unroll
    for (int k = 0; k <= 2 * CH; ++k) pb[k] = slot_of(gz + k - CH) * CTPL;
    const int gid = lin(b, gx, gy, gz);
    // the partial residual, and the fused update's state and register, before the arithmetic
    T oh[5], ol[5];
    if (active && !first) {
#pragma unroll
      for (int v = FUSE ? 0 : V0; v < 5; ++v) r_load(b, v, gid, oh[v], ol[v]);
    }
    double fq[5], fo[5];
    if constexpr (FUSE) {
      if (active) {
#pragma unroll
        for (int v = 0; v < 5; ++v) {
          fq[v] = b.q[v][gid];
          fo[v] = rf.a_zero ? 0.0 : b.rk[v][gid];
        }
      }
    }
    T du[3][3];
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
        const int r = ty < 2 ? ty : ty + CTY;
        const int at = r * CSX + tx + CH;
        Sy[r * CX + tx] = dp(Fd::U + 0, 0, 2, at) + dz(Fd::U + 2, at);
      } else if (ty == 4) {
        const int r = tx >> 2, c = (tx & 3) < 2 ? (tx & 3) : CX + (tx & 3);
        const int at = (r + CH) * CSX + c;
        Sx[r * CSX + c] = dp(Fd::U + 1, 1, 2, at) + dz(Fd::U + 2, at);
      }
      __syncthreads();
    }
    // every thread reaches the barriers of an iteration at the same call sites: the point update is
    // guarded, never skipped with a jump past a barrier
    if (active) {
      const T* c = sm + pb[2] + own;
      // stencil values along j: f(m) at m = -2 .. 2
      auto F = [&](int f, int j, int m) -> T {
        return j == 2 ? sm[f * FS + pb[m + CH] + own] : c[f * FS + m * (j == 0 ? 1 : CSX)];
      };
      auto D1 = [&](int f, int j) -> T { return d1(j, F(f, j, -2), F(f, j, -1), F(f, j, 1), F(f, j, 2)); };
      T racc[5] = {L_(0.0), L_(0.0), L_(0.0), L_(0.0), L_(0.0)};
      const T uc[3] = {c[0], c[FS], c[2 * FS]};
      T lap[3] = {L_(0.0), L_(0.0), L_(0.0)}, dT[3], dmu[3], lapT = L_(0.0);
      T divm = L_(0.0), cm[3] = {L_(0.0), L_(0.0), L_(0.0)}, ce = L_(0.0), cr = L_(0.0);
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        T u[3][5];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
#pragma unroll
          for (int m = 0; m < 5; ++m) u[i][m] = m == 2 ? uc[i] : F(Fd::U + i, j, m - 2);
          if (!VISC || i != j) du[i][j] = d1(j, u[i][0], u[i][1], u[i][3], u[i][4]);
          if (VISC) {
            const T s = d2(j, u[i][0], u[i][1], u[i][2], u[i][3], u[i][4]);
            lap[i] = i == j ? fmat(L_(4.0 / 3.0), s, lap[i]) : lap[i] + s;
          }
        }
        if (VISC) {
          const T t[5] = {F(Fd::TT, j, -2), F(Fd::TT, j, -1), c[Fd::TT * FS], F(Fd::TT, j, 1), F(Fd::TT, j, 2)};
          lapT += d2(j, t[0], t[1], t[2], t[3], t[4]);
          if (VISC == 1) {
            dT[j] = d1(j, t[0], t[1], t[3], t[4]);
            dmu[j] = D1(Fd::MU, j);
          }
        }
        if (CONV) {
          T mm[3][4];
#pragma unroll
          for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int k = 0; k < 4; ++k) mm[i][k] = F(Fd::M + i, j, k < 2 ? k - 2 : k - 1);
          const T mj = c[(Fd::M + j) * FS];
          const T dmj = d1(j, mm[j][0], mm[j][1], mm[j][2], mm[j][3]);
          divm += dmj;
          T pr[4];
          if (CONV == 1) {
            // R_rho -= D_j m_j ; R_m_i -= 1/2 [D_j(m_i u_j + 2 p delta_ij) + u_i D_j m_j + m_j D_j u_i]
            // R_E -= D_j((p + E/2) u_j) + 1/2 [m_j D_j(E/rho) + (E/rho) D_j m_j]
#pragma unroll
            for (int i = 0; i < 3; ++i) {
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                const int m = k < 2 ? k - 2 : k - 1;
                pr[k] = i == j ? fmat(mm[i][k], u[j][m + 2], F(Fd::P, j, m)) : mm[i][k] * u[j][m + 2];
              }
              cm[i] += fmat(mj, du[i][j], d1(j, pr[0], pr[1], pr[2], pr[3]));
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const int m = k < 2 ? k - 2 : k - 1;
              pr[k] = F(Fd::HH, j, m) * u[j][m + 2];
            }
            ce += fmat(L_(0.5) * mj, D1(Fd::EE, j), d1(j, pr[0], pr[1], pr[2], pr[3]));
          } else {
            // R_rho = -1/2 sum_j [D_j m_j + rho D_j u_j + u_j D_j rho]
            // R_m_i = -D_i p - 1/4 sum_j [D_j(u_i m_j) + rho D_j(u_i u_j) + u_i D_j m_j + u_j D_j m_i
            //                             + m_i D_j u_j + m_j D_j u_i + u_i u_j D_j rho]
            // R_E = -1/4 sum_j [D_j(H m_j) + rho D_j(H u_j) + H D_j m_j + u_j D_j(H rho) + m_j D_j H
            //                   + H rho D_j u_j + H u_j D_j rho]
            const T r0 = c[Fd::HH * FS], H0 = c[Fd::EE * FS], uj = uc[j];
            T g[4], hh[4], rr[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const int m = k < 2 ? k - 2 : k - 1;
              g[k] = fmat(r0, u[j][m + 2], mm[j][k]);
              hh[k] = F(Fd::EE, j, m);
              rr[k] = F(Fd::HH, j, m);
            }
            const T drho = d1(j, rr[0], rr[1], rr[2], rr[3]);
            const T s = fmat(uj, drho, dmj);  // D_j m_j + u_j D_j rho
            cr += fmat(r0, du[j][j], s);
#pragma unroll
            for (int i = 0; i < 3; ++i) {
#pragma unroll
              for (int k = 0; k < 4; ++k) pr[k] = u[i][k < 2 ? k : k + 1] * g[k];
              T a = d1(j, pr[0], pr[1], pr[2], pr[3]);
              a = fmat(uc[i], s, a);
              a = fmat(uj, i == j ? dmj : d1(j, mm[i][0], mm[i][1], mm[i][2], mm[i][3]), a);
              a = fmat(c[(Fd::M + i) * FS], du[j][j], a);
              cm[i] += fmat(mj, du[i][j], a);
            }
            T a;
#pragma unroll
            for (int k = 0; k < 4; ++k) pr[k] = hh[k] * g[k];
            a = d1(j, pr[0], pr[1], pr[2], pr[3]);
#pragma unroll
            for (int k = 0; k < 4; ++k) pr[k] = hh[k] * rr[k];
            a = fmat(uj, d1(j, pr[0], pr[1], pr[2], pr[3]), a);
            a = fmat(mj, d1(j, hh[0], hh[1], hh[2], hh[3]), a);
            ce += fmat(H0, fmat(r0, du[j][j], s), a);
          }
        }
      }
      if (CONV == 1) {
        racc[0] = -divm;
#pragma unroll
        for (int i = 0; i < 3; ++i) racc[1 + i] = -L_(0.5) * fmat(uc[i], divm, cm[i]);
        racc[4] = -fmat(L_(0.5) * divm, c[Fd::EE * FS], ce);
      }
      if (CONV == 2) {
        racc[0] = -L_(0.5) * cr;
#pragma unroll
        for (int i = 0; i < 3; ++i) racc[1 + i] = -fmat(L_(0.25), cm[i], D1(Fd::P, i));
        racc[4] = -L_(0.25) * ce;
      }
      if (VISC) {
        const T* px = Sx + ty * CSX + tx + CH;
        const T* py = Sy + (ty + CH) * CX + tx;
        lap[0] = fmat(L_(1.0 / 3.0), d1(0, px[-2], px[-1], px[1], px[2]), lap[0]);
        lap[1] = fmat(L_(1.0 / 3.0), d1(1, py[-2 * CX], py[-CX], py[CX], py[2 * CX]), lap[1]);
        lap[2] = fmat(L_(1.0 / 3.0), d1(2, sz[0], sz[1], sz[3], sz[4]), lap[2]);
        const T invRe = cpar<T>(cp.invRe, cp.invRe_f), kheat = cpar<T>(cp.kheat, cp.kheat_f);
        const T mu = VISC == 1 ? c[Fd::MU * FS] : cpar<T>(cp.mu_c, cp.mu_c_f);
        const T div3 = L_(2.0 / 3.0) * (du[0][0] + du[1][1] + du[2][2]);
        const T t01 = du[0][1] + du[1][0], t02 = du[0][2] + du[2][0], t12 = du[1][2] + du[2][1];
        const T t0 = fmat(L_(2.0), du[0][0], -div3), t1 = fmat(L_(2.0), du[1][1], -div3),
                t2 = fmat(L_(2.0), du[2][2], -div3);
        T m[3] = {mu * lap[0], mu * lap[1], mu * lap[2]};
        if (VISC == 1) {
          m[0] += t0 * dmu[0] + t01 * dmu[1] + t02 * dmu[2];
          m[1] += t01 * dmu[0] + t1 * dmu[1] + t12 * dmu[2];
          m[2] += t02 * dmu[0] + t12 * dmu[1] + t2 * dmu[2];
        }
        const T phi = t0 * du[0][0] + t1 * du[1][1] + t2 * du[2][2] + t01 * t01 + t02 * t02 + t12 * t12;
        const T e = mu * phi + uc[0] * m[0] + uc[1] * m[1] + uc[2] * m[2];
        T h = mu * lapT;
        if (VISC == 1) h += dT[0] * dmu[0] + dT[1] * dmu[1] + dT[2] * dmu[2];
#pragma unroll
        for (int i = 0; i < 3; ++i) racc[1 + i] = fmat(m[i], invRe, racc[1 + i]);
        racc[4] += e * invRe + h * kheat;
        if (cp.forced) {
          T w = L_(0.0);
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            const T fi = cpar<T>(cp.force[i], cp.force_f[i]);
            racc[1 + i] -= fi;
            w += fi * uc[i];
          }
          racc[4] -= w;
        }
      }
      if constexpr (FUSE) {
        // the central scheme's only residual kernel starts from zero, the viscous terms of a
        // shock-capturing block from the sweeps' partial residual
        unsigned nb = 0;
        rk_modes(rf, [&](auto mode) {
          constexpr int MODE = decltype(mode)::value;
#pragma unroll
          for (int v = 0; v < 5; ++v) {
            float h = racc[v], l = 0.f;
            if constexpr (CONV == 0) {
              h = oh[v];
              l = ol[v];
              if (v >= V0) rp_final(racc[v], h, l);
            }
            nb += rk_point<MODE>(b, rf, v, gid, h, l, fq[v], fo[v]);
          }
        });
        if (nb) atomicAdd(rf.bad, (unsigned long long)nb);
      } else if (first) {
#pragma unroll
        for (int v = V0; v < 5; ++v) acc_point(b, v, gid, racc[v], 1);
      } else {
#pragma unroll
        for (int v = V0; v < 5; ++v) rp_store(b, v, gid, racc[v], oh[v], ol[v]);
      }
    }
    __syncthreads();  // the next iteration overwrites plane gz-2 and the sums
  }
  if constexpr (BULK) {
    // only a broken CTA can end with copies in flight: wait for them (bounded) before its
    // shared memory is released
#pragma unroll
    for (int s2 = 0; s2 < 2; ++s2)
      if (pend & (1u << s2)) mbar_wait_bounded(&bar[s2], (ppar >> s2) & 1u);
  }
}

}  // namespace osb
