// osb_central.cu -- launches of the central 4th-order convective / viscous kernel, compiled
// once per precision (OSB_CENTRAL_T).
#include "osb_closures.h"
#include "osb_internal.h"
#include "osb_central_tile.cuh"

#include <algorithm>
#include <cmath>

namespace osb {
namespace {

// Faces whose central derivatives take the one-sided closures (ModifyCentralDerivative walls).
inline bool is_wall(int kind) { return kind == OSB_BC_ISOTHERMAL_WALL || kind == OSB_BC_ADIABATIC_WALL; }

// Constants of one block's central terms; WALL: with the closures at its wall faces.
template <bool WALL>
CentralParams central_params(const Block& bl) {
  CentralParams cp{};
  const osb_block_desc& d = bl.d;
  cp.gama = d.gama;
  cp.M2 = d.Minf * d.Minf;
  cp.mu_c = d.mu_const;
  cp.invRe = 1.0 / d.Re;
  cp.kheat = 1.0 / (d.Pr * d.Re * d.Minf * d.Minf * (d.gama - 1.0));
  cp.gama_f = (float)cp.gama;
  cp.M2_f = (float)cp.M2;
  cp.mu_c_f = (float)cp.mu_c;
  cp.invRe_f = (float)cp.invRe;
  cp.kheat_f = (float)cp.kheat;
  cp.mu_pow = d.viscous == OSB_VISC_POWER_LAW ? d.visc_power : 0.0;
  cp.mu_pow_f = (float)cp.mu_pow;
  cp.forced = d.forcing[0] != 0.0 || d.forcing[1] != 0.0 || d.forcing[2] != 0.0;
  for (int i = 0; i < 3; ++i) {
    cp.force[i] = d.forcing[i];
    cp.force_f[i] = (float)d.forcing[i];
  }
  for (int i = 0; i < 3; ++i) {
    cp.invd[i] = bl.k.invd[i];
    cp.inv2d[i] = bl.k.inv2d[i];
    cp.invd_f[i] = (float)cp.invd[i];
    cp.inv2d_f[i] = (float)cp.inv2d[i];
  }
  if (WALL) {
    cp.wall_lo = is_wall(bl.d.bc[1][0]);
    cp.wall_hi = is_wall(bl.d.bc[1][1]);
    const Closures& cl = closures();
    for (int r = 0; r < 4; ++r)
      for (int m = 0; m < 6; ++m) {
        cp.c1[r][m] = cl.c1[r][m];
        cp.c1f[r][m] = (float)cl.c1[r][m];
      }
    for (int r = 0; r < 2; ++r)
      for (int m = 0; m < 5; ++m) {
        cp.c2[r][m] = cl.c2[r][m];
        cp.c2f[r][m] = (float)cl.c2[r][m];
      }
  }
  return cp;
}

// Launch shape of a kernel on 32 x rows columns: z chunks per column so the CTAs fill whole waves (a
// chunk starts by staging four planes, `start` computed planes' worth).  Chunks of at least four planes,
// but shorter ones while each CTA has an SM of its own: a 24^3 block is 3 columns, and its 18 chunks of
// four planes left 134 SMs idle (FP64 KGP 1.07 ms in 2 steps, 0.39 in 72 chunks of one; FP32 0.101
// and 0.054).  Two such CTAs on an SM share its FP64 pipe: 48^3 viscous 0.78 ms in chunks of two, 0.68 of four.
struct ColumnGrid {
  dim3 grid;
  int czc;
};
template <typename K>
ColumnGrid column_grid(osb_ctx* c, const BlockK& k, K kern, int rows, size_t smem, double start) {
  const unsigned nx = (k.n[0] + CX - 1) / CX, ny = (k.n[1] + rows - 1) / rows;
  const long slots = (long)resident_ctas(kern, CX * rows, smem) * c->sm_count;
  int nz = wave_chunks(k.n[2], (long)nx * ny, slots, start, 4);
  if ((long)nx * ny * nz < c->sm_count) nz = wave_chunks(k.n[2], (long)nx * ny, c->sm_count, start, 1);
  const int czc = (k.n[2] + nz - 1) / nz;
  return {dim3(nx, ny, (k.n[2] + czc - 1) / czc), czc};
}

template <typename T, int VISC, bool FUSE>
int launch_wall(osb_ctx* c, Block& bl, int first, const RkFuse& rf) {
  auto kern = k_central_wall<T, VISC, FUSE>;
  constexpr size_t smem = (size_t)WallFields::N * CRING * CPL * sizeof(T);
  OSB_CK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const ColumnGrid g = column_grid(c, bl.k, kern, CWY, smem, 1.4);
  timing_begin(c, FAM_CENTRAL);
  kern<<<g.grid, CX * CWY, smem, c->stream>>>(bl.k, central_params<true>(bl), first, g.czc, rf);
  timing_end(c);
  c->launches++;
  return OSB_OK;
}

template <typename T, int CONV, int VISC, bool FUSE, bool BULK, bool WRAP = false>
int launch_tile(osb_ctx* c, Block& bl, int first, const RkFuse& rf) {
  if constexpr (CONV != 0 && !BULK && !WRAP) {
    if (bl.k.wrap) return launch_tile<T, CONV, VISC, FUSE, BULK, true>(c, bl, first, rf);
  }
  auto kern = k_central<T, CONV, VISC, FUSE, BULK, WRAP>;
  constexpr size_t smem = ct_smem<T, CONV, VISC, BULK>();
  OSB_CK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const ColumnGrid g = column_grid(c, bl.k, kern, CTY, smem, sizeof(T) == 8 ? 0.9 : 1.4);
  timing_begin(c, FAM_CENTRAL);
  kern<<<g.grid, CTT, smem, c->stream>>>(bl.k, central_params<false>(bl), first, g.czc, rf);
  timing_end(c);
  c->launches++;
  return OSB_OK;
}

// With rf (FP32 path) the kernel applies the RK update instead of storing the residual; its
// planes come in by register loads or, after osb_set_central_staging(1), by bulk copies.
template <typename T, int CONV, int VISC>
int launch_central_t(osb_ctx* c, Block& bl, int first, const RkFuse* rf) {
  if (is_wall(bl.d.bc[1][0]) || is_wall(bl.d.bc[1][1])) {
    if constexpr (CONV == 0 && VISC != 0) {
      if constexpr (sizeof(T) == 4)
        if (rf) return launch_wall<T, VISC, true>(c, bl, first, *rf);
      return launch_wall<T, VISC, false>(c, bl, first, RkFuse{});
    }
    return fail(OSB_ENOTSUP, "walls are implemented for shock-capturing schemes");
  }
  if constexpr (sizeof(T) == 4) {
    if (rf && c->central_bulk) return launch_tile<T, CONV, VISC, true, true>(c, bl, first, *rf);
    if (rf) return launch_tile<T, CONV, VISC, true, false>(c, bl, first, *rf);
  }
  return launch_tile<T, CONV, VISC, false, false>(c, bl, first, RkFuse{});
}

template <typename T>
int launch_central(osb_ctx* c, Block& bl, bool conv, int first, const RkFuse* rf) {
  const int visc = bl.d.viscous;
  if (conv && bl.d.split_form == OSB_SPLIT_KGP) {
    if (visc == OSB_VISC_SUTHERLAND || visc == OSB_VISC_POWER_LAW) return launch_central_t<T, 2, 1>(c, bl, first, rf);
    if (visc == OSB_VISC_CONSTANT) return launch_central_t<T, 2, 2>(c, bl, first, rf);
    return launch_central_t<T, 2, 0>(c, bl, first, rf);
  }
  if (conv) {
    if (visc == OSB_VISC_SUTHERLAND || visc == OSB_VISC_POWER_LAW) return launch_central_t<T, 1, 1>(c, bl, first, rf);
    if (visc == OSB_VISC_CONSTANT) return launch_central_t<T, 1, 2>(c, bl, first, rf);
    return launch_central_t<T, 1, 0>(c, bl, first, rf);
  }
  if (visc == OSB_VISC_SUTHERLAND || visc == OSB_VISC_POWER_LAW) return launch_central_t<T, 0, 1>(c, bl, first, rf);
  if (visc == OSB_VISC_CONSTANT) return launch_central_t<T, 0, 2>(c, bl, first, rf);
  return OSB_OK;
}

}  // namespace

#ifndef OSB_CENTRAL_T
#define OSB_CENTRAL_T double
#define OSB_CENTRAL_NAME central_f64
#endif

int OSB_CENTRAL_NAME(osb_ctx* c, Block& bl, bool conv, int first, const RkFuse* rf) {
  return launch_central<OSB_CENTRAL_T>(c, bl, conv, first, rf);
}

}  // namespace osb
