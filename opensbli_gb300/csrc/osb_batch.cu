// osb_batch.cu -- persistent fused RK stage for batches of 2D periodic blocks (FP32-residual
// path).
//
// One launch advances every block of the context by one RK stage.  The grid is persistent
// (ctas_per_sm x SMs CTAs); each CTA claims tiles of up to 32 x ty points of any block from a work
// list (one tile per CTA where they suffice, else statically strided or through an atomic counter)
// and, per tile,
//   1. stages the FP32 state of the tile plus 3 points on every side in shared memory with the
//      primitives of each point (formed once), reading
//      the periodic images directly from the opposite interior (equivalent to the periodic
//      halo exchange of periodic.py:53-71, so no boundary kernel runs between stages),
//   2. computes the characteristic LLF fluxes of every x- and y-interface of the tile into shared
//      memory, one interface per thread and round, both directions in one list (char_flux, each
//      flux once),
//   3. forms -(dF_x/dx + dF_y/dy) per point as a float-float pair (exact flux differences),
//      applies the FP64 low-storage / SBLI RK update to the caller's state and register (the
//      first low-storage stage, A = 0, does not read the register), and
//      writes the FP32 state of the next stage into the other buffer of a ping-pong pair.
// The residual never goes to HBM.  Tiles read one FP32 buffer and write the other, so a stage
// has no intra-launch dependencies and needs no grid-wide barrier.
//
// Bound by the latency of the flux arithmetic at few warps: with a sliding window per thread a tile
// gave each of its 128 threads nine interfaces in a row on 8 warps per SM (issue 40 %).  One interface
// per thread and round fits 80 registers: 384 threads, 24 warps per SM with the default two CTAs,
// three rounds for the 1 072 interfaces of a 32 x 16 tile.  The phases between the rounds wait on
// memory, so a tile's FP64 rows and the next tile's FP32 rows are prefetched into L2.
// TENO (generated_order) forms the window's primitives in each direction's own frame, in 117 (TENO6
// 150) registers and one CTA per SM: 97 x 120, 10 steps 0.38 ms, WENO5-Z 0.26.
//
// The tiling / schedule knobs (ty, CTAs per SM, static or dynamic claiming, work order) are
// the analogue of OPS's cache-blocking tiling parameters (OPS_TILING, OPS_TILESIZE_X/Y) and are
// chosen per workload by opensbli_gb300/autotune.py.
#include <algorithm>
#include <cstring>
#include <numeric>
#include <vector>

#include "osb_internal.h"

namespace osb {

constexpr int BTX = 32;        // largest tile width (points)
constexpr int BTHREADS = 384;  // threads per CTA
constexpr int BH = 3;          // stencil reach of the flux difference
constexpr int BPITCH = BTX + 2 * BH;
constexpr int BNF = 8;         // staged fields: rho, m0, m1, E, u0, u1, p, a

struct BatchBlock {
  int n0, n1;       // interior size
  int st1, off0;    // OPS-layout row stride and linear index of (0, 0)
  int depth;        // exchange depth of its (periodic) faces, one for all; 0: they differ
  long alloc;       // allocated points per array
  float invd0, invd1;
  double* q[4];
  double* rk[4];
  const float* qin[4];
  float* qout[4];
};

// Periodic image of x in [0, n) for x >= -n.
__device__ __forceinline__ int wrapi(int x, int n) { return x < 0 ? x + n : (x < n ? x : x % n); }

__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

template <int SCH, int AVG>
__global__ void __launch_bounds__(BTHREADS, generated_order<2, SCH>() ? 1 : 2) k_batch2d(const BatchBlock* __restrict__ blocks,
                                                      const int4* __restrict__ work, int nwork, int* counter,
                                                      int ty, SchemeParams spd, int kind, double A, double B,
                                                      float dt_h, float dt_l, int save, unsigned long long* bad) {
  constexpr int NV = 4;
  const SP<float> sp(spd);
  extern __shared__ __align__(16) unsigned char osb_smem[];
  const int SR = ty + 2 * BH;    // state rows
  const int SPL = SR * BPITCH;   // one staged field
  float* S = reinterpret_cast<float*>(osb_smem);  // [BNF][SR][BPITCH]
  float* Fx = S + BNF * SPL;                      // [NV][ty][BTX + 1]
  float* Fy = Fx + NV * ty * (BTX + 1);           // [NV][ty + 1][BTX]
  __shared__ int s_w;
  const int t = threadIdx.x;
  const float gm = sp.gama;
  unsigned long long nbad = 0;
  // dynamic claiming takes the next tile while the current one is computed (the first one is the
  // CTA's own number: the counter starts at the grid size)
  int w = blockIdx.x;
  while (w < nwork) {
    if (counter && t == 0) s_w = atomicAdd(counter, 1) + gridDim.x;
    const int4 wk = work[w];
    const BatchBlock& bk = blocks[wk.x];
    const int x0 = wk.y, y0 = wk.z;
    const int n0 = bk.n0, n1 = bk.n1;
    const int tw = min(wk.w & 0xffff, n0 - x0), th = min(wk.w >> 16, n1 - y0);  // the tile's points
    // 1. stage the tile (periodic images read from the interior); the FP64 rows of phase 3 start
    // towards L2 meanwhile
    for (int idx = t; idx < (th + 2 * BH) * BPITCH; idx += BTHREADS) {
      const int c = idx % BPITCH, r = idx / BPITCH;
      if (c >= tw + 2 * BH) continue;
      const int id = bk.off0 + wrapi(x0 - BH + c, n0) + wrapi(y0 - BH + r, n1) * bk.st1;
      Pt<float, 2> s;
#pragma unroll
      for (int v = 0; v < NV; ++v) s.q[v] = __ldg(bk.qin[v] + id);
      make_pt<float, 2>(s, gm);
      float* at = S + idx;
#pragma unroll
      for (int v = 0; v < NV; ++v) at[v * SPL] = s.q[v];
      at[4 * SPL] = s.u[0];
      at[5 * SPL] = s.u[1];
      at[6 * SPL] = s.p;
      at[7 * SPL] = s.a;
    }
    for (int idx = t; idx < th * 2 * NV * 3; idx += BTHREADS) {
      const int k = idx % 3, v = (idx / 3) % (2 * NV), r = idx / (6 * NV);
      if (k * 16 < tw) prefetch_l2((v < NV ? bk.q[v] : bk.rk[v - NV]) + bk.off0 + x0 + k * 16 + (y0 + r) * bk.st1);
    }
    __syncthreads();
    w = counter ? s_w : w + gridDim.x;
    if (w < nwork) {  // the next tile's FP32 rows towards L2
      const int4 nk = work[w];
      const BatchBlock& nb = blocks[nk.x];
      const int nw = min(nk.w & 0xffff, nb.n0 - nk.y), nh = min(nk.w >> 16, nb.n1 - nk.z);
      for (int idx = t; idx < (nh + 2 * BH) * NV * 2; idx += BTHREADS) {
        const int k = idx & 1, v = (idx >> 1) % NV, r = idx / (2 * NV);
        if (k == 0 || nw > 1)
          prefetch_l2(nb.qin[v] + nb.off0 + nk.y + (k ? nw - 1 : 0) + wrapi(nk.z - BH + r, nb.n1) * nb.st1);
      }
    }
    // 2. x-interfaces i = 0 .. tw of each row (left of point i), then y-interfaces j = 0 .. th of
    // each column; the local frame of y has u1 as the normal velocity
    const int nx = (tw + 1) * th, nall = nx + tw * (th + 1);
    for (int k = t; k < nall; k += BTHREADS) {
      const bool yd = k >= nx;
      const int kk = yd ? k - nx : k, wd = yd ? tw : tw + 1;
      const int r = kk / wd, c = kk - r * wd;
      // first point of the window: three left of (below) the interface's right (upper) point
      const float* s = S + (yd ? r * BPITCH + c + BH : (r + BH) * BPITCH + c);
      const int st = yd ? BPITCH : 1;
      const int fn = yd ? 2 : 1, ft = 3 - fn;
      Pt<float, 2> win[6];
#pragma unroll
      for (int m = 0; m < 6; ++m) {
        const float* a = s + m * st;
        win[m].q[0] = a[0];
        win[m].q[1] = a[fn * SPL];
        win[m].q[2] = a[ft * SPL];
        win[m].q[3] = a[3 * SPL];
        if constexpr (generated_order<2, SCH>()) {  // in each direction's own frame, as the sweeps
          make_pt<float, 2, true>(win[m], gm);
        } else {
          win[m].u[0] = a[(3 + fn) * SPL];
          win[m].u[1] = a[(3 + ft) * SPL];
          win[m].p = a[6 * SPL];
          win[m].a = a[7 * SPL];
        }
      }
      float fh[NV];
      char_flux<float, 2, SCH, AVG>(win, sp, fh);
      float* f = yd ? Fy + r * BTX + c : Fx + r * (BTX + 1) + c;
      const int fs = yd ? (ty + 1) * BTX : ty * (BTX + 1);
      f[0] = fh[0];
      f[fn * fs] = fh[1];
      f[ft * fs] = fh[2];
      f[3 * fs] = fh[3];
    }
    __syncthreads();
    // 3. residual (float-float) and FP64 RK update of the tile's points
    for (int p = t; p < BTX * th; p += BTHREADS) {
      const int r = p / BTX, c = p % BTX;
      if (c >= tw) continue;
      const int id = bk.off0 + x0 + c + (y0 + r) * bk.st1;
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        float p1, e1, p2, e2;
        ff_flux_diff(Fx[(v * ty + r) * (BTX + 1) + c + 1], Fx[(v * ty + r) * (BTX + 1) + c], bk.invd0, p1, e1);
        ff_flux_diff(Fy[(v * (ty + 1) + r + 1) * BTX + c], Fy[(v * (ty + 1) + r) * BTX + c], bk.invd1, p2, e2);
        float h = __fadd_rn(p1, e1);
        float l = __fsub_rn(e1, __fsub_rn(h, p1));
        ff_add(h, l, p2, e2);
        const double x = dt_residual(h, l, dt_h, dt_l);  // as rk_point
        double q = bk.q[v][id];
        double o;
        if (kind == 0) {
          o = A == 0.0 ? x : __fma_rn(A, bk.rk[v][id], x);
          q = __fma_rn(B, o, q);
        } else {
          o = save ? q : bk.rk[v][id];
          q = __fma_rn(A, x, o);
          o = __fma_rn(B, x, o);
        }
        bk.rk[v][id] = o;
        bk.q[v][id] = q;
        bk.qout[v][id] = d2f_rn(q);
        if ((((unsigned)__double2hiint(q) >> 20) & 0x7ffu) == 0x7ffu) ++nbad;
      }
    }
    __syncthreads();  // the next tile reuses the shared arrays (and s_w)
  }
  if (nbad) atomicAdd(bad, nbad);
}

// FP32 state <- FP64 state of every block, whole allocations (k_q2qf of all blocks in one launch;
// blockIdx.y = 4 * block + variable).
__global__ void k_batch_q2qf(const BatchBlock* __restrict__ blocks) {
  const BatchBlock& b = blocks[blockIdx.y >> 2];
  const int v = blockIdx.y & 3, n = (int)b.alloc;
  float* f = const_cast<float*>(b.qin[v]);
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) f[t] = d2f_rn(b.q[v][t]);
}

// Periodic halo shells of every block, FP64 and FP32 state (k_periodic_shell of all blocks in one
// launch; blockIdx.y = block): y faces over the full row, then x faces of the interior rows.
__global__ void k_batch_halo(const BatchBlock* __restrict__ blocks) {
  const BatchBlock& b = blocks[blockIdx.y];
  const int D = b.depth, n0 = b.n0, n1 = b.n1, e0 = n0 + 2 * D;
  const int cy = 2 * D * e0, total = cy + 2 * D * n1;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
    int x, y;
    if (t < cy) {
      x = t % e0 - D;
      y = t / e0;
      y = y < D ? y - D : n1 + y - D;
    } else {
      const int u = t - cy;
      x = u % (2 * D);
      x = x < D ? x - D : n0 + x - D;
      y = u / (2 * D);
    }
    const int di = b.off0 + x + y * b.st1, si = b.off0 + wrapi(x, n0) + wrapi(y, n1) * b.st1;
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      b.q[v][di] = b.q[v][si];
      float* f = const_cast<float*>(b.qin[v]);
      f[di] = f[si];
    }
  }
}

size_t batch_smem(int ty) {
  const int NV = 4;
  return sizeof(float) *
         ((size_t)BNF * (ty + 2 * BH) * BPITCH + (size_t)NV * ty * (BTX + 1) + (size_t)NV * (ty + 1) * BTX);
}

namespace {

template <int SCH, int AVG>
int launch_batch_t(osb_ctx* c, const BatchBlock* tab, const SchemeParams& sp, int kind, double A, double B, double dt,
                   int save) {
  const float dt_h = (float)dt, dt_l = (float)(dt - (double)dt_h);
  auto kern = k_batch2d<SCH, AVG>;
  const int ty = c->batch.ty;
  const size_t smem = batch_smem(ty);
  OSB_CK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int* counter = nullptr;
  const int grid = std::max(1, std::min(c->batch.nwork, c->sched.ctas_per_sm * c->sm_count));
  if (c->sched.dynamic && grid < c->batch.nwork) {  // a CTA per tile has nothing to claim
    OSB_CK(cudaMemsetAsync(c->batch.counter, 0, sizeof(int), c->stream));
    counter = c->batch.counter;
  }
  timing_begin(c, FAM_PERSISTENT);
  kern<<<grid, BTHREADS, smem, c->stream>>>(tab, c->batch.work, c->batch.nwork, counter, ty, sp, kind, A, B, dt_h,
                                            dt_l, save, c->bad);
  timing_end(c);
  c->launches++;
  OSB_CK(cudaGetLastError());
  return OSB_OK;
}

}  // namespace

bool batch_eligible(const osb_ctx* c, std::string* why) {
  auto no = [&](const char* w) {
    if (why) *why = w;
    return false;
  };
  if (c->prec != OSB_PREC_FP32_RESIDUAL) return no("the persistent stage is an FP32-residual path");
  if (c->blocks.empty()) return no("no blocks");
  for (const auto& bl : c->blocks) {
    if (bl.d.ndim != 2) return no("the persistent stage takes 2D blocks");
    if (bl.k.m[9]) return no("the persistent stage takes Cartesian blocks");
    if (bl.d.scheme == OSB_SCHEME_CENTRAL4 || bl.d.viscous != OSB_VISC_NONE || bl.d.flux_type != OSB_FLUX_LLF)
      return no("the persistent stage takes the characteristic LLF Euler flux");
    for (int d = 0; d < 2; ++d)
      if (bl.d.bc[d][0] != OSB_BC_PERIODIC || bl.d.bc[d][1] != OSB_BC_PERIODIC)
        return no("the persistent stage takes fully periodic blocks");
  }
  return true;
}

// Builds the per-parity block tables, the second FP32 buffer of every block and the tile
// work list for the current schedule.
int batch_build(osb_ctx* c) {
  batch_free(c);
  if (c->sched.tile_y != 8 && c->sched.tile_y != 16 && c->sched.tile_y != 32)
    return fail(OSB_EINVAL, "tile_y must be 8, 16 or 32");
  const int nb = (int)c->blocks.size();
  // Tiles are at most 32 x tile_y points, a block's extents cut evenly.  Where tiles of that height
  // do not give every SM one, lower ones do: the launch then lasts as long as one tile, and the
  // extra y-interface per column of a lower tile costs less than the idle SMs (97 x 120 points: 32
  // tiles of height 16 took 27 us a stage, see the header for the time now).
  auto parts = [](int n, int most) { return (n + most - 1) / most; };
  auto tiles = [&](int h) {
    long n = 0;
    for (const auto& bl : c->blocks) n += (long)parts(bl.k.n[0], BTX) * parts(bl.k.n[1], h);
    return n;
  };
  int ty = c->sched.tile_y;
  while (ty > 2 && tiles(ty) < c->sm_count) ty /= 2;
  c->batch.ty = ty;
  std::vector<BatchBlock> tab[2];
  for (int ib = 0; ib < nb; ++ib) {
    Block& bl = c->blocks[ib];
    if (!bl.qf_alt) return fail(OSB_EINVAL, "block %d has no FP32 state buffers", ib);
    float* buf[2] = {bl.qf_base, bl.qf_alt};
    for (int p = 0; p < 2; ++p) {
      BatchBlock b;
      memset(&b, 0, sizeof b);
      b.n0 = bl.k.n[0];
      b.n1 = bl.k.n[1];
      b.st1 = bl.k.st[1];
      b.off0 = bl.k.off0;
      b.alloc = bl.k.alloc;
      b.depth = bl.periodic_depth();
      b.invd0 = (float)bl.k.invd[0];
      b.invd1 = (float)bl.k.invd[1];
      for (int v = 0; v < 4; ++v) {
        b.q[v] = bl.k.q[v];
        b.rk[v] = bl.k.rk[v];
        b.qin[v] = buf[p] + (size_t)v * bl.k.alloc;
        b.qout[v] = buf[p ^ 1] + (size_t)v * bl.k.alloc;
      }
      tab[p].push_back(b);
    }
  }
  // tile list
  std::vector<int> order(nb);
  std::iota(order.begin(), order.end(), 0);
  auto npts = [&](int i) { return (long)c->blocks[i].k.n[0] * c->blocks[i].k.n[1]; };
  if (c->sched.order == 1)
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return npts(a) > npts(b); });
  std::vector<std::vector<int4>> per(nb);
  for (int ib = 0; ib < nb; ++ib) {
    const BlockK& k = c->blocks[ib].k;
    const int tw = parts(k.n[0], parts(k.n[0], BTX)), th = parts(k.n[1], parts(k.n[1], ty));
    for (int y = 0; y < k.n[1]; y += th)
      for (int x = 0; x < k.n[0]; x += tw) per[ib].push_back(make_int4(ib, x, y, tw | th << 16));
  }
  std::vector<int4> work;
  if (c->sched.order == 2) {
    // interleaved: one tile of each block in turn
    size_t maxn = 0;
    for (auto& p : per) maxn = std::max(maxn, p.size());
    for (size_t i = 0; i < maxn; ++i)
      for (int ib : order)
        if (i < per[ib].size()) work.push_back(per[ib][i]);
  } else {
    for (int ib : order) work.insert(work.end(), per[ib].begin(), per[ib].end());
  }
  c->batch.nwork = (int)work.size();
  c->batch.one_depth = true;
  c->batch.max_alloc = 0;
  for (const auto& bl : c->blocks) {
    c->batch.one_depth = c->batch.one_depth && bl.periodic_depth() > 0;
    c->batch.max_alloc = std::max(c->batch.max_alloc, bl.k.alloc);
  }
  for (int p = 0; p < 2; ++p) {
    OSB_CK(cudaMalloc(&c->batch.tab[p], sizeof(BatchBlock) * nb));
    OSB_CK(cudaMemcpyAsync(c->batch.tab[p], tab[p].data(), sizeof(BatchBlock) * nb, cudaMemcpyHostToDevice,
                           c->stream));
  }
  OSB_CK(cudaMalloc(&c->batch.work, sizeof(int4) * work.size()));
  OSB_CK(cudaMemcpyAsync(c->batch.work, work.data(), sizeof(int4) * work.size(), cudaMemcpyHostToDevice, c->stream));
  OSB_CK(cudaMalloc(&c->batch.counter, sizeof(int)));
  OSB_CK(cudaStreamSynchronize(c->stream));  // host vectors go out of scope
  c->batch.ready = true;
  return OSB_OK;
}

void batch_free(osb_ctx* c) {
  for (int p = 0; p < 2; ++p)
    if (c->batch.tab[p]) {
      cudaFree(c->batch.tab[p]);
      c->batch.tab[p] = nullptr;
    }
  if (c->batch.work) cudaFree(c->batch.work);
  if (c->batch.counter) cudaFree(c->batch.counter);
  c->batch.work = nullptr;
  c->batch.counter = nullptr;
  c->batch.nwork = 0;
  c->batch.ready = false;
}

// The FP32 state of every block from its FP64 state, and the halos of both at the end of a call, each
// in one launch (128 launches for 64 instances before, 0.9 ms of a 5-step call).  False where the
// tables do not allow it: the caller then goes block by block.
bool batch_sync_shadow(osb_ctx* c) {
  if (!c->batch.ready || c->blocks.size() > 16383) return false;
  const dim3 grid((unsigned)std::min(grid_for(c, c->batch.max_alloc, 256), 64), (unsigned)(4 * c->blocks.size()));
  k_batch_q2qf<<<grid, 256, 0, c->stream>>>(c->batch.tab[c->qf_parity]);
  c->launches++;
  return true;
}
bool batch_halo(osb_ctx* c) {
  if (!c->batch.ready || !c->batch.one_depth || c->blocks.size() > 65535) return false;
  timing_begin(c, FAM_BC);
  k_batch_halo<<<dim3(8, (unsigned)c->blocks.size()), 256, 0, c->stream>>>(c->batch.tab[c->qf_parity]);
  timing_end(c);
  c->launches++;
  return true;
}

// Points BlockK::qf of every block at FP32 buffer `parity` (0: the original one).
void batch_set_parity(osb_ctx* c, int parity) {
  c->qf_parity = parity;
  for (auto& bl : c->blocks) {
    float* buf = parity ? bl.qf_alt : bl.qf_base;
    for (int v = 0; v < bl.d.ndim + 2; ++v) bl.k.qf[v] = buf + (size_t)v * bl.k.alloc;
  }
}

// One RK stage of every block in one persistent launch; flips the FP32 buffer parity.
int batch_stage(osb_ctx* c, int s, double dt) {
  if (!c->batch.ready) {
    int rc = batch_build(c);
    if (rc) return rc;
  }
  const Block& f = c->blocks[0];
  SchemeParams sp = scheme_params(f.d.gama, f.d.eps, f.d.teno_ct, f.d.shock_filter_control, 1e-12);
  const int kind = c->rk_kind == OSB_RK_LOW_STORAGE ? 0 : 1;
  const int save = (kind == 1 && s == 0) ? 1 : 0;
  const BatchBlock* tab = c->batch.tab[c->qf_parity];
  const int sch = f.d.scheme, avg = f.d.averaging;
  int rc;
  if (avg == OSB_AVG_ROE) {
    if (sch == OSB_SCHEME_WENO5_JS) rc = launch_batch_t<SCH_WENO5_JS, AVG_ROE>(c, tab, sp, kind, c->A[s], c->B[s], dt, save);
    else if (sch == OSB_SCHEME_WENO5_Z) rc = launch_batch_t<SCH_WENO5_Z, AVG_ROE>(c, tab, sp, kind, c->A[s], c->B[s], dt, save);
    else if (sch == OSB_SCHEME_TENO6) rc = launch_batch_t<SCH_TENO6, AVG_ROE>(c, tab, sp, kind, c->A[s], c->B[s], dt, save);
    else rc = launch_batch_t<SCH_TENO5, AVG_ROE>(c, tab, sp, kind, c->A[s], c->B[s], dt, save);
  } else {
    if (sch == OSB_SCHEME_WENO5_JS) rc = launch_batch_t<SCH_WENO5_JS, AVG_SIMPLE>(c, tab, sp, kind, c->A[s], c->B[s], dt, save);
    else if (sch == OSB_SCHEME_WENO5_Z) rc = launch_batch_t<SCH_WENO5_Z, AVG_SIMPLE>(c, tab, sp, kind, c->A[s], c->B[s], dt, save);
    else if (sch == OSB_SCHEME_TENO6) rc = launch_batch_t<SCH_TENO6, AVG_SIMPLE>(c, tab, sp, kind, c->A[s], c->B[s], dt, save);
    else rc = launch_batch_t<SCH_TENO5, AVG_SIMPLE>(c, tab, sp, kind, c->A[s], c->B[s], dt, save);
  }
  if (rc) return rc;
  batch_set_parity(c, c->qf_parity ^ 1);
  return OSB_OK;
}

}  // namespace osb
