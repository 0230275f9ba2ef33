// mbm_tile.cuh -- the Heun stage in tiles, for grids that leave the row march
// (mbm_stage.cuh) short of warps, and the step loop around it as one persistent kernel;
// compiled once per arithmetic mode, like the march, whose results it equals bit for bit.
// 4 x 61^2 cells, a step: 124 us bitwise and 62 us fast with the march of 8-row segments, two
// fill launches, a controller launch and a graph's loop; 24 and 15 us like this.
//
// The march gives a warp a strip of 28 columns and walks it up a segment of rows, 4 rows of
// warm-up per segment, each row a chain of primitives, slopes, two fluxes and an update:
// 2 us a row (fast) to 4 us (bitwise) with few warps on an SM, 12 rows at the least.  Here
// a CTA of 256 threads takes a tile of 28 x 4 output cells and does each of those once, side
// by side, with a barrier between:
//   A  the 32 x 8 cells of the tile with its halo: projected primitives; the relaxation
//      terms of the update of the output cells
//   B  the slopes: rows of cells in warps, three components at a time (30 tasks)
//   C  the fluxes: 29 x 4 x-faces and 28 x 5 y-faces, 256 in all, one per thread; a y face is
//      an x face of states with x and y swapped, so that a warp that holds both kinds runs
//      one path
//   D  the update of the 28 x 4 cells
// The halo makes it evaluate the primitives 2.3 times per output cell (the march 1.3 times)
// and the fluxes 1.14 times (1.16), so large grids stay with the march; the line is drawn at
// TILE_MOST_* (mbm_internal.h), where both are measured.  What bounds it: with one tile per CTA
// the chain through the four phases, 6,000 cycles fast and 14,000 bitwise per stage, and the
// barrier over the grid, 2,500 (a step of 14 tiles: 21,200 and 34,000 cycles); with more, two
// CTAs per SM share the FP64 and issue slots.
// Two CTAs per SM leave a thread 128 registers: 122 to 126 fast, no spills; bitwise 128 with 344
// bytes of spill stores and 308 of loads in the step loop (one CTA per SM, without them, ran as
// fast with one tile a CTA and slower with more).
//
// tile_steps runs whole Steps calls of such grids (src/Main.c:189-244): a cooperative grid
// whose CTAs keep a few tiles each, with a barrier over the grid after each Heun stage.  The
// dt controller runs in every CTA, on a copy of the case's state in shared memory and the
// maxima all CTAs have left in global memory, so that nothing but the barrier stands between
// the last flux and the next stage.  Ghost cells are not filled between the stages: a tile
// reads a ghost cell's value from the cell that SetBoundary would have copied it from (or the
// Dirichlet row), through the resolved ghost map.  The ghosts of all three layers are filled
// once, at the end.
#pragma once

#include "mbm_stage.cuh"
#if !MBM_FAST_ARITH
#include "mbm_stage_exact.cuh"
#endif
#include "mbm_step.cuh"

namespace mbm {
namespace MBM_ARITH {

constexpr int TILE_THREADS = 256;
#ifndef TILE_CTAS
#define TILE_CTAS 2
#endif
constexpr int TILE_COLS = 32, TILE_HALO_ROWS = TILE_ROWS + 4;   // of the halo tile
constexpr int XF = (STRIP + 1) * TILE_ROWS;                      // x faces of a tile
static_assert(TILE_COLS * TILE_HALO_ROWS == TILE_THREADS && XF + STRIP * (TILE_ROWS + 1) == TILE_THREADS,
              "one thread per halo cell and per face");

struct TileShared {
  double P[NV][TILE_THREADS];                    // projected primitives of the halo tile
  double S[NV][TILE_COLS * (2 * TILE_ROWS + 2)]; // slopes: x of the 4 output rows, y of 6 rows (swapped)
  double F[NV][TILE_THREADS];                    // fluxes, by face (y faces swapped)
  double R[NV][TILE_COLS * TILE_ROWS];           // relaxation terms of the update
  unsigned long long part[3][8];                 // the warps' largest lambda_x, lambda_y, production
};

// what a tile needs of its case
struct TileCase {
  double dt, F, Kn;
  int lim, cur;
  bool gather;       // ghost cells of the stage's input are read through the ghost map
};

// a cell's moments: from the layer, or, for a ghost cell of a gathered layer, from where the
// ghost fill takes it
__device__ __forceinline__ void tile_load(const StageArgs& a, const BlockDev& B, int goff, const double* layer,
                                          bool gather, int I, int J, double (&U)[NV]) {
  const double* p = layer + B.off + (long long)J * B.pitch + I + 1;
  long long stride = B.plane;
  unsigned fx = 0u, fy = 0u;
  const bool inner = I >= NG && I < B.nxp - NG && J >= NG && J < B.nyp - NG;
  if (gather && !inner) {
    const int w = B.nxp - 2 * NG, top = J - (B.nyp - NG);
    // the map lists a block's ghost cells row by row
    const int pos = J < NG ? J * B.nxp + I
                  : top < 0 ? NG * B.nxp + (J - NG) * 2 * NG + (I < NG ? I : I - w)
                            : NG * B.nxp + (B.nyp - 2 * NG) * 2 * NG + top * B.nxp + I;
    const GhostEntry e = a.ghosts[goff + pos];
    if (e.src >= 0) {
      const BlockDev& S = a.blk[e.src_blk_flags & 0xffff];
      p = layer + S.off + e.src;
      stride = S.plane;
    } else {
      p = a.dirichlet + (size_t)(-(e.src + 1)) * NV;
      stride = 1;
    }
    fx = ((e.src_blk_flags >> 16) & 1) ? 0x80000000u : 0u;
    fy = ((e.src_blk_flags >> 17) & 1) ? 0x80000000u : 0u;
  }
#pragma unroll
  for (int m = 0; m < NV; m++) U[m] = __ldcg(p + m * stride);
  if (gather) {
#pragma unroll
    for (int m = 0; m < NV; m++) {
      const unsigned f = ((m == 1 || m == 5 || m == 7) ? fx : 0u) ^ ((m == 2 || m == 5 || m == 8) ? fy : 0u);
      U[m] = __hiloint2double(__double2hiint(U[m]) ^ (int)f, __double2loint(U[m]));
    }
  }
}

// Phase B: ten rows of slopes in slots, 0 .. 3 the x slopes of the output rows, 4 .. 9 the y
// slopes of the halo tile's rows 1 .. 6 (stored with x and y swapped).  Each of the 8 warps
// does one of the first eight, nine components at fixed offsets; the last two go in groups of
// three components, {0,1,2}, {3,4,6}, {5,7,8} (in each the swap exchanges the last two), to
// six of the warps.
template <int LIM, int N>
__device__ __forceinline__ void slope_set(const double (&d1)[N], const double (&d2)[N], const Recip& h,
                                          double (&S)[N]) {
#if MBM_FAST_ARITH
#pragma unroll
  for (int i = 0; i < N; i++) S[i] = limit<LIM>(d1[i], d2[i]);
#else
  slopes<LIM>(d1, d2, h, S);
#endif
}

template <int LIM>
__device__ __forceinline__ void tile_slopes(TileShared& sh, int warp, int lane, const Recip& rdx, const Recip& rdy) {
  constexpr int SP = TILE_COLS * (2 * TILE_ROWS + 2);
  const bool x = warp < TILE_ROWS, yl = lane >= 2 && lane <= 29;
  if (x ? lane >= 1 && lane <= 30 : yl) {
    const double* p = &sh.P[0][(x ? warp + 2 : warp - TILE_ROWS + 1) * TILE_COLS + lane];
    const int st = x ? 1 : TILE_COLS, d = x ? 0 : SP;
    double* const o = &sh.S[0][warp * TILE_COLS + lane];
    double *const ou = o + d, *const od = o - d, *const ou2 = ou + d, *const od2 = od - d;
    double* const at[NV] = {o, ou, od, o, ou2, o, od2, ou, od};
    double d1[NV], d2[NV], S[NV];
#pragma unroll
    for (int n = 0; n < NV; n++) {
      const double p0 = p[n * TILE_THREADS];
      d1[n] = p0 - p[n * TILE_THREADS - st];
      d2[n] = p[n * TILE_THREADS + st] - p0;
    }
    slope_set<LIM>(d1, d2, x ? rdx : rdy, S);
#pragma unroll
    for (int n = 0; n < NV; n++) at[n][n * SP] = S[n];
  }
  if (warp < 6 && yl) {
    const int g = warp >= 3 ? warp - 3 : warp, r = warp >= 3 ? 6 : 5;      // group, row of the halo tile
    const int c[3] = {g == 0 ? 0 : (g == 1 ? 3 : 5), g == 0 ? 1 : (g == 1 ? 4 : 7), g == 0 ? 2 : (g == 1 ? 6 : 8)};
    const double* p = &sh.P[0][r * TILE_COLS + lane];
    double* o = &sh.S[0][(TILE_ROWS + r - 1) * TILE_COLS + lane];
    double d1[3], d2[3], S[3];
#pragma unroll
    for (int i = 0; i < 3; i++) {
      const double p0 = p[c[i] * TILE_THREADS];
      d1[i] = p0 - p[c[i] * TILE_THREADS - TILE_COLS];
      d2[i] = p[c[i] * TILE_THREADS + TILE_COLS] - p0;
    }
    slope_set<LIM>(d1, d2, rdy, S);
    o[c[0] * SP] = S[0];
    o[c[2] * SP] = S[1];
    o[c[1] * SP] = S[2];
  }
}

// one tile of stage HEUN; every thread of the CTA calls it
template <int HEUN>
__device__ __forceinline__ void tile_stage(const StageArgs& a, const Work w, const BlockDev& B, int goff,
                                           const TileCase& cs, TileShared& sh) {
  const int t = threadIdx.x, lane = t & 31, row = t >> 5;
  const int nxp = B.nxp, nyp = B.nyp;
  const double* layer = layer_ptr(a.buf, phys_layer(a.sel_in, cs.cur));
  const double dt = cs.dt, Fx = cs.F;
  // the output cell of this thread, rows 2 .. 5 of the halo tile
  const int I = w.I0 - 2 + lane, J = w.J0 - 2 + row;
  const long long idx = (long long)J * B.pitch + I + 1;
  const bool out_cell = row >= 2 && row < 2 + TILE_ROWS && lane >= 2 && lane <= 29 && I >= NG && I <= nxp - 1 - NG &&
                        J >= NG && J <= nyp - 1 - NG;
  double prod = 0.0, lamx = 0.0, lamy = 0.0;
  // A
  {
    double U[NV], Q[NV], R0[NV];
    const bool ok = I >= 0 && I < nxp && J >= 0 && J < nyp;
    const bool rlx_rd = HEUN == 1 && a.rlx_read;
    if (ok) tile_load(a, B, goff, layer, cs.gather, I, J, U);
    else benign(U);
    if (HEUN == 1 && out_cell) {       // Data0's relaxation term, or Data0
      const double* d0 = rlx_rd ? a.rlx + B.off + idx : layer_ptr(a.buf, phys_layer(a.sel_d0, cs.cur)) + B.off + idx;
#pragma unroll
      for (int n = 0; n < NV; n++) R0[n] = __ldcg(d0 + n * B.plane);
    }
    const Recip Kn(cs.Kn);
    primitive(U, Q);
    const bool ring = I == 0 || I == nxp - 1 || J == 0 || J == nyp - 1;
    const bool cell = ok && !ring;     // relaxation range (src/Main.c:320-321)
    const double z = coll_of(Q, dt, Kn);
    double R[NV];
#if MBM_FAST_ARITH
    const double g = dt * Fx;
    if (HEUN == 0) {
      const Damp01 dm(z);
      if (cell) prod = fmax(prod, 0.5 * (1 - dm.d2_0));
      if (out_cell) {
        relaxed_moments(Q, dm.d1_0, dm.d2_0, R);
        if (a.rlx) {
#pragma unroll
          for (int n = 0; n < NV; n++) __stcg(a.rlx + B.off + idx + n * B.plane, R[n]);
        }
      }
      if (!ring) {
        const double th = Q[3];
        Q[4] = fma(dm.d1_1, Q[4] - th, th);
        Q[5] = dm.d1_1 * Q[5];
        Q[6] = fma(dm.d1_1, Q[6] - th, th);
        Q[7] = dm.d2_1 * Q[7];
        Q[8] = dm.d2_1 * Q[8];
      }
    } else {
#pragma unroll
      for (int n = 0; n < NV; n++) R[n] = U[n];
      if (!ring) project3(Q, z);
    }
    if (out_cell && g != 0.0) {
      double V[NV];
      push_moments(R, g, V);
#pragma unroll
      for (int n = 0; n < NV; n++) R[n] = V[n];
    }
#else
    double d1u, d2u, d1p, d2p;
    if (HEUN == 0) {
      damp01(z, d1u, d1p);
      damp01(2.0 / 3 * z, d2u, d2p);
    } else {
      damp23(z, d1u, d1p);
      damp23(2.0 / 3 * z, d2u, d2p);
    }
    if (cell) prod = fmax(prod, 0.5 * (1 - d2u));
    if (out_cell) {
      if (HEUN == 0 && a.rlx) {
        relax_d<-1>(Q, R, dt, Fx, d1u, d2u);
#pragma unroll
        for (int n = 0; n < NV; n++) __stcg(a.rlx + B.off + idx + n * B.plane, R[n]);
      }
      relax_d<2 * HEUN>(Q, R, dt, Fx, d1u, d2u);
    }
    if (!ring) {
      double V[NV];
      relax_d<2 * HEUN + 1>(Q, V, dt, Fx, d1p, d2p);
      primitive(V, Q);
    }
#endif
#pragma unroll
    for (int n = 0; n < NV; n++) sh.P[n][t] = Q[n];
    if (out_cell) {
      if (HEUN == 1) {
        if (!rlx_rd) {
          double V[NV];
#pragma unroll
          for (int n = 0; n < NV; n++) U[n] = R0[n];
          primitive(U, V);
          relax_m1(V, R0, dt, Kn, Fx);
        }
#pragma unroll
        for (int n = 0; n < NV; n++) R[n] += R0[n];
      }
#pragma unroll
      for (int n = 0; n < NV; n++) sh.R[n][t - 2 * TILE_COLS] = R[n];
    }
  }
  __syncthreads();
  // B
  {
    const Recip rdx(B.dx), rdy(B.dy);
    const int warp = __shfl_sync(0xffffffffu, row, 0);
    switch (cs.lim) {
      case 0: tile_slopes<0>(sh, warp, lane, rdx, rdy); break;
      case 1: tile_slopes<1>(sh, warp, lane, rdx, rdy); break;
      case 2: tile_slopes<2>(sh, warp, lane, rdx, rdy); break;
      case 3: tile_slopes<3>(sh, warp, lane, rdx, rdy); break;
      default: tile_slopes<4>(sh, warp, lane, rdx, rdy); break;
    }
  }
  __syncthreads();
  // C
  {
    const bool y = t >= XF;
    const int u = y ? t - XF : t, per = y ? STRIP : STRIP + 1;
    const int fr = u / per, fc = u - fr * per;
    const int col = y ? 2 + fc : 1 + fc, r = y ? 1 + fr : 2 + fr;       // the lower or left cell
    const int st = y ? TILE_COLS : 1;
    const int pL = r * TILE_COLS + col, sL = (y ? TILE_ROWS + fr : fr) * TILE_COLS + col;
    // the swap exchanges planes 1 and 2, 4 and 6, 7 and 8: plane m of a y face at 0, +d or -d, ...
    const int d = y ? TILE_THREADS : 0;
    const double* p0 = &sh.P[0][pL];
    const double *pu = p0 + d, *pd = p0 - d, *pu2 = pu + d, *pd2 = pd - d, *s0 = &sh.S[0][sL];
    const double* const at[NV] = {p0, pu, pd, p0, pu2, p0, pd2, pu, pd};
    constexpr int SP = TILE_COLS * (2 * TILE_ROWS + 2);
    double PL[NV], PR[NV], f[NV];
#if !MBM_FAST_ARITH
    const double hd = 0.5 * (y ? B.dy : B.dx);
#endif
#pragma unroll
    for (int n = 0; n < NV; n++) {
      const double l = at[n][n * TILE_THREADS], rr = at[n][n * TILE_THREADS + st];
      const double sl = s0[n * SP], sr = s0[n * SP + st];
#if MBM_FAST_ARITH
      PL[n] = fma(0.5, sl, l);
      PR[n] = fma(-0.5, sr, rr);
#else
      PL[n] = l + hd * sl;
      PR[n] = rr - hd * sr;
#endif
    }
#if MBM_FAST_ARITH
    const double lam = hll<1>(PL, PR, f);
#else
    const double lam = hll_swapped(PL, PR, y, f);
#endif
    const int C = w.I0 - 2 + col, Jf = w.J0 - 2 + r;
    if (C >= 1 && C <= nxp - 3 && Jf >= 1 && Jf <= nyp - 3) {       // face loop range (src/Main.c:353-354)
      if (y) lamy = lam > 0.0 ? lam : 0.0;
      else lamx = lam > 0.0 ? lam : 0.0;
    }
#pragma unroll
    for (int n = 0; n < NV; n++) sh.F[n][t] = f[n];
    const unsigned long long mx[3] = {warp_max(lamx), warp_max(lamy), warp_max(prod)};
    if (lane == 0) {
#pragma unroll
      for (int k = 0; k < 3; k++) sh.part[k][row] = mx[k];
    }
  }
  __syncthreads();
  // the block's maxima: one atomic each per tile (8 lanes of warp 0, which has no cell to
  // update, per value)
  unsigned long long* slot = a.lam + ((size_t)w.blk * 2 + HEUN) * 3;
  if (t < 24) {
    unsigned long long v = sh.part[t >> 3][t & 7];
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
      const unsigned long long u = __shfl_xor_sync(0x00ffffffu, v, o);
      v = u > v ? u : v;
    }
    if ((t & 7) == 0 && v != 0ull) atomicMax(slot + (t >> 3), v);
  }
  // D
  int expmax = 0;
  if (out_cell) {
    double* out = layer_ptr(a.buf, phys_layer(a.sel_out, cs.cur)) + B.off + idx;
    constexpr int swap[NV] = {0, 2, 1, 3, 6, 5, 4, 8, 7};
    const double dtdx = div_rn(dt, B.dx), dtdy = div_rn(dt, B.dy);
    const int c = lane - 2, fx = (row - 2) * (STRIP + 1) + c, fy = XF + (row - 2) * STRIP + c;
#pragma unroll
    for (int n = 0; n < NV; n++) {
      double v = accumulate(sh.R[n][t - 2 * TILE_COLS], dtdx, dtdy, sh.F[n][fx], sh.F[swap[n]][fy],
                            sh.F[swap[n]][fy + STRIP], sh.F[n][fx + 1]);
      if (HEUN == 1) v = 0.5 * v;
      __stcg(out + n * B.plane, v);
      expmax = max(expmax, __double2hiint(v) & 0x7ff00000);
    }
  }
  // a NaN or infinity written: the step loop's maxima carry the flag, else the case
  if (expmax == 0x7ff00000) {
    if (a.goff) atomicMax(slot + 2, LAM_NONFINITE);
    else atomicOr(&a.cases[B.case_id].nonfinite, 1);
  }
}

// one stage of every live block, a tile per CTA
template <int HEUN>
__global__ void __launch_bounds__(TILE_THREADS, TILE_CTAS) tile_kernel(const StageArgs a) {
  pdl_enter();
  extern __shared__ __align__(128) unsigned char stage_shared[];
  TileShared& sh = *reinterpret_cast<TileShared*>(stage_shared);
  for (int w = blockIdx.x; w < a.nwork; w += gridDim.x) {
    const Work wk = a.work[w];
    const BlockDev B = a.blk[wk.blk];
    const CaseDev& c = a.cases[B.case_id];
    if (c.done) continue;
    tile_stage<HEUN>(a, wk, B, 0, TileCase{c.dt, c.F, c.Kn, c.limiter, c.cur, false}, sh);
  }
}

cudaError_t launch_tiles(const StageArgs& a, cudaStream_t s) {
  const dim3 g(a.nwork), b(TILE_THREADS);
  return a.heun ? launch_k(tile_kernel<1>, g, b, sizeof(TileShared), s, a)
                : launch_k(tile_kernel<0>, g, b, sizeof(TileShared), s, a);
}

// ------------------------------------------------------------------- the step loop --
// Barrier over the grid, `phase` the number of barriers passed with this one.  A wait gives up
// after wait_ns of device time (sync[2] is then set and the CTA returns).  Thread 0's
// release and acquire order the CTA's accesses, as in a cooperative grid's own barrier.

__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ bool tile_barrier(unsigned* sync, unsigned phase, unsigned long long wait_ns) {
  __syncthreads();
  int ok = 1;
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;\n" ::"l"(sync) : "memory");
    const unsigned target = phase * gridDim.x;
    unsigned long long t0 = 0;
    for (unsigned k = 0; (int)(ld_acquire(sync) - target) < 0; k++) {      // the count may wrap
      if ((k & 1023u) != 1023u) continue;
      const unsigned long long t = global_ns();
      if (t0 == 0) t0 = t;
      if (t - t0 > wait_ns || k > (1u << 30)) { ok = 0; break; }
    }
    if (!ok) atomicExch(sync + 2, 1u);
  }
  return __syncthreads_and(ok);
}

// a tile of the CTA, and the state of its case as this CTA's controller keeps it
struct TileMeta {
  Work w;
  BlockDev B;
  int goff, slot;    // slot: the case in ctl
};

struct TileLoopShared {
  TileMeta tile[TILE_MAX];
  CaseDev ctl[TILE_MAX];
  int id[TILE_MAX];      // the case of each slot
  int owner[TILE_MAX];   // this CTA has the case's first tile: it writes the records
  int ntile, ncase, stop;
};

// The step loop (see the head of this file).  lam is triple-buffered by attempt: an attempt's
// maxima are read by every CTA after its second barrier, and zeroed by the case's owner one
// attempt later, when no CTA can still be reading them.  They also carry whether a stage
// wrote a NaN or infinity (a flag of the case's own could be set by a CTA that is ahead).
__global__ void __launch_bounds__(TILE_THREADS, TILE_CTAS) tile_steps(const TileLoop L) {
  extern __shared__ __align__(128) unsigned char stage_shared[];
  TileShared& sh = *reinterpret_cast<TileShared*>(stage_shared);
  TileLoopShared& ls = *reinterpret_cast<TileLoopShared*>(stage_shared + sizeof(TileShared));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (L.drop && blockIdx.x == 0) return;
  StageArgs a = L.st;
  if (tid < TILE_MAX) {
    const int w = blockIdx.x + tid * gridDim.x;
    if (w < a.nwork) {
      ls.tile[tid].w = a.work[w];
      ls.tile[tid].B = a.blk[a.work[w].blk];
      ls.tile[tid].goff = a.goff[a.work[w].blk];
    }
  }
  __syncthreads();
  if (tid == 0) {
    int n = 0, nc = 0;
    for (int w = blockIdx.x; w < a.nwork && n < TILE_MAX; w += gridDim.x, n++) {
      const int id = ls.tile[n].B.case_id;
      int k = 0;
      while (k < nc && ls.id[k] != id) k++;
      if (k == nc) {
        ls.id[k] = id;
        ls.ctl[k] = a.cases[id];
        ls.owner[k] = 0;
        nc++;
      }
      ls.tile[n].slot = k;
      if (ls.tile[n].w.blk == ls.ctl[k].blk0 && ls.tile[n].w.I0 == 1 && ls.tile[n].w.J0 == 1) ls.owner[k] = 1;
    }
    ls.ntile = n;
    ls.ncase = nc;
    ls.stop = 0;
    // cases that were done before the loop count as done for the others
    for (int k = 0; k < nc; k++)
      if (ls.owner[k] && ls.ctl[k].done) atomicAdd(L.sync + 3, 1u);
  }
  __syncthreads();
  const int ntile = ls.ntile;
  unsigned phase = 0;
  for (int k = 0;; k++) {
    a.lam = L.lam + (size_t)(k % 3) * 6 * L.nblk;
    a.sel_in = SEL_CUR; a.sel_d0 = SEL_CUR; a.sel_out = SEL_TMP;
#pragma unroll 1
    for (int i = 0; i < ntile; i++) {
      const TileMeta& m = ls.tile[i];
      const CaseDev& c = ls.ctl[m.slot];
      // DATA's own ghosts until this call has accepted a step (a caller may have set them)
      if (!c.done)
        tile_stage<0>(a, m.w, m.B, m.goff, TileCase{c.dt, c.F, c.Kn, c.limiter, c.cur, c.nstep > 0}, sh);
    }
    if (!tile_barrier(L.sync, ++phase, L.wait_ns)) return;
    if (L.ncase > 1) {      // every case done, as of the last attempt
      if (tid == 0) ls.stop = __ldcg(L.sync + 3) == (unsigned)L.ncase;
      __syncthreads();
      if (ls.stop) break;
    }
    a.sel_in = SEL_TMP; a.sel_d0 = SEL_CUR; a.sel_out = SEL_OTHER;
#pragma unroll 1
    for (int i = 0; i < ntile; i++) {
      const TileMeta& m = ls.tile[i];
      const CaseDev& c = ls.ctl[m.slot];
      if (!c.done) tile_stage<1>(a, m.w, m.B, m.goff, TileCase{c.dt, c.F, c.Kn, c.limiter, c.cur, true}, sh);
    }
    if (!tile_barrier(L.sync, ++phase, L.wait_ns)) return;
    // controllers: a warp per case of this CTA
    for (int j = warp; j < ls.ncase; j += TILE_THREADS / 32) {
      CaseDev& c = ls.ctl[j];
      if (c.done) continue;
      bool bad;
      const double cfl = case_cfl(c, a.blk, a.lam, lane, bad);
      if (lane == 0) {
        c.nonfinite = bad;
        control_case(c, cfl, ls.owner[j] ? L.trace + (size_t)ls.id[j] * MAX_TRACE * 4 : nullptr);
        if (c.done && ls.owner[j] && L.ncase > 1) atomicAdd(L.sync + 3, 1u);
      }
      if (ls.owner[j]) {
        unsigned long long* z = L.lam + ((size_t)((k + 2) % 3) * L.nblk + c.blk0) * 6;
        for (int q = lane; q < 6 * c.nblk; q += 32) z[q] = 0ull;
      }
    }
    __syncthreads();
    if (L.ncase == 1 && ls.ctl[0].done) break;
  }
  // the owners' records, then SetBoundary of the layers the loop wrote: TMP, DATA if a step was
  // accepted, and the third layer unless it still is the state the call started from
  if (tid < ls.ncase && ls.owner[tid]) a.cases[ls.id[tid]] = ls.ctl[tid];
  if (!tile_barrier(L.sync, ++phase, L.wait_ns)) return;
  for (int i = blockIdx.x * blockDim.x + tid; i < 3 * L.nghost; i += gridDim.x * blockDim.x) {
    const int which = i / L.nghost;
    const GhostEntry e = a.ghosts[i - which * L.nghost];
    const CaseDev* c = a.cases + a.blk[e.dst_blk].case_id;
    const int nstep = __ldcg(&c->nstep), ran = __ldcg(&c->attempts) > 0;
    const bool fill = which == 0 ? ran : which == 1 ? nstep >= 1 : ran && (nstep != 1 || !__ldcg(&c->accepted));
    if (!fill) continue;
    const int cur = __ldcg(&c->cur);
    ghost_fill(a.blk, e, layer_ptr(a.buf, which == 0 ? 2 : which == 1 ? cur : 1 - cur), a.dirichlet, nullptr);
  }
}

constexpr int TILE_STEPS_SMEM = (int)(sizeof(TileShared) + sizeof(TileLoopShared));

// resident CTAs of tile_steps per SM; called at context creation, with the device current
int tile_ctas_per_sm() {
  static std::mutex mu;
  static unsigned long long done = 0;
  int dev = 0;
  cudaGetDevice(&dev);
  {
    std::lock_guard<std::mutex> g(mu);
    const unsigned long long bit = dev < 64 ? (1ull << dev) : 0ull;
    if (!bit || !(done & bit)) {
      cudaFuncSetAttribute(tile_kernel<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TileShared));
      cudaFuncSetAttribute(tile_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TileShared));
      cudaFuncSetAttribute(tile_steps, cudaFuncAttributeMaxDynamicSharedMemorySize, TILE_STEPS_SMEM);
      done |= bit;
    }
  }
  int n = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, tile_steps, TILE_THREADS, TILE_STEPS_SMEM);
  return n;
}

// L.sync and L.lam must be zero; grid: at most the CTAs that are resident at once, at least a
// TILE_MAX-th of the tiles
cudaError_t launch_tile_steps(const TileLoop& L, int grid, cudaStream_t s) {
  TileLoop l = L;
  void* args[] = {&l};
  return cudaLaunchCooperativeKernel(tile_steps, dim3(grid), dim3(TILE_THREADS), args, TILE_STEPS_SMEM, s);
}

}  // namespace MBM_ARITH
}  // namespace mbm
