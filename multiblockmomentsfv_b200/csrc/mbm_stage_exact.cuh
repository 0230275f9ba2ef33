// mbm_stage_exact.cuh -- the bitwise Heun stage of large grids (Update, src/Main.c:297-396): the
// row march of mbm_stage.cuh, written for a small body of code.
//
// One warp owns a strip of 28 output columns plus a 2-column halo on each side (lane l <->
// column I0 - 2 + l) and a segment of rows, and marches up the segment; iteration r forms the
// projected primitives of row r, the y slopes of row r-1 and the y-face flux between rows r-2
// and r-1, then the x slopes and x-face fluxes of row r-2 and its update.
//
// The unfused, exactly rounded arithmetic takes 126 M warp instructions a stage of 4 x 512^2 cells
// where the fast mode takes 52 M.  Written out straight, each direction with code of its own, a
// row is 44 KB of instructions, more than an SM keeps close: its warps waited for instructions a
// fifth of the time.  So the two directions are one loop, x and y swapped in the y pass (hll_swapped).  The
// moments of the next row and Data0 of the row to be updated are copied to shared memory
// while a row is worked on (the next row's without a condition: lanes and rows outside the grid
// copy the nearest cell), and the update's other term is loaded before the fluxes.
//
// What bounds it: fixed-latency dependencies and the FP64 pipe (49 % of an SM's active cycles) at
// two warps per scheduler.  4 x 1024^2 cells, harmonic: 886 -> 815 us a stage (4 x 256^2: 78 ->
// 71); with copies under a condition and a state at rest in place of the missing cells 838,
// without the copies 884; three warps per scheduler (168 registers; both sides of a face
// one loop too, its states and partial sums in shared memory; no room for the copies, 20-100
// bytes of spills) 930-1,020: the tighter allocation leaves less to issue between dependent
// operations than the third warp brings.
#pragma once

#include "mbm_stage.cuh"

namespace mbm {
namespace bitwise {

// Rolling state of one warp, lane fastest (conflict-free 8-byte accesses)
struct ExactWindow {
  double P[3][NV][32];      // projected primitives of rows r, r-1, r-2
  double lo[2][NV][32];     // upper y-face state of a row (x and y swapped), by parity of r; the
                            // one of the finished face then holds the left x-face states
  double hi[NV][32];        // lower y-face state of row r-1 (swapped); then the right x-face states
  double G[2][NV][32];      // y fluxes below and above row r-2 (swapped), by parity of r
  double Ua[NV][32];        // the moments of the next row, copied there asynchronously
  double D0a[NV][32];       // stage 2: Data0 (or its stored relaxation term) of the row to be updated
};

// two CTAs of four warps per SM: 240 to 254 registers, no spills
constexpr int EXACT_WARPS = 4, EXACT_CTAS = 2;
constexpr int EXACT_SMEM = (int)sizeof(ExactWindow) * EXACT_WARPS;

template <int HEUN, int LIM>
__device__ __forceinline__ void exact_item(const StageArgs& a, const Work w, const int wi, const int lane,
                                           ExactWindow& win) {
  const BlockDev B = a.blk[w.blk];
  const CaseDev& cs = a.cases[B.case_id];
  if (cs.done) return;
  const int cur = cs.cur;
  const double dt = cs.dt, Fx = cs.F;
  const int lim = cs.limiter;
  const Recip Kn(cs.Kn);
  const double* __restrict__ in = layer_ptr(a.buf, phys_layer(a.sel_in, cur)) + B.off;
  const double* __restrict__ d0 = layer_ptr(a.buf, phys_layer(a.sel_d0, cur)) + B.off;
  double* __restrict__ out = layer_ptr(a.buf, phys_layer(a.sel_out, cur)) + B.off;
  // the relaxation term of the stage-1 input (flag -1), written by stage 1; stage 2 reads it
  // with rlx_read in place of forming it from Data0.  Null: not stored.
  double* __restrict__ rlx = a.rlx ? a.rlx + B.off : nullptr;
  const bool rlx_rd = HEUN == 1 && a.rlx_read;
  const double* __restrict__ d0src = rlx_rd ? rlx : d0;
  const int nxp = B.nxp, nyp = B.nyp, pitch = B.pitch;
  const long long plane = B.plane;
  const int C = w.I0 - 2 + lane;
  const bool col_in = C >= 0 && C < nxp;
  const bool col_ring = C == 0 || C == nxp - 1;
  const bool col_face = C >= 1 && C <= nxp - 3;      // face loop range (src/Main.c:353-354)
  const bool col_cell = C >= 1 && C <= nxp - 2;      // relaxation range (src/Main.c:320-321)
  const bool col_out = lane >= 2 && lane <= 29 && C >= NG && C <= nxp - 1 - NG;
  const double dtdx = div_rn(dt, B.dx), dtdy = div_rn(dt, B.dy);
  const Recip rdx(B.dx), rdy(B.dy);   // dx, dy in the safe range (checked at creation)
  double lamx = 0.0, lamy = 0.0, prod = 0.0;
  int expmax = 0;     // largest exponent field (high word & 0x7ff00000) written: all ones = NaN or inf
  const int rs = w.J0 >= 2 ? w.J0 - 2 : w.J0 - 1;
  int s0 = rs % 3;                 // window slot of row r
  auto u_fetch = [&](int rr) {
    // lanes and rows outside the grid: the nearest cell's values, unused
    const long long idx = (long long)min(rr, nyp - 1) * pitch + min(max(C, 0), nxp - 1) + 1;
#pragma unroll
    for (int n = 0; n < NV; n++) cp_async8(&win.Ua[n][lane], in + n * plane + idx);
    cp_async_commit();
  };
  u_fetch(rs);
#pragma unroll 1
  for (int r = rs; r <= w.J1 + 1; r++) {
    const int sm1 = s0 == 0 ? 2 : s0 - 1, sm2 = sm1 == 0 ? 2 : sm1 - 1;
    const int J = r - 2;
    const bool row = J >= w.J0 && J < w.J1;
    const bool upd = row && col_out && J >= NG && J <= nyp - 1 - NG;      // this lane updates a cell
    // (a) projected primitives of row r: Aux.Prim (src/Main.c:314-336)
    {
      double U[NV], Q[NV];
      const bool ok = col_in && r >= 0 && r < nyp;
      cp_async_wait_all();
#pragma unroll
      for (int n = 0; n < NV; n++) U[n] = win.Ua[n][lane];
      if (HEUN == 1 && upd) {
#pragma unroll
        for (int n = 0; n < NV; n++) cp_async8(&win.D0a[n][lane], d0src + n * plane + (long long)J * pitch + C + 1);
        cp_async_commit();
      }
      u_fetch(r + 1);                      // into the slot just read
      primitive(U, Q);
      // one collision number serves every ProductionsDirect of this cell in this stage,
      // each flag's damping factors formed from it with the reference's expressions:
      // the CFL share and the update's relaxation term (flag 2 HEUN, parked in the
      // output layer until the update of this row two iterations later), stage 1's
      // relaxation of Data0 for stage 2 (flag -1: flag 0 without the force) and the
      // projection (flag 2 HEUN + 1)
      const double z = coll_of(Q, dt, Kn);
      double d1u, d2u, d1p, d2p;      // flags 2 HEUN and 2 HEUN + 1, at z and 2z/3
      if (HEUN == 0) {
        damp01(z, d1u, d1p);
        damp01(2.0 / 3 * z, d2u, d2p);
      } else {
        damp23(z, d1u, d1p);
        damp23(2.0 / 3 * z, d2u, d2p);
      }
      if (ok && col_cell && r >= 1 && r <= nyp - 2) {
        const double c = 0.5 * (1 - d2u);
        if (c > prod) prod = c;
      }
      if (ok && col_out && r >= NG && r <= nyp - 1 - NG && r >= w.J0 && r < w.J1) {
        const long long idx = (long long)r * pitch + C + 1;
        double R[NV];
        relax_d<2 * HEUN>(Q, R, dt, Fx, d1u, d2u);
#pragma unroll
        for (int n = 0; n < NV; n++) out[n * plane + idx] = R[n];
        if (HEUN == 0 && rlx) {
          relax_d<-1>(Q, R, dt, Fx, d1u, d2u);
#pragma unroll
          for (int n = 0; n < NV; n++) rlx[n * plane + idx] = R[n];
        }
      }
      if (!(col_ring || r == 0 || r == nyp - 1)) {
        double V[NV];
        relax_d<2 * HEUN + 1>(Q, V, dt, Fx, d1p, d2p);
        primitive(V, Q);
      }
#pragma unroll
      for (int n = 0; n < NV; n++) win.P[s0][n][lane] = Q[n];
    }
    __syncwarp();
    // (b) y slopes of row r-1 (src/Main.c:348-349) and the y face (r-2 | r-1), then (c) x slopes
    // of row r-2 and its faces C | C+1 (src/Main.c:346-347, 372-378)
    double flx[NV], R[NV];
    const long long idx = (long long)J * pitch + C + 1;
    if (upd) {                              // relax<2 HEUN> of the cell, wanted after the fluxes
#pragma unroll
      for (int n = 0; n < NV; n++) R[n] = out[n * plane + idx];
    }
#pragma unroll 1
    for (int f = 0; f < 2; f++) {
      const bool y = f == 0;
      if (y ? r < rs + 2 : !row) continue;
      // planes 1 and 2, 4 and 6, 7 and 8 exchanged for y: plane n at 32 n, + d or - d, ...
      const int d = y ? 32 : 0;
      const int off[NV] = {0, 32 + d, 64 - d, 96, 128 + 2 * d, 160, 192 - 2 * d, 224 + d, 256 - d};
      const double* pc = &win.P[y ? sm1 : sm2][0][lane];
      const double* pm = y ? &win.P[sm2][0][lane] : &win.P[sm2][0][(lane + 31) & 31];
      const double* pp = y ? &win.P[s0][0][lane] : &win.P[sm2][0][(lane + 1) & 31];
      double* const pl = &win.lo[(r - 1) & 1][0][lane];
      {
        double d1[NV], d2[NV], S[NV], p0[NV];
#pragma unroll
        for (int n = 0; n < NV; n++) {
          p0[n] = pc[off[n]];
          d1[n] = p0[n] - pm[off[n]];
          d2[n] = pp[off[n]] - p0[n];
        }
        const double h = 0.5 * (y ? B.dy : B.dx);
        slopes_of<LIM>(d1, d2, y ? rdy : rdx, lim, S);
        double* const up = y ? &win.lo[r & 1][0][lane] : pl;
#pragma unroll
        for (int n = 0; n < NV; n++) {
          up[n * 32] = p0[n] + h * S[n];
          win.hi[n][lane] = p0[n] - h * S[n];
        }
      }
      __syncwarp();
      if (y ? r >= rs + 3 && lane >= 2 && lane <= 29 : lane >= 1 && lane <= 29) {
        const double* pr = &win.hi[0][y ? lane : lane + 1];
        double L[NV], R_[NV];
#pragma unroll
        for (int n = 0; n < NV; n++) {
          L[n] = pl[n * 32];
          R_[n] = pr[n * 32];
        }
        const double lam = hll_swapped(L, R_, y, flx);
        if (col_face && J >= 1 && J <= nyp - 3) {
          if (y) lamy = lam > lamy ? lam : lamy;
          else lamx = lam > lamx ? lam : lamx;
        }
        if (y) {
#pragma unroll
          for (int n = 0; n < NV; n++) win.G[r & 1][n][lane] = flx[n];
        }
      }
      __syncwarp();
    }
    // cell update of row J (src/Main.c:323-331, 367-393)
    if (row) {
      double Fm[NV];
#pragma unroll
      for (int n = 0; n < NV; n++) Fm[n] = __shfl_up_sync(0xffffffffu, flx[n], 1);
      if (upd) {
        if constexpr (HEUN == 1) {
          double R0[NV];
          cp_async_wait_one();              // Data0 has landed (the next row may still be on its way)
#pragma unroll
          for (int n = 0; n < NV; n++) R0[n] = win.D0a[n][lane];
          if (!rlx_rd) {                    // not stored: relax<-1>(Data0)
            double U[NV], Q[NV];
#pragma unroll
            for (int n = 0; n < NV; n++) U[n] = R0[n];
            primitive(U, Q);
            relax_m1(Q, R0, dt, Kn, Fx);
          }
#pragma unroll
          for (int n = 0; n < NV; n++) R[n] += R0[n];
        }
        constexpr int swap[NV] = {0, 2, 1, 3, 6, 5, 4, 8, 7};
#pragma unroll
        for (int n = 0; n < NV; n++) {
          double v = accumulate(R[n], dtdx, dtdy, Fm[n], win.G[(r - 1) & 1][swap[n]][lane],
                                win.G[r & 1][swap[n]][lane], flx[n]);
          if (HEUN == 1) v = 0.5 * v;
          out[n * plane + idx] = v;
          expmax = max(expmax, __double2hiint(v) & 0x7ff00000);
        }
      }
    }
    s0 = s0 == 2 ? 0 : s0 + 1;
  }
  cp_async_wait_all();                      // nothing in flight past the work item
  if (a.gs_item) scatter_item(a, wi, lane, out - B.off, out, plane);
  stage_maxima<HEUN>(a, w.blk, B.case_id, lane, lamx, lamy, prod, expmax);
}

template <int HEUN, int LIM>
__global__ void __launch_bounds__(32 * EXACT_WARPS, EXACT_CTAS) stage_exact(const StageArgs a) {
  pdl_enter();
  extern __shared__ __align__(128) unsigned char stage_shared[];
  ExactWindow* win = reinterpret_cast<ExactWindow*>(stage_shared);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (;;) {
    int w = 0;
    if (lane == 0) w = atomicAdd(a.queue, 1);
    w = __shfl_sync(0xffffffffu, w, 0);
    if (w >= a.nwork) break;
    exact_item<HEUN, LIM>(a, a.work[w], w, lane, win[warp]);
  }
}

template <int HEUN, int LIM>
static void exact_attr() {
  cudaFuncSetAttribute(stage_exact<HEUN, LIM>, cudaFuncAttributeMaxDynamicSharedMemorySize, EXACT_SMEM);
}

// as the fast mode's (mbm_stage.cuh)
int stage_ctas_per_sm(int heun) {
  static std::mutex mu;
  static unsigned long long done = 0;     // one bit per device ordinal < 64
  int dev = 0;
  cudaGetDevice(&dev);
  {
    std::lock_guard<std::mutex> g(mu);
    const unsigned long long bit = dev < 64 ? (1ull << dev) : 0ull;
    if (!bit || !(done & bit)) {
      exact_attr<0, 0>(); exact_attr<0, 1>(); exact_attr<0, 2>(); exact_attr<0, 3>(); exact_attr<0, 4>();
      exact_attr<0, LIM_ANY>(); exact_attr<1, LIM_ANY>();
      exact_attr<1, 0>(); exact_attr<1, 1>(); exact_attr<1, 2>(); exact_attr<1, 3>(); exact_attr<1, 4>();
      done |= bit;
    }
  }
  int n = 0;
  if (heun) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, stage_exact<1, 4>, 32 * EXACT_WARPS, EXACT_SMEM);
  else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, stage_exact<0, 4>, 32 * EXACT_WARPS, EXACT_SMEM);
  return n > 0 ? n : 1;
}

int stage_cta_warps() { return EXACT_WARPS; }

template <int HEUN>
static cudaError_t launch_exact(int lim, const StageArgs& a, int grid, cudaStream_t s) {
  const dim3 g(grid), b(32 * EXACT_WARPS);
  switch (lim) {
    case 0: return launch_k(stage_exact<HEUN, 0>, g, b, EXACT_SMEM, s, a);
    case 1: return launch_k(stage_exact<HEUN, 1>, g, b, EXACT_SMEM, s, a);
    case 2: return launch_k(stage_exact<HEUN, 2>, g, b, EXACT_SMEM, s, a);
    case 3: return launch_k(stage_exact<HEUN, 3>, g, b, EXACT_SMEM, s, a);
    case LIM_ANY: return launch_k(stage_exact<HEUN, LIM_ANY>, g, b, EXACT_SMEM, s, a);
    default: return launch_k(stage_exact<HEUN, 4>, g, b, EXACT_SMEM, s, a);
  }
}

cudaError_t launch_stage(int lim, const StageArgs& a, int grid, cudaStream_t s) {
  return a.heun ? launch_exact<1>(lim, a, grid, s) : launch_exact<0>(lim, a, grid, s);
}

}  // namespace bitwise
}  // namespace mbm
