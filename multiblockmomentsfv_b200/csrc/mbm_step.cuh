// mbm_step.cuh -- what a step does between its stages: the ghost fill of one cell and the dt
// controller, for the kernels that launch them by themselves (mbm_kernels.cu) and for the
// persistent step loop (mbm_tile.cuh).  No multiply-add here may be contracted.
#pragma once

#include "mbm_div.cuh"
#include "mbm_internal.h"

namespace mbm {

// SetBoundary (src/Boundary.c:173-193) of one ghost cell: the host resolved the two
// sweeps into the final source of every ghost cell (an interior cell of some
// block, with the composed wall signs of src/Scenario.c:57-63, or a Dirichlet row).
__device__ __forceinline__ void ghost_fill(const BlockDev* __restrict__ blk, const GhostEntry& e, double* layer,
                                           const double* __restrict__ dirichlet, const double* __restrict__ recv) {
  const BlockDev D = blk[e.dst_blk];
  double* dst = layer + D.off + e.dst;
  const int sblk = e.src_blk_flags & 0xffff;
  const bool fx = (e.src_blk_flags >> 16) & 1, fy = (e.src_blk_flags >> 17) & 1;
  const double* p;
  long long stride = 1;
  if (e.src_blk_flags & GHOST_REMOTE) {          // a source cell on another rank
    p = recv + (size_t)e.src * NV;
  } else if (e.src >= 0) {
    p = layer + blk[sblk].off + e.src;
    stride = blk[sblk].plane;
  } else {
    p = dirichlet + (size_t)(-(e.src + 1)) * NV;
  }
  double v[NV];
#pragma unroll
  for (int m = 0; m < NV; m++) v[m] = p[m * stride];
#pragma unroll
  for (int m = 0; m < NV; m++) {
    const bool flip = (fx && (m == 1 || m == 5 || m == 7)) != (fy && (m == 2 || m == 5 || m == 8));
    dst[m * D.plane] = flip ? -v[m] : v[m];
  }
}

// CFL of an attempt of case c (src/Main.c:253-283): the maximum over stages and blocks of
// dt*lx/dx + dt*ly/dy + prod, `width` lanes (those of mask) over the blocks (the maximum is
// order-free).
// The values are >= 0 or NaN, which never passes a '>' test.  bad: a maximum that tile_steps
// flagged (a NaN or infinity was written).
constexpr unsigned long long LAM_NONFINITE = ~0ull;

__device__ __forceinline__ double case_cfl(const CaseDev& c, const BlockDev* __restrict__ blk,
                                           const unsigned long long* lam, int lane, bool& bad, int width = 32,
                                           unsigned mask = 0xffffffffu) {
  const double dt = c.dt;
  bad = false;
  double cfl = 0.0;
  for (int b = c.blk0 + lane; b < c.blk0 + c.nblk; b += width) {
    const unsigned long long* s = lam + (size_t)b * 6;
    double v[6];
#pragma unroll
    for (int k = 0; k < 6; k++) {
      const unsigned long long u = __ldcg(s + k);
      bad = bad || u == LAM_NONFINITE;
      v[k] = __longlong_as_double((long long)u);
    }
    const double dx = blk[b].dx, dy = blk[b].dy;
    const double v1 = div_rn(dt * v[0], dx) + div_rn(dt * v[1], dy) + v[2];
    const double v2 = div_rn(dt * v[3], dx) + div_rn(dt * v[4], dy) + v[5];
    if (v1 > cfl) cfl = v1;
    if (v2 > cfl) cfl = v2;
  }
  const unsigned h = (unsigned)__double2hiint(cfl), hm = __reduce_max_sync(mask, h);
  const unsigned lm = __reduce_max_sync(mask, h == hm ? (unsigned)__double2loint(cfl) : 0u);
  bad = __any_sync(mask, bad);
  return __hiloint2double((int)hm, (int)lm);
}

// One Steps iteration's bookkeeping of a case (src/Main.c:196-216): reject if CFL > CFLmax,
// else accept, swap DATA/NEW and advance t; next dt = dt*CFLreg/CFL.  trace: the case's
// progress records (null: kept by another CTA).
__device__ __forceinline__ void control_case(CaseDev& cs, double cfl, double* trace) {
  const double dt = cs.dt;
  cs.cfl_last = cfl;
  cs.attempts++;
  cs.accepted = 0;
  if (cs.nonfinite) {       // a stage wrote a NaN or infinity: stop before accepting it
    // bit 2: a bounded wait for a bulk copy ran out (MBM_ETIMEOUT), else MBM_ENONFINITE
    cs.status = (cs.nonfinite & 2) ? 3 : 2;
    cs.done = 1;
  } else if (cfl > cs.CFLmax) {
    cs.dt = div_rn(dt * cs.CFLreg, cfl);
    cs.nrej++;
  } else {
    cs.t += dt;
    double nd = div_rn(dt * cs.CFLreg, cfl);
    if (cs.t + nd > cs.tend) nd = cs.tend - cs.t;
    cs.dt = nd;
    cs.nstep++;
    cs.cur = 1 - cs.cur;
    cs.accepted = 1;
    if (cs.dtlog && cs.nstep <= cs.dtlog_cap) cs.dtlog[cs.nstep - 1] = dt;   // frozen for the adjoint
    if (cs.show_every > 0 && cs.nstep % cs.show_every == 0 && cs.trace_n < MAX_TRACE) {
      if (trace) {
        double* r = trace + (size_t)cs.trace_n * 4;
        r[0] = cs.nstep; r[1] = cfl; r[2] = cs.t; r[3] = cs.dt;
      }
      cs.trace_n++;
    }
    if (!(cs.t < cs.tend) || (cs.step_cap > 0 && cs.nstep >= cs.step_cap)) cs.done = 1;
  }
  if (!cs.done) {
    if (!isfinite(cfl) || !isfinite(cs.dt) || !(cs.dt > 0.0)) {
      cs.status = 2;  // MBM_ENONFINITE
      cs.done = 1;
    } else if (cs.attempts >= cs.max_attempts) {
      cs.status = 5;  // MBM_ESTEPLIMIT
      cs.done = 1;
    }
  }
}

// The controllers' one CTA, and the lanes of each case's, as a power of two: up to a warp while
// they fit the CTA side by side, and no fewer than the cases have blocks on average.
constexpr int CONTROL_THREADS = 256;

inline int control_lanes_log2(int ncases, int nblk) {
  int k = 5;
  while (k > 0 && (long long)ncases << k > CONTROL_THREADS && (long long)ncases << (k - 1) >= nblk) k--;
  return k;
}

// The controllers of every case, called by all threads of one CTA; clears the maxima.  Returns,
// in every thread, whether a case is still live.  A case gets 1 << lanes_log2 lanes: one case a
// warp, a batch of 512 one-block cases a thread each.  A chain of dependent loads and divisions,
// 2.4 us a case, is what bounds it, so many cases must run side by side: a step attempt of 512
// one-block cases of 24^2 cells, fast, 279 us with a warp per case, 124 like this.
__device__ __forceinline__ int control_cases(CaseDev* cases, int ncases, const BlockDev* __restrict__ blk,
                                             unsigned long long* lam, double* trace, const double* cfl_ext,
                                             int lanes_log2) {
  int live = 0;
  const int width = 1 << lanes_log2, lane = threadIdx.x & (width - 1);
  const unsigned mask = (width == 32 ? 0xffffffffu : (1u << width) - 1u) << (threadIdx.x & 31 & ~(width - 1));
  for (int c = threadIdx.x >> lanes_log2; c < ncases; c += blockDim.x >> lanes_log2) {
    CaseDev& cs = cases[c];
    if (cs.done) continue;
    bool flagged;      // (never here: the stages' kernels flag cs.nonfinite)
    const double cfl = case_cfl(cs, blk, lam, lane, flagged, width, mask);
    for (int q = lane; q < 6 * cs.nblk; q += width) lam[(size_t)cs.blk0 * 6 + q] = 0ull;
    __syncwarp(mask);
    if (lane != 0) continue;
    // a case split over ranks brings the max over all ranks (single-case contexts)
    control_case(cs, cfl_ext ? *cfl_ext : cfl, trace + (size_t)c * MAX_TRACE * 4);
    if (!cs.done) live = 1;
  }
  return __syncthreads_or(live);
}

}  // namespace mbm
