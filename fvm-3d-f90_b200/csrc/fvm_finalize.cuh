// fvm_finalize.cuh — the end of a time step for one case, as a CTA-wide
// device function: ClassIteration%reset_residual / compute_residual per
// block in block order / update (class_iteration.f90, file-local 195-259),
// time += dt, the stop checks of converged (:180-188) and the next step's dt.
// Run by finalize_kernel, one CTA of 256 threads per case. Every FP64
// operation is an explicitly rounded intrinsic, so the result does not depend
// on the contraction or fast-math flags of the including translation unit.
#pragma once
#include <cuda_runtime.h>

#include "fvm_types.h"

namespace fvm {

// What bounds it: memory round trips (partials, then the case state) and the
// serial fold; the bytes are negligible. So the warps of the CTA share the
// blocks evenly: with fewer blocks than warps each block's task partials are
// cut into kMaxW / nblocks slices, one warp each (a warp's lanes stride its
// slice, kU partials in flight per lane, then a butterfly), and the fold runs
// on six lanes of warp 0 at once, one per norm, over the blocks in order, as
// the reference accumulates them. A fixed order: the slices depend on the
// block and task counts only. One warp per block, with thread 0 folding all
// six norms, took 30.7 us (launched alone, launch included) on a block of 1,936
// tasks (701^2 cells in 2D) and 34.8 us on one of 128^3 cells, now 12.3 and
// 14.3; the steps went from 144.6 to 127.0 and from 1094 to 1068 us. Sixteen
// warps were no faster.
// The CTA of case 0 also zeroes the stage work-queue counters for the next
// step. The descriptors (case, block list, block sizes and task ranges)
// change only when the engine re-plans between steps, and the case state only
// here, so they are read before `wait` (the programmatic-launch wait for the
// step's last kernel; every stage kernel of the step waited for the previous
// finalize) and their memory round trips overlap that kernel's tail; partials
// and counters are touched only after it.
template <class Wait>
__device__ __forceinline__ void finalize_case(int c, const DevBlock* blocks, const DevCase* cases, const int* case_blk,
                                              DevCaseState* st, const double* partials, int* counters,
                                              int ncounters, Wait wait) {
  constexpr int kMaxW = 8;
  __shared__ double red[kMaxW][6];  // per warp: five sums of rhs^2, the wave-speed maximum
  __shared__ double s_npt[kMaxW];   // per warp: cells of its block
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int NW = min(kMaxW, (int)(blockDim.x >> 5));
  const DevCase& C = cases[c];
  const int nblocks = C.nblocks, block0 = C.block0, ts_set = C.timestep_set;
  const double dt_fixed = C.dt_fixed, cfl = C.cfl;
  const int S = nblocks > 0 && nblocks < NW ? NW / nblocks : 1;  // slices (warps) per block
  const int per = NW / S;                                        // blocks in flight
  const int slice = warp % S;
  // the first block of this warp
  int pf_task0 = 0, pf_ntask = 0;
  double pf_npt = 1.0;
  if (warp < per * S && warp / S < nblocks) {
    const DevBlock& B = blocks[case_blk[block0 + warp / S]];
    pf_task0 = B.task0;
    pf_ntask = B.ntask;
    pf_npt = (double)((int64_t)B.n[0] * B.n[1] * B.n[2]);
  }
  double S_t = 0.0, S_dt = 0.0, S_abs0 = 1.0;
  long long S_step = 0;
  if (tid < 6 && nblocks > 0) {
    S_t = st[c].t;
    S_dt = st[c].dt;
    S_step = st[c].step;
    S_abs0 = st[c].res_abs0[tid];
  }
  wait();
  if (c == 0)
    for (int i = tid; i < ncounters; i += blockDim.x) counters[i] = 0;
  if (nblocks == 0) return;  // removed case (uniform over the CTA)
  double res = 0.0;          // lane e of warp 0: norm e (5: total)
  double wmax = 0.0;
  for (int b0 = 0; b0 < nblocks; b0 += per) {
    const int bb = b0 + warp / S;
    if (warp < per * S && bb < nblocks) {
      int task0 = pf_task0, ntask = pf_ntask;
      double npt = pf_npt;
      if (b0 > 0) {
        const DevBlock& B = blocks[case_blk[block0 + bb]];
        task0 = B.task0;
        ntask = B.ntask;
        npt = (double)((int64_t)B.n[0] * B.n[1] * B.n[2]);
      }
      // each lane loads kU partials before adding them (in a fixed order), so
      // a slice costs one memory round trip per 32 * kU of its tasks
      constexpr int kU = 8;
      double s[5] = {0, 0, 0, 0, 0}, m = 0.0;
      for (int t = slice * 32 + lane; t < ntask; t += 32 * S * kU) {
        double2 q[kU][3];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
          const int tt = t + 32 * S * u;
          if (tt < ntask) {
            const double2* p = reinterpret_cast<const double2*>(partials + (int64_t)(task0 + tt) * kPartStride);
#pragma unroll
            for (int v = 0; v < 3; ++v) q[u][v] = p[v];
          } else {
#pragma unroll
            for (int v = 0; v < 3; ++v) q[u][v] = make_double2(0.0, 0.0);  // adds nothing
          }
        }
#pragma unroll
        for (int u = 0; u < kU; ++u) {
          s[0] = __dadd_rn(s[0], q[u][0].x);
          s[1] = __dadd_rn(s[1], q[u][0].y);
          s[2] = __dadd_rn(s[2], q[u][1].x);
          s[3] = __dadd_rn(s[3], q[u][1].y);
          s[4] = __dadd_rn(s[4], q[u][2].x);
          m = fmax(m, q[u][2].y);
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
        for (int v = 0; v < 5; ++v) s[v] = __dadd_rn(s[v], __shfl_xor_sync(0xffffffffu, s[v], o));
        m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
      }
      if (lane == 0) {
#pragma unroll
        for (int v = 0; v < 5; ++v) red[warp][v] = s[v];
        red[warp][5] = m;
        s_npt[warp] = npt;
      }
    }
    __syncthreads();
    if (warp == 0) {
      for (int b = 0; b < per && b0 + b < nblocks; ++b) {
        // lanes 0..4: the block's squared norm of one variable; lane 5: their mean
        const int e = min(lane, 5);
        double r2 = 0.0;
        for (int q = 0; q < S; ++q) {
          if (e < 5) r2 = __dadd_rn(r2, red[b * S + q][e]);
          wmax = fmax(wmax, red[b * S + q][5]);
        }
        r2 = __ddiv_rn(r2, s_npt[b * S]);
        double sum = 0.0;
#pragma unroll
        for (int v = 0; v < 5; ++v) sum = __dadd_rn(sum, __shfl_sync(0xffffffffu, r2, v));
        if (e == 5) r2 = __ddiv_rn(sum, 5.0);
        res = __dsqrt_rn(__dadd_rn(__dmul_rn(res, res), r2));
      }
    }
    __syncthreads();
  }
  if (tid < 6) {
    DevCaseState& D = st[c];
    S_step += 1;
    if (S_step == 1) {
      S_abs0 = res;
      D.res_abs0[tid] = res;
    }
    D.res_abs[tid] = res;
    D.res_rel[tid] = __ddiv_rn(res, S_abs0);
    if (tid == 0) {
      D.step = S_step;
      D.t = __dadd_rn(S_t, S_dt);
      D.dt_last = S_dt;
      D.dt = (ts_set == 0) ? dt_fixed : __ddiv_rn(cfl, wmax);
    }
    if (tid == 5) {
      if (isnan(res))
        D.status = 4;  // FVM_ERR_NONFINITE
      else if (res > 1.0E10)
        D.status = 5;  // FVM_ERR_DIVERGED
    }
  }
}

}  // namespace fvm
