// plain_kernel.cu - the plain FP64 form's SIMPLE outer iteration as one
// persistent cooperative launch: every solve by a team of CTAs (wide_team.cuh)
// as wide as its grid can use, up to the whole GPU.
//
// Phases, with the reference functions they mirror (phases.cuh holds the
// arithmetic per cell): face values and gradients; momentum assembly,
// relaxation and residuals; red-black Gauss-Seidel for u and v; Rhie-Chow
// fluxes; pressure-correction assembly; the pressure CG (wide_cg.cuh);
// correction; SST blending, assembly, the k and omega sweeps (row_sweeps.cuh),
// floors and eddy viscosity. A phase is a grid-stride pass over the team's
// cells between two barriers (1.0 us each); the CG, 200 exchanges an
// iteration, is most of the time.
//
// Every sum is formed in an order that depends on the grid alone, so a solve
// gives the same bits on any number of CTAs, alone or in a batch.

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <string>

#include "common.hpp"
#include "phases.cuh"
#include "row_sweeps.cuh"
#include "solver.hpp"
#include "wide_cg.cuh"
#include "wide_plan.hpp"

namespace cfdb {
namespace {

/// The pressure-correction system as the CG loads it.
struct PressureSystem {
  const Instance& I;
  DEV int wake(int i) const { return I.acrossJ0[i]; }
  DEV double north(int i, int j) const {
    if (j == I.NJ || (j == 0 && I.acrossJ0[i] < 0)) return 0.0;
    return I.pN[j * I.NI + i];
  }
  DEV double east(int i, int j) const { return (i > 0 && i < I.NI) ? I.pE[j * (I.NI + 1) + i] : 0.0; }
  DEV double first(int c, int, int) const { return I.pB[c]; }
};

/// One colour of a red-black Gauss-Seidel sweep of the momentum system for u
/// and v together (one matrix, two right-hand sides; LinearSystem.cpp:77-116
/// per cell, off-diagonals summed S, E, N, W). With an even row length every
/// pair of cells (2m, 2m + 1) holds one of each colour, so threads take only
/// the colour's cells, two at a time with every load first; a missing
/// neighbour's index is clamped to the cell itself and its term left out.
DEV void gsColour(const Instance& I, const WideTeam& t, int colour) {
  const double* __restrict__ D = I.aD;
  const double* __restrict__ cS = I.aS;
  const double* __restrict__ cN = I.aN;
  const double* __restrict__ cW = I.aW;
  const double* __restrict__ cE = I.aE;
  const double* __restrict__ bu = I.bU;
  const double* __restrict__ bv = I.bV;
  double* __restrict__ u = I.u;
  double* __restrict__ v = I.v;
  const int NI = I.NI;
  const bool paired = (NI & 1) == 0;
  const int first = paired ? t.c0 / 2 : t.c0, last = paired ? t.c1 / 2 : t.c1;
  constexpr int kPair = 2;
  for (int q0 = first + t.tid; q0 < last; q0 += kPair * t.T) {
    int cell[kPair], nb[kPair][4];
    bool ok[kPair];
    double d[kPair], a[kPair][4], b1[kPair], b2[kPair], x1[kPair][4], x2[kPair][4];
#pragma unroll
    for (int e = 0; e < kPair; ++e) {
      const int q = min(q0 + e * t.T, last - 1);
      int c = paired ? 2 * q : q;
      const int j = c / NI;
      int i = c - j * NI;
      const int shift = (i + j + colour) & 1;  // 1: the cell itself has the other colour
      ok[e] = q0 + e * t.T < last && (paired || shift == 0);
      if (paired) {
        c += shift;
        i += shift;
      }
      cell[e] = c;
      nb[e][0] = across(I, c, i, j, 0);  // S
      nb[e][1] = across(I, c, i, j, 3);  // E
      nb[e][2] = across(I, c, i, j, 1);  // N
      nb[e][3] = across(I, c, i, j, 2);  // W
      d[e] = D[c];
      a[e][0] = cS[c];
      a[e][1] = cE[c];
      a[e][2] = cN[c];
      a[e][3] = cW[c];
      b1[e] = bu[c];
      b2[e] = bv[c];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int n = (nb[e][k] >= 0) ? nb[e][k] : c;
        x1[e][k] = u[n];
        x2[e][k] = v[n];
      }
    }
#pragma unroll
    for (int e = 0; e < kPair; ++e) {
      if (!ok[e] || !(fabs(d[e]) > 0.0)) continue;
      double o1 = 0.0, o2 = 0.0;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (nb[e][k] >= 0) {
          o1 += a[e][k] * x1[e][k];
          o2 += a[e][k] * x2[e][k];
        }
      }
      u[cell[e]] = (b1[e] - o1) / d[e];
      v[cell[e]] = (b2[e] - o2) / d[e];
    }
  }
}

/// The reference's two-reduction Jacobi-PCG (kernel flag bit 3; kept to compare
/// with): the next direction d' = z + beta d is formed redundantly for each
/// neighbour from z and d, which are both stable across the barrier.
DEV int cgTwoReductions(const Instance& I, WideTeam& t) {
  double init[2];
  wideSums<2>(t, init, [&](int c, int, int, double (&acc)[2]) {
    const double b = I.pB[c], zc = precondition(b, I.pD[c]);
    I.r[c] = b;
    I.z[c] = zc;
    I.d0[c] = zc;
    acc[0] += fabs(b);
    acc[1] += b * zc;
  });
  const double initial = init[0];
  double rz = init[1], beta = 0.0;
  if (!(initial > 0.0)) return 0;
  int iterations = 0;
  double *dCur = I.d0, *dNext = I.d1;
  for (int iter = 0; iter < I.cgMax; ++iter) {
    double dAd[1];
    wideSums<1>(t, dAd, [&](int c, int i, int j, double (&acc)[1]) {
      auto dir = [&](int n) { return (iter == 0) ? dCur[n] : I.z[n] + beta * dCur[n]; };
      const double dc = dir(c);
      double y = I.pD[c] * dc;
      const int n = (j > 0) ? c - I.NI : I.acrossJ0[i];
      if (n >= 0) y += I.pN[j * I.NI + i] * dir(n);
      if (j < I.NJ - 1) y += I.pN[(j + 1) * I.NI + i] * dir(c + I.NI);
      if (i > 0) y += I.pE[j * (I.NI + 1) + i] * dir(c - 1);
      if (i < I.NI - 1) y += I.pE[j * (I.NI + 1) + i + 1] * dir(c + 1);
      if (iter > 0) dNext[c] = dc;
      I.q[c] = y;
      acc[0] += dc * y;
    });
    if (iter > 0) {
      double* swap = dCur;
      dCur = dNext;
      dNext = swap;
    }
    if (!(fabs(dAd[0]) > 0.0)) break;
    const double step = rz / dAd[0];
    double rr[2];
    wideSums<2>(t, rr, [&](int c, int, int, double (&acc)[2]) {
      I.x[c] += step * dCur[c];
      const double rc = I.r[c] - step * I.q[c], zc = precondition(rc, I.pD[c]);
      I.r[c] = rc;
      I.z[c] = zc;
      acc[0] += fabs(rc);
      acc[1] += rc * zc;
    });
    iterations = iter + 1;
    if (rr[0] <= I.cgTol * initial) break;
    if (!(fabs(rz) > 0.0)) break;
    beta = rr[1] / rz;
    rz = rr[1];
  }
  return iterations;
}

/// One solve of a launch, by every thread of its team: `iterations` outer
/// iterations or fewer (`stopStage` ends the first early; `tolerance` >= 0 stops
/// at convergence or divergence as SolverWorker does, SolverWorker.cpp:164-185).
DEV void plainSolve(const Instance& I, WideTeam& t, int iterations, int stopStage, double tolerance, int smemBytes,
                    int flags) {
  extern __shared__ double dyn[];
  const bool sst = I.model == 2;
  const bool leader = t.rank == 0 && t.tid == 0;
  int done = 0;
  const int limit = min(I.iterLimit, iterations);
  const double stopTol = (tolerance >= 0.0) ? tolerance : I.stopTol;
  for (int it = 0; it < limit; ++it) {
    // the iteration's monitor, written as its values become known
    double* const mon = I.history + static_cast<std::size_t>(it) * kMonSlots;
    if (leader) {
      for (int s = 0; s < kMonSlots; ++s) mon[s] = 0.0;
    }
    auto note = [&](int slot, double value) {
      if (leader) mon[slot] = value;
    };
    double residuals[3] = {0.0, 0.0, 0.0};  // continuity, momentum x and y

    // 1. face values and gradients; velocity scale.
    double scale;
    {
      double v1[1] = {0.0};
      wideCells(t, [&](int c, int i, int j) { gradientsCell(I, c, i, j, v1[0]); });
      wideMax(t, v1);
      scale = smax(0.0, v1[0]);
      if (!(scale > 0.0)) scale = 1.0;
      note(kMonMomX, scale);  // the scale itself when the iteration ends here
    }
    if (stopStage == kStageGradients) { done = it + 1; break; }

    // 2. momentum assembly + relaxation + residuals (u and v together).
    {
      double v3[3];
      wideSums<3>(t, v3, [&](int c, int i, int j, double (&acc)[3]) {
        momentumCell<false>(I, c, i, j, acc[0], acc[1], acc[2]);
      });
      const double s = v3[2] * scale;
      residuals[1] = v3[0] / smax(s, kTinySolver);
      residuals[2] = v3[1] / smax(s, kTinySolver);
      note(kMonMomX, residuals[1]);
      note(kMonMomY, residuals[2]);
    }
    if (stopStage == kStageMomentumAssembly) { done = it + 1; break; }

    // 3. Gauss-Seidel sweeps, red-black, u and v together.
    for (int half = 0; half < 2 * I.sweeps; ++half) {
      gsColour(I, t, half & 1);
      wideBarrier(t);
    }
    if (stopStage == kStageMomentumSolve) { done = it + 1; break; }

    // 4. Rhie-Chow face fluxes.
    wideCells(t, [&](int c, int i, int j) { rhieChowCell(I, c, i, j); });
    wideBarrier(t);
    if (stopStage == kStageRhieChow) { done = it + 1; break; }

    bool stopped = false;
    const int passes = (I.nCorr > 1) ? I.nCorr : 1;
    for (int pass = 0; pass < passes && !stopped; ++pass) {
      // 5. pressure-correction assembly; the CG starts from x = 0.
      double v2[2];
      wideSums<2>(t, v2, [&](int c, int i, int j, double (&acc)[2]) {
        I.x[c] = 0.0;
        pressureAssemblyCell(I, c, i, j, acc[0], acc[1]);
      });
      if (pass == 0) {
        residuals[0] = v2[0] / I.refMassFlow;
        note(kMonMassImbalance, v2[0]);
        note(kMonContinuity, residuals[0]);
      }
      if (!I.hasPRef) {
        const double mean = v2[1] / static_cast<double>(I.N);
        wideCells(t, [&](int c, int, int) { I.pB[c] -= mean; });
        wideBarrier(t);
      }
      if (stopStage == kStagePressureAssembly) { stopped = true; break; }

      // 6. the pressure correction: Jacobi-preconditioned CG (LinearSystem.cpp:118-210).
      int cgIters;
      if (flags & kFlagTwoReductionCg) {
        cgIters = cgTwoReductions(I, t);
      } else {
        const PressureSystem load{I};
        const bool any = (flags & kFlagSharedCg) != 0;
        const WideCgSystem S{I.pD, false, I.x, nullptr, I.spill,
                             wideCgSpill(I.NI, I.NJ, t.R, t.T, smemBytes, any), I.cgTol, I.cgMax};
        if (flags & kFlagHaloWaitTest) {
          // test: a wait for a count nothing sets, which gives up and reports it
          if (t.tid == 0) {
            int polls = 0;
            while (*static_cast<volatile unsigned*>(&t.sh->never) == 0u && ++polls < (1 << 24)) {
            }
            if (polls >= (1 << 24)) atomicOr(t.faultWord, kFaultHaloWait);
          }
          __syncthreads();
        }
        cgIters = wideCg(t, S, load, smemBytes, any).iterations;
      }
      wideBarrier(t);
      if (leader) mon[kMonPressureIterations] += static_cast<double>(cgIters);
      if (!I.hasPRef) {
        double sx[1];
        wideSums<1>(t, sx, [&](int c, int, int, double (&acc)[1]) { acc[0] += I.x[c]; });
        const double m = sx[0] / static_cast<double>(I.N);
        wideCells(t, [&](int c, int, int) { I.x[c] -= m; });
        wideBarrier(t);
      }
      if (stopStage == kStagePressureSolve) { stopped = true; break; }

      // 7. correct p, u, v and the face fluxes.
      wideCells(t, [&](int c, int i, int j) { correctCell(I, c, i, j); });
      wideBarrier(t);
      if (stopStage == kStageCorrect) { stopped = true; break; }
    }
    if (stopped) {
      done = it + 1;
      break;
    }

    // 8. divergence (+ SST strain, gradients of k and omega, blending, production).
    if (sst) {
      double v1[1] = {0.0};
      wideCells(t, [&](int c, int i, int j) { sstBlendingCell(I, c, i, j, v1[0]); });
      wideMax(t, v1);
      note(kMonMaxDivergence, smax(0.0, v1[0]));
      if (stopStage == kStageSstBlending) { done = it + 1; break; }

      // the rows go to the sweeps' layouts, divided by their diagonals, and the
      // values with them; the message tag is this iteration's
      const unsigned tag = t.epoch;
      const RowSweepShape z = rowSweepShape(I.NI);
      const RowSweepSystem systems[2] = {{I.kC, I.kV, I.k}, {I.wC, I.wV, I.om}};
      double a4[4];
      wideSums<4>(t, a4, [&](int c, int i, int j, double (&acc)[4]) {
        sstAssemblyCell(I, c, i, j, acc,
                        [&](double dK, const double (&oK)[4], double bK, double dW, const double (&oW)[4], double bW,
                            double, double) {
                          I.kD[c] = dK;
                          I.kB[c] = bK;
                          I.wD[c] = dW;
                          I.wB[c] = bW;
                          rowSweepStoreRow(systems[0], z, I.NI, i, j, dK, oK, bK, I.k[c], tag);
                          rowSweepStoreRow(systems[1], z, I.NI, i, j, dW, oW, bW, I.om[c], tag);
                        });
      });
      note(kMonTurbFirst, a4[0] / smax(a4[1] * smax(I.kIn, kTinySst), kTinySst));
      note(kMonTurbSecond, a4[2] / smax(a4[3] * smax(I.wIn, kTinySst), kTinySst));
      if (stopStage == kStageSstAssembly) { done = it + 1; break; }

      // k and omega sweep in the reference's cell order: their floors and the
      // wall-cell omega override act after the sweeps, so the converged state
      // depends on the order (a colouring would move it by ~1e-3).
      const bool waitTest = (flags & kFlagChainWaitTest) != 0;
      if (flags & (kFlagSequentialRows | kFlagBarrierSweeps)) {
        for (int s = 0; s < kSweeps; ++s) {
          rowSweeps(I, t, systems, tag, s, waitTest && s == 1, reinterpret_cast<char*>(dyn), smemBytes);
          wideBarrier(t);
        }
      } else {
        rowSweeps(I, t, systems, tag, -1, waitTest, reinterpret_cast<char*>(dyn), smemBytes);
        wideBarrier(t);
      }
      if (stopStage == kStageSstSolve) { done = it + 1; break; }

      double m8[8];
#pragma unroll
      for (int s = 0; s < 8; ++s) m8[s] = -INFINITY;
      m8[5] = 0.0;
      m8[7] = 0.0;
      wideCells(t, [&](int c, int i, int j) { sstFinishCell<false>(I, c, i, j, m8); });
      wideMax(t, m8);
      note(kMonMaxK, m8[0]); note(kMonMinK, -m8[1]);
      note(kMonMaxW, m8[2]); note(kMonMinW, -m8[3]);
      note(kMonMaxMut, m8[4]); note(kMonMinMut, -m8[6]);
      note(kMonMaxYPlus, m8[5]);
      note(kMonMaxRatio, m8[7]);
    } else {
      double v1[1] = {0.0};
      wideCells(t, [&](int c, int i, int j) { v1[0] = smax(v1[0], fabs(cellDivergence(I, c, i, j))); });
      wideMax(t, v1);
      note(kMonMaxDivergence, smax(0.0, v1[0]));
    }

    done = it + 1;
    if (stopTol >= 0.0) {
      const double a = residuals[0], b = residuals[1], cc = residuals[2];
      if (!isfinite(a) || !isfinite(b) || !isfinite(cc)) break;
      if (smax(smax(fabs(a), fabs(b)), fabs(cc)) < stopTol) break;
    }
  }
  if (leader) *I.iterations = done;
}

/// CTA b runs solves plan[b].begin .. plan[b].end of `list` (indices into
/// `instances`) one after another, as CTA plan[b].rank of each one's team of
/// plan[b].R; without a plan the whole grid is the team of instance 0.
__global__ void __launch_bounds__(kWideThreads, 1)
plainKernel(const Instance* __restrict__ instances, const WideCta* __restrict__ plan, const int* __restrict__ list,
            int iterations, int stopStage, double tolerance, int smemBytes, int flags) {
  __shared__ WideShared sh;
  const WideCta me = (plan != nullptr) ? plan[blockIdx.x]
                                       : WideCta{0, 1, static_cast<int>(blockIdx.x), static_cast<int>(gridDim.x)};
  if (threadIdx.x == 0) sh.ahead = 0.0;
  for (int k = me.begin; k < me.end; ++k) {
    const Instance& I = instances[(list != nullptr) ? list[k] : k];
    const int R = wideUsefulCtas(I.NI, I.NJ, min(me.R, I.wideMost), static_cast<int>(blockDim.x));
    const double outer = outerBound(I.NI, I.NJ, R, static_cast<int>(blockDim.x),
                                    wideEffort(false, I.nCorr, I.cgMax, I.mgCap, I.sweeps));
    if (me.rank >= R) {
      // the rest of the team is at work on it: a wait of the next one is behind that
      if (threadIdx.x == 0) sh.ahead += outer;
      continue;
    }
    WideTeam t;
    wideJoin(t, I.wide, I.iterations + 1, &sh, me.rank, R, I.NI, I.NJ, iterations, outer);
    plainSolve(I, t, iterations, stopStage, tolerance, smemBytes, flags);
    wideLeave(t);
    __syncthreads();
  }
}

}  // namespace

Status preparePlainKernel() {
  static PerDeviceOnce once;
  return once.run([]() -> Status {
    const cudaError_t e = cudaFuncSetAttribute(plainKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxWideSmem);
    return (e == cudaSuccess) ? ok() : fail(CFD_INITIALIZATION_FAILURE, cudaGetErrorString(e));
  });
}

Status launchPlain(const Instance* dInstances, const WidePlan& plan, const WideCta* dPlan, const int* dList,
                   int threads, int iterations, int stopStage, double tolerance, cudaStream_t stream) {
  if (Status st = preparePlainKernel(); st != CFD_OK) return st;
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(static_cast<unsigned>(plan.ctas.size()), 1, 1);
  config.blockDim = dim3(static_cast<unsigned>(threads), 1, 1);
  config.dynamicSmemBytes = static_cast<size_t>(plan.smemBytes);
  config.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  config.attrs = attr;
  config.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&config, plainKernel, dInstances, dPlan, dList, iterations, stopStage,
                                           tolerance, plan.smemBytes, kernelFlags());
  if (e != cudaSuccess) {
    return fail(CFD_INITIALIZATION_FAILURE, std::string("SIMPLE kernel launch: ") + cudaGetErrorString(e));
  }
  return CFD_OK;
}

}  // namespace cfdb
