// simple_kernel.cu - the SIMPLE outer iteration (laminar and k-omega SST) as
// one persistent cooperative kernel per launch: the mixed FP32/FP64 form.
//
// A SIMPLE iteration is ~15 dependent phases and a pressure solve of ~16
// multigrid V-cycles, each a chain of small phases over the levels: 5-point
// stencils and reductions over 1e4-1e5 cells, far too little work to hide a
// kernel launch. The launch is cooperative and persistent: a solve has a team of
// CTAs (wide_team.cuh), one per SM and up to the whole GPU, that meet in
// barriers through L2, and a batch's solves share the launch by a plan. One
// thread-block cluster of 16 CTAs per solve has cheaper barriers (0.7 us against
// 1.0) but leaves 132 SMs idle beside a lone solve: a phase over 768x192 cells
// took 6 us there, and an outer iteration 2.6 ms.
//
// Arithmetic
// ----------
// The plain FP64 form is built with contraction off (no FMA) and evaluates
// every per-cell and per-face expression with the operands, association and
// accumulation order the reference uses, so each non-reduction stage gives
// the reference's values to the last bit. Face quantities are recomputed by
// every cell that touches the face (the owner and the neighbour compute the
// identical value) instead of being scattered, so no atomics are needed and
// a cell's sums are accumulated in the reference's face order:
//   Green-Gauss, assembly, net flux, divergence: S, N, W, E
//     (j-faces before i-faces, ascending index; Mesh.cpp:138-170)
//   Gauss-Seidel off-diagonal sum:               S, E, N, W
//     (Mesh::cellFaces order, Mesh.cpp:172-181; LinearSystem.cpp:94-112)
// Reductions (residual norms, CG dots, maxima) are deterministic: sums in an
// order that depends on the grid alone (wide_team.cuh); every CTA derives the
// same bits, so control flow that depends on them (CG exit, convergence) is
// uniform, and a solve gives the same bits on any number of CTAs. Gauss-Seidel is red-black instead of lexicographic: exact with the
// wake cut because cellsI is even on a C-grid, so partners across the cut have
// opposite colours. It changes the iterate path but not the converged answer.

#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <cstdlib>

#include <algorithm>
#include <string>

#include "common.hpp"
#include "instance.hpp"
#include "mixed_sweeps.cuh"
#include "phases.cuh"
#include "solver.hpp"
#include "wide_plan.hpp"
#include "wide_team.cuh"

namespace cfdb {
namespace {

/// One red-black colour pass of the momentum corrections (A du = ru, A dv = rv
/// in FP32, shared rows). The last pass of the last sweep also adds both
/// corrections to the FP64 velocities of every own cell: the other colour's
/// corrections are final by then and no neighbour reads u or v during the
/// sweeps. Cells in pairs as in the plain form's gsColour.
DEV void gsColourMixed(const Instance& I, const WideTeam& t, int colour, bool last) {
  const Rows32& m = I.mom;
  const float* __restrict__ D = m.D;
  const float* __restrict__ cS = m.S;
  const float* __restrict__ cN = m.N;
  const float* __restrict__ cW = m.W;
  const float* __restrict__ cE = m.E;
  const float* __restrict__ ru = m.r;
  const float* __restrict__ rv = I.momRv;
  float* __restrict__ xu = m.x;
  float* __restrict__ xv = I.momXv;
  const int NI = I.NI;
  const bool paired = (NI & 1) == 0;
  const int first = paired ? t.c0 / 2 : t.c0, end = paired ? t.c1 / 2 : t.c1;
  constexpr int kPair = 2;
  for (int q0 = first + t.tid; q0 < end; q0 += kPair * t.T) {
    int cell[kPair], nb[kPair][4];
    bool ok[kPair];
    float d[kPair], a[kPair][4], b1[kPair], b2[kPair], x1[kPair][4], x2[kPair][4];
#pragma unroll
    for (int e = 0; e < kPair; ++e) {
      const int q = min(q0 + e * t.T, end - 1);
      int c = paired ? 2 * q : q;
      const int j = c / NI;
      int i = c - j * NI;
      const int shift = (i + j + colour) & 1;  // 1: the cell itself has the other colour
      ok[e] = q0 + e * t.T < end && (paired || shift == 0);
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
      b1[e] = ru[c];
      b2[e] = rv[c];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int n = (nb[e][k] >= 0) ? nb[e][k] : c;
        x1[e][k] = xu[n];
        x2[e][k] = xv[n];
      }
    }
#pragma unroll
    for (int e = 0; e < kPair; ++e) {
      if (!ok[e] || d[e] == 0.0f) continue;
      float ou = 0.0f, ov = 0.0f;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (nb[e][k] >= 0) {
          ou += a[e][k] * x1[e][k];
          ov += a[e][k] * x2[e][k];
        }
      }
      xu[cell[e]] = (b1[e] - ou) / d[e];
      xv[cell[e]] = (b2[e] - ov) / d[e];
    }
  }
  if (last) {
    // the corrections of the CTA's cells (it wrote all of them) onto u, v
    __syncthreads();
    for (int c = t.c0 + t.tid; c < t.c1; c += t.T) {
      I.u[c] += static_cast<double>(xu[c]);
      I.v[c] += static_cast<double>(xv[c]);
    }
  }
}

#include "pressure_mg.cuh"

// ---- the kernel -----------------------------------------------------------------

/// One solve of a launch, by every thread of its team: `iterations` outer
/// iterations or fewer (`stopStage` ends the first early; `tolerance` >= 0 stops
/// at convergence or divergence as SolverWorker does, SolverWorker.cpp:164-185).
DEV void mixedSolve(const Instance& I, WideTeam& t, int iterations, int stopStage, double tolerance, int smemBytes,
                    int flags) {
  const bool sst = (I.model == 2);
  const bool leader = (t.rank == 0 && t.tid == 0);

  int done = 0;
  const int limit = (I.iterLimit < iterations) ? I.iterLimit : iterations;
  const double stopTol = (tolerance >= 0.0) ? tolerance : I.stopTol;
  for (int it = 0; it < limit; ++it) {
    // the iteration's monitor, written as its values become known (16 doubles
    // per thread fewer to keep than with one write at the end)
    double* const mon = I.history + static_cast<std::size_t>(it) * kMonSlots;
    if (leader) {
      for (int s = 0; s < kMonSlots; ++s) mon[s] = 0.0;
    }
    auto note = [&](int slot, double value) {
      if (leader) mon[slot] = value;
    };
    double continuity = 0.0, momentumX = 0.0, momentumY = 0.0;

    // 1. face values and gradients; velocity scale.
    {
      double v1[1] = {0.0};
      wideCells(t, [&](int c, int i, int j) { gradientsCell(I, c, i, j, v1[0]); });
      wideMax(t, v1);
      double scale = smax(0.0, v1[0]);
      if (!(scale > 0.0)) scale = 1.0;
      momentumX = scale;  // held until the residuals are known
      note(kMonMomX, scale);
    }
    if (stopStage == kStageGradients) { done = it + 1; break; }

    // 2. momentum assembly + relaxation + residuals (u and v together).
    {
      double v3[3];
      wideSums(t, v3, [&](int c, int i, int j, double (&acc)[3]) {
        momentumCell<true>(I, c, i, j, acc[0], acc[1], acc[2]);
      });
      const double scale = v3[2] * momentumX;
      momentumX = v3[0] / smax(scale, kTinySolver);
      momentumY = v3[1] / smax(scale, kTinySolver);
      note(kMonMomX, momentumX);
      note(kMonMomY, momentumY);
    }
    if (stopStage == kStageMomentumAssembly) { done = it + 1; break; }

    // 3. Gauss-Seidel sweeps, red-black, u and v together.
    for (int sweep = 0; sweep < I.sweeps; ++sweep) {
      for (int colour = 0; colour < 2; ++colour) {
        gsColourMixed(I, t, colour, sweep == I.sweeps - 1 && colour == 1);
        wideBarrier(t);
      }
    }
    if (stopStage == kStageMomentumSolve) { done = it + 1; break; }

    // 4. Rhie-Chow face fluxes.
    wideCells(t, [&](int c, int i, int j) { rhieChowCell(I, c, i, j); });
    wideBarrier(t);
    if (stopStage == kStageRhieChow) { done = it + 1; break; }

    bool stopped = false;
    const int passes = (I.nCorr > 1) ? I.nCorr : 1;
    for (int pass = 0; pass < passes && !stopped; ++pass) {
      // 5. pressure-correction assembly; the solve starts from x = 0, r = b.
      double v2[2];
      wideSums(t, v2, [&](int c, int i, int j, double (&acc)[2]) {
        pressureAssemblyCell(I, c, i, j, acc[0], acc[1]);
      });
      if (pass == 0) {
        continuity = v2[0] / I.refMassFlow;
        note(kMonMassImbalance, v2[0]);
        note(kMonContinuity, continuity);
      }
      const double mean = I.hasPRef ? 0.0 : v2[1] / static_cast<double>(I.N);
      double init[1];
      wideSums(t, init, [&](int c, int, int, double (&acc)[1]) {
        double b = I.pB[c];
        if (!I.hasPRef) {
          b -= mean;
          I.pB[c] = b;
        }
        I.x[c] = 0.0;
        I.r[c] = b;
        acc[0] += fabs(b);
      });
      if (stopStage == kStagePressureAssembly) { stopped = true; break; }

      // 6. the pressure correction: multigrid CG (pressure_mg.cuh).
      const double initial = init[0];
      const int cgIters = (initial > 0.0) ? pressureMixed(I, t, initial, (flags & kFlagPhasedCycle) != 0) : 0;
      if (leader) mon[kMonPressureIterations] += static_cast<double>(cgIters);
      if (!I.hasPRef) {
        double sx[1];
        wideSums(t, sx, [&](int c, int, int, double (&acc)[1]) { acc[0] += I.x[c]; });
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
    if (stopped) { done = it + 1; break; }

    // 8. divergence (+ SST strain, gradients of k and omega, blending, production).
    if (sst) {
      double v1[1] = {0.0};
      wideCells(t, [&](int c, int i, int j) { sstBlendingCell(I, c, i, j, v1[0]); });
      wideMax(t, v1);
      note(kMonMaxDivergence, smax(0.0, v1[0]));
      if (stopStage == kStageSstBlending) { done = it + 1; break; }

      const unsigned tag = t.epoch;  // of this iteration's sweep messages
      const bool rowwise = !(flags & kFlagPlainWavefront) && I.NI <= 8 * t.T && mixedRowsFit(I.NI, I.mg.coarseBytes);
      const bool chained = rowwise && !(flags & (kFlagSequentialRows | kFlagBarrierSweeps)) &&
                           mixedChained(I, t, smemBytes);
      const ChainShape z = chainShape(I.NI, t.T);
      double a4[4];
      wideSums(t, a4, [&](int c, int i, int j, double (&acc)[4]) {
        sstAssemblyCell(I, c, i, j, acc,
                        [&](double dK, const double (&oK)[4], double bK, double dW, const double (&oW)[4], double bW,
                            double yk, double yw) {
          I.kD[c] = dK; I.kS[c] = oK[0]; I.kN[c] = oK[1]; I.kW[c] = oK[2]; I.kE[c] = oK[3]; I.kB[c] = bK;
          I.wD[c] = dW; I.wS[c] = oW[0]; I.wN[c] = oW[1]; I.wW[c] = oW[2]; I.wE[c] = oW[3]; I.wB[c] = bW;
          const float rk = static_cast<float>(bK - yk), rw = static_cast<float>(bW - yw);
          auto put = [&](const Rows32& a, float4* rows, double d, const double (&o)[4], float r) {
            const float D = static_cast<float>(d), S = static_cast<float>(o[0]), N = static_cast<float>(o[1]);
            const float W = static_cast<float>(o[2]), E = static_cast<float>(o[3]);
            if (chained) {
              chainStoreRow(rows, z, i, j, D, S, N, W, E, r);
            } else {
              a.D[c] = D; a.S[c] = S; a.N[c] = N; a.W[c] = W; a.E[c] = E; a.r[c] = r;
            }
            a.x[c] = 0.0f;
          };
          put(I.tk, I.tkC, dK, oK, rk);
          put(I.tw, I.twC, dW, oW, rw);
        });
      });
      note(kMonTurbFirst, a4[0] / smax(a4[1] * smax(I.kIn, kTinySst), kTinySst));
      note(kMonTurbSecond, a4[2] / smax(a4[3] * smax(I.wIn, kTinySst), kTinySst));
      if (stopStage == kStageSstAssembly) { done = it + 1; break; }

      // k and omega sweep in the reference's cell order: their floors and
      // the wall-cell omega override act after the sweeps, so the converged
      // state depends on the order (a colouring would move it by ~1e-3).
      if (chained) {
        chainedSweeps(I, t, tag, (flags & kFlagChainWaitTest) != 0);
      } else if (rowwise) {
        sequentialSweeps(I, t);
      } else {
        gsWavefrontSweeps(I, t, 3, I.kD, I.kS, I.kN, I.kW, I.kE, I.kB, I.k, I.wD, I.wS, I.wN,
                          I.wW, I.wE, I.wB, I.om);
      }
      wideBarrier(t);
      if (stopStage == kStageSstSolve) { done = it + 1; break; }

      double m8[8];
#pragma unroll
      for (int s = 0; s < 8; ++s) m8[s] = -INFINITY;
      m8[5] = 0.0;
      m8[7] = 0.0;
      wideCells(t, [&](int c, int i, int j) { sstFinishCell<true>(I, c, i, j, m8); });
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
      const double a = continuity, b = momentumX, cc = momentumY;
      if (!isfinite(a) || !isfinite(b) || !isfinite(cc)) break;
      if (smax(smax(fabs(a), fabs(b)), fabs(cc)) < stopTol) break;
    }
  }
  if (leader) *I.iterations = done;
}

/// The launch, as plainKernel's (plain_kernel.cu): CTA b runs solves
/// plan[b].begin .. plan[b].end of `list` one after another; without a plan the
/// whole grid is the team of instance 0.
__global__ void __launch_bounds__(kWideThreads, 1)
simpleKernel(const Instance* __restrict__ instances, const WideCta* __restrict__ plan, const int* __restrict__ list,
             int iterations, int stopStage, double tolerance, int smemBytes, int flags) {
  __shared__ WideShared sh;
  const WideCta me = (plan != nullptr) ? plan[blockIdx.x]
                                       : WideCta{0, 1, static_cast<int>(blockIdx.x), static_cast<int>(gridDim.x)};
  if (threadIdx.x == 0) sh.ahead = 0.0;
  for (int k = me.begin; k < me.end; ++k) {
    const Instance& I = instances[(list != nullptr) ? list[k] : k];
    const int R = min(me.R, I.wideMost);
    const double outer = outerBound(I.NI, I.NJ, R, static_cast<int>(blockDim.x),
                                    wideEffort(true, I.nCorr, I.cgMax, I.mgCap, I.sweeps));
    if (me.rank >= R) {
      // the rest of the team is at work on it: a wait of the next one is behind that
      if (threadIdx.x == 0) sh.ahead += outer;
      continue;
    }
    WideTeam t;
    wideJoin(t, I.wide, I.iterations + 1, &sh, me.rank, R, I.NI, I.NJ, iterations, outer);
    mixedSolve(I, t, iterations, stopStage, tolerance, smemBytes, flags);
    wideLeave(t);
    __syncthreads();
  }
}

}  // namespace

/// Brute-force distance from each cell centroid to the nearest no-slip wall
/// face centre (TurbulenceModel.cpp:28-65). One thread per cell.
__global__ void wallDistanceKernel(int n, const double* __restrict__ centroid,
                                   int walls, const double* __restrict__ wallCentre,
                                   double far, double* __restrict__ out) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n) return;
  if (walls == 0) {
    out[c] = far;
    return;
  }
  const double cx = centroid[2 * c], cy = centroid[2 * c + 1];
  double best = 1.7976931348623157e308;
  for (int w = 0; w < walls; ++w) {
    const double dx = cx - wallCentre[2 * w];
    const double dy = cy - wallCentre[2 * w + 1];
    const double sq = dx * dx + dy * dy;
    best = smin(best, sq);
  }
  out[c] = sqrt(best);
}

}  // namespace cfdb

// ---- launch helpers ---------------------------------------------------------------

namespace cfdb {

int chooseClusterSize(int cells) {
  // About four cells per thread at 512 threads per CTA before another CTA is
  // added; 16 is the largest (non-portable) cluster.
  int r = 1;
  while (r < 16 && cells > r * 512 * 4) r *= 2;
  return r;
}

int kernelFlags() {
  // Implementation choices for comparisons and tests. Bits 2 and 5 run the
  // three k/omega sweeps one after another (the same bits). Plain form: bit 7
  // the pressure CG in its form for any shape (all in memory; the same bits),
  // bit 3 the reference's two-reduction CG (the same to rounding). Mixed form:
  // bit 1 the plain wavefront sweeps, bit 9 the V-cycle with a phase per half
  // sweep (the same bits). Bit 6 is for tests: a k/omega sweep also waits for a
  // count that nothing sets, so that wait gives up and the launch reports its
  // fault word; bit 8 does the same before the plain form's pressure CG. Other
  // bits are accepted and have no effect.
  const char* env = std::getenv("CFD_KERNEL_FLAGS");
  return (env != nullptr) ? std::atoi(env) : 0;
}

/// Dynamic shared memory at most: what 227 KB leave beside the static tables
/// and the multigrid's descriptor.
constexpr int kMaxMixedSmem = 220928;

int mixedSmemBytes(int NI, int threads, int multigridBytes) {
  // the coarse levels, the sweeps' copies (a row's two vectors at least)
  long long bytes = std::max<long long>(multigridBytes, (2LL * NI + 64) * 4);
  const long long chain = chainBytes(NI, threads);
  if (chainable(NI, threads) && chain <= kMaxMixedSmem) bytes = std::max(bytes, chain);
  return static_cast<int>(std::min<long long>(bytes, kMaxMixedSmem));
}

Status prepareSimpleKernel() {
  static PerDeviceOnce once;
  return once.run([]() -> Status {
    const cudaError_t e = cudaFuncSetAttribute(simpleKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxMixedSmem);
    return (e == cudaSuccess) ? ok() : fail(CFD_INITIALIZATION_FAILURE, cudaGetErrorString(e));
  });
}

Status launchSimple(const Instance* dInstances, const WidePlan& plan, const WideCta* dPlan, const int* dList,
                    int threads, int iterations, int stopStage, double tolerance, cudaStream_t stream) {
  if (Status st = prepareSimpleKernel(); st != CFD_OK) return st;
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
  const cudaError_t e = cudaLaunchKernelEx(&config, simpleKernel, dInstances, dPlan, dList, iterations, stopStage,
                                           tolerance, plan.smemBytes, kernelFlags());
  if (e != cudaSuccess) {
    return fail(CFD_INITIALIZATION_FAILURE, std::string("SIMPLE kernel launch: ") + cudaGetErrorString(e));
  }
  return CFD_OK;
}

Status launchWallDistance(int n, const double* centroid, int walls, const double* wallCentre,
                          double far, double* out, cudaStream_t stream) {
  const int block = 256;
  wallDistanceKernel<<<(n + block - 1) / block, block, 0, stream>>>(n, centroid, walls, wallCentre, far, out);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(CFD_INITIALIZATION_FAILURE, cudaGetErrorString(e));
  return CFD_OK;
}

}  // namespace cfdb
