// phases.cuh - the stages of a SIMPLE iteration (laminar and k-omega SST) for
// one cell, shared by the plain and the mixed form's kernels. Each is the
// reference's expression for expression, with its accumulation order; see
// simple_kernel.cu on the arithmetic.
#pragma once

#include <cmath>
#include <cstdint>

#include "cfd_gpu.h"
#include "instance.hpp"
#include "team.cuh"

namespace cfdb {
namespace {

constexpr double kTinySolver = 1e-300;  // SimpleSolver.cpp:16
constexpr double kTinySst = 1.0e-30;    // KOmegaSST.cpp:22
constexpr double kMinOmega = 1.0e-10;   // KOmegaSST.cpp:20
// SSTConstants (KOmegaSST.hpp:147-171)
constexpr double kSigmaK1 = 0.85, kSigmaW1 = 0.5, kBeta1 = 0.075;
constexpr double kSigmaK2 = 1.0, kSigmaW2 = 0.856, kBeta2 = 0.0828;
constexpr double kBetaStar = 0.09, kKappa = 0.41, kA1 = 0.31, kProdLimit = 10.0;

// BoundaryKind values the kernel tests for (cfd_gpu.h CFD_BC_*; outlet and
// internal faces need no test of their own).
constexpr int kInlet = CFD_BC_INLET, kFarField = CFD_BC_FARFIELD, kWall = CFD_BC_NOSLIP_WALL;

// ---- faces of a cell ----------------------------------------------------------

struct Face {
  int fam;     // 0 N-face, 1 E-face
  int idx;     // index within its family
  int owner;   // owning cell
  int nb;      // neighbour cell of an interior face, else -1
  int other;   // nb, or the cell across the wake cut, else -1
  bool mine;   // the cell being processed owns this face
};

DEV Face faceS(const Instance& I, int c, int i, int j) {
  Face f;
  f.fam = 0;
  f.idx = j * I.NI + i;
  if (j > 0) {
    f.owner = c - I.NI; f.nb = c; f.other = c; f.mine = false;
  } else {
    f.owner = c; f.nb = -1; f.other = I.acrossJ0[i]; f.mine = true;
  }
  return f;
}
DEV Face faceN(const Instance& I, int c, int i, int j) {
  Face f;
  f.fam = 0;
  f.idx = (j + 1) * I.NI + i;
  f.owner = c;
  f.mine = true;
  f.nb = (j < I.NJ - 1) ? c + I.NI : -1;
  f.other = f.nb;
  return f;
}
DEV Face faceW(const Instance& I, int c, int i, int j) {
  Face f;
  f.fam = 1;
  f.idx = j * (I.NI + 1) + i;
  if (i > 0) {
    f.owner = c - 1; f.nb = c; f.mine = false;
  } else {
    f.owner = c; f.nb = -1; f.mine = true;
  }
  f.other = f.nb;
  return f;
}
DEV Face faceE(const Instance& I, int c, int i, int j) {
  Face f;
  f.fam = 1;
  f.idx = j * (I.NI + 1) + i + 1;
  f.owner = c;
  f.mine = true;
  f.nb = (i < I.NI - 1) ? c + 1 : -1;
  f.other = f.nb;
  return f;
}

DEV const FaceGeo& geo(const Instance& I, const Face& f) { return f.fam ? I.gE : I.gN; }
DEV double massFlux(const Instance& I, const Face& f) { return f.fam ? I.mfE[f.idx] : I.mfN[f.idx]; }
DEV double* massFluxPtr(const Instance& I, const Face& f) { return f.fam ? I.mfE + f.idx : I.mfN + f.idx; }
DEV int kindOf(const Instance& I, const Face& f) { return f.fam ? I.kindE[f.idx] : I.kindN[f.idx]; }
DEV double bcU(const Instance& I, const Face& f) { return f.fam ? I.bcuE[f.idx] : I.bcuN[f.idx]; }
DEV double bcV(const Instance& I, const Face& f) { return f.fam ? I.bcvE[f.idx] : I.bcvN[f.idx]; }
DEV double bcP(const Instance& I, const Face& f) { return f.fam ? I.bcpE[f.idx] : I.bcpN[f.idx]; }

/// SimpleSolver::imposesVelocity (SimpleSolver.cpp:247-262) for a boundary face.
DEV bool imposesVelocity(const Instance& I, const Face& f) {
  const int kind = kindOf(I, f);
  if (kind == kWall || kind == kInlet) return true;
  if (kind == kFarField) {
    const double dead = f.fam ? I.deadE[f.idx] : I.deadN[f.idx];
    return massFlux(I, f) < dead;
  }
  return false;
}

/// Accumulate a face's Green-Gauss contribution S*phi into the cell's sum:
/// added for the owner, subtracted for the neighbour (Gradient.cpp:29-40).
DEV void ggAdd(const Face& f, double Sx, double Sy, double phi, double& gx, double& gy) {
  const double cx = Sx * phi, cy = Sy * phi;
  if (f.mine) {
    gx += cx; gy += cy;
  } else {
    gx -= cx; gy -= cy;
  }
}

DEV void ggFinish(double vol, double& gx, double& gy) {
  if (vol > 0.0) {
    const double s = 1.0 / vol;
    gx *= s;
    gy *= s;
  }
}

/// Cell on the other side of face k (0 S, 1 N, 2 W, 3 E) of cell (i, j), or -1.
DEV int across(const Instance& I, int c, int i, int j, int k) {
  switch (k) {
    case 0: return (j > 0) ? c - I.NI : I.acrossJ0[i];
    case 1: return (j < I.NJ - 1) ? c + I.NI : -1;
    case 2: return (i > 0) ? c - 1 : -1;
    default: return (i < I.NI - 1) ? c + 1 : -1;
  }
}

// ---- phase: face values + Green-Gauss gradients of u, v, p ---------------------

/// interpolateFaceValues (SimpleSolver.cpp:268-304) for one face.
DEV void faceUVP(const Instance& I, const Face& f, double& fu, double& fv, double& fp) {
  const int o = f.owner;
  if (f.other >= 0) {
    const double w = geo(I, f).w[f.idx];
    const int n = f.other;
    fu = w * I.u[o] + (1.0 - w) * I.u[n];
    fv = w * I.v[o] + (1.0 - w) * I.v[n];
    fp = w * I.p[o] + (1.0 - w) * I.p[n];
    return;
  }
  if (imposesVelocity(I, f)) {
    fu = bcU(I, f);
    fv = bcV(I, f);
    fp = I.p[o];
  } else {
    fu = I.u[o];
    fv = I.v[o];
    fp = bcP(I, f);
  }
}

DEV void gradientsCell(const Instance& I, int c, int i, int j, double& speedMax) {
  double ux = 0.0, uy = 0.0, vx = 0.0, vy = 0.0, px = 0.0, py = 0.0;
  const Face fs[4] = {faceS(I, c, i, j), faceN(I, c, i, j), faceW(I, c, i, j), faceE(I, c, i, j)};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const Face& f = fs[k];
    double fu, fv, fp;
    faceUVP(I, f, fu, fv, fp);
    const FaceGeo& g = geo(I, f);
    const double Sx = g.Sx[f.idx], Sy = g.Sy[f.idx];
    ggAdd(f, Sx, Sy, fu, ux, uy);
    ggAdd(f, Sx, Sy, fv, vx, vy);
    ggAdd(f, Sx, Sy, fp, px, py);
  }
  const double vol = I.vol[c];
  ggFinish(vol, ux, uy);
  ggFinish(vol, vx, vy);
  ggFinish(vol, px, py);
  I.gux[c] = ux; I.guy[c] = uy;
  I.gvx[c] = vx; I.gvy[c] = vy;
  I.gpx[c] = px; I.gpy[c] = py;
  speedMax = smax(speedMax, hypot(I.u[c], I.v[c]));
}

// ---- phase: momentum assembly (u and v share the matrix), relaxation, residual --

template <bool kMixed>
DEV void momentumCell(const Instance& I, int c, int i, int j, double& resU, double& resV, double& diagL1) {
  double diag = 0.0, sU = 0.0, sV = 0.0;
  double off[4] = {0.0, 0.0, 0.0, 0.0};  // coefficient on the S, N, W, E cell
  const Face fs[4] = {faceS(I, c, i, j), faceN(I, c, i, j), faceW(I, c, i, j), faceE(I, c, i, j)};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const Face& f = fs[k];
    const FaceGeo& g = geo(I, f);
    const int o = f.owner;
    const double flux = massFlux(I, f);
    if (f.other >= 0) {
      const int n = f.other;
      const double w = g.w[f.idx];
      const double vis = w * I.mu[o] + (1.0 - w) * I.mu[n];
      const double dif = vis * g.D[f.idx];
      const double outward = smax(flux, 0.0);
      const double inward = smax(-flux, 0.0);
      const double Tx = g.Tx[f.idx], Ty = g.Ty[f.idx];
      const double fgux = I.gux[o] * w + I.gux[n] * (1.0 - w);
      const double fguy = I.guy[o] * w + I.guy[n] * (1.0 - w);
      const double fgvx = I.gvx[o] * w + I.gvx[n] * (1.0 - w);
      const double fgvy = I.gvy[o] * w + I.gvy[n] * (1.0 - w);
      const double cu = I.blend * vis * (fgux * Tx + fguy * Ty);
      const double cv = I.blend * vis * (fgvx * Tx + fgvy * Ty);
      if (f.nb >= 0) {
        double du = 0.0, dv = 0.0;
        if (I.sou) {
          const double uo = I.u[o], un = I.u[n], vo = I.v[o], vn = I.v[n];
          du = flux * ((w * uo + (1.0 - w) * un) - ((flux >= 0.0) ? uo : un));
          dv = flux * ((w * vo + (1.0 - w) * vn) - ((flux >= 0.0) ? vo : vn));
        }
        if (f.mine) {
          diag += outward + dif;
          off[k] = 0.0 + (-inward - dif);
          sU += cu; sV += cv;
          if (I.sou) { sU -= du; sV -= dv; }
        } else {
          diag += inward + dif;
          off[k] = 0.0 + (-outward - dif);
          sU -= cu; sV -= cv;
          if (I.sou) { sU += du; sV += dv; }
        }
      } else {
        // Wake cut: the owner's row only (SimpleSolver.cpp:379-398).
        diag += outward + dif;
        off[k] = 0.0 + (-inward - dif);
        sU += cu; sV += cv;
      }
      continue;
    }
    // Boundary face (SimpleSolver.cpp:400-416).
    const double vis = I.mu[o];
    const double dif = vis * g.D[f.idx];
    if (imposesVelocity(I, f)) {
      const double iu = bcU(I, f), iv = bcV(I, f);
      const double Tx = g.Tx[f.idx], Ty = g.Ty[f.idx];
      sU -= flux * iu; sV -= flux * iv;
      diag += dif;
      sU += dif * iu; sV += dif * iv;
      sU += I.blend * vis * (I.gux[o] * Tx + I.guy[o] * Ty);
      sV += I.blend * vis * (I.gvx[o] * Tx + I.gvy[o] * Ty);
    } else {
      diag += flux;
    }
  }
  const double vol = I.vol[c];
  sU -= I.gpx[c] * vol;
  sV -= I.gpy[c] * vol;
  // applyRelaxation (SimpleSolver.cpp:425-443).
  const double uc = I.u[c], vc = I.v[c];
  if (!(fabs(diag) > 0.0)) {
    diag = 1.0;
  } else {
    const double relaxed = diag / I.alphaU;
    sU += (relaxed - diag) * uc;
    sV += (relaxed - diag) * vc;
    diag = relaxed;
  }
  I.aD[c] = diag; I.aS[c] = off[0]; I.aN[c] = off[1]; I.aW[c] = off[2]; I.aE[c] = off[3];
  I.bU[c] = sU; I.bV[c] = sV;
  // residualL1 (LinearSystem.cpp:45-54): y = A x in multiply's face order.
  double yu = diag * uc, yv = diag * vc;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int n = across(I, c, i, j, k);
    if (n >= 0) {
      yu += off[k] * I.u[n];
      yv += off[k] * I.v[n];
    }
  }
  resU += fabs(sU - yu);
  resV += fabs(sV - yv);
  diagL1 += fabs(diag);
  if constexpr (kMixed) {
    // FP32 rows and residuals for the correction-form sweeps.
    const Rows32& m = I.mom;
    m.D[c] = static_cast<float>(diag);
    m.S[c] = static_cast<float>(off[0]);
    m.N[c] = static_cast<float>(off[1]);
    m.W[c] = static_cast<float>(off[2]);
    m.E[c] = static_cast<float>(off[3]);
    m.r[c] = static_cast<float>(sU - yu);
    I.momRv[c] = static_cast<float>(sV - yv);
    m.x[c] = 0.0f;
    I.momXv[c] = 0.0f;
  }
}

// ---- phase: Rhie-Chow face fluxes (SimpleSolver.cpp:445-496) -------------------

DEV void rhieChowFace(const Instance& I, const Face& f) {
  const FaceGeo& g = geo(I, f);
  const int o = f.owner;
  const double Sx = g.Sx[f.idx], Sy = g.Sy[f.idx], D = g.D[f.idx];
  double* mf = massFluxPtr(I, f);
  if (f.other >= 0) {
    const int n = f.other;
    const double w = g.w[f.idx];
    const double ix = I.u[o] * w + I.u[n] * (1.0 - w);
    const double iy = I.v[o] * w + I.v[n] * (1.0 - w);
    const double dens = w * I.rho[o] + (1.0 - w) * I.rho[n];
    const double mob = w * (I.vol[o] / I.aD[o]) + (1.0 - w) * (I.vol[n] / I.aD[n]);
    const double sgx = I.gpx[o] * w + I.gpx[n] * (1.0 - w);
    const double sgy = I.gpy[o] * w + I.gpy[n] * (1.0 - w);
    const double compact = (I.p[n] - I.p[o]) * D;
    const double smooth = sgx * Sx + sgy * Sy;
    *mf = dens * (ix * Sx + iy * Sy) - dens * mob * (compact - smooth);
    return;
  }
  const double dens = I.rho[o];
  if (imposesVelocity(I, f)) {
    *mf = dens * (bcU(I, f) * Sx + bcV(I, f) * Sy);
  } else {
    const double mob = I.vol[o] / I.aD[o];
    const double compact = (bcP(I, f) - I.p[o]) * D;
    const double smooth = I.gpx[o] * Sx + I.gpy[o] * Sy;
    *mf = dens * (I.u[o] * Sx + I.v[o] * Sy) - dens * mob * (compact - smooth);
  }
}

DEV void rhieChowCell(const Instance& I, int c, int i, int j) {
  if (j == 0) rhieChowFace(I, faceS(I, c, i, j));
  rhieChowFace(I, faceN(I, c, i, j));
  if (i == 0) rhieChowFace(I, faceW(I, c, i, j));
  rhieChowFace(I, faceE(I, c, i, j));
}

// ---- phase: pressure-correction assembly (SimpleSolver.cpp:498-580) ------------

/// rho_f * mobility_f * D for a face with a cell on each side (the same
/// coefficient the flux correction uses).
DEV double pressureCoefficient(const Instance& I, const Face& f, int n) {
  const FaceGeo& g = geo(I, f);
  const int o = f.owner;
  const double w = g.w[f.idx];
  const double dens = w * I.rho[o] + (1.0 - w) * I.rho[n];
  const double mob = w * (I.vol[o] / I.aD[o]) + (1.0 - w) * (I.vol[n] / I.aD[n]);
  return dens * mob * g.D[f.idx];
}

DEV void pressureAssemblyCell(const Instance& I, int c, int i, int j, double& netL1, double& bSum) {
  double net = 0.0, diag = 0.0;
  const Face fs[4] = {faceS(I, c, i, j), faceN(I, c, i, j), faceW(I, c, i, j), faceE(I, c, i, j)};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const Face& f = fs[k];
    const double flux = massFlux(I, f);
    if (f.mine) net += flux; else net -= flux;
    if (f.other >= 0) {
      const double coef = pressureCoefficient(I, f, f.other);
      diag += coef;
      if (f.mine) {
        double* slot = f.fam ? I.pE + f.idx : I.pN + f.idx;
        *slot = 0.0 + (-coef);
      }
      continue;
    }
    if (imposesVelocity(I, f)) continue;
    const double mob = I.vol[c] / I.aD[c];
    diag += I.rho[c] * mob * geo(I, f).D[f.idx];
  }
  I.net[c] = net;
  I.pD[c] = diag;
  I.pB[c] = -net;
  netL1 += fabs(net);
  bSum += -net;
}

/// y = A x for the pressure-correction matrix, in multiply's face order.
DEV double pressureRow(const Instance& I, int c, int i, int j, const double* xv, double xc) {
  double y = I.pD[c] * xc;
  if (j > 0) y += I.pN[j * I.NI + i] * xv[c - I.NI];
  else if (I.acrossJ0[i] >= 0) y += I.pN[i] * xv[I.acrossJ0[i]];
  if (j < I.NJ - 1) y += I.pN[(j + 1) * I.NI + i] * xv[c + I.NI];
  if (i > 0) y += I.pE[j * (I.NI + 1) + i] * xv[c - 1];
  if (i < I.NI - 1) y += I.pE[j * (I.NI + 1) + i + 1] * xv[c + 1];
  return y;
}

// ---- phase: correction (SimpleSolver.cpp:582-660) ------------------------------

DEV void correctFace(const Instance& I, const Face& f) {
  const FaceGeo& g = geo(I, f);
  const int o = f.owner;
  double* mf = massFluxPtr(I, f);
  if (f.other >= 0) {
    const int n = f.other;
    const double w = g.w[f.idx];
    const double dens = w * I.rho[o] + (1.0 - w) * I.rho[n];
    const double mob = w * (I.vol[o] / I.aD[o]) + (1.0 - w) * (I.vol[n] / I.aD[n]);
    *mf -= dens * mob * g.D[f.idx] * (I.x[n] - I.x[o]);
    return;
  }
  if (imposesVelocity(I, f)) return;
  const double mob = I.vol[o] / I.aD[o];
  *mf -= I.rho[o] * mob * g.D[f.idx] * (0.0 - I.x[o]);
}

DEV void correctCell(const Instance& I, int c, int i, int j) {
  double gx = 0.0, gy = 0.0;
  const Face fs[4] = {faceS(I, c, i, j), faceN(I, c, i, j), faceW(I, c, i, j), faceE(I, c, i, j)};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const Face& f = fs[k];
    const FaceGeo& g = geo(I, f);
    double fc;
    if (f.other >= 0) {
      const double w = g.w[f.idx];
      fc = w * I.x[f.owner] + (1.0 - w) * I.x[f.other];
    } else if (imposesVelocity(I, f)) {
      fc = I.x[f.owner];
    } else {
      fc = 0.0;
    }
    ggAdd(f, g.Sx[f.idx], g.Sy[f.idx], fc, gx, gy);
  }
  ggFinish(I.vol[c], gx, gy);
  I.p[c] += I.alphaP * I.x[c];
  const double mob = I.vol[c] / I.aD[c];
  I.u[c] -= gx * mob;
  I.v[c] -= gy * mob;
  if (j == 0) correctFace(I, fs[0]);
  correctFace(I, fs[1]);
  if (i == 0) correctFace(I, fs[2]);
  correctFace(I, fs[3]);
}

// ---- divergence (SimpleSolver.cpp:796-817) -------------------------------------

DEV double cellDivergence(const Instance& I, int c, int i, int j) {
  double net = 0.0;
  const Face fs[4] = {faceS(I, c, i, j), faceN(I, c, i, j), faceW(I, c, i, j), faceE(I, c, i, j)};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const Face& f = fs[k];
    const double dens = smax(I.rho[f.owner], kTinySolver);
    const double vf = massFlux(I, f) / dens;
    if (f.mine) net += vf; else net -= vf;
  }
  const double area = I.vol[c];
  return (area > 0.0) ? net / area : 0.0;
}

// ---- k-omega SST (KOmegaSST.cpp) -----------------------------------------------

/// Face value of k or omega (KOmegaSST.cpp:26-68, with the no-slip override
/// of :236-241 for omega). isOmega selects the wall treatment.
DEV double sstFaceValue(const Instance& I, const Face& f, const double* phi, bool isOmega) {
  const int o = f.owner;
  if (f.nb >= 0) {
    const double w = geo(I, f).w[f.idx];
    return w * phi[o] + (1.0 - w) * phi[f.nb];
  }
  if (f.other >= 0) {
    const double w = 1.0;  // ownerWeight() of a face without a neighbour
    return w * phi[o] + (1.0 - w) * phi[f.other];
  }
  const double inflow = isOmega ? I.wIn : I.kIn;
  switch (kindOf(I, f)) {
    case kWall: return isOmega ? phi[o] : 0.0;
    case kInlet: return inflow;
    case kFarField: return (massFlux(I, f) < 0.0) ? inflow : phi[o];
    default: return phi[o];
  }
}

DEV void sstBlendingCell(const Instance& I, int c, int i, int j, double& divMax) {
  divMax = smax(divMax, fabs(cellDivergence(I, c, i, j)));
  // computeStrain (:202-216), gradients from the start of the iteration.
  const double s11 = I.gux[c], s22 = I.gvy[c];
  const double s12 = 0.5 * (I.guy[c] + I.gvx[c]);
  const double S = sqrt(2.0 * (s11 * s11 + s22 * s22 + 2.0 * s12 * s12));
  I.strain[c] = S;
  // Green-Gauss gradients of k and omega (:224-244).
  double kx = 0.0, ky = 0.0, wx = 0.0, wy = 0.0;
  const Face fs[4] = {faceS(I, c, i, j), faceN(I, c, i, j), faceW(I, c, i, j), faceE(I, c, i, j)};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const Face& f = fs[k];
    const FaceGeo& g = geo(I, f);
    const double Sx = g.Sx[f.idx], Sy = g.Sy[f.idx];
    ggAdd(f, Sx, Sy, sstFaceValue(I, f, I.k, false), kx, ky);
    ggAdd(f, Sx, Sy, sstFaceValue(I, f, I.om, true), wx, wy);
  }
  const double vol = I.vol[c];
  ggFinish(vol, kx, ky);
  ggFinish(vol, wx, wy);
  I.gkx[c] = kx; I.gky[c] = ky; I.gwx[c] = wx; I.gwy[c] = wy;
  // Cross-diffusion and the blending functions (:247-286).
  const double d = smax(I.wallDist[c], kTinySst);
  const double rho = I.rho[c];
  const double nu = I.muMol[c] / smax(rho, kTinySst);
  const double omega = smax(I.om[c], kMinOmega);
  const double energy = smax(I.k[c], 0.0);
  const double cdv = 2.0 * rho * kSigmaW2 * (kx * wx + ky * wy) / omega;
  const double cdp = smax(cdv, 1.0e-10);
  const double term1 = sqrt(smax(energy, 0.0)) / (kBetaStar * omega * d);
  const double term2 = 500.0 * nu / (d * d * omega);
  const double term3 = 4.0 * rho * kSigmaW2 * energy / (cdp * d * d);
  const double arg1 = smin(smax(term1, term2), term3);
  const double F1 = tanh(sclamp(arg1 * arg1 * arg1 * arg1, 0.0, 50.0));
  const double arg2 = smax(2.0 * term1, term2);
  const double F2 = tanh(sclamp(arg2 * arg2, 0.0, 50.0));
  I.cd[c] = cdv;
  I.f1[c] = F1;
  I.f2[c] = F2;
  // Limited production (:362-368).
  const double raw = I.mut[c] * S * S;
  const double ceiling = kProdLimit * kBetaStar * rho * smax(I.k[c], 0.0) * smax(I.om[c], kMinOmega);
  I.prod[c] = smin(raw, ceiling);
}

DEV double blendF1(double f1, double nearValue, double farValue) { return f1 * nearValue + (1.0 - f1) * farValue; }

/// Assemble, relax and measure one row of the k and of the omega equation
/// (KOmegaSST.cpp:378-466); both equations in one pass over the faces.
/// The rows go to store(dK, oK, bK, dW, oW, bW, yk, yw).
template <typename Store>
DEV void sstAssemblyCell(const Instance& I, int c, int i, int j, double (&acc)[4], Store&& store) {
  const double relax = sclamp(I.alphaT, 0.05, 1.0);
  double dK = 0.0, bK = 0.0, dW = 0.0, bW = 0.0;
  double oK[4] = {0.0, 0.0, 0.0, 0.0}, oW[4] = {0.0, 0.0, 0.0, 0.0};
  const Face fs[4] = {faceS(I, c, i, j), faceN(I, c, i, j), faceW(I, c, i, j), faceE(I, c, i, j)};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const Face& f = fs[k];
    const FaceGeo& g = geo(I, f);
    const int o = f.owner;
    const double flux = massFlux(I, f);
    const double Dt = g.Dt[f.idx];
    if (f.other >= 0) {
      const int n = f.other;
      const double w = (f.nb >= 0) ? g.w[f.idx] : 1.0;
      const double f1o = I.f1[o], f1n = I.f1[n];
      const double sko = blendF1(f1o, kSigmaK1, kSigmaK2), skn = blendF1(f1n, kSigmaK1, kSigmaK2);
      const double swo = blendF1(f1o, kSigmaW1, kSigmaW2), swn = blendF1(f1n, kSigmaW1, kSigmaW2);
      const double muo = I.muMol[o], mun = I.muMol[n], mto = I.mut[o], mtn = I.mut[n];
      const double difK = (w * (muo + sko * mto) + (1.0 - w) * (mun + skn * mtn)) * Dt;
      const double difW = (w * (muo + swo * mto) + (1.0 - w) * (mun + swn * mtn)) * Dt;
      const double outward = smax(flux, 0.0);
      const double inward = smax(-flux, 0.0);
      if (f.mine) {
        dK += outward + difK;
        dW += outward + difW;
        oK[k] = 0.0 + (-inward - difK);
        oW[k] = 0.0 + (-inward - difW);
      } else {
        dK += inward + difK;
        dW += inward + difW;
        oK[k] = 0.0 + (-outward - difK);
        oW[k] = 0.0 + (-outward - difW);
      }
      continue;
    }
    const double f1o = I.f1[o];
    const double difK = (I.muMol[o] + blendF1(f1o, kSigmaK1, kSigmaK2) * I.mut[o]) * Dt;
    const double difW = (I.muMol[o] + blendF1(f1o, kSigmaW1, kSigmaW2) * I.mut[o]) * Dt;
    const int kind = kindOf(I, f);
    const bool imposed = kind == kWall || kind == kInlet || (kind == kFarField && flux < 0.0);
    if (imposed) {
      const double valK = (kind == kWall) ? 0.0 : I.kIn;
      const double valW = I.wIn;  // the omega equation's wall value is its inflow value
      dK += difK + smax(flux, 0.0);
      bK += (difK - smin(flux, 0.0)) * valK;
      dW += difW + smax(flux, 0.0);
      bW += (difW - smin(flux, 0.0)) * valW;
    } else {
      dK += smax(flux, 0.0);
      dW += smax(flux, 0.0);
    }
  }
  // Sources (:446-453): explicit production, implicit destruction.
  const double vol = I.vol[c];
  const double rho = I.rho[c];
  const double F1 = I.f1[c];
  const double omPos = smax(I.om[c], kMinOmega);
  const double S = I.strain[c];
  bK += I.prod[c] * vol;
  dK += kBetaStar * rho * omPos * vol;
  const double gamma = blendF1(F1, I.gamma1, I.gamma2);
  const double beta = blendF1(F1, kBeta1, kBeta2);
  double wProd = gamma * rho * S * S;
  wProd += (1.0 - F1) * I.cd[c];
  bW += wProd * vol;
  dW += beta * rho * omPos * vol;
  // Implicit under-relaxation (:455-463).
  const double kc = I.k[c], wc = I.om[c];
  if (fabs(dK) > kTinySst) {
    const double relaxed = dK / relax;
    bK += (relaxed - dK) * kc;
    dK = relaxed;
  }
  if (fabs(dW) > kTinySst) {
    const double relaxed = dW / relax;
    bW += (relaxed - dW) * wc;
    dW = relaxed;
  }
  double yk = dK * kc, yw = dW * wc;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int n = across(I, c, i, j, k);
    if (n >= 0) {
      yk += oK[k] * I.k[n];
      yw += oW[k] * I.om[n];
    }
  }
  acc[0] += fabs(bK - yk);
  acc[1] += fabs(dK);
  acc[2] += fabs(bW - yw);
  acc[3] += fabs(dW);
  store(dK, oK, bK, dW, oW, bW, yk, yw);
}

/// wallOmega (KOmegaSST.cpp:86-92).
DEV double wallOmega(const Instance& I, double nu, double distance, double energy) {
  const double d = smax(distance, kTinySst);
  const double viscous = 6.0 * nu / (kBeta1 * d * d);
  const double logarithmic = sqrt(smax(energy, 0.0)) / (I.betaStarQuarter * kKappa * d);
  return sqrt(viscous * viscous + logarithmic * logarithmic);
}

/// Floors, wall conditions, eddy viscosity, ranges (KOmegaSST.cpp:289-345,
/// :469-471, :513-529; SimpleSolver.cpp:232-245, :782-790).
template <bool kMixed>
DEV void sstFinishCell(const Instance& I, int c, int i, int j, double (&mx)[8]) {
  double kRaw = I.k[c], wRaw = I.om[c];
  if constexpr (kMixed) {
    kRaw += static_cast<double>(I.tk.x[c]);
    wRaw += static_cast<double>(I.tw.x[c]);
  }
  double kc = smax(kRaw, 0.0);
  double wc = smax(wRaw, kMinOmega);
  const uint8_t mask = I.wallMask[c];
  if (mask != 0) {
    const double d = smax(I.wallDist[c], kTinySst);
    const double rho = smax(I.rho[c], kTinySst);
    const double mu = I.muMol[c];
    const double nu = mu / rho;
    wc = wallOmega(I, nu, d, kc);
    const double uc = I.u[c], vc = I.v[c];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (!(mask & (1u << k))) continue;
      const Face f = (k == 0) ? faceS(I, c, i, j) : (k == 1) ? faceN(I, c, i, j)
                               : (k == 2) ? faceW(I, c, i, j) : faceE(I, c, i, j);
      const FaceGeo& g = geo(I, f);
      const double nX = g.nx[f.idx] * -1.0, nY = g.ny[f.idx] * -1.0;
      const double dn = uc * nX + vc * nY;
      const double px = uc - nX * dn, py = vc - nY * dn;
      const double tangential = hypot(px, py);
      const double shear = mu * tangential / d;
      const double fv = sqrt(shear / rho);
      mx[5] = smax(mx[5], fv * d / smax(nu, kTinySst));
    }
  }
  I.k[c] = kc;
  I.om[c] = wc;
  const double denom = smax(kA1 * smax(wc, kMinOmega), I.strain[c] * I.f2[c]);
  const double mut = I.rho[c] * kA1 * smax(kc, 0.0) / smax(denom, kTinySst);
  I.mut[c] = mut;
  I.mu[c] = I.muMol[c] + mut;
  // ranges: max of (k, omega, mut) and of their negatives (for the minima)
  mx[0] = smax(mx[0], kc); mx[1] = smax(mx[1], -kc);
  mx[2] = smax(mx[2], wc); mx[3] = smax(mx[3], -wc);
  mx[4] = smax(mx[4], mut); mx[6] = smax(mx[6], -mut);
  const double muMol = I.muMol[c];
  if (muMol > 0.0) mx[7] = smax(mx[7], mut / muMol);
}

DEV double precondition(double rc, double dg) { return (fabs(dg) > 0.0) ? rc / dg : rc; }


}  // namespace
}  // namespace cfdb
