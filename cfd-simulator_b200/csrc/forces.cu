// forces.cu - wall surface data and force integration on the device, FP64:
// post::extractSurface and post::integrateForces (src/post/SurfaceData.cpp:101-348,
// src/post/Forces.cpp:23-130) on the solver's current field.
//
// Everything that depends only on the mesh (the wall stations in contour
// order, their normals, tangents and lengths, the two wall distances of the
// shear fit, the leading edge) is tabulated on the host once, in the
// reference's arithmetic. The device reads the wall-adjacent cells, finds the
// stagnation station, evaluates each station in parallel and then sums the
// forces and moments in the reference's order (upper surface from the
// leading edge, then the lower surface outwards from it) so the coefficients
// round as the reference's do.

#include <cuda_runtime.h>

#include <cmath>

#include "forces.hpp"

namespace cfdb {
namespace {

#define FDEV __device__ __forceinline__

struct ForceParams {
  double dynamicPressure, referencePressure, chord, cosA, sinA;
};

constexpr int kForceThreads = 512;

/// Per station: Cp, wall shear, Cf and the force/moment increments, in wall
/// order, by one block. What bounds it is latency: everything that does not
/// depend on an order is a parallel pass (the stagnation station is the highest
/// owner pressure, first of equals; each side's separation the first pair that
/// qualifies), and the six sums, whose order is the reference's, run down shared
/// memory in six lanes. A call on 510 stations takes 58 us, 202 with
/// one thread for all of that.
__global__ void __launch_bounds__(kForceThreads)
forcesKernel(WallTable w, const double* __restrict__ p, const double* __restrict__ u, const double* __restrict__ v,
             const double* __restrict__ mu, ForceParams fp, double* __restrict__ station, double* __restrict__ out) {
  __shared__ double increments[6][kForceThreads];
  __shared__ double highest[kForceThreads / 32];
  __shared__ int where[kForceThreads / 32];
  __shared__ int firstPair[2];
  const int S = w.count, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // the highest pressure above the lowest double, at the lowest index (S: none)
  double high = -1.7976931348623157e308;
  int best = S;
  auto better = [&](double value, int at) {
    if (value > high || (value == high && at < best && best < S)) {
      high = value;
      best = at;
    }
  };
  for (int k = threadIdx.x; k < S; k += blockDim.x) better(p[w.owner[k]], k);
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const double value = __shfl_xor_sync(0xffffffffu, high, off);
    const int at = __shfl_xor_sync(0xffffffffu, best, off);
    if (at < S) better(value, at);
  }
  if (lane == 0) {
    highest[warp] = high;
    where[warp] = best;
  }
  if (threadIdx.x < 2) firstPair[threadIdx.x] = 0x7fffffff;
  __syncthreads();
  for (int q = 0; q < kForceThreads / 32; ++q) {
    if (where[q] < S) better(highest[q], where[q]);
  }
  const int stag = (best < S) ? best : 0;
  for (int k = threadIdx.x; k < S; k += blockDim.x) {
    const int o = w.owner[k];
    const double nx = w.nx[k], ny = w.ny[k];
    // flowTangent (SurfaceData.cpp:278-288)
    double tx = w.tx[k], ty = w.ty[k];
    const bool forward = (k == stag) ? (k >= w.leadingEdge) : (k > stag);
    if (!forward) {
      tx = tx * -1.0;
      ty = ty * -1.0;
    }
    const double pressure = p[o];
    const double cp = (fp.dynamicPressure > 0.0) ? (pressure - fp.referencePressure) / fp.dynamicPressure : 0.0;
    const double uc = u[o], vc = v[o];
    const double dn = uc * nx + vc * ny;
    const double px = uc - nx * dn, py = vc - ny * dn;
    double shear = 0.0;
    const double d1 = w.wallDistance[k];
    if (d1 > 0.0) {
      double gradient = (px * tx + py * ty) / d1;
      const int second = w.second[k];
      if (second >= 0) {
        const double d2 = w.outerDistance[k];
        if (d2 > d1 * 1.05) {
          const double ou = u[second], ov = v[second];
          const double odn = ou * nx + ov * ny;
          const double opx = ou - nx * odn, opy = ov - ny * odn;
          const double u1 = px * tx + py * ty;
          const double u2 = opx * tx + opy * ty;
          gradient = (u1 * d2 * d2 - u2 * d1 * d1) / (d1 * d2 * (d2 - d1));
        }
      }
      shear = mu[o] * gradient;
    }
    const double cf = (fp.dynamicPressure > 0.0) ? shear / fp.dynamicPressure : 0.0;
    double* s = station + static_cast<size_t>(k) * kStationValues;
    s[0] = pressure;
    s[1] = cp;
    s[2] = shear;
    s[3] = cf;
    s[4] = tx;
    s[5] = ty;
  }
  __syncthreads();
  // Accumulator::add over upper then lower (Forces.cpp:23-45, :76-80): station q
  // of that order, a block's worth at a time. A station without length adds 0,
  // which changes no sum.
  const double refX = 0.25 * fp.chord, refY = 0.0;
  const int upper = S - w.leadingEdge;
  double sum = 0.0;  // of lanes 0 .. 5 of the first warp
  int stations = 0;
  for (int first = 0; first < S; first += kForceThreads) {
    const int q = first + static_cast<int>(threadIdx.x);
    double dpx = 0.0, dpy = 0.0, dfx = 0.0, dfy = 0.0, dpm = 0.0, dfm = 0.0;
    bool counts = false;
    if (q < S) {
      const int k = (q < upper) ? w.leadingEdge + q : w.leadingEdge - 1 - (q - upper);
      const double* s = station + static_cast<size_t>(k) * kStationValues;
      const double ds = w.length[k];
      counts = ds > 0.0;
      if (counts) {
        const double scale = -(s[0] - fp.referencePressure) * ds;
        dpx = w.nx[k] * scale;
        dpy = w.ny[k] * scale;
        const double fs = s[2] * ds;
        dfx = s[4] * fs;
        dfy = s[5] * fs;
        const double ax = w.cx[k] - refX, ay = w.cy[k] - refY;
        dpm = ax * dpy - ay * dpx;
        dfm = ax * dfy - ay * dfx;
      }
    }
    increments[0][threadIdx.x] = dpx;
    increments[1][threadIdx.x] = dpy;
    increments[2][threadIdx.x] = dfx;
    increments[3][threadIdx.x] = dfy;
    increments[4][threadIdx.x] = dpm;
    increments[5][threadIdx.x] = dfm;
    stations += __syncthreads_count(counts);
    if (threadIdx.x < 6) {
      const int n = min(S - first, kForceThreads);
#pragma unroll 8
      for (int m = 0; m < n; ++m) sum = sum + increments[threadIdx.x][m];
    }
    __syncthreads();
  }
  // findSeparation (SurfaceData.cpp:179-203) on each surface, walked from the
  // leading edge: the first pair of stations, neither of them the stagnation
  // station, whose wall shear goes from positive to negative
  for (int side = 0; side < 2; ++side) {
    const int count = (side == 0) ? upper : w.leadingEdge;
    for (int m = 1 + static_cast<int>(threadIdx.x); m < count; m += static_cast<int>(blockDim.x)) {
      const int k = (side == 0) ? w.leadingEdge + m : w.leadingEdge - 1 - m;
      const int kp = (side == 0) ? k - 1 : k + 1;  // the station before it
      if (k == stag || kp == stag) continue;
      const double before = station[static_cast<size_t>(kp) * kStationValues + 2];
      const double after = station[static_cast<size_t>(k) * kStationValues + 2];
      if (before > 0.0 && after < 0.0) {
        atomicMin(&firstPair[side], m);
        break;
      }
    }
  }
  __syncthreads();
  if (warp != 0) return;
  const double pfx = __shfl_sync(0xffffffffu, sum, 0), pfy = __shfl_sync(0xffffffffu, sum, 1);
  const double ffx = __shfl_sync(0xffffffffu, sum, 2), ffy = __shfl_sync(0xffffffffu, sum, 3);
  const double pm = __shfl_sync(0xffffffffu, sum, 4), fm = __shfl_sync(0xffffffffu, sum, 5);
  if (lane != 0) return;
  const double pd = pfx * fp.cosA + pfy * fp.sinA;
  const double fd = ffx * fp.cosA + ffy * fp.sinA;
  const double pl = pfy * fp.cosA - pfx * fp.sinA;
  const double fl = ffy * fp.cosA - ffx * fp.sinA;
  const double drag = pd + fd;
  const double lift = pl + fl;
  const double moment = -pm - fm;
  const double forceScale = fp.dynamicPressure * fp.chord;
  const double momentScale = forceScale * fp.chord;
  out[0] = lift / forceScale;
  out[1] = drag / forceScale;
  out[2] = moment / momentScale;
  out[3] = pd / forceScale;
  out[4] = fd / forceScale;
  out[5] = lift;
  out[6] = drag;
  out[7] = moment;
  out[8] = (fp.chord > 0.0) ? w.cx[stag] / fp.chord : w.cx[stag];
  out[9] = static_cast<double>(stations);
  // separation: the chordwise station is interpolated linearly between the pair;
  // -1 where none is found
  for (int side = 0; side < 2; ++side) {
    double found = -1.0;
    const int m = firstPair[side];
    if (m != 0x7fffffff) {
      const int k = (side == 0) ? w.leadingEdge + m : w.leadingEdge - 1 - m;
      const int kp = (side == 0) ? k - 1 : k + 1;
      const double before = station[static_cast<size_t>(kp) * kStationValues + 2];
      const double after = station[static_cast<size_t>(k) * kStationValues + 2];
      const double span = before - after;
      const double fraction = (span > 0.0) ? before / span : 0.0;
      const double xp = (fp.chord > 0.0) ? w.cx[kp] / fp.chord : w.cx[kp];
      const double xk = (fp.chord > 0.0) ? w.cx[k] / fp.chord : w.cx[k];
      found = xp + fraction * (xk - xp);
    }
    out[10 + side] = found;
  }
}

}  // namespace

Status buildWallTable(const HostMesh& m, const double* nodes, HostWallTable* out) {
  HostWallTable& t = *out;
  t = HostWallTable{};
  if (nodes == nullptr) return ok();
  const int ni = m.nodesI, NI = ni - 1, NJ = m.nodesJ - 1;
  const int jFaces = NI * m.nodesJ;
  // collectWallFaces (SurfaceData.cpp:27-59): the j = 0 faces marked Wall.
  for (int i = 0; i < NI; ++i) {
    const int f = i;
    if (m.boundary[f] != 1) continue;  // mesh::BoundaryType::Wall
    const double ax = nodes[2 * i], ay = nodes[2 * i + 1];
    const double bx = nodes[2 * (i + 1)], by = nodes[2 * (i + 1) + 1];
    const double alx = bx - ax, aly = by - ay;
    const double len = std::hypot(alx, aly);
    if (!(len > 0.0)) continue;
    const int owner = m.owner[f];
    const double cx = m.faceCentre[2 * f], cy = m.faceCentre[2 * f + 1];
    const double nx = m.faceNormal[2 * f] * -1.0, ny = m.faceNormal[2 * f + 1] * -1.0;
    t.face.push_back(f);
    t.owner.push_back(owner);
    t.cx.push_back(cx);
    t.cy.push_back(cy);
    t.tx.push_back(alx * (1.0 / len));
    t.ty.push_back(aly * (1.0 / len));
    t.nx.push_back(nx);
    t.ny.push_back(ny);
    t.length.push_back(len);
    t.node0x.push_back(ax);
    // wall distance of the owner centroid (SurfaceData.cpp:118-119)
    const double ox = m.centroid[2 * owner] - cx, oy = m.centroid[2 * owner + 1] - cy;
    t.wallDistance.push_back(std::abs(ox * nx + oy * ny));
    // secondCellFromWall (SurfaceData.cpp:67-98): the cell across the owner's
    // face that points most nearly along the wall normal (alignment > 0.5),
    // faces visited below, right, above, left.
    const int oi = owner % NI, oj = owner / NI;
    const int cellFaces[4] = {oj * NI + oi, jFaces + (oi + 1) * NJ + oj, (oj + 1) * NI + oi,
                              jFaces + oi * NJ + oj};
    int best = -1;
    double bestAlignment = 0.5;
    for (int q = 0; q < 4; ++q) {
      const int g = cellFaces[q];
      if (g == f) continue;
      int across = m.neighbour[g];
      if (across < 0 && m.boundary[g] == 4 && m.partner[g] >= 0) across = m.owner[m.partner[g]];
      if (across < 0 || across == owner) continue;
      double ux = m.faceNormal[2 * g], uy = m.faceNormal[2 * g + 1];
      if (m.owner[g] != owner) {
        ux = ux * -1.0;
        uy = uy * -1.0;
      }
      const double alignment = ux * nx + uy * ny;
      if (alignment > bestAlignment) {
        bestAlignment = alignment;
        best = across;
      }
    }
    t.second.push_back(best);
    double d2 = 0.0;
    if (best >= 0) {
      const double qx = m.centroid[2 * best] - cx, qy = m.centroid[2 * best + 1] - cy;
      d2 = std::abs(qx * nx + qy * ny);
    }
    t.outerDistance.push_back(d2);
  }
  // leading edge: the first station whose first node is furthest forward
  // (SurfaceData.cpp:238-250)
  double forward = 1.7976931348623157e308;
  t.leadingEdge = 0;
  for (std::size_t k = 0; k < t.node0x.size(); ++k) {
    if (t.node0x[k] < forward) {
      forward = t.node0x[k];
      t.leadingEdge = static_cast<int>(k);
    }
  }
  return ok();
}

Status launchForces(const WallTable& w, const double* p, const double* u, const double* v,
                    const double* mu, double dynamicPressure, double referencePressure,
                    double chord, double cosA, double sinA, double* station, double* out,
                    cudaStream_t stream) {
  ForceParams fp{dynamicPressure, referencePressure, chord, cosA, sinA};
  forcesKernel<<<1, kForceThreads, 0, stream>>>(w, p, u, v, mu, fp, station, out);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(CFD_INITIALIZATION_FAILURE, cudaGetErrorString(e));
  return ok();
}

}  // namespace cfdb
