// streamlines.cu - post::traceStreamlines (src/post/Streamlines.cpp:80-197)
// on the device: classical RK4 through the piecewise-constant cell velocity
// of a structured block, with the reference's point location (a walk out of
// the worst edge from a hint cell, across the wake cut, and a first-cell scan
// where no hint is usable; Streamlines.cpp:47-100).
//
// One thread per seed and direction, alone in its warp (a curve is a serial
// chain; curves that share a warp wait for one another's branches), with the
// corners and the velocity of the cells that it is in kept in registers: most of
// a step's five locations end in the cell they start from. The seeds are placed first by a scan in
// which every (seed, cell) pair is tested and the lowest containing cell wins,
// which is the cell the reference's sequential scan finds. Arithmetic follows
// the reference's expressions and their order (no contraction), so curves
// agree with the reference's to rounding: the speed is CUDA's hypot (within
// its documented error of the host's std::hypot), the one operation that may
// round differently.

#include <cuda_runtime.h>

#include <cmath>

#include "streamlines.hpp"

namespace cfdb {
namespace {

#define SDEV __device__ __forceinline__

struct Block {
  int NI, NJ;           // cells
  const double* nodes;  // (x, y) per node, node (i, j) at j*(NI+1) + i
  const double* area;   // per cell
  const int* acrossJ0;  // cell across the j = 0 face of column i, or -1
  const double *u, *v;  // per cell
};

/// -turn(a, b, p): how far p lies outside the edge a -> b of an anticlockwise
/// cell (Streamlines.cpp:13-29), negative inside.
SDEV double edgeDistance(const Block& B, int c, int k, double px, double py) {
  const int i = c % B.NI, j = c / B.NI;
  const int stride = B.NI + 1;
  // corners (i, j), (i+1, j), (i+1, j+1), (i, j+1) (Mesh.cpp:130-136)
  const int corner[5] = {j * stride + i, j * stride + i + 1, (j + 1) * stride + i + 1,
                         (j + 1) * stride + i, j * stride + i};
  const double ax = B.nodes[2 * corner[k]], ay = B.nodes[2 * corner[k] + 1];
  const double bx = B.nodes[2 * corner[k + 1]], by = B.nodes[2 * corner[k + 1] + 1];
  const double ex = bx - ax, ey = by - ay;
  const double qx = px - ax, qy = py - ay;
  return -(ex * qy - ey * qx);
}

/// A cell with what the walk and the trace read of it.
struct Place {
  int i, j;
  double x[4], y[4];  // corners (i, j), (i+1, j), (i+1, j+1), (i, j+1) (Mesh.cpp:130-136)
  double u, v, area;
};
SDEV Place placeOf(const Block& B, int i, int j) {
  Place q;
  q.i = i;
  q.j = j;
  const int stride = B.NI + 1, at = j * stride + i, c = j * B.NI + i;
  const int corner[4] = {at, at + 1, at + stride + 1, at + stride};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    q.x[k] = B.nodes[2 * corner[k]];
    q.y[k] = B.nodes[2 * corner[k] + 1];
  }
  q.u = B.u[c];
  q.v = B.v[c];
  q.area = B.area[c];
  return q;
}

/// locateCell (Streamlines.cpp:47-100): from a hint, walk towards the point,
/// leaving each cell through the edge it lies furthest beyond (edges 0 below, 1
/// right, 2 above, 3 left: Mesh::cellFaces order, Mesh.cpp:204-213; across the
/// wake cut to the partner; false when that is a real boundary); after 4096
/// steps without arriving the first cell that contains the point (a scan: rare
/// on a walk, and costly, but it is the reference's answer). `at`: the hint in,
/// the cell out (unchanged when there is none).
SDEV bool locate(const Block& B, double px, double py, Place& at) {
  Place q = at;
  for (int step = 0; step < 4096; ++step) {
    double outside[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const double ax = q.x[k], ay = q.y[k], bx = q.x[(k + 1) & 3], by = q.y[(k + 1) & 3];
      const double ex = bx - ax, ey = by - ay;
      const double qx = px - ax, qy = py - ay;
      outside[k] = -(ex * qy - ey * qx);
    }
    int worstEdge = -1;
    double worst = 0.0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (outside[k] > worst) {
        worst = outside[k];
        worstEdge = k;
      }
    }
    if (worstEdge < 0) {
      at = q;
      return true;
    }
    int i = q.i, j = q.j;
    if (worstEdge == 0) {
      if (j > 0) {
        --j;
      } else {
        const int c = B.acrossJ0[i];
        if (c < 0) return false;
        i = c % B.NI;
        j = c / B.NI;
      }
    } else if (worstEdge == 1) {
      if (++i >= B.NI) return false;
    } else if (worstEdge == 2) {
      if (++j >= B.NJ) return false;
    } else {
      if (--i < 0) return false;
    }
    q = placeOf(B, i, j);
  }
  const int cells = B.NI * B.NJ;
  for (int c = 0; c < cells; ++c) {
    bool inside = true;
    for (int k = 0; k < 4 && inside; ++k) inside = !(edgeDistance(B, c, k, px, py) > 0.0);
    if (inside) {
      at = placeOf(B, c % B.NI, c / B.NI);
      return true;
    }
  }
  return false;
}

/// Lowest-index cell containing each seed (the reference's scan), by atomicMin.
__global__ void seedKernel(Block B, int seeds, const double* __restrict__ xy, int* __restrict__ cell) {
  const long long t = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const long long cells = static_cast<long long>(B.NI) * B.NJ;
  if (t >= cells * seeds) return;
  const int s = static_cast<int>(t / cells);
  const int c = static_cast<int>(t % cells);
  const double px = xy[2 * s], py = xy[2 * s + 1];
  for (int k = 0; k < 4; ++k) {
    if (edgeDistance(B, c, k, px, py) > 0.0) return;
  }
  atomicMin(cell + s, c);
}

/// One seed in one direction (odd blocks downstream, even upstream): the
/// points from the seed onwards, at most maxSteps + 1 (Streamlines.cpp:132-183).
/// A block of one warp, one lane of it at work. Both ways, 200 steps on 384x96: 1,000
/// seeds take 0.42 ms, 5,000 0.75; 1.01 and 0.96 as threads of blocks of 128, which
/// read all corners again for every location (20,000 seeds: 1.03 and 0.98).
__global__ void traceKernel(Block B, int seeds, const double* __restrict__ xy, const int* __restrict__ seedCell,
                            StreamlineSettings o, double* __restrict__ points, int* __restrict__ lengths) {
  const int t = blockIdx.x;
  if (threadIdx.x != 0) return;
  const int s = t >> 1;
  const bool downstream = (t & 1) != 0;
  double* out = points + static_cast<long long>(t) * 2 * (o.maxSteps + 1);
  const int start = seedCell[s];
  if (start < 0 || start >= B.NI * B.NJ || (!downstream && !o.traceBackwards)) {
    lengths[t] = 0;
    return;
  }
  const double sense = downstream ? 1.0 : -1.0;
  double px = xy[2 * s], py = xy[2 * s + 1];
  Place cell = placeOf(B, start % B.NI, start / B.NI);
  int n = 0;
  out[2 * n] = px;
  out[2 * n + 1] = py;
  ++n;
  // velocityAt: the cell holding the point (walking from the carried cell),
  // its velocity times the sense; zero outside the domain
  auto velocityAt = [&](double x, double y, Place& carried, double& vx, double& vy) {
    if (!locate(B, x, y, carried)) {
      vx = 0.0;
      vy = 0.0;
      return;
    }
    vx = carried.u * sense;
    vy = carried.v * sense;
  };
  for (int step = 0; step < o.maxSteps; ++step) {
    Place probe = cell;
    double k1x, k1y;
    velocityAt(px, py, probe, k1x, k1y);
    const double speed = hypot(k1x, k1y);
    if (!(speed > o.stallSpeed)) break;
    const double step0 = o.stepFraction * sqrt(fmax(cell.area, 0.0));
    const double dt = (speed > 0.0) ? step0 / speed : 0.0;
    if (!(dt > 0.0)) break;
    double k2x, k2y;
    velocityAt(px + k1x * (0.5 * dt), py + k1y * (0.5 * dt), probe, k2x, k2y);
    double k3x, k3y;
    velocityAt(px + k2x * (0.5 * dt), py + k2y * (0.5 * dt), probe, k3x, k3y);
    double k4x, k4y;
    velocityAt(px + k3x * dt, py + k3y * dt, probe, k4x, k4y);
    const double h = dt / 6.0;
    const double ax = (((k1x + k2x * 2.0) + k3x * 2.0) + k4x) * h;
    const double ay = (((k1y + k2y * 2.0) + k3y * 2.0) + k4y) * h;
    const double nx = px + ax, ny = py + ay;
    if (!locate(B, nx, ny, cell)) break;  // left the domain
    px = nx;
    py = ny;
    out[2 * n] = px;
    out[2 * n + 1] = py;
    ++n;
  }
  lengths[t] = n;
}

}  // namespace

Status launchStreamlines(int NI, int NJ, const double* nodes, const double* area, const int* acrossJ0,
                         const double* u, const double* v, int seeds, const double* seedXY,
                         const StreamlineSettings& o, int* seedCell, double* points, int* lengths,
                         cudaStream_t stream) {
  const Block B{NI, NJ, nodes, area, acrossJ0, u, v};
  const long long pairs = static_cast<long long>(NI) * NJ * seeds;
  const int block = 256;
  cudaError_t e = cudaMemsetAsync(seedCell, 0x7f, sizeof(int) * seeds, stream);  // above any cell index
  if (e != cudaSuccess) return fail(CFD_INITIALIZATION_FAILURE, cudaGetErrorString(e));
  seedKernel<<<static_cast<unsigned>((pairs + block - 1) / block), block, 0, stream>>>(B, seeds, seedXY, seedCell);
  traceKernel<<<2 * seeds, 32, 0, stream>>>(B, seeds, seedXY, seedCell, o, points, lengths);
  e = cudaGetLastError();
  if (e != cudaSuccess) return fail(CFD_INITIALIZATION_FAILURE, cudaGetErrorString(e));
  return CFD_OK;
}

}  // namespace cfdb
