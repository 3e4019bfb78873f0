// wide_plan.cu - how many CTAs a wide team gets (host side).

#include "wide_plan.hpp"

#include "common.hpp"
#include "solver.hpp"
#include "wide_cg.cuh"

namespace cfdb {

int wideCapacity() {
  static PerDeviceOnce once;
  static int sms[64] = {};
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 64) return 0;
  const Status st = once.run([&]() -> Status {
    int n = 0, cooperative = 0;
    cudaError_t e = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&cooperative, cudaDevAttrCooperativeLaunch, device);
    if (e != cudaSuccess) return fail(CFD_INITIALIZATION_FAILURE, cudaGetErrorString(e));
    sms[device] = cooperative ? std::min(n, kMaxWideCtas) : 0;
    return ok();
  });
  return (st == CFD_OK) ? sms[device] : 0;
}

double wideCgMicroseconds(int NI, int NJ, int R) {
  const WideCgShape s = wideCgShape(NI, NJ, R, kWideThreads);
  return 1.2 + 0.15 * s.rounds * s.K * s.passes + ((R > 1) ? 0.2 : 0.0);
}

int wideChooseCtas(int NI, int NJ, int capacity) {
  const int columns = wideCgShape(NI, NJ, 1, kWideThreads).columnTiles;
  int best = columns;
  for (int R = columns; R <= capacity; R += columns) {
    if (wideCgMicroseconds(NI, NJ, R) < wideCgMicroseconds(NI, NJ, best)) best = R;
  }
  return best;
}

}  // namespace cfdb
