// wide_plan.cu - how many CTAs a wide team gets, and how a launch shares the
// GPU between solves (host side).

#include "wide_plan.hpp"

#include <atomic>
#include <functional>
#include <map>
#include <numeric>
#include <queue>
#include <utility>

#include "common.hpp"
#include "row_sweeps.cuh"
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
  const int cells = s.rounds * s.K * s.passes, form = wideCgForm(s, kWideThreads, kMaxWideSmem);
  if (form == 0) return 2.0 + 1.3 * cells;
  return (form % 8 == 0) ? 1.2 + 0.5 * cells : 1.2 + 1.0 * cells;
}

int wideLeastCtas(int NI, int NJ, int threads) { return wideCgShape(NI, NJ, 1, threads).columnTiles; }

int wideMostCtas(int NI, int NJ, int threads) {
  const WideCgShape s = wideCgShape(NI, NJ, 1, threads);
  return std::min(s.columnTiles * s.unitRows, kMaxWideCtas / s.columnTiles * s.columnTiles);
}

int mixedMostCtas(int NI, int NJ) {
  // 512 cells a CTA, one a thread: more CTAs gain nothing (two iterations at
  // 384x96 on 72 CTAs 1.66 ms, on 144 1.67; at 192x48 on 18 1.22, on 36 1.22),
  // fewer do lose (1.75 on 36, 1.25 on 9), and a batch holds more solves side by
  // side. Six, for the sweeps.
  const int chunks = static_cast<int>((static_cast<long long>(NI) * NJ + 511) / 512);
  return std::min(std::max(chunks, 6), kMaxWideCtas);
}

int wideChooseCtas(int NI, int NJ, int capacity) {
  const int columns = wideLeastCtas(NI, NJ, kWideThreads);
  int best = columns;
  for (int R = columns; R <= capacity; R += columns) {
    if (wideCgMicroseconds(NI, NJ, R) < wideCgMicroseconds(NI, NJ, best)) best = R;
  }
  return best;
}

long long wideSpillDoubles(int NI, int NJ, int most, int threads) {
  long long doubles = 0;
  const int columns = wideLeastCtas(NI, NJ, threads);
  for (int R = columns; R <= std::max(most, columns); ++R) {
    doubles = std::max(doubles, R * wideCgSpill(NI, NJ, R, threads, kMaxWideSmem, true));
  }
  return doubles;
}

namespace {

int usefulCtas(const WideJob& job, int width, int threads) {
  if (job.mixedSmem > 0) return std::min(width, job.most);
  return wideUsefulCtas(job.NI, job.NJ, std::min(width, job.most), threads);
}

/// Modelled microseconds of one outer iteration: the CG, ~17 barriers, the
/// other phases' passes (0.54 ms on 16 CTAs at 768x192), the sweeps' rows.
double outerMicroseconds(const WideJob& job, int R) {
  const double cells = static_cast<double>(job.NI) * job.NJ;
  if (job.mixedSmem > 0) {
    // 16 V-cycles of ~8 barriers and a coarse cycle each
    return 16.0 * (30.0 + 3.3 * cells / R / 512.0) + 30.0 + cells / R / 512.0 * (job.sst ? 30.0 : 15.0) +
           (job.sst ? 0.4 * job.NJ : 0.0);
  }
  return 200.0 * wideCgMicroseconds(job.NI, job.NJ, R) + 30.0 + cells / R / 512.0 * (job.sst ? 30.0 : 15.0) +
         (job.sst ? 0.4 * job.NJ : 0.0);
}

int smemBytes(const WideJob& job, int R, int threads) {
  if (job.mixedSmem > 0) return job.mixedSmem;
  const bool any = (kernelFlags() & kFlagSharedCg) != 0;
  long long bytes = wideCgBytes(job.NI, job.NJ, R, threads, kMaxWideSmem, any);
  {
    // whatever the model is now: it can be changed after a batch is planned
    const RowSweepShape z = rowSweepShape(job.NI);
    const int warps = threads / 32, perCta = (2 * kSweeps + R - 1) / R;
    long long sweeps = static_cast<long long>(std::min(perCta, warps)) * rowSweepBytes(z);
    if (perCta == 1 && warps >= z.chunks && rowSweepRingBytes(z) <= kMaxWideSmem) sweeps = rowSweepRingBytes(z);
    bytes = std::max(bytes, std::min<long long>(sweeps, kMaxWideSmem));
  }
  return static_cast<int>(bytes);
}

}  // namespace

WidePlan planWide(const std::vector<WideJob>& jobs, int threads, int capacity) {
  WidePlan plan;
  const int count = static_cast<int>(jobs.size());
  capacity = std::max(capacity, 1);
  // side by side, each at its widest
  std::vector<int> widths(jobs.size());
  int total = 0;
  for (int k = 0; k < count; ++k) {
    widths[k] = usefulCtas(jobs[k], std::min(jobs[k].most, capacity), threads);
    total += widths[k];
  }
  if (total <= capacity) {
    for (int k = 0; k < count; ++k) {
      for (int r = 0; r < widths[k]; ++r) plan.ctas.push_back(WideCta{k, k + 1, r, widths[k]});
      plan.list.push_back(k);
      plan.smemBytes = std::max(plan.smemBytes, smemBytes(jobs[k], widths[k], threads));
    }
    return plan;
  }
  // teams of equal width, each with a list of solves: longest first to the
  // team that is free first. The number of teams that finishes first wins (the
  // fewest of equals); a solve's bits do not depend on it. A solve's cost follows
  // from its kind and the width, and numbers of teams are tried in the order of
  // what they take at least, so most are not tried at all: 512 coarse solves 0.5
  // ms, 20 with every number tried and every solve priced for it.
  int least = 1;
  std::vector<WideJob> kinds;
  std::vector<int> kindOf(jobs.size()), members;
  for (int k = 0; k < count; ++k) {
    std::size_t kind = 0;
    while (kind < kinds.size() && !(kinds[kind] == jobs[k])) ++kind;
    if (kind == kinds.size()) {
      kinds.push_back(jobs[k]);
      members.push_back(0);
      if (jobs[k].mixedSmem == 0) least = std::max(least, wideLeastCtas(jobs[k].NI, jobs[k].NJ, threads));
    }
    kindOf[k] = static_cast<int>(kind);
    ++members[kind];
  }
  std::map<int, std::vector<double>> priced;  // width -> cost of each kind
  auto costs = [&](int width) -> const std::vector<double>& {
    std::vector<double>& cost = priced[width];
    if (cost.empty()) {
      for (const WideJob& job : kinds) cost.push_back(outerMicroseconds(job, usefulCtas(job, width, threads)));
    }
    return cost;
  };
  std::vector<std::pair<double, int>> tries;  // what so many teams take at least
  for (int teams = 1; teams <= std::min(count, capacity / least); ++teams) {
    const std::vector<double>& cost = costs(capacity / teams);
    double sum = 0.0;
    for (std::size_t kind = 0; kind < kinds.size(); ++kind) sum += members[kind] * cost[kind];
    // (less a little: sums of the same numbers in other orders)
    tries.emplace_back(std::max(sum / teams * (1.0 - 1e-9), *std::max_element(cost.begin(), cost.end())), teams);
  }
  std::sort(tries.begin(), tries.end());
  double best = -1.0;
  int bestTeams = 1;
  std::vector<std::vector<int>> bestLists;
  for (const auto& [atLeast, teams] : tries) {
    if (best >= 0.0 && atLeast > best) break;
    const std::vector<double>& cost = costs(capacity / teams);
    std::vector<int> order(jobs.size());
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return cost[kindOf[a]] > cost[kindOf[b]]; });
    std::vector<std::vector<int>> lists(static_cast<std::size_t>(teams));
    std::priority_queue<std::pair<double, int>, std::vector<std::pair<double, int>>, std::greater<>> load;
    for (int team = 0; team < teams; ++team) load.emplace(0.0, team);
    double makespan = 0.0;
    for (int k : order) {
      const auto [until, team] = load.top();
      load.pop();
      lists[team].push_back(k);
      load.emplace(until + cost[kindOf[k]], team);
      makespan = std::max(makespan, until + cost[kindOf[k]]);
    }
    if (best < 0.0 || makespan < best || (makespan == best && teams < bestTeams)) {
      best = makespan;
      bestTeams = teams;
      bestLists = std::move(lists);
    }
  }
  const int width = capacity / bestTeams;
  for (const std::vector<int>& solves : bestLists) {
    const int begin = static_cast<int>(plan.list.size());
    int widest = 0;
    for (int k : solves) {
      plan.list.push_back(k);
      const int R = usefulCtas(jobs[k], width, threads);
      widest = std::max(widest, R);
      plan.smemBytes = std::max(plan.smemBytes, smemBytes(jobs[k], R, threads));
    }
    const int end = static_cast<int>(plan.list.size());
    for (int r = 0; r < widest; ++r) plan.ctas.push_back(WideCta{begin, end, r, width});
  }
  return plan;
}

int wideShare(const WideJob& job, int threads, int together, int capacity) {
  const std::vector<WideJob> all(static_cast<std::size_t>(std::min(std::max(together, 1), kMaxWideCtas)), job);
  const WidePlan plan = planWide(all, threads, capacity);
  return plan.ctas.empty() ? job.most : std::min(plan.ctas.front().R, job.most);
}

namespace {
std::atomic<int> g_inFlight[64];
}

WideFlight::WideFlight() {
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 64) return;
  device_ = device;
  g_inFlight[device_].fetch_add(1, std::memory_order_relaxed);
}
WideFlight::~WideFlight() {
  if (device_ >= 0) g_inFlight[device_].fetch_sub(1, std::memory_order_relaxed);
}
int WideFlight::together() const {
  return (device_ >= 0) ? std::max(g_inFlight[device_].load(std::memory_order_relaxed), 1) : 1;
}

}  // namespace cfdb
