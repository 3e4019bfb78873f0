// plan_check.cu - the host side of the launches' shapes, for tests on a machine
// without a GPU: reads one query a line, answers in one line.
//
//   plan CAPACITY THREADS {NI NJ SST}...   CTAs, shared memory, teams of the plain
//                                          form's plan; 1 if the plan is sound
//   teams CAPACITY THREADS {NI NJ SST}...  its teams: the solves in order as solve
//                                          CTAs pairs, -1 after each team
//   tiles THREADS NJ NI0 NI1               blocks of NI0 .. NI1 columns with a column
//                                          tile that holds no column, or more units
//                                          than sums are kept of; the first of them
//   whole CAPACITY THREADS NI NJ           1 if every team such a block can get is
//                                          whole rows of CTAs with a unit each
//   sweeps NI                              shared memory of one k or omega sweep
//   share CAPACITY THREADS TOGETHER NI NJ SST  CTAs of a lone launch beside others
//   waits CAPACITY THREADS ITERATIONS CAP {NI NJ SST}...  of any CTA's longest wait
//                                          for the solves before its own, as
//                                          modelled, the permille of its limit
#include <cstdio>
#include <iostream>
#include <sstream>
#include <string>

#include "row_sweeps.cuh"
#include "wide_cg.cuh"
#include "wide_plan.hpp"

using namespace cfdb;

namespace {

/// Every solve is in one range, the CTAs that name a range have ranks 0 .. n-1
/// and one R, and there are as many of them as the widest solve of it uses.
bool sound(const WidePlan& plan, const std::vector<WideJob>& jobs) {
  std::vector<int> seen(jobs.size(), 0);
  int listed = 0;
  for (std::size_t b = 0; b < plan.ctas.size(); ++b) {
    const WideCta& c = plan.ctas[b];
    if (c.begin < 0 || c.end <= c.begin || c.end > static_cast<int>(plan.list.size())) return false;
    if (c.rank == 0) {
      if (c.begin != listed) return false;
      listed = c.end;
    } else if (b == 0 || plan.ctas[b - 1].begin != c.begin || plan.ctas[b - 1].rank != c.rank - 1 ||
               plan.ctas[b - 1].R != c.R) {
      return false;
    }
  }
  if (listed != static_cast<int>(plan.list.size())) return false;
  for (int k : plan.list) {
    if (k < 0 || k >= static_cast<int>(jobs.size()) || seen[static_cast<std::size_t>(k)]++) return false;
  }
  return plan.list.size() == jobs.size();
}

int ctasOf(const WideJob& job, int width, int threads) {
  return wideUsefulCtas(job.NI, job.NJ, std::min(width, job.most), threads);
}

/// Modelled milliseconds of `iterations` of a solve with `cap` CG iterations each.
double milliseconds(const WideJob& job, int R, int iterations, int cap) {
  return 1e-3 * iterations * (cap * wideCgMicroseconds(job.NI, job.NJ, R) + (job.sst ? 1.5 * job.NJ : 0.0));
}

double waits(const WidePlan& plan, const std::vector<WideJob>& jobs, int threads, int iterations, int cap) {
  double worst = 0.0;
  for (const WideCta& c : plan.ctas) {
    double behind = 0.0, ahead = 0.0;
    for (int k = c.begin; k < c.end; ++k) {
      const WideJob& job = jobs[static_cast<std::size_t>(plan.list[static_cast<std::size_t>(k)])];
      const int R = ctasOf(job, c.R, threads);
      const double outer = outerBound(job.NI, job.NJ, R, threads, wideEffort(false, 1, cap, 16, 3));
      // a poll is 0.4 us at least, a unit of the limit 2^20 ns
      const double limit = kWideSpinLimit * 0.4e-3 + wideWaitLimit(outer + iterations * ahead) * 1.048576;
      worst = std::max(worst, behind / limit);
      behind += milliseconds(job, R, iterations, cap);
      ahead += outer;
    }
  }
  return worst;
}

}  // namespace

int main() {
  std::string line;
  while (std::getline(std::cin, line)) {
    std::istringstream in(line);
    std::string what;
    in >> what;
    if (what == "whole") {
      int capacity = 0, threads = 0, NI = 0, NJ = 0;
      in >> capacity >> threads >> NI >> NJ;
      auto whole = [&](int R, int T) {
        const WideCgShape s = wideCgShape(NI, NJ, R, T);
        return s.RT >= 1 && R == s.columnTiles * s.RT;
      };
      bool ok = capacity < wideLeastCtas(NI, NJ, kWideThreads) ||
                whole(wideChooseCtas(NI, NJ, capacity), kWideThreads);
      const int most = wideMostCtas(NI, NJ, threads);
      for (int width = wideLeastCtas(NI, NJ, threads); width <= capacity; ++width) {
        ok = ok && whole(wideUsefulCtas(NI, NJ, std::min(width, most), threads), threads);
      }
      std::printf("%d\n", ok ? 1 : 0);
    } else if (what == "share") {
      int capacity = 0, threads = 0, together = 0, NI = 0, NJ = 0, sst = 0;
      in >> capacity >> threads >> together >> NI >> NJ >> sst;
      const WideJob job{NI, NJ, wideMostCtas(NI, NJ, threads), sst != 0, 0};
      const int share = wideShare(job, threads, together, capacity);
      std::printf("%d %d %d\n", share, wideLeastCtas(NI, NJ, threads), ctasOf(job, share, threads));
    } else if (what == "sweeps") {
      int NI = 0;
      in >> NI;
      std::printf("%d\n", rowSweepBytes(rowSweepShape(NI)));
    } else if (what == "tiles") {
      int threads = 0, NJ = 0, first = 0, last = 0, bad = 0, where = 0;
      in >> threads >> NJ >> first >> last;
      for (int NI = first; NI <= last; ++NI) {
        const WideCgShape s = wideCgShape(NI, NJ, kMaxWideCtas, threads);
        const bool ok = s.columnTiles >= 1 && s.columnTiles <= kMaxColumnTiles && (s.columnTiles - 1) * s.width < NI &&
                        s.columnTiles * s.width >= NI && s.columnTiles * s.unitRows <= kMaxUnits &&
                        s.unitRows * s.B >= NJ && (s.unitRows - 1) * s.B < NJ;
        if (!ok && bad++ == 0) where = NI;
      }
      std::printf("%d %d\n", bad, where);
    } else if (what == "plan" || what == "teams" || what == "waits") {
      int capacity = 0, threads = 0, iterations = 0, cap = 0;
      in >> capacity >> threads;
      if (what == "waits") in >> iterations >> cap;
      std::vector<WideJob> jobs;
      for (int NI, NJ, sst; in >> NI >> NJ >> sst;) {
        jobs.push_back(WideJob{NI, NJ, wideMostCtas(NI, NJ, threads), sst != 0, 0});
      }
      const WidePlan plan = planWide(jobs, threads, capacity);
      if (what == "waits") {
        std::printf("%d\n", static_cast<int>(1000.0 * waits(plan, jobs, threads, iterations, cap)));
        continue;
      }
      if (what == "teams") {
        for (const WideCta& c : plan.ctas) {
          if (c.rank != 0) continue;
          for (int k = c.begin; k < c.end; ++k) {
            const int job = plan.list[static_cast<std::size_t>(k)];
            std::printf("%d %d ", job, ctasOf(jobs[static_cast<std::size_t>(job)], c.R, threads));
          }
          std::printf("-1 ");
        }
        std::printf("\n");
        continue;
      }
      int teams = 0;
      for (const WideCta& c : plan.ctas) teams += (c.rank == 0) ? 1 : 0;
      std::printf("%zu %d %d %d\n", plan.ctas.size(), plan.smemBytes, teams, sound(plan, jobs) ? 1 : 0);
    } else {
      std::printf("?\n");
    }
  }
  return 0;
}
