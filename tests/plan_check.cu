// plan_check.cu - the host side of the launches' shapes, for tests on a machine
// without a GPU: reads one query a line, answers in one line.
//
//   plan CAPACITY THREADS {NI NJ SST}...   CTAs, shared memory, teams of the plain
//                                          form's plan; 1 if the plan is sound
#include <cstdio>
#include <iostream>
#include <sstream>
#include <string>

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

}  // namespace

int main() {
  std::string line;
  while (std::getline(std::cin, line)) {
    std::istringstream in(line);
    std::string what;
    in >> what;
    if (what == "plan") {
      int capacity = 0, threads = 0;
      in >> capacity >> threads;
      std::vector<WideJob> jobs;
      for (int NI, NJ, sst; in >> NI >> NJ >> sst;) {
        jobs.push_back(WideJob{NI, NJ, wideMostCtas(NI, NJ, threads), sst != 0, 0});
      }
      const WidePlan plan = planWide(jobs, threads, capacity);
      int teams = 0;
      for (const WideCta& c : plan.ctas) teams += (c.rank == 0) ? 1 : 0;
      std::printf("%zu %d %d %d\n", plan.ctas.size(), plan.smemBytes, teams, sound(plan, jobs) ? 1 : 0);
    } else {
      std::printf("?\n");
    }
  }
  return 0;
}
