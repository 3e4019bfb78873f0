// wide_plan.hpp - how many CTAs a wide team gets, and its scratch (host side).
#pragma once

#include <algorithm>
#include <cstddef>
#include <vector>

#include "instance.hpp"

namespace cfdb {

/// Dynamic shared memory of a wide kernel: what 227 KB leave beside its
/// static tables.
constexpr int kMaxWideSmem = 222032;

/// CTAs the current device runs at once with one wide CTA per SM (at most
/// kMaxWideCtas); 0 with an error set when the device cannot be asked.
int wideCapacity();

/// The layout of a wide team's scratch, with `messages` messages in a set.
struct WideScratchLayout {
  std::size_t epoch, arrived, left, slots, chunkSums, set, bytes;
  WideScratchLayout(int NI, int NJ, long long messages) {
    std::size_t at = 0;
    auto take = [&](std::size_t n) {
      const std::size_t here = at;
      at += (n + 255) & ~std::size_t{255};
      return here;
    };
    epoch = take(sizeof(unsigned long long));
    arrived = take(sizeof(unsigned));  // a line each
    left = take(sizeof(unsigned));
    slots = take(2 * kMaxWideCtas * 8 * sizeof(double));
    chunkSums = take(2 * 4 * ((static_cast<std::size_t>(NI) * NJ + 255) / 256) * sizeof(double));
    set = take(2 * static_cast<std::size_t>(messages) * sizeof(ulonglong2));
    bytes = at;
  }
  WideScratch at(char* base) const {
    return WideScratch{reinterpret_cast<unsigned long long*>(base + epoch),
                       reinterpret_cast<unsigned*>(base + arrived),
                       reinterpret_cast<unsigned*>(base + left),
                       reinterpret_cast<double*>(base + slots),
                       reinterpret_cast<double*>(base + chunkSums),
                       reinterpret_cast<ulonglong2*>(base + set)};
  }
};

/// Modelled microseconds of one CG iteration on R CTAs of 512 threads: the
/// cells of a thread, and the exchange between CTAs.
double wideCgMicroseconds(int NI, int NJ, int R);

/// CTAs for a lone system: the count with the smallest modelled time.
int wideChooseCtas(int NI, int NJ, int capacity);

/// CTAs a solve can use at most (a CG unit each) and needs at least (a column
/// tile each), for blocks of `threads`.
int wideMostCtas(int NI, int NJ, int threads);
int wideLeastCtas(int NI, int NJ, int threads);

/// Doubles of spill a solve needs whatever the number of its CTAs up to `most`.
long long wideSpillDoubles(int NI, int NJ, int most, int threads);

/// CTAs a solve of the mixed form can use at most.
int mixedMostCtas(int NI, int NJ);

/// A solve as the planner sees it.
struct WideJob {
  int NI, NJ;
  int most;  // CTAs at most
  bool sst;
  int mixedSmem;  // mixed form: its dynamic shared memory; 0: plain form
  bool operator==(const WideJob& o) const {
    return NI == o.NI && NJ == o.NJ && most == o.most && sst == o.sst && mixedSmem == o.mixedSmem;
  }
};
struct WidePlan {
  std::vector<WideCta> ctas;
  std::vector<int> list;  // solves in the order the CTAs' ranges name them
  int smemBytes{0};
  bool operator==(const WidePlan& o) const {
    auto same = [](const WideCta& a, const WideCta& b) {
      return a.begin == b.begin && a.end == b.end && a.rank == b.rank && a.R == b.R;
    };
    return smemBytes == o.smemBytes && list == o.list &&
           std::equal(ctas.begin(), ctas.end(), o.ctas.begin(), o.ctas.end(), same);
  }
};
/// How one launch runs these solves (of one form) on `capacity` CTAs (wideCapacity()):
/// side by side when the GPU holds them all at their widest, else in teams that take
/// one solve after another.
WidePlan planWide(const std::vector<WideJob>& jobs, int threads, int capacity);

/// CTAs of a launch of one solve beside `together - 1` others, from other host
/// threads: as many as it would get in one launch with as many of its kind. A
/// launch as wide as the GPU would make the others wait for all of it. Seven
/// threads, each a lone SST solve, ms per solve and iteration: plain 384x96 0.94 as
/// wide as it goes, 0.36 so, 768x192 1.67 and 0.82; mixed 0.42 and 0.21, 1.28 and 0.47.
int wideShare(const WideJob& job, int threads, int together, int capacity);

/// The launches of lone solves that this process has in flight on a device, this
/// one included, while it lives.
class WideFlight {
 public:
  WideFlight();
  ~WideFlight();
  WideFlight(const WideFlight&) = delete;
  WideFlight& operator=(const WideFlight&) = delete;
  int together() const;

 private:
  int device_{-1};
};

}  // namespace cfdb
