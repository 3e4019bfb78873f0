// wide_plan.hpp - how many CTAs a wide team gets, and its scratch (host side).
#pragma once

#include <algorithm>
#include <cstddef>

#include "instance.hpp"

namespace cfdb {

/// Dynamic shared memory of a wide kernel: what 227 KB leave beside its
/// static tables.
constexpr int kMaxWideSmem = 223120;

/// CTAs the current device runs at once with one wide CTA per SM (at most
/// kMaxWideCtas); 0 with an error set when the device cannot be asked.
int wideCapacity();

/// The layout of a wide team's scratch, with `messages` messages in a set.
struct WideScratchLayout {
  std::size_t epoch, flags, slots, rowSums, set, bytes;
  WideScratchLayout(int NJ, long long messages) {
    std::size_t at = 0;
    auto take = [&](std::size_t n) {
      const std::size_t here = at;
      at += (n + 255) & ~std::size_t{255};
      return here;
    };
    epoch = take(sizeof(unsigned long long));
    flags = take(kMaxWideCtas * sizeof(unsigned));
    slots = take(2 * kMaxWideCtas * 8 * sizeof(double));
    rowSums = take(2 * 4 * static_cast<std::size_t>(NJ) * sizeof(double));
    set = take(2 * static_cast<std::size_t>(messages) * sizeof(ulonglong2));
    bytes = at;
  }
  WideScratch at(char* base) const {
    return WideScratch{reinterpret_cast<unsigned long long*>(base + epoch),
                       reinterpret_cast<unsigned*>(base + flags),
                       reinterpret_cast<double*>(base + slots),
                       reinterpret_cast<double*>(base + rowSums),
                       reinterpret_cast<ulonglong2*>(base + set)};
  }
};

/// Modelled microseconds of one CG iteration on R CTAs of 512 threads: the
/// cells of a thread, and the exchange between CTAs.
double wideCgMicroseconds(int NI, int NJ, int R);

/// CTAs for a lone system: the count with the smallest modelled time.
int wideChooseCtas(int NI, int NJ, int capacity);

}  // namespace cfdb
