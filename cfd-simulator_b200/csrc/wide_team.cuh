// wide_team.cuh - any number of CTAs of one cooperative launch working on one
// solve: barriers, maxima, row-ordered sums and tagged messages through
// global memory.
//
// Why not a thread-block cluster: a cluster is at most 16 CTAs and must fit
// in one GPC, so a lone 768x192 solve keeps 132 of the 148 SMs idle and its
// state (1.2 MB per array) in L2. Spread over ~100 SMs the state of the
// pressure CG fits on chip, and what a step costs is one exchange through L2
// (an iteration of the CG takes 4.6 us, of which a round trip is under 1) instead
// of the streaming of 900 KB per SM.
//
// Messages are tagged: every double travels as two 64-bit words, each half of
// it beside a 32-bit tag, so a reader that sees the tag in both words has the
// value; no flag, fence or acknowledgement is needed. (Each 64-bit word is a
// single-copy-atomic access; the two may arrive apart.) Tags come from the
// team's epoch, which every exchange increments and the solve's scratch keeps
// between launches, so a stale message never carries the tag waited for.
//
// Every CTA of a team must be resident: the launch is cooperative, one CTA
// per SM. All waits are bounded (kWideSpinLimit polls, then wideWaitLimit): one
// that gives up sets a code in the solve's fault word, after which the CTA waits no
// more, so a launch always ends and the host reports it.
//
// Sums are formed per chunk of 256 consecutive cells and the chunks' sums in one
// fixed order, so their bits do not depend on how many CTAs share the cells.
#pragma once

#include <cuda_runtime.h>

#include "instance.hpp"
#include "team.cuh"

namespace cfdb {

constexpr int kChunkCells = 256;  // cells whose sums are formed together, by as many threads
constexpr int kChunkBatch = 16;   // chunks of a CTA whose partial sums are held at once
constexpr int kMaxSums = 4;
constexpr int kWideThreads = 512;
/// Polls after which a wait is overdue, each an L2 round trip (0.4 us or more): ~1 s.
/// From there on it goes by the clock (wideWaitLimit).
constexpr int kWideSpinLimit = 1 << 21;

/// What a solve's settings let one outer iteration do.
struct WideEffort {
  double exchanges;  // of the CG (plain form)
  double cycles;     // of the multigrid (mixed form)
  int sweeps;        // of the momentum system
};
__host__ __device__ inline WideEffort wideEffort(bool mixed, int corrections, int cgMax, int mgCap, int sweeps) {
  const double passes = (corrections > 1) ? corrections : 1;
  return WideEffort{mixed ? 0.0 : passes * (cgMax + 1.0), mixed ? passes * (mgCap + 3.0) : 0.0, sweeps};
}
/// Microseconds that one outer iteration of a solve takes at most on R CTAs of T
/// threads, per cell of a thread where it streams. Measured at 768x192: an iteration
/// of the CG 4.6 us on 144 CTAs (2 cells a thread), in a full GPU 12 on 36, 30 on 24
/// and 88 on 12 (24 cells), bounded by 5 + 5 a cell; a V-cycle 38 us, by 200 + 20; the rows of
/// the sweeps 1.1 to 3.5 us each, by 5 + 5 a cell of the row for each of the six.
__host__ __device__ inline double outerBound(int NI, int NJ, int R, int T, const WideEffort& e) {
  const double cells = static_cast<double>(NI) * NJ / (static_cast<double>(R) * T) + 1.0;
  double us = 1000.0 + e.exchanges * (5.0 + 5.0 * cells) + e.cycles * (200.0 + 20.0 * cells);
  us += (50.0 + 2.0 * e.sweeps) * (2.0 + 2.0 * cells) + 6.0 * NJ * (10.0 + 5.0 * NI / T);
  if (e.cycles > 0.0) {  // as wavefronts of diagonals
    us += 6.0 * (static_cast<double>(NI) + NJ) * (2.0 + 2.0 * ((NI < NJ) ? NI : NJ) / T);
  }
  return us;
}
/// How long an overdue wait still waits behind `microseconds` of other work (its own
/// solve's phases, and the earlier solves of its team that it has no part in): two
/// seconds and four times that, in 2^20 ns.
__host__ __device__ inline int wideWaitLimit(double microseconds) {
  const double limit = 2000.0 + 4.0e-3 * microseconds;
  return (limit < 5e8) ? static_cast<int>(limit) : 500000000;
}

constexpr int kUnitBatch = 8;       // units of the CG whose partial sums are held at once
constexpr int kUnitWarps = 8;       // warps that share a unit
constexpr int kSumLine = 8;         // messages from one unit's sums to the next: a 128-byte line
constexpr int kSumCopies = 4;       // copies of every unit's sums, each polled by its share of the CTAs

struct WideShared {
  union {
    double chunkPart[kChunkBatch][kChunkCells / 32][kMaxSums];
    double groupPart[kMaxSums][256];
    double unitPart[kUnitBatch][kUnitWarps][4];
  };
  double warpPart[kWideThreads / 32][kRedSlots];
  double result[kRedSlots];
  double ahead;    // microseconds an iteration of the earlier solves of the CTA's list, at most
  int waitLimit;
  int fault;       // a wait of this CTA gave up
  unsigned never;  // stays 0: the wait tests' condition
};

struct WideTeam {
  int rank, R, tid, T;
  int NI, NJ, N;
  int chunks;            // of the block
  int chunk0, chunk1;    // own ones
  int c0, c1;            // own cells: whole chunks
  unsigned epoch;
  unsigned barriers;  // of this launch so far
  WideScratch mem;
  int* faultWord;
  WideShared* sh;
};

/// `iterations` of this solve, each of `outer` microseconds at most, behind as many
/// of the solves before it (sh->ahead).
DEV void wideJoin(WideTeam& t, const WideScratch& mem, int* faultWord, WideShared* sh, int rank, int R, int NI,
                  int NJ, int iterations, double outer) {
  t.rank = rank;
  t.R = R;
  t.tid = static_cast<int>(threadIdx.x);
  t.T = static_cast<int>(blockDim.x);
  t.NI = NI;
  t.NJ = NJ;
  t.N = NI * NJ;
  t.chunks = (t.N + kChunkCells - 1) / kChunkCells;
  t.chunk0 = static_cast<int>(static_cast<long long>(t.chunks) * rank / R);
  t.chunk1 = static_cast<int>(static_cast<long long>(t.chunks) * (rank + 1) / R);
  t.c0 = t.chunk0 * kChunkCells;
  t.c1 = min(t.chunk1 * kChunkCells, t.N);
  if (t.c0 > t.c1) t.c0 = t.c1;
  t.mem = mem;
  t.faultWord = faultWord;
  t.sh = sh;
  t.epoch = static_cast<unsigned>(*mem.epoch);
  t.barriers = 0u;
  __syncthreads();
  if (t.tid == 0) {
    sh->waitLimit = wideWaitLimit(outer + iterations * sh->ahead);
    sh->ahead += outer;
    sh->fault = 0;
    sh->never = 0u;
  }
  __syncthreads();
}

/// Keep the epoch for the next launch. After a launch that gave up, CTAs can
/// differ: the largest is kept. The last CTA to leave clears the barrier's count
/// (nobody waits for it any more).
DEV void wideLeave(WideTeam& t) {
  if (t.tid == 0) {
    const unsigned long long was = *t.mem.epoch;
    const unsigned moved = t.epoch - static_cast<unsigned>(was);
    if (moved < 0x80000000u) atomicMax(t.mem.epoch, was + moved);
    __threadfence();
    if (atomicAdd(t.mem.left, 1u) == static_cast<unsigned>(t.R) - 1u) {
      __threadfence();
      atomicExch(t.mem.arrived, 0u);
      atomicExch(t.mem.left, 0u);
    }
  }
}

/// An overdue wait: `polls` counted up to its number, from then on it holds the time
/// that was, below 0. The next `polls`, or 0 when the wait is given up.
DEV int wideOverdue(WideShared* sh, int* faultWord, int polls, int code) {
  constexpr int kLowest = -2147483647 - 1, kTime = (1 << 30) - 1;
  unsigned long long ns;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(ns));
  const int now = static_cast<int>(ns >> 20) & kTime;
  if (polls > 0) return kLowest + now;
  if (((now - (polls - 1 - kLowest)) & kTime) < *static_cast<volatile int*>(&sh->waitLimit)) return polls - 1;
  *static_cast<volatile int*>(&sh->fault) = 1;
  atomicOr(faultWord, code);
  return 0;
}
static __device__ __noinline__ int wideOverdueFar(WideShared* sh, int* faultWord, int polls, int code) {
  return wideOverdue(sh, faultWord, polls, code);
}
/// One more unsuccessful poll: true when the wait is over (given up now or before).
/// kFar: what an overdue wait does lies in a function of its own. The mixed form's
/// waits and the barrier are 1 % of an iteration faster so, the CG's 8 % slower
/// (192x48), whose registers a call would spill.
template <unsigned kPolls = static_cast<unsigned>(kWideSpinLimit), bool kFar = false>
DEV bool wideGiveUp(WideTeam& t, int& polls, int code) {
  if (*static_cast<volatile int*>(&t.sh->fault) != 0) return true;
  if (static_cast<unsigned>(++polls) < kPolls) return false;
  polls = kFar ? wideOverdueFar(t.sh, t.faultWord, polls, code) : wideOverdue(t.sh, t.faultWord, polls, code);
  return polls == 0;
}
DEV bool wideGiveUpFar(WideTeam& t, int& polls, int code) { return wideGiveUp<kWideSpinLimit, true>(t, polls, code); }

// ---- tagged messages ------------------------------------------------------------

DEV void messageStore(ulonglong2* slot, double v, unsigned tag) {
  const unsigned long long bits = static_cast<unsigned long long>(__double_as_longlong(v));
  const unsigned long long t = static_cast<unsigned long long>(tag) << 32;
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(slot), "l"(t | (bits & 0xffffffffull)),
               "l"(t | (bits >> 32))
               : "memory");
}
DEV ulonglong2 messageLoad(const ulonglong2* slot) {
  ulonglong2 m;
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(m.x), "=l"(m.y) : "l"(slot) : "memory");
  return m;
}
DEV bool messageReady(const ulonglong2& m, unsigned tag) {
  return static_cast<unsigned>(m.x >> 32) == tag && static_cast<unsigned>(m.y >> 32) == tag;
}
DEV double messageValue(const ulonglong2& m) {
  return __longlong_as_double(static_cast<long long>((m.x & 0xffffffffull) | (m.y << 32)));
}
/// Wait for the value of `slot` with this tag, given a first look at it.
DEV double messageWait(WideTeam& t, const ulonglong2* slot, ulonglong2 m, unsigned tag, int code) {
  int polls = 0;
  while (!messageReady(m, tag)) {
    if (wideGiveUp(t, polls, code)) return 0.0;
    m = messageLoad(slot);
  }
  return messageValue(m);
}
/// The value of a message; `code` is the fault of a wait that gives up.
DEV double messageWait(WideTeam& t, const ulonglong2* slot, unsigned tag, int code) {
  ulonglong2 m = messageLoad(slot);
  int polls = 0;
  while (!messageReady(m, tag)) {
    if (wideGiveUp(t, polls, code)) return 0.0;
    m = messageLoad(slot);
  }
  return messageValue(m);
}
/// The values of N messages set[from[k]] (-1: none), waited for together:
/// every look loads all that are still missing, so the wait ends one L2 round
/// trip after the last has arrived.
template <int N>
DEV void messageWaitAll(WideTeam& t, const ulonglong2* set, const int (&from)[N], unsigned tag, int code,
                        double (&value)[N]) {
  unsigned missing = 0;
#pragma unroll
  for (int k = 0; k < N; ++k) missing |= (from[k] >= 0) ? 1u << k : 0u;
  int polls = 0;
  while (missing != 0u) {
    ulonglong2 m[N];
#pragma unroll
    for (int k = 0; k < N; ++k) {
      if (missing & (1u << k)) m[k] = messageLoad(set + from[k]);
    }
#pragma unroll
    for (int k = 0; k < N; ++k) {
      if ((missing & (1u << k)) && messageReady(m[k], tag)) {
        missing &= ~(1u << k);
        value[k] = messageValue(m[k]);
      }
    }
    if (missing != 0u && wideGiveUp(t, polls, code)) break;
  }
}

// ---- barrier ----------------------------------------------------------------------

/// Every CTA's global writes before it are visible to every CTA after it. Each
/// CTA adds one to a count that its first thread then polls; the count starts at
/// 0 in every launch (wideLeave). The release orders the block's writes before
/// its arrival and the acquire the peers' before its reads. One poll a CTA: with
/// a flag per CTA, polled by as many threads, the 148 x 5 polls of the flags'
/// lines queue up behind one another and a barrier of 148 CTAs takes 4 to 5 us
/// (1.7 us of 36).
DEV void wideBarrier(WideTeam& t) {
  ++t.epoch;
  ++t.barriers;
  __syncthreads();
  if (t.R == 1) return;
  if (t.tid == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(t.mem.arrived) : "memory");
    const unsigned all = t.barriers * static_cast<unsigned>(t.R);
    int polls = 0;
    for (;;) {
      unsigned v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(t.mem.arrived) : "memory");
      if (static_cast<int>(v - all) >= 0) break;
      if (wideGiveUpFar(t, polls, kFaultTeamWait)) break;
    }
  }
  __syncthreads();
}

// ---- reductions ---------------------------------------------------------------------

/// Maximum of v[k] over every thread of the team, in every thread. Also a barrier.
template <int K>
DEV void wideMax(WideTeam& t, double (&v)[K]) {
  const int lane = t.tid & 31, warp = t.tid >> 5, warps = t.T >> 5;
#pragma unroll
  for (int k = 0; k < K; ++k) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v[k] = smax(v[k], __shfl_down_sync(0xffffffffu, v[k], off));
    if (lane == 0) t.sh->warpPart[warp][k] = v[k];
  }
  __syncthreads();
  double* slots = t.mem.slots + ((t.epoch + 1u) & 1u) * kMaxWideCtas * kRedSlots;
  if (t.tid < K) {
    double a = t.sh->warpPart[0][t.tid];
    for (int w = 1; w < warps; ++w) a = smax(a, t.sh->warpPart[w][t.tid]);
    slots[t.rank * kRedSlots + t.tid] = a;
  }
  wideBarrier(t);
  for (int k = warp; k < K; k += warps) {
    double a = -INFINITY;
    for (int r = lane; r < t.R; r += 32) a = smax(a, __ldcg(slots + r * kRedSlots + k));
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) a = smax(a, __shfl_down_sync(0xffffffffu, a, off));
    if (lane == 0) t.sh->result[k] = a;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < K; ++k) v[k] = t.sh->result[k];
}

/// The sum of a CG unit over its `warps` warps, once they have all been stored.
DEV double unitTotal(const WideTeam& t, int slot, int k, int warps) {
  double a[kUnitWarps];
#pragma unroll
  for (int w = 0; w < kUnitWarps; ++w) a[w] = (w < warps) ? t.sh->unitPart[slot][w][k] : 0.0;
  return ((a[0] + a[1]) + (a[2] + a[3])) + ((a[4] + a[5]) + (a[6] + a[7]));
}

/// f(c, i, j) for every own cell.
template <typename F>
DEV void wideCells(const WideTeam& t, F&& f) {
  for (int c = t.c0 + t.tid; c < t.c1; c += t.T) {
    const int j = c / t.NI;
    f(c, c - j * t.NI, j);
  }
}

/// Items 0 .. count-1 in chunks of 256, and this CTA's share of the chunks.
struct WideRange {
  int count, chunks, chunk0, chunk1;
};
DEV WideRange wideRange(const WideTeam& t, int count) {
  const int chunks = (count + kChunkCells - 1) / kChunkCells;
  return WideRange{count, chunks, static_cast<int>(static_cast<long long>(chunks) * t.rank / t.R),
                   static_cast<int>(static_cast<long long>(chunks) * (t.rank + 1) / t.R)};
}
/// f(m) for every own item.
template <typename F>
DEV void wideItems(const WideTeam& t, const WideRange& range, F&& f) {
  const int end = min(range.chunk1 * kChunkCells, range.count);
  for (int m = range.chunk0 * kChunkCells + t.tid; m < end; m += t.T) f(m);
}

/// item(m, acc) over every own item, adding to its chunk's sums; the team's
/// totals in every thread. Also a barrier. A chunk's sums are a tree over its
/// items, 32 chunks' a tree, and those are added in order. At most as many
/// items as the block has cells.
template <int K, typename F>
DEV void wideItemSums(WideTeam& t, const WideRange& range, double (&out)[K], F&& item) {
  const int lane = t.tid & 31, warp = t.tid >> 5, warps = t.T >> 5;
  const int team = min(t.T, kChunkCells), teams = t.T / team, mine = t.tid / team, lt = t.tid - mine * team;
  double* sums = t.mem.chunkSums + static_cast<std::size_t>((t.epoch + 1u) & 1u) * kMaxSums * t.chunks;
  for (int base = range.chunk0; base < range.chunk1; base += kChunkBatch) {
    const int n = min(range.chunk1 - base, kChunkBatch);
    for (int slot = mine; slot < n && mine < teams; slot += teams) {
      // the same 32 items share a warp's part whatever the number of threads
      for (int first = lt; first < kChunkCells; first += team) {
        const int m = (base + slot) * kChunkCells + first;
        double acc[K] = {};
        if (m < range.count) item(m, acc);
        __syncwarp();
#pragma unroll
        for (int k = 0; k < K; ++k) {
#pragma unroll
          for (int off = 16; off > 0; off >>= 1) acc[k] += __shfl_down_sync(0xffffffffu, acc[k], off);
          if (lane == 0) t.sh->chunkPart[slot][first >> 5][k] = acc[k];
        }
      }
    }
    __syncthreads();
    for (int m = t.tid; m < n * K; m += t.T) {
      const int slot = m / K, k = m - slot * K;
      double a[kChunkCells / 32];
#pragma unroll
      for (int w = 0; w < kChunkCells / 32; ++w) a[w] = t.sh->chunkPart[slot][w][k];
      sums[k * range.chunks + base + slot] = ((a[0] + a[1]) + (a[2] + a[3])) + ((a[4] + a[5]) + (a[6] + a[7]));
    }
    if (base + kChunkBatch < range.chunk1) __syncthreads();
  }
  wideBarrier(t);
  const int groups = (range.chunks + 31) / 32;
  double total[K] = {};
  for (int first = 0; first < groups; first += 256) {
    const int n = min(groups - first, 256);
    for (int m = warp; m < K * n; m += warps) {
      const int k = m / n, group = first + m - k * n, at = group * 32 + lane;
      double a = (at < range.chunks) ? __ldcg(sums + k * range.chunks + at) : 0.0;
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) a += __shfl_down_sync(0xffffffffu, a, off);
      if (lane == 0) t.sh->groupPart[k][group - first] = a;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < K; ++k) {
      for (int g = 0; g < n; ++g) total[k] += t.sh->groupPart[k][g];
    }
    __syncthreads();
  }
#pragma unroll
  for (int k = 0; k < K; ++k) out[k] = total[k];
}

/// The sums over every cell of the block, cell(c, i, j, acc).
template <int K, typename F>
DEV void wideSums(WideTeam& t, double (&out)[K], F&& cell) {
  wideItemSums(t, WideRange{t.N, t.chunks, t.chunk0, t.chunk1}, out, [&](int c, double (&acc)[K]) {
    const int j = c / t.NI;
    cell(c, c - j * t.NI, j, acc);
  });
}

}  // namespace cfdb
