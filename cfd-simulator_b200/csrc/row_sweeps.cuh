// row_sweeps.cuh - the plain form's k and omega Gauss-Seidel sweeps in the
// reference's cell order (LinearSystem.cpp:77-116), by a wide team.
//
// With row j-1 already swept and row j+1 and the east neighbours still old,
// the cell-order update of row j is the first-order recurrence
//   x_i = p_i + q_i x_(i-1),  p_i = (b_i - aN x_N - aE x_E - aS x_S) / aP,  q_i = -aW / aP,
// a composition of affine maps. The rows are a serial chain (192 of them at
// 768x192, three sweeps, two equations), so what counts is the time from one
// row to the next, and everything that does not depend on the row before is
// taken off it:
//   * the coefficients are divided by aP in the assembly, where every SM works,
//     and laid out in the order the lanes read them;
//   * a warp owns a chunk of 32 to 128 columns for all rows. It scans its own
//     part of the row with shuffles, and only then needs the value entering
//     from the chunk to its west, which passed it a tagged value through shared
//     memory: the chunks of one row form a wavefront, with no block barrier;
//   * the three sweeps of both equations run at once on six CTAs, each a few
//     rows behind the one it reads. Their values travel as tagged messages
//     (wide_team.cuh) in whole-grid buffers, so no stage ever waits for the
//     stage it feeds;
//   * a row's coefficients arrive in shared memory by asynchronous copies
//     issued kSweepDepth rows ahead, the previous sweep's values in registers
//     three rows ahead.
// A row took 3.5 us as a block-wide scan of one CTA with a barrier on either
// side.
//
// Row 0 is split at NI/2: the wake-cut partner (NI-1-i, 0) of (i, 0) comes later
// in the row for i < NI/2 (old value) and earlier for i >= NI/2 (new value). A
// cell with aP = 0 keeps its value. The chunks depend on NI alone, so the bits
// do not depend on how many CTAs or warps share the work.
#pragma once

#include "wide_team.cuh"

namespace cfdb {

constexpr int kSweeps = 3;      // KOmegaSST.cpp:469-512: three sweeps of each equation
constexpr int kSweepDepth = 4;  // rows whose coefficients are on their way
constexpr int kAhead = 3;       // rows whose old values are on their way

struct RowSweepShape {
  int per, width, chunks, padded;  // cells per lane, columns per chunk, chunks, columns with padding
  int edges;                       // rows whose chunk edges are kept on chip
};
/// Shared memory of one sweep at most: what a wide kernel has (kMaxWideSmem).
constexpr int kMaxSweepBytes = 222032;
__host__ __device__ inline RowSweepShape rowSweepShape(int NI) {
  RowSweepShape s;
  s.per = (NI + 255) / 256;
  if (s.per > 4) s.per = 4;
  s.width = 32 * s.per;
  s.chunks = (NI + s.width - 1) / s.width;
  s.padded = s.chunks * s.width;
  s.edges = (s.chunks <= 16) ? 64 : 16;
  // more than 816 chunks (104,448 columns): not on chip at all, a chunk's west
  // value is then its west neighbour's message (rowSweep)
  if (s.chunks > kMaxSweepBytes / (s.edges * 16 + 16)) s.edges = 0;
  return s;
}
/// Place of column i in a row of the packed layouts: lane-contiguous cells,
/// stored so that a warp reads 32 consecutive values per cell of a lane.
__host__ __device__ inline int rowSweepPlace(const RowSweepShape& s, int i) {
  const int chunk = i / s.width, r = i - chunk * s.width;
  return chunk * s.width + (r % s.per) * 32 + r / s.per;
}
/// Doubles of one equation's packed coefficients, messages of its values.
__host__ __device__ inline long long rowSweepCoefficients(int NI, int NJ) {
  return 5LL * rowSweepShape(NI).padded * NJ;
}
__host__ __device__ inline long long rowSweepMessages(int NI, int NJ) {
  return static_cast<long long>(kSweeps + 1) * rowSweepShape(NI).padded * NJ;
}
/// Shared memory of one sweep: the chunks' edges and progress.
__host__ __device__ inline int rowSweepBytes(const RowSweepShape& s) {
  return (s.edges > 0) ? s.chunks * (s.edges * 16 + 16) : 0;
}
/// And with the coefficients of kSweepDepth rows of every chunk.
__host__ __device__ inline int rowSweepRingBytes(const RowSweepShape& s) {
  return rowSweepBytes(s) + s.chunks * kSweepDepth * 5 * s.width * 8;
}

/// One equation in the packed layouts.
struct RowSweepSystem {
  const double* c;      // b, aS, aE, aN, -aW over aP: [row][chunk][5][width]
  ulonglong2* values;   // [kSweeps + 1][row][padded]: the start, and what each sweep leaves
  double* x;            // the unknowns, natural order
};

DEV void rowSweepStoreRow(const RowSweepSystem& y, const RowSweepShape& z, int NI, int i, int j, double diag,
                          const double (&off)[4], double b, double x, unsigned tag) {
  const int place = rowSweepPlace(z, i), chunk = i / z.width;
  double* c = const_cast<double*>(y.c) + (static_cast<long long>(j) * z.chunks + chunk) * 5 * z.width +
              (place - chunk * z.width);
  const bool solve = fabs(diag) > 0.0;
  c[0] = solve ? b / diag : x;
  c[z.width] = solve ? off[0] / diag : 0.0;
  c[2 * z.width] = solve ? off[3] / diag : 0.0;
  c[3 * z.width] = solve ? off[1] / diag : 0.0;
  c[4 * z.width] = (solve && i > 0) ? -off[2] / diag : 0.0;
  messageStore(y.values + static_cast<long long>(j) * z.padded + place, x, tag);
}

/// Polls of shared memory after which a wait is overdue: eight and more to one of L2.
constexpr unsigned kEdgePolls = 1u << 24;

/// A chunk's last value of a row, tagged j + 1, in shared memory.
DEV void edgeStore(volatile unsigned long long* slot, double v, unsigned tag) {
  const unsigned long long bits = static_cast<unsigned long long>(__double_as_longlong(v));
  const unsigned long long t = static_cast<unsigned long long>(tag) << 32;
  slot[0] = t | (bits & 0xffffffffull);
  slot[1] = t | (bits >> 32);
}
DEV double edgeWait(WideTeam& t, volatile unsigned long long* slot, unsigned tag) {
  int polls = 0;
  for (;;) {
    const unsigned long long a = slot[0], b = slot[1];
    if (static_cast<unsigned>(a >> 32) == tag && static_cast<unsigned>(b >> 32) == tag) {
      return __longlong_as_double(static_cast<long long>((a & 0xffffffffull) | (b << 32)));
    }
    if (wideGiveUp<kEdgePolls>(t, polls, kFaultChainWait)) return 0.0;
  }
}

/// Wait until the next chunk has taken the edges of `rows` rows.
DEV void edgeRoom(WideTeam& t, volatile int* progress, int rows) {
  int polls = 0;
  while (*progress < rows) {
    if (wideGiveUp<kEdgePolls>(t, polls, kFaultChainWait)) return;
  }
}

/// One sweep's chunk in flight: what a warp carries from row to row.
template <int PER>
struct ChunkRow {
  double p[PER], q[PER];      // the row's affine maps, cell by cell of the lane
  double x[PER];              // its new values
};

/// Solve the chunk's part of a row from its maps: scan, then the value from the
/// west; the chunk's last value comes back in every lane. `active` bit e: cell e
/// takes part (others are skipped and keep x).
template <int PER>
DEV double chunkSolve(ChunkRow<PER>& c, unsigned active, double west) {
  const int lane = threadIdx.x & 31;
  double P = 0.0, Q = 1.0;
#pragma unroll
  for (int e = 0; e < PER; ++e) {
    if (active & (1u << e)) {
      P = fma(c.q[e], P, c.p[e]);
      Q = c.q[e] * Q;
    }
  }
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const double pp = __shfl_up_sync(0xffffffffu, P, off), qq = __shfl_up_sync(0xffffffffu, Q, off);
    if (lane >= off) {
      P = fma(Q, pp, P);
      Q = Q * qq;
    }
  }
  double before = __shfl_up_sync(0xffffffffu, P, 1), scale = __shfl_up_sync(0xffffffffu, Q, 1);
  if (lane == 0) {
    before = 0.0;
    scale = 1.0;
  }
  double x = fma(scale, west, before);
#pragma unroll
  for (int e = 0; e < PER; ++e) {
    if (active & (1u << e)) {
      x = fma(c.q[e], x, c.p[e]);
      c.x[e] = x;
    }
  }
  return fma(__shfl_sync(0xffffffffu, Q, 31), west, __shfl_sync(0xffffffffu, P, 31));
}

DEV void copyAsync16(double* to, const double* from) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(static_cast<unsigned>(__cvta_generic_to_shared(to))),
               "l"(from)
               : "memory");
}

/// Sweep s of one equation by the `warps` warps from this thread's slot on
/// (warp `w` of them). kRing: a warp has one chunk, its coefficients arrive by
/// asynchronous copies; else a warp has every warps-th chunk and loads as it goes.
/// kOnChip: the chunks' edges are kept on chip (RowSweepShape::edges).
template <int PER, bool kRing, bool kOnChip>
__device__ __noinline__ void rowSweep(const Instance& I, const WideTeam& team, const RowSweepSystem& system, int s,
                                      unsigned tag, int w, int warps, char* smem) {
  WideTeam t = team;
  const RowSweepSystem y = system;
  const RowSweepShape z = rowSweepShape(I.NI);
  const int NI = I.NI, NJ = I.NJ, lane = threadIdx.x & 31;
  const int half = NI / 2;
  volatile unsigned long long* edges = reinterpret_cast<unsigned long long*>(smem);
  volatile int* progress = reinterpret_cast<int*>(smem + z.chunks * z.edges * 16);
  const ulonglong2* in = y.values + static_cast<long long>(s) * NJ * z.padded;
  ulonglong2* out = y.values + static_cast<long long>(s + 1) * NJ * z.padded;
  const long long rowCoefs = static_cast<long long>(z.chunks) * 5 * z.width;
  double* ring = reinterpret_cast<double*>(smem + rowSweepBytes(z)) + w * kSweepDepth * 5 * z.width;

  // the previous sweep's value at (row j, place), cell `i` of the row
  auto value = [&](int j, int place, bool exists, const ulonglong2& first) {
    if (!exists) return 0.0;
    const ulonglong2* slot = in + static_cast<long long>(j) * z.padded + place;
    ulonglong2 m = first;
    int polls = 0;
    while (!messageReady(m, tag)) {
      if (wideGiveUp(t, polls, kFaultChainWait)) return 0.0;
      m = messageLoad(slot);
    }
    return messageValue(m);
  };
  auto look = [&](int j, int place, bool exists) {
    return (exists && j < NJ) ? messageLoad(in + static_cast<long long>(j) * z.padded + place) : ulonglong2{0, 0};
  };

  // Where no edges are kept, the value that enters a chunk's part of a row: its west
  // neighbour's last message.
  auto neighbour = [&](int chunk, int j) {
    const ulonglong2* slot = out + static_cast<long long>(j) * z.padded + rowSweepPlace(z, chunk * z.width - 1);
    return messageWait(t, slot, tag, kFaultChainWait);
  };
  // What a row leaves: progress, its values, and at the last sweep the unknowns.
  auto finish = [&](int chunk, int j, unsigned exists, const double (&x)[PER]) {
    // every lane has the value from the west: its place may be used again
    __syncwarp();
    if (kOnChip && lane == 0) progress[chunk] = j + 1;
    const long long at = static_cast<long long>(j) * z.padded + chunk * z.width + lane;
    const long long cell = static_cast<long long>(j) * NI + chunk * z.width + lane * PER;
#pragma unroll
    for (int e = 0; e < PER; ++e) {
      if (!((exists >> e) & 1u)) continue;
      if (!kRing || s + 1 < kSweeps || j == 0) messageStore(out + at + e * 32, x[e], tag);
      if (s + 1 == kSweeps) y.x[cell + e] = x[e];
    }
  };
  // The part of a row's maps that no new value enters, from its coefficients
  // (lane-strided) and the old values: base, aS, q.
  auto maps = [&](const double* co, const double (&old)[PER], double oldEast, const double (&north)[PER],
                  double (&base)[PER], double (&cs)[PER], double (&q)[PER]) {
#pragma unroll
    for (int e = 0; e < PER; ++e) {
      const double east = (e + 1 < PER) ? old[(e + 1 < PER) ? e + 1 : e] : oldEast;
      const double b = co[e * 32 + lane], ce = co[2 * z.width + e * 32 + lane], cn = co[3 * z.width + e * 32 + lane];
      cs[e] = co[z.width + e * 32 + lane];
      q[e] = co[4 * z.width + e * 32 + lane];
      base[e] = fma(-cn, north[e], fma(-ce, east, b));
    }
  };
  // A row after the first: x from the row before (south) and the west.
  auto row = [&](int chunk, int j, const double* co, const double (&old)[PER], double oldEast,
                 const double (&north)[PER], const double (&south)[PER], double (&x)[PER]) {
    double p[PER], cs[PER], q[PER];
    maps(co, old, oldEast, north, p, cs, q);
    double P = 0.0, Q = 1.0;
#pragma unroll
    for (int e = 0; e < PER; ++e) {
      p[e] = fma(-cs[e], south[e], p[e]);
      P = fma(q[e], P, p[e]);
      Q = q[e] * Q;
    }
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const double pp = __shfl_up_sync(0xffffffffu, P, off), qq = __shfl_up_sync(0xffffffffu, Q, off);
      if (lane >= off) {
        P = fma(Q, pp, P);
        Q = Q * qq;
      }
    }
    double before = __shfl_up_sync(0xffffffffu, P, 1), scale = __shfl_up_sync(0xffffffffu, Q, 1);
    if (lane == 0) {
      before = 0.0;
      scale = 1.0;
    }
    double x0;
    if constexpr (kOnChip) {
      volatile unsigned long long* mine = edges + (chunk * z.edges + j % z.edges) * 2;
      x0 = (chunk > 0) ? edgeWait(t, mine - 2 * z.edges, static_cast<unsigned>(j) + 1u) : 0.0;
      if (lane == 31 && chunk + 1 < z.chunks) {
        if (j >= z.edges) edgeRoom(t, progress + chunk + 1, j - z.edges + 1);
        edgeStore(mine, fma(Q, x0, P), static_cast<unsigned>(j) + 1u);  // the chunk's last value
      }
    } else {
      x0 = (chunk > 0) ? neighbour(chunk, j) : 0.0;
    }
    double v = fma(scale, x0, before);
    unsigned exists = 0;
#pragma unroll
    for (int e = 0; e < PER; ++e) {
      v = fma(q[e], v, p[e]);
      const bool there = chunk * z.width + lane * PER + e < NI;
      x[e] = there ? v : 0.0;
      exists |= there ? 1u << e : 0u;
    }
    finish(chunk, j, exists, x);
  };
  // Row 0, in two halves: a wake partner's value is this sweep's where it lies
  // to the west (the first half), else the previous sweep's.
  auto row0 = [&](int chunk, const double* co, const double (&old)[PER], double oldEast, const double (&north)[PER],
                  double (&x)[PER]) {
    const int i0 = chunk * z.width + lane * PER;
    ChunkRow<PER> c;
    double base[PER], cs[PER];
    maps(co, old, oldEast, north, base, cs, c.q);
    unsigned exists = 0;
#pragma unroll
    for (int e = 0; e < PER; ++e) exists |= (i0 + e < NI) ? 1u << e : 0u;
    volatile unsigned long long* mine = edges + chunk * z.edges * 2;
    double x0 = 0.0;
    if (chunk > 0) x0 = kOnChip ? edgeWait(t, mine - 2 * z.edges, 1u) : neighbour(chunk, 0);
    double last = 0.0;
    for (int part = 0; part < 2; ++part) {
      const int from = part ? half : 0, to = part ? NI : half;
      if (chunk * z.width >= to || (chunk + 1) * z.width <= from) continue;
      unsigned active = 0;
#pragma unroll
      for (int e = 0; e < PER; ++e) {
        const int i = i0 + e;
        if (i < from || i >= to) continue;
        active |= 1u << e;
        const int a = I.acrossJ0[i];
        double partner = 0.0;
        if (a >= 0) {
          const int place = rowSweepPlace(z, a);
          const ulonglong2* slot = ((a < i) ? out : in) + place;
          ulonglong2 m = messageLoad(slot);
          int polls = 0;
          while (!messageReady(m, tag) && !wideGiveUp(t, polls, kFaultChainWait)) m = messageLoad(slot);
          partner = messageValue(m);
        }
        c.p[e] = fma(-cs[e], partner, base[e]);
      }
      __syncwarp();
      x0 = last = chunkSolve<PER>(c, active, x0);
      if (part == 0) {
#pragma unroll
        for (int e = 0; e < PER; ++e) {
          if (active & (1u << e)) messageStore(out + chunk * z.width + e * 32 + lane, c.x[e], tag);
        }
      }
    }
    if (kOnChip && lane == 31 && chunk + 1 < z.chunks) edgeStore(mine, last, 1u);
#pragma unroll
    for (int e = 0; e < PER; ++e) x[e] = ((exists >> e) & 1u) ? c.x[e] : 0.0;
    finish(chunk, 0, exists, x);
  };

  if constexpr (kRing) {
    const int chunk = w;
    if (chunk >= z.chunks) return;
    const int i0 = chunk * z.width + lane * PER, place = chunk * z.width + lane;
    const bool hasEast = lane == 31 && (chunk + 1) * z.width < NI;
    const int eastPlace = (chunk + 1) * z.width;  // the next chunk's first cell
    const double* co = y.c + static_cast<long long>(chunk) * 5 * z.width;
    auto fetch = [&](int j) {
      if (j < NJ) {
        double* to = ring + (j % kSweepDepth) * 5 * z.width;
        const double* from = co + j * rowCoefs;
        for (int m = lane; m < 5 * z.width / 2; m += 32) copyAsync16(to + 2 * m, from + 2 * m);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int j = 0; j < kSweepDepth - 1; ++j) fetch(j);
    double old[PER], north[PER], south[PER];
    // messages on their way, kAhead rows of them; the loop below is unrolled by
    // kAhead so that each stays in the register it was loaded into
    ulonglong2 ahead[kAhead][PER], aheadEast[kAhead];
#pragma unroll
    for (int e = 0; e < PER; ++e) old[e] = value(0, place + e * 32, i0 + e < NI, look(0, place + e * 32, i0 + e < NI));
    double east = value(0, eastPlace, hasEast, look(0, eastPlace, hasEast));
#pragma unroll
    for (int d = 0; d < kAhead; ++d) {
#pragma unroll
      for (int e = 0; e < PER; ++e) ahead[d][e] = look(1 + d, place + e * 32, i0 + e < NI);
      aheadEast[d] = look(1 + d, eastPlace, hasEast);
    }
    auto step = [&](int j, ulonglong2 (&next)[PER], ulonglong2& nextE, bool first) {
#pragma unroll
      for (int e = 0; e < PER; ++e) north[e] = value(j + 1, place + e * 32, i0 + e < NI && j + 1 < NJ, next[e]);
      const double nextEast = value(j + 1, eastPlace, hasEast && j + 1 < NJ, nextE);
      asm volatile("cp.async.wait_group %0;" ::"n"(kSweepDepth - 2) : "memory");
      __syncwarp();
#pragma unroll
      for (int e = 0; e < PER; ++e) next[e] = look(j + 1 + kAhead, place + e * 32, i0 + e < NI);
      nextE = look(j + 1 + kAhead, eastPlace, hasEast);
      fetch(j + kSweepDepth - 1);  // into the slot whose row is done
      double oldEast = __shfl_down_sync(0xffffffffu, old[0], 1);
      if (lane == 31) oldEast = east;
      const double* const c = ring + (j % kSweepDepth) * 5 * z.width;
      if (first) row0(chunk, c, old, oldEast, north, south);
      else row(chunk, j, c, old, oldEast, north, south, south);
#pragma unroll
      for (int e = 0; e < PER; ++e) old[e] = north[e];
      east = nextEast;
    };
    step(0, ahead[0], aheadEast[0], true);
    for (int j0 = 1; j0 < NJ; j0 += kAhead) {
#pragma unroll
      for (int d = 0; d < kAhead; ++d) {
        if (j0 + d < NJ) step(j0 + d, ahead[(1 + d) % kAhead], aheadEast[(1 + d) % kAhead], false);
      }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
  } else {
    double x[PER];
    for (int j = 0; j < NJ; ++j) {
      for (int chunk = w; chunk < z.chunks; chunk += warps) {
        const int i0 = chunk * z.width + lane * PER, place = chunk * z.width + lane;
        const bool hasEast = lane == 31 && (chunk + 1) * z.width < NI;
        const int eastPlace = (chunk + 1) * z.width;
        double old[PER], north[PER], south[PER];
#pragma unroll
        for (int e = 0; e < PER; ++e) {
          const bool have = i0 + e < NI;
          const int at = place + e * 32;
          const ulonglong2 a = look(j, at, have), b = look(j + 1, at, have);
          south[e] = 0.0;
          if (j > 0 && have) {
            // this lane's own value of the row before
            const ulonglong2* slot = out + static_cast<long long>(j - 1) * z.padded + at;
            ulonglong2 m = messageLoad(slot);
            int polls = 0;
            while (!messageReady(m, tag) && !wideGiveUp(t, polls, kFaultChainWait)) m = messageLoad(slot);
            south[e] = messageValue(m);
          }
          old[e] = value(j, at, have, a);
          north[e] = value(j + 1, at, have && j + 1 < NJ, b);
        }
        const double east = value(j, eastPlace, hasEast, look(j, eastPlace, hasEast));
        __syncwarp();
        double oldEast = __shfl_down_sync(0xffffffffu, old[0], 1);
        if (lane == 31) oldEast = east;
        const double* const c = y.c + j * rowCoefs + static_cast<long long>(chunk) * 5 * z.width;
        if (j == 0) row0(chunk, c, old, oldEast, north, x);
        else row(chunk, j, c, old, oldEast, north, south, x);
        __syncwarp();
      }
    }
  }
}

template <bool kRing>
DEV void rowSweepAny(const Instance& I, const WideTeam& t, const RowSweepSystem& y, int s, unsigned tag, int w, int warps,
                     char* smem) {
  const RowSweepShape z = rowSweepShape(I.NI);
  switch (z.per) {
    case 1: rowSweep<1, kRing, true>(I, t, y, s, tag, w, warps, smem); break;
    case 2: rowSweep<2, kRing, true>(I, t, y, s, tag, w, warps, smem); break;
    case 3: rowSweep<3, kRing, true>(I, t, y, s, tag, w, warps, smem); break;
    default:
      if (kRing || z.edges > 0) rowSweep<4, kRing, true>(I, t, y, s, tag, w, warps, smem);
      else rowSweep<4, false, false>(I, t, y, s, tag, w, warps, smem);
      break;
  }
}

/// The six sweeps (equation, sweep) of the team: one per CTA where it has six,
/// else several at once on a CTA's warps. The caller ends with a barrier. With
/// `onlySweep` >= 0 only that sweep of both equations runs (tests: one after
/// another). `waitTest`: the second sweep also waits for a count nothing sets.
DEV void rowSweeps(const Instance& I, WideTeam& t, const RowSweepSystem (&systems)[2], unsigned tag, int onlySweep,
                   bool waitTest, char* smem, int smemBytes) {
  const RowSweepShape z = rowSweepShape(I.NI);
  const int units = 2 * kSweeps, perCta = (units + t.R - 1) / t.R, first = t.rank * perCta;
  if (first >= units) return;
  const int warps = t.T >> 5, warp = t.tid >> 5;
  const bool ring = perCta == 1 && warps >= z.chunks && rowSweepRingBytes(z) <= smemBytes;
  const int region = rowSweepBytes(z);
  int slots = min(perCta, warps);
  while (slots > 1 && slots * region > smemBytes) --slots;
  const int slotWarps = warps / slots, slot = warp / slotWarps;
  if (waitTest) {
    if (t.tid == 0 && first <= 1 && 1 < first + perCta) {
      int polls = 0;
      while (*static_cast<volatile unsigned*>(&t.sh->never) == 0u && ++polls < (1 << 24)) {
      }
      if (polls >= (1 << 24)) atomicOr(t.faultWord, kFaultChainWait);
    }
    __syncthreads();
  }
  for (int base = first; base < min(first + perCta, units); base += slots) {
    // edges and progress cleared, whatever the memory held
    __syncthreads();
    for (int m = t.tid; m < slots * region / 4; m += t.T) reinterpret_cast<int*>(smem)[m] = 0;
    __syncthreads();
    const int unit = base + slot;
    if (slot < slots && unit < min(first + perCta, units) && (onlySweep < 0 || unit % kSweeps == onlySweep)) {
      char* mine = smem + slot * region;
      const RowSweepSystem& y = systems[unit / kSweeps];
      const int w = warp - slot * slotWarps;
      if (ring) rowSweepAny<true>(I, t, y, unit % kSweeps, tag, w, slotWarps, mine);
      else rowSweepAny<false>(I, t, y, unit % kSweeps, tag, w, slotWarps, mine);
    }
  }
}

}  // namespace cfdb
