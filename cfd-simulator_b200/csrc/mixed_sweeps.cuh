// mixed_sweeps.cuh - the mixed form's k and omega sweeps: FP32 corrections to
// the FP64 unknowns, in the reference's cell order (LinearSystem.cpp:77-116).
//
// A row of a sweep is a first-order recurrence solved by a scan over one CTA's
// threads (gsRowSolve below says which); the rows are a serial chain, so what
// counts is the time from one row to the next. rowChain runs the three sweeps
// of both equations at once on six CTAs, each a few rows behind the one it
// reads, with everything off the chain that does not depend on the row before:
// the coefficients come by asynchronous copies kChainDepth rows ahead, the
// previous sweep's values as tagged messages (value and tag in one 64-bit word)
// loaded kChainAhead rows ahead, the row below from the thread's own registers.
// What is left is the scan, with one barrier in it: every warp composes the
// warps' totals for itself.
#pragma once

#include "phases.cuh"
#include "wide_team.cuh"

namespace cfdb {
namespace {

/// Lexicographic Gauss-Seidel, executed as wavefronts: cells with i + j = d
/// for d = 0, 1, ... Within a wavefront no cell depends on another; every
/// cell sees its S and W neighbours already updated and its N and E
/// neighbours not yet, exactly as in cell-index order. Across the wake cut,
/// the partner (NI-1-i, 0) of (i, 0) lies on an earlier wavefront exactly when
/// its cell index is smaller, so that coupling is reproduced too. The result
/// is the reference's sweep (LinearSystem.cpp:77-116) to the last bit.
///
/// One CTA runs one system: rank 0 sweeps x1, rank 1 (or rank 0 again when
/// the team has one CTA) sweeps x2. The caller ends with a barrier.
DEV void gsWavefrontSweeps(const Instance& I, const WideTeam& t, int sweeps, const double* D,
                           const double* cS, const double* cN, const double* cW,
                           const double* cE, const double* b1, double* x1, const double* D2,
                           const double* cS2, const double* cN2, const double* cW2,
                           const double* cE2, const double* b2, double* x2) {
  const bool one = (t.R == 1);
  if (!one && t.rank > 1) return;
  const int fronts = I.NI + I.NJ - 1;
  for (int sweep = 0; sweep < sweeps; ++sweep) {
    for (int d = 0; d < fronts; ++d) {
      const int jLo = (d - (I.NI - 1) > 0) ? d - (I.NI - 1) : 0;
      const int jHi = (d < I.NJ - 1) ? d : I.NJ - 1;
      const int count = jHi - jLo + 1;
      const int work = one ? 2 * count : count;
      for (int k = t.tid; k < work; k += t.T) {
        const bool second = one ? (k >= count) : (t.rank == 1);
        const int j = jLo + (one ? (k % count) : k);
        const int i = d - j;
        const int c = j * I.NI + i;
        const double* Dv = second ? D2 : D;
        const double dd = Dv[c];
        if (!(fabs(dd) > 0.0)) continue;
        const double* aS = second ? cS2 : cS;
        const double* aN = second ? cN2 : cN;
        const double* aW = second ? cW2 : cW;
        const double* aE = second ? cE2 : cE;
        double* x = second ? x2 : x1;
        const double* b = second ? b2 : b1;
        const int nS = across(I, c, i, j, 0), nE = across(I, c, i, j, 3);
        const int nN = across(I, c, i, j, 1), nW = across(I, c, i, j, 2);
        double off = 0.0;
        if (nS >= 0) off += aS[c] * x[nS];
        if (nE >= 0) off += aE[c] * x[nE];
        if (nN >= 0) off += aN[c] * x[nN];
        if (nW >= 0) off += aW[c] * x[nW];
        x[c] = (b[c] - off) / dd;
      }
      __syncthreads();
    }
  }
}

/// Block-wide exclusive scan of affine maps x -> p + q x composed in thread
/// order: each thread passes the composition (p, q) of its own elements
/// (identity (0, 1) if none) and receives the composition of all elements of
/// lower threads. Uses sc[0 .. 2*warps) of shared memory; two __syncthreads.
template <typename T>
DEV void blockAffineExclusiveScan(T& p, T& q, T* sc) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nwarps = (blockDim.x + 31) >> 5;
  // inclusive scan within the warp (later maps applied after earlier ones)
  T ip = p, iq = q;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const T pp = __shfl_up_sync(0xffffffffu, ip, off);
    const T qq = __shfl_up_sync(0xffffffffu, iq, off);
    if (lane >= off) {
      ip = ip + iq * pp;
      iq = iq * qq;
    }
  }
  // exclusive within the warp
  T ep = __shfl_up_sync(0xffffffffu, ip, 1);
  T eq = __shfl_up_sync(0xffffffffu, iq, 1);
  if (lane == 0) {
    ep = T(0);
    eq = T(1);
  }
  if (lane == 31) {
    sc[2 * warp] = ip;
    sc[2 * warp + 1] = iq;
  }
  __syncthreads();
  if (warp == 0) {
    T wp = (lane < nwarps) ? sc[2 * lane] : T(0);
    T wq = (lane < nwarps) ? sc[2 * lane + 1] : T(1);
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const T pp = __shfl_up_sync(0xffffffffu, wp, off);
      const T qq = __shfl_up_sync(0xffffffffu, wq, off);
      if (lane >= off) {
        wp = wp + wq * pp;
        wq = wq * qq;
      }
    }
    T xp = __shfl_up_sync(0xffffffffu, wp, 1);
    T xq = __shfl_up_sync(0xffffffffu, wq, 1);
    if (lane == 0) {
      xp = T(0);
      xq = T(1);
    }
    if (lane < nwarps) {
      sc[2 * lane] = xp;
      sc[2 * lane + 1] = xq;
    }
  }
  __syncthreads();
  // earlier warps first, then the earlier lanes of this warp
  const T wp = sc[2 * warp], wq = sc[2 * warp + 1];
  p = ep + eq * wp;
  q = eq * wq;
}

/// One row of a lexicographic Gauss-Seidel sweep (LinearSystem.cpp:77-116).
/// With row j-1 already updated and row j+1 and the east neighbours still
/// holding their old values, the cell-order update of row j is the
/// first-order recurrence x_i = p_i + q_i x_{i-1},
///   p_i = (b_i - aS x_S - aE x_E - aN x_N) / a_P,  q_i = -aW / a_P,
/// solved by a block-wide scan. Row 0 is split in two: the wake-cut partner
/// (NI-1-i, 0) of (i, 0) comes later in the row for i < NI/2 (old value) and
/// earlier for i >= NI/2 (new value), so the second half is solved after the
/// first. A cell with a_P = 0 keeps its value (p = x, q = 0). This is the
/// reference's sweep map; only the rounding differs from cell-by-cell order.
///
/// Run by every thread of one CTA; rowPrev holds row j-1's new values,
/// oldRow and northRow rows j and j+1 as the previous sweep left them (the
/// unknowns themselves, or a copy). Needs NI <= 8 * blockDim.x. Leaves row
/// j's new values in rowNew and ends with a barrier; the caller publishes.
template <typename T>
struct SysView {
  const T *D, *S, *N, *W, *E, *b;
  T* x;
};

/// The row solve for any cells per thread (up to 8), loading as it goes.
template <typename T>
DEV void gsRowSolveAny(const Instance& I, int j, const SysView<T>& y, const T* oldRow, const T* northRow, T* rowNew,
                       const T* rowPrev, T* sc) {
  const T *D = y.D, *cS = y.S, *cN = y.N, *cW = y.W, *cE = y.E, *b = y.b;
  const int NI = I.NI, NJ = I.NJ;
  const int nt = blockDim.x;
  const int per = (NI + nt - 1) / nt;  // contiguous cells per thread
  const int i0 = threadIdx.x * per;
  const int segments = (j == 0) ? 2 : 1;
  T carry = T(0);
  for (int seg = 0; seg < segments; ++seg) {
    const int lo = (segments == 1) ? 0 : (seg == 0 ? 0 : NI / 2);
    const int hi = (segments == 1) ? NI : (seg == 0 ? NI / 2 : NI);
    T pv[8], qv[8];
    T P = T(0), Q = T(1);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      pv[e] = T(0);
      qv[e] = T(1);
      const int i = i0 + e;
      if (e >= per || i < lo || i >= hi) continue;
      const int c = j * NI + i;
      const T d = D[c];
      if (!(fabs(d) > T(0))) {
        pv[e] = oldRow[i];
        qv[e] = T(0);
      } else {
        T off = T(0);
        if (j > 0) {
          off += cS[c] * rowPrev[i];
        } else {
          const int a = I.acrossJ0[i];
          if (a >= 0) off += cS[c] * ((a < i) ? rowNew[a] : oldRow[a]);
        }
        if (i < NI - 1) off += cE[c] * oldRow[i + 1];
        if (j < NJ - 1) off += cN[c] * northRow[i];
        pv[e] = (b[c] - off) / d;
        qv[e] = (i > 0) ? -cW[c] / d : T(0);
      }
      P = pv[e] + qv[e] * P;
      Q = qv[e] * Q;
    }
    blockAffineExclusiveScan(P, Q, sc);
    T xv = P + Q * carry;  // value entering this thread's chunk
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int i = i0 + e;
      if (e >= per || i < lo || i >= hi) continue;
      xv = pv[e] + qv[e] * xv;
      rowNew[i] = xv;
    }
    __syncthreads();
    if (hi > lo) carry = rowNew[hi - 1];
  }
}

/// The row solve for at most MAXPER cells per thread. Every operand of the
/// thread's cells is loaded before any is used (indices clamped into the row;
/// values of cells outside it are never used), so the loads overlap instead
/// of waiting behind the branch on the diagonal.
template <typename T, int MAXPER>
DEV void gsRowSolveN(const Instance& I, int j, const SysView<T>& y, const T* oldRow, const T* northRow, T* rowNew,
                     const T* rowPrev, T* sc) {
  const T* __restrict__ D = y.D;
  const T* __restrict__ cS = y.S;
  const T* __restrict__ cN = y.N;
  const T* __restrict__ cW = y.W;
  const T* __restrict__ cE = y.E;
  const T* __restrict__ b = y.b;
  const int NI = I.NI, NJ = I.NJ;
  const int nt = blockDim.x;
  const int per = (NI + nt - 1) / nt;  // contiguous cells per thread
  const int i0 = threadIdx.x * per;
  const bool hasNorth = j < NJ - 1;
  const long long rowBase = static_cast<long long>(j) * NI;
  T dv[MAXPER], sv[MAXPER], ev[MAXPER], nv[MAXPER], wv[MAXPER], bv[MAXPER];
  T oldI[MAXPER], oldE[MAXPER], northI[MAXPER], prevI[MAXPER];
  int wake[MAXPER];
#pragma unroll
  for (int e = 0; e < MAXPER; ++e) {
    const int i = min(i0 + e, NI - 1);
    const long long c = rowBase + i;
    dv[e] = D[c];
    sv[e] = cS[c];
    ev[e] = cE[c];
    nv[e] = cN[c];
    wv[e] = cW[c];
    bv[e] = b[c];
    oldI[e] = oldRow[i];
    oldE[e] = oldRow[min(i + 1, NI - 1)];
    northI[e] = hasNorth ? northRow[i] : T(0);
    prevI[e] = (j > 0) ? rowPrev[i] : T(0);
    wake[e] = (j == 0) ? I.acrossJ0[i] : -1;
  }
  const int segments = (j == 0) ? 2 : 1;
  T carry = T(0);
  for (int seg = 0; seg < segments; ++seg) {
    const int lo = (segments == 1) ? 0 : (seg == 0 ? 0 : NI / 2);
    const int hi = (segments == 1) ? NI : (seg == 0 ? NI / 2 : NI);
    T pv[MAXPER], qv[MAXPER];
    T P = T(0), Q = T(1);
#pragma unroll
    for (int e = 0; e < MAXPER; ++e) {
      pv[e] = T(0);
      qv[e] = T(1);
      const int i = i0 + e;
      if (e >= per || i < lo || i >= hi) continue;
      const T d = dv[e];
      if (!(fabs(d) > T(0))) {
        pv[e] = oldI[e];
        qv[e] = T(0);
      } else {
        T off = T(0);
        if (j > 0) {
          off += sv[e] * prevI[e];
        } else {
          const int a = wake[e];
          if (a >= 0) off += sv[e] * ((a < i) ? rowNew[a] : oldRow[a]);
        }
        if (i < NI - 1) off += ev[e] * oldE[e];
        if (hasNorth) off += nv[e] * northI[e];
        pv[e] = (bv[e] - off) / d;
        qv[e] = (i > 0) ? -wv[e] / d : T(0);
      }
      P = pv[e] + qv[e] * P;
      Q = qv[e] * Q;
    }
    blockAffineExclusiveScan(P, Q, sc);
    T xv = P + Q * carry;  // value entering this thread's chunk
#pragma unroll
    for (int e = 0; e < MAXPER; ++e) {
      const int i = i0 + e;
      if (e >= per || i < lo || i >= hi) continue;
      xv = pv[e] + qv[e] * xv;
      rowNew[i] = xv;
    }
    __syncthreads();
    if (hi > lo) carry = rowNew[hi - 1];
  }
}

template <typename T>
DEV void gsRowSolve(const Instance& I, int j, const SysView<T>& y, const T* oldRow, const T* northRow, T* rowNew,
                    const T* rowPrev, T* sc) {
  if (I.NI <= 2 * static_cast<int>(blockDim.x)) {
    gsRowSolveN<T, 2>(I, j, y, oldRow, northRow, rowNew, rowPrev, sc);
  } else {
    gsRowSolveAny(I, j, y, oldRow, northRow, rowNew, rowPrev, sc);
  }
}

/// One row of the sweep on the unknowns in place: solve from the unknowns,
/// then publish row j to global memory (east/north reads of later rows and
/// the next sweep) and to rowPrev (the south values of row j + 1). Every
/// read of this row's old values and of rowPrev happened before the scan's
/// barriers. Ends without a barrier (the caller synchronises before the
/// next row).
template <typename T>
DEV void gsRow(const Instance& I, int j, const SysView<T>& y, T* rowNew, T* rowPrev, T* sc) {
  T* x = y.x;
  const int NI = I.NI;
  gsRowSolve(I, j, y, x + static_cast<long long>(j) * NI, x + static_cast<long long>(j + 1) * NI, rowNew, rowPrev,
             sc);
  for (int i = threadIdx.x; i < NI; i += blockDim.x) {
    x[j * NI + i] = rowNew[i];
    rowPrev[i] = rowNew[i];
  }
}

/// Bring row j's coefficients and right-hand side (fixed during the sweeps)
/// towards this SM's L1 ahead of its scan, one prefetch per 128-byte line,
/// spread over the CTA's threads. A hint only: it changes no value.
template <typename T>
DEV void prefetchRow(const Instance& I, int j, const SysView<T>& y) {
  if (j < 0 || j >= I.NJ) return;
  constexpr int perLine = 128 / static_cast<int>(sizeof(T));
  const int lines = (I.NI + perLine - 1) / perLine;
  const T* arrays[6] = {y.D, y.S, y.N, y.W, y.E, y.b};
  for (int q = threadIdx.x; q < 6 * lines; q += blockDim.x) {
    const T* line = arrays[q / lines] + static_cast<long long>(j) * I.NI + (q % lines) * perLine;
    asm volatile("prefetch.global.L1 [%0];" ::"l"(line));
  }
}

/// `sweeps` lexicographic sweeps of one system by one CTA, row after row.
/// Needs 2 * NI + 2 * warps doubles of shared memory.
template <typename T>
DEV void gsRowScanSweeps(const Instance& I, int sweeps, const SysView<T>& y, T* smem) {
  T* rowNew = smem;          // row j, new values
  T* rowPrev = smem + I.NI;  // row j - 1, new values
  T* sc = smem + 2 * I.NI;
  for (int sweep = 0; sweep < sweeps; ++sweep) {
    for (int j = 0; j < I.NJ; ++j) {
      gsRow(I, j, y, rowNew, rowPrev, sc);
      prefetchRow(I, (j + 1 < I.NJ) ? j + 1 : 0, y);
      __syncthreads();
    }
  }
}


// ---- the three sweeps of both equations at once ---------------------------------

constexpr int kChainDepth = 4;  // rows whose coefficients are on their way or in use
constexpr int kChainAhead = 3;  // rows whose old values are on their way

/// How a row of NI lies on a CTA of T threads: thread q has cells q * per ..
/// (per of them), as `cells` places of a kernel unrolled that far.
struct ChainShape {
  int per, cells, threads, words;  // words: 16-byte words of coefficients per thread and row
};
__host__ __device__ inline ChainShape chainShape(int NI, int T) {
  ChainShape z;
  z.per = (NI + T - 1) / T;
  z.cells = (z.per <= 2) ? z.per : 4;
  z.threads = ((NI + z.per - 1) / z.per + 31) / 32 * 32;
  z.words = z.cells + (z.cells + 1) / 2;
  return z;
}
/// Whether a row can be chained (at most 4 cells per thread), and the shared
/// memory of rowChain: the warps' totals, row 0, the copies.
__host__ __device__ inline bool chainable(int NI, int T) { return NI <= 4 * T; }
__host__ __device__ inline long long chainBytes(int NI, int T) {
  const ChainShape z = chainShape(NI, T);
  return 4 * (128LL + (NI + 31) / 32 * 32) + 16LL * kChainDepth * z.words * z.threads;
}

/// A cell's row of the corrections' system where rowChain reads it, and off the
/// chain what does not depend on the row before: the west coefficient over the
/// diagonal. A thread's words of a row lie a word of every thread apart: (S, E,
/// N, b) of each cell, then (D, q) of two cells each.
DEV void chainStoreRow(float4* rows, const ChainShape& z, int i, int j, float D, float S, float N, float W, float E,
                       float b) {
  const int q = i / z.per, e = i - q * z.per;
  float4* const row = rows + static_cast<long long>(j) * z.words * z.threads + q;
  row[e * z.threads] = make_float4(S, E, N, b);
  float2* const tail = reinterpret_cast<float2*>(row + (z.cells + e / 2) * z.threads);
  tail[e & 1] = make_float2(D, (fabsf(D) > 0.0f && i > 0) ? -W / D : 0.0f);
}

/// A message: each value beside the tag in one 64-bit word.
DEV unsigned long long chainWord(float v, unsigned tag) {
  return (static_cast<unsigned long long>(tag) << 32) | static_cast<unsigned long long>(__float_as_uint(v));
}
template <int CELLS>
DEV void chainStore(unsigned long long* to, const float (&v)[CELLS], unsigned tag) {
  if constexpr (CELLS == 1) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(to), "l"(chainWord(v[0], tag)) : "memory");
  } else {
#pragma unroll
    for (int e = 0; e < CELLS; e += 2) {
      asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(to + e), "l"(chainWord(v[e], tag)),
                   "l"(chainWord(v[e + 1], tag))
                   : "memory");
    }
  }
}
DEV unsigned long long chainLoad(const unsigned long long* from) {
  unsigned long long word;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(word) : "l"(from) : "memory");
  return word;
}
template <int CELLS>
DEV void chainLoad(const unsigned long long* from, unsigned long long (&word)[CELLS]) {
  if constexpr (CELLS == 1) {
    word[0] = chainLoad(from);
  } else {
#pragma unroll
    for (int e = 0; e < CELLS; e += 2) {
      asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];"
                   : "=l"(word[e]), "=l"(word[e + 1])
                   : "l"(from + e)
                   : "memory");
    }
  }
}
DEV bool chainReady(unsigned long long word, unsigned tag) { return static_cast<unsigned>(word >> 32) == tag; }
DEV float chainValue(unsigned long long word) { return __uint_as_float(static_cast<unsigned>(word)); }
/// The value of a message.
DEV float chainWait(WideTeam& t, const unsigned long long* from, unsigned long long word, unsigned tag) {
  int polls = 0;
  while (!chainReady(word, tag)) {
    if (wideGiveUpFar(t, polls, kFaultChainWait)) return 0.0f;
    word = chainLoad(from);
  }
  return chainValue(word);
}
DEV void copyAsync16(float4* to, const float4* from) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(static_cast<unsigned>(__cvta_generic_to_shared(to))),
               "l"(from)
               : "memory");
}

/// One sweep of one system by one CTA: old values from `in` (null: all zero),
/// new ones to `out` (null: to the unknowns x). The scan's tree is
/// blockAffineExclusiveScan's, so the bits are gsRowScanSweeps'. What bounds a
/// row is the instructions that every warp issues for it, and their latencies one
/// after another; a missing neighbour has coefficient and value zero, so nothing
/// but row 0 needs a test. The six sweeps of 96 rows of 384 take 120 us (239 as a
/// block scan with four barriers a row), of 192 rows of 768 290 (508).
template <int CELLS>
__device__ __noinline__ void rowChain(const Instance& I, WideTeam& team, const float4* rows, float* x,
                                      const unsigned long long* in, unsigned long long* out, unsigned tag) {
  extern __shared__ __align__(16) double dyn[];
  WideTeam t = team;
  const int NI = I.NI, NJ = I.NJ;
  const ChainShape z = chainShape(NI, t.T);
  const int threads = z.threads, per = z.per;
  if (t.tid >= threads) return;
  constexpr int kWords = CELLS + (CELLS + 1) / 2;
  const int tid = t.tid, lane = tid & 31, warp = tid >> 5, warps = threads >> 5, i0 = tid * per;
  float2* const totals = reinterpret_cast<float2*>(dyn);  // [2][32]
  float* const rowNew = reinterpret_cast<float*>(dyn) + 128;
  float4* const ring = reinterpret_cast<float4*>(rowNew + (NI + 31) / 32 * 32) + tid;
  const float4* const mine = rows + tid;
  auto copyRow = [&](int j) {
    if (j < NJ) {
      const float4* const from = mine + static_cast<long long>(j) * kWords * threads;
      float4* const to = ring + (j % kChainDepth) * kWords * threads;
#pragma unroll
      for (int a = 0; a < kWords; ++a) copyAsync16(to + a * threads, from + a * threads);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto meet = [&] { asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory"); };

  // Values of the sweep before: a thread waits for its cells', the last lane also
  // for its east neighbour's.
  const int exists = min(max(NI - i0, 0), per);  // the thread's cells
  const bool hasOld = in != nullptr && exists > 0;
  const bool hasEast = hasOld && lane == 31 && i0 + per < NI;
  auto slot = [&](int j) { return in + (static_cast<long long>(j) * threads + tid) * CELLS; };
  auto look = [&](int j, unsigned long long (&raw)[CELLS], unsigned long long& rawEast) {
    if (j >= NJ) return;
    if (hasOld) chainLoad<CELLS>(slot(j), raw);
    if (hasEast) rawEast = chainLoad(slot(j) + CELLS);
  };
  auto take = [&](int j, unsigned long long (&raw)[CELLS], unsigned long long rawEast, float (&value)[CELLS],
                  float& east) {
    east = 0.0f;
#pragma unroll
    for (int e = 0; e < CELLS; ++e) value[e] = 0.0f;
    if (hasOld && j < NJ) {
      int polls = 0;
      for (;;) {
        bool ready = true;
#pragma unroll
        for (int e = 0; e < CELLS; ++e) ready = ready && (e >= exists || chainReady(raw[e], tag));
        if (ready || wideGiveUpFar(t, polls, kFaultChainWait)) break;
        chainLoad<CELLS>(slot(j), raw);
      }
#pragma unroll
      for (int e = 0; e < CELLS; ++e) value[e] = (e < exists) ? chainValue(raw[e]) : 0.0f;
      if (hasEast) east = chainWait(t, slot(j) + CELLS, rawEast, tag);
    }
    __syncwarp();
  };
#pragma unroll
  for (int d = 0; d < kChainDepth - 1; ++d) copyRow(d);
  float old[CELLS], prev[CELLS], oldEast;
  // rows on their way; the loop below is unrolled by kChainAhead so that each
  // stays in the registers it was loaded into (moving it would wait for it)
  unsigned long long raw[kChainAhead][CELLS], rawEast[kChainAhead];
  {
    unsigned long long row0[CELLS], east0 = 0;
    look(0, row0, east0);
#pragma unroll
    for (int d = 0; d < kChainAhead; ++d) look(1 + d, raw[d], rawEast[d]);
    take(0, row0, east0, old, oldEast);
  }
#pragma unroll
  for (int e = 0; e < CELLS; ++e) prev[e] = 0.0f;
  int scans = 0;
  auto step = [&](int j, unsigned long long (&next)[CELLS], unsigned long long& nextEast, bool first) {
    copyRow(j + kChainDepth - 1);
    float north[CELLS], northEast;
    take(j + 1, next, nextEast, north, northEast);
    look(j + 1 + kChainAhead, next, nextEast);
    asm volatile("cp.async.wait_group %0;" ::"n"(kChainDepth - 1) : "memory");
    const float4* const row = ring + (j % kChainDepth) * kWords * threads;
    float4 c[CELLS], tail[(CELLS + 1) / 2];
#pragma unroll
    for (int e = 0; e < CELLS; ++e) c[e] = row[e * threads];
#pragma unroll
    for (int e = 0; e < (CELLS + 1) / 2; ++e) tail[e] = row[(CELLS + e) * threads];
    float east = __shfl_down_sync(0xffffffffu, old[0], 1);
    if (lane == 31) east = oldEast;
    float carry = 0.0f, xs[CELLS];
#pragma unroll
    for (int e = 0; e < CELLS; ++e) xs[e] = 0.0f;
    // row 0 in two parts: the second half's partners across the cut are in the first
    for (int part = 0; part < (first ? 2 : 1); ++part) {
      const int lo = (part == 0) ? 0 : NI / 2, hi = (first && part == 0) ? NI / 2 : NI;
      float pv[CELLS], qv[CELLS], P = 0.0f, Q = 1.0f;
#pragma unroll
      for (int e = 0; e < CELLS; ++e) {
        float south = prev[e];
        if (first && i0 + e < NI) {
          const int a = I.acrossJ0[i0 + e];
          south = 0.0f;
          if (a >= 0 && a < i0 + e) south = rowNew[a];
          else if (a >= 0 && in != nullptr) {
            const unsigned long long* at = in + static_cast<long long>(a / per) * CELLS + a % per;
            south = chainWait(t, at, chainLoad(at), tag);
          }
        }
        const float D = (e & 1) ? tail[e / 2].z : tail[e / 2].x, q = (e & 1) ? tail[e / 2].w : tail[e / 2].y;
        const float eastOld = (e + 1 < CELLS && e + 1 < per) ? old[(e + 1) % CELLS] : east;
        const float off = (c[e].x * south + c[e].y * eastOld) + c[e].z * north[e];
        pv[e] = (fabsf(D) > 0.0f) ? (c[e].w - off) / D : old[e];
        qv[e] = q;
        if (e >= per || (first && (i0 + e < lo || i0 + e >= hi))) {
          pv[e] = 0.0f;
          qv[e] = 1.0f;
        }
        P = pv[e] + qv[e] * P;
        Q = qv[e] * Q;
      }
      // the scan: inclusive within the warp, the warps' totals to every warp,
      // which composes the totals before its own
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const float pp = __shfl_up_sync(0xffffffffu, P, off), qq = __shfl_up_sync(0xffffffffu, Q, off);
        if (lane >= off) {
          P = P + Q * pp;
          Q = Q * qq;
        }
      }
      float2* const set = totals + 32 * (scans++ & 1);
      if (lane == 31) set[warp] = make_float2(P, Q);
      float ep = __shfl_up_sync(0xffffffffu, P, 1), eq = __shfl_up_sync(0xffffffffu, Q, 1);
      if (lane == 0) {
        ep = 0.0f;
        eq = 1.0f;
      }
      meet();
      const float2 total = (lane < warps) ? set[lane] : make_float2(0.0f, 1.0f);
      float wp = total.x, wq = total.y;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        if (off >= warps) break;
        const float pp = __shfl_up_sync(0xffffffffu, wp, off), qq = __shfl_up_sync(0xffffffffu, wq, off);
        if (lane >= off) {
          wp = wp + wq * pp;
          wq = wq * qq;
        }
      }
      wp = __shfl_sync(0xffffffffu, wp, max(warp - 1, 0));
      wq = __shfl_sync(0xffffffffu, wq, max(warp - 1, 0));
      if (warp == 0) {
        wp = 0.0f;
        wq = 1.0f;
      }
      float xv = (ep + eq * wp) + (eq * wq) * carry;
#pragma unroll
      for (int e = 0; e < CELLS; ++e) {
        const int i = i0 + e;
        xv = pv[e] + qv[e] * xv;
        if (!first) {
          xs[e] = xv;
        } else if (e < per && i >= lo && i < hi) {
          xs[e] = xv;
          rowNew[i] = xv;
        }
      }
      if (first) {
        meet();
        if (hi > lo) carry = rowNew[hi - 1];
      }
    }
    if (out != nullptr) {
      chainStore<CELLS>(out + (static_cast<long long>(j) * threads + tid) * CELLS, xs, tag);
    } else {
#pragma unroll
      for (int e = 0; e < CELLS; ++e) {
        if (e < exists) x[static_cast<long long>(j) * NI + i0 + e] = xs[e];
      }
    }
#pragma unroll
    for (int e = 0; e < CELLS; ++e) {
      prev[e] = xs[e];
      old[e] = north[e];
    }
    oldEast = northEast;
  };
  step(0, raw[0], rawEast[0], true);
  for (int j0 = 1; j0 < NJ; j0 += kChainAhead) {
#pragma unroll
    for (int d = 0; d < kChainAhead; ++d) {
      if (j0 + d < NJ) step(j0 + d, raw[(1 + d) % kChainAhead], rawEast[(1 + d) % kChainAhead], false);
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

/// Whether the corrections are swept row by row rather than as wavefronts of the
/// FP64 systems: a rule of the grid alone (it decides the rounding), two rows
/// within the larger of the coarse levels at 32 bytes a cell and six rows.
DEV bool mixedRowsFit(int NI, int coarseBytes) {
  const long long six = (6LL * NI + 64) * 4;
  return (2LL * NI + 64) * 8 <= max(static_cast<long long>(coarseBytes), (six <= 210 * 1024) ? six : 0LL);
}

/// Whether a team's k and omega sweeps run chained, on six CTAs.
DEV bool mixedChained(const Instance& I, const WideTeam& t, int smemBytes) {
  return t.R >= 6 && chainable(I.NI, t.T) && chainBytes(I.NI, t.T) <= smemBytes;
}
/// The chained sweeps, from the rows that chainStoreRow stored; the caller ends
/// with a barrier. With `waitTest` the second sweeps also wait once for a count
/// that nothing sets, which gives up and reports it.
DEV void chainedSweeps(const Instance& I, WideTeam& t, unsigned tag, bool waitTest) {
  if (t.rank >= 6) return;
  const int s = t.rank % 3;
  const bool omega = t.rank >= 3;
  const float4* const rows = omega ? I.twC : I.tkC;
  float* const x = omega ? I.tw.x : I.tk.x;
  unsigned long long* const values = omega ? I.twV : I.tkV;
  const long long sweep = chainSlots(I.NI, I.NJ);
  const unsigned long long* in = (s > 0) ? values + (s - 1) * sweep : nullptr;
  unsigned long long* out = (s < 2) ? values + s * sweep : nullptr;
  if (waitTest && s == 1 && t.tid == 0) {
    int polls = 0;
    while (*static_cast<volatile unsigned*>(&t.sh->never) == 0u && ++polls < (1 << 24)) {
    }
    if (polls >= (1 << 24)) atomicOr(t.faultWord, kFaultChainWait);
  }
  const int cells = chainShape(I.NI, t.T).cells;
  if (cells == 1) rowChain<1>(I, t, rows, x, in, out, tag);
  else if (cells == 2) rowChain<2>(I, t, rows, x, in, out, tag);
  else rowChain<4>(I, t, rows, x, in, out, tag);
}
/// The same sweeps with a CTA per system, one sweep after another. Needs
/// NI <= 8 * T.
DEV void sequentialSweeps(const Instance& I, const WideTeam& t) {
  extern __shared__ __align__(16) double dyn[];
  float* rows = reinterpret_cast<float*>(dyn);
  auto system = [](const Rows32& r) { return SysView<float>{r.D, r.S, r.N, r.W, r.E, r.r, r.x}; };
  if (t.rank == 0) gsRowScanSweeps(I, 3, system(I.tk), rows);
  if (t.rank == ((t.R > 1) ? 1 : 0)) gsRowScanSweeps(I, 3, system(I.tw), rows);
}

}  // namespace
}  // namespace cfdb
