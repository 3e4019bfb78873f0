// wide_cg.cuh - the reference's Jacobi-preconditioned conjugate gradient
// (LinearSystem.cpp:118-210) by a wide team (wide_team.cuh), one exchange per
// iteration.
//
// The iteration is Chronopoulos and Gear's single-reduction arrangement
// (J. Comput. Appl. Math. 25, 1989): with u = M^-1 r and w = A u, one reduction
// gives gamma = r.u, delta = w.u and rho = sum |r|;
//   beta_k = gamma_k / gamma_(k-1),  d.Ad_k = delta_k - beta_k^2 d.Ad_(k-1),
//   alpha_k = gamma_k / d.Ad_k,
//   p = u + beta p,  s = w + beta s (= A p),  x += alpha p,  r -= alpha s,
// with the reference's stopping rule (rho <= tolerance * rho_0, tested after
// each update), its cap and its breakdown guards (d.Ad = 0 before an update,
// r.z = 0 before forming beta).
//
// Tiles. The block is cut into column tiles of at most 256 columns and unit
// rows of B rows; a CTA has one column tile and some consecutive unit rows, a
// thread one column and K consecutive rows of a unit, 256 threads a unit.
// Column tiles and B depend on the block alone (about as many units as the GPU
// has SMs), and the sums are formed per unit and added in unit order, so the
// bits are the same however many CTAs share the units.
//
// One round trip per iteration. The only values a CTA needs from its
// neighbours are the u of the cells bordering its tile. It forms those
// itself, from copies of their r and s that it updates as the owner does and
// from their w, which the owner publishes with its sums: the border exchange
// and the reduction wait for the same L2 latency. A unit's sums have a line of
// their own: with several writers a line the polls of it queue up (2,100
// cycles a load instead of 350 to 700).
//
// Three forms of the same arithmetic. One unit per CTA: 256 threads hold the
// cells' state in registers, the other 256 the border's, and wait for the
// messages. Two to eight units: every thread holds cells. Any shape: every
// array in memory, shared as far as it reaches, then global.
#pragma once

#include "wide_team.cuh"

namespace cfdb {

/// How a block is tiled and how a team of R CTAs of T threads shares it.
struct WideCgShape {
  int columnTiles, width, passes, G;  // tiles of `width` columns: G threads, `passes` columns each
  int teams, groups;                  // teams of threads with a unit each; rows of threads in a team
  int B, K, unitRows;                 // rows of a unit, of it per thread; units down a column tile
  int RT, units;                      // CTAs down a column tile, units of the busiest CTA
  int rounds;                         // units per team
};

constexpr int kMaxColumnTiles = 64;
constexpr int kMaxUnits = 160;  // of a block: 144 as tiled below
constexpr int kUnitThreads = 32 * kUnitWarps;

/// The tiling of the block in `columnTiles` column tiles (rows of a unit and
/// units included), for teams of `team` threads.
__host__ __device__ inline WideCgShape wideCgTiles(int NI, int NJ, int columnTiles, int team) {
  WideCgShape s;
  s.width = (NI + columnTiles - 1) / columnTiles;
  s.columnTiles = (NI + s.width - 1) / s.width;  // as many as hold a column at that width
  s.passes = (s.width + team - 1) / team;
  s.G = ((s.width + s.passes - 1) / s.passes + 31) / 32 * 32;
  s.groups = team / s.G;
  // units: as many as fit the SMs (144 of 148 leave a column-tile remainder),
  // and two rows a thread at least, below which the exchange is all there is
  const int down = (144 / s.columnTiles > 1) ? 144 / s.columnTiles : 1;
  const int rows = (NJ + down - 1) / down;
  s.K = (rows + s.groups - 1) / s.groups;
  if (s.K < 2) s.K = 2;
  s.B = s.K * s.groups;
  s.unitRows = (NJ + s.B - 1) / s.B;
  return s;
}
/// The block's tiling is a rule of the block and the threads alone: column tiles
/// as wide as a team, half or a quarter of it, whichever leaves a thread the
/// fewest rows; above two rows a thread, of those the shortest border. 768x192 in
/// 144 units of 64x16 cells has 160 border cells a unit, in units of 256x4 it has
/// 520: 1,000 iterations 4.7 against 5.2 ms; 642x151 gets 3 rows a thread instead
/// of 4. With two rows a thread wide tiles stay: a side's messages are stored a
/// row at a time, 16 bytes each, and cost more than the shorter border saves
/// (384x96, 200 iterations and the rest of an SST iteration: 0.93 ms in tiles
/// of 192x2, 1.01 in tiles of 64x8).
__host__ __device__ inline WideCgShape wideCgShape(int NI, int NJ, int R, int T) {
  const int team = (T < kUnitThreads) ? T : kUnitThreads;
  WideCgShape s;
  int best = 0;
  for (int w = team; w >= 32 && w >= team / 4; w /= 2) {
    int tiles = (NI + w - 1) / w;
    if (w < team && (w % 32 != 0 || tiles > 144)) break;
    if (tiles > kMaxColumnTiles) tiles = kMaxColumnTiles;  // then several columns a thread
    const WideCgShape z = wideCgTiles(NI, NJ, tiles, team);
    const int cost = 4096 * z.K * z.passes + ((z.K > 2) ? 2 * (z.width + z.B) : 0);
    if (w == team || cost < best) {
      s = z;
      best = cost;
    }
  }
  s.teams = T / team;
  s.RT = R / s.columnTiles;
  if (s.RT > s.unitRows) s.RT = s.unitRows;
  s.units = (s.RT > 0) ? (s.unitRows + s.RT - 1) / s.RT : s.unitRows;
  s.rounds = (s.units + s.teams - 1) / s.teams;
  return s;
}

/// The fewest CTAs up to `width` that leave a CTA no more units than `width`
/// CTAs would (and at least one per column tile).
__host__ __device__ inline int wideUsefulCtas(int NI, int NJ, int width, int T) {
  WideCgShape s = wideCgShape(NI, NJ, width, T);
  if (s.RT < 1) return s.columnTiles;
  return s.columnTiles * ((s.unitRows + s.units - 1) / s.units);
}

/// The messages of one exchange: bottom and top rows of every CTA row, left
/// and right columns of every column tile, the units' three sums.
__host__ __device__ inline long long wideMessages(int NI, int NJ, int R, int T) {
  const WideCgShape s = wideCgShape(NI, NJ, R, T);
  return (2LL * s.RT * NI + 2LL * s.columnTiles * NJ + kSumLine - 1) / kSumLine * kSumLine +
         static_cast<long long>(kSumLine) * kSumCopies * s.columnTiles * s.unitRows;
}

/// An array in a tile's geometry: one border row and column on every side.
__host__ __device__ inline long long wideCgPlane(const WideCgShape& s) {
  return (static_cast<long long>(s.units) * s.B + 2) * (s.width + 2);
}
__host__ __device__ inline long long wideCgBorder(const WideCgShape& s) {
  return 2LL * s.units * s.B + 2LL * s.width;
}
/// Shared memory, in bytes, of the unrolled forms with C cells per thread: u
/// and the border's r, s, 1/D; p and x above 3 cells, and where they are not
/// in registers (`all`) the coefficients and 1/D.
__host__ __device__ inline long long wideCgUnrolledBytes(const WideCgShape& s, int C, int T, bool all) {
  long long n = wideCgPlane(s) + 3 * wideCgBorder(s);
  if (!all) n += 2 * wideCgPlane(s) + 3LL * C * T;
  else if (C > 3) n += 2LL * C * T;
  return 8 * n;
}
/// Doubles of the form for any shape: u, both coefficients, the border, six
/// arrays of the thread's cells.
__host__ __device__ inline long long wideCgAnyDoubles(const WideCgShape& s, int T) {
  return 3 * wideCgPlane(s) + 3 * wideCgBorder(s) + 6LL * s.rounds * s.K * s.passes * T;
}
/// Which form takes the shape in `most` bytes: 8 K + units per team of the
/// unrolled ones (in the split one, 0 units), or 0 for the form for any shape.
__host__ __device__ inline int wideCgForm(const WideCgShape& s, int T, long long most) {
  if (T != kWideThreads || s.passes != 1 || s.RT < 1) return 0;
  auto fits = [&](int C, bool all) { return wideCgUnrolledBytes(s, C, T, all) <= most; };
  if (s.units == 1) return (s.K <= 4 && fits(s.K, true)) ? 8 * s.K : 0;
  if (s.units > kUnitBatch) return 0;
  const int rounds = (s.rounds == 3) ? 4 : s.rounds;
  if (s.K == 2 && rounds <= 4 && fits(2 * rounds, rounds == 1)) return 16 + rounds;
  if (s.K == 4 && rounds <= 2 && fits(4 * rounds, false)) return 32 + rounds;
  return 0;
}
__host__ __device__ inline long long wideCgFormBytes(const WideCgShape& s, int T, int form) {
  const int K = form / 8, rounds = form % 8;
  if (form == 0) return 8 * wideCgAnyDoubles(s, T);
  return wideCgUnrolledBytes(s, K * ((rounds > 0) ? rounds : 1), T, rounds == 0 || K * rounds <= 2);
}
/// Dynamic shared memory for a team of R CTAs, and doubles of global memory
/// per CTA for what does not fit there (0: everything does). `any`: with the
/// form for any shape (a wake map that couples to other rows needs it).
__host__ __device__ inline long long wideCgBytes(int NI, int NJ, int R, int T, long long most, bool any) {
  const WideCgShape s = wideCgShape(NI, NJ, R, T);
  const long long n = wideCgFormBytes(s, T, any ? 0 : wideCgForm(s, T, most));
  return (n < most) ? n : most;
}
__host__ __device__ inline long long wideCgSpill(int NI, int NJ, int R, int T, long long most, bool any) {
  const WideCgShape s = wideCgShape(NI, NJ, R, T);
  if (!any && wideCgForm(s, T, most) != 0) return 0;
  return (8 * wideCgAnyDoubles(s, T) <= most) ? 0 : wideCgAnyDoubles(s, T);
}

/// One system; every pointer is global. The coefficients come from a loader:
/// north(i, j) and east(i, j) of face (i, j), zero on boundary faces except
/// the wake cut's; wake(i), the cell across the j = 0 face of column i or -1;
/// and first(c, i, j), the residual the solve starts from.
struct WideCgSystem {
  const double* D;    // diagonal, per cell
  bool wakeAnywhere;  // wake entries may name cells outside row 0
  double* x;          // the start in, the solution out
  double* u;          // a cell each: read by the other CTAs when wakeAnywhere
  double* spill;      // per CTA `spillStride` doubles for the arrays that do not fit on chip
  long long spillStride;
  double tolerance;
  int cap;
};

struct WideCgResult {
  int iterations;
  double initial, final;
  bool converged;
};

/// M^-1 r for a diagonal without a usable reciprocal, as the reference writes it.
DEV double wideCgPrecondition(double r, double D) { return (fabs(D) > 0.0) ? r / D : r; }
/// 1/D, or infinity where the reference does not divide (D zero or not a number).
DEV double wideCgReciprocal(double D) { return (fabs(D) > 0.0) ? 1.0 / D : INFINITY; }

/// Three sums over the warp at once, in 7 shuffles instead of 15: the first
/// two steps halve the number of values a lane carries while they add. Lane 0
/// gets the first, lane 1 the second, lane 2 the third.
DEV double warpSum3(double a, double b, double c) {
  const int lane = threadIdx.x & 31;
  const bool odd = (lane & 1) != 0, upper = (lane & 2) != 0;
  // pairs: even lanes keep a, odd lanes b; c is summed in both
  double ab = odd ? b : a;
  ab += __shfl_xor_sync(0xffffffffu, odd ? a : b, 1);
  c += __shfl_xor_sync(0xffffffffu, c, 1);
  // fours: lanes 0, 1 keep ab, lanes 2, 3 keep c
  double v = upper ? c : ab;
  v += __shfl_xor_sync(0xffffffffu, upper ? ab : c, 2);
#pragma unroll
  for (int off = 4; off < 32; off <<= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}

/// Where a CTA's tile lies, and where its messages go and come from.
struct WideCgTile {
  WideCgShape z;
  int ct, rt, unit0, units;
  int i0, width, j0, rows, stride;  // rows of `stride` doubles: a border column on either side
  bool splitWake;                   // the wake's partners may lie in another tile: border cells
  int topRows, leftCols, rightCols, sums, unitCount, set;  // offsets in a message set, its size
  int team, lt, q, g;               // this thread: its team, its place there, its first column and row group
  bool working;

  DEV WideCgTile(const WideTeam& t, bool wakeAnywhere) {
    z = wideCgShape(t.NI, t.NJ, t.R, t.T);
    ct = t.rank % z.columnTiles;
    rt = t.rank / z.columnTiles;
    unit0 = z.unitRows * rt / z.RT;
    units = z.unitRows * (rt + 1) / z.RT - unit0;
    j0 = unit0 * z.B;
    rows = min((unit0 + units) * z.B, t.NJ) - j0;
    i0 = ct * z.width;
    width = min(z.width, t.NI - i0);
    stride = z.width + 2;
    splitWake = z.columnTiles > 1 && !wakeAnywhere;
    topRows = z.RT * t.NI;
    leftCols = 2 * topRows;
    rightCols = leftCols + z.columnTiles * t.NJ;
    sums = (rightCols + z.columnTiles * t.NJ + kSumLine - 1) / kSumLine * kSumLine;
    unitCount = z.columnTiles * z.unitRows;
    set = sums + kSumLine * kSumCopies * unitCount;
    const int teamThreads = min(t.T, kUnitThreads);
    team = t.tid / teamThreads;
    lt = t.tid - team * teamThreads;
    q = lt % z.G;
    g = lt / z.G;
    working = team < z.teams && g < z.groups && q < width;
  }
  DEV int border() const { return 2 * width + 2 * rows; }
  /// Border cell h: the row below (0 .. width), above, the column left, right.
  /// Its cell in the block or -1; its place among the tile's cells; the message
  /// that carries its w.
  template <typename Loader>
  DEV int cell(const WideTeam& t, const Loader& load, int h) const {
    if (h < width) return (j0 > 0) ? (j0 - 1) * t.NI + i0 + h : (splitWake ? load.wake(i0 + h) : -1);
    if (h < 2 * width) return (j0 + rows < t.NJ) ? (j0 + rows) * t.NI + i0 + h - width : -1;
    if (h < 2 * width + rows) return (i0 > 0) ? (j0 + h - 2 * width) * t.NI + i0 - 1 : -1;
    return (i0 + width < t.NI) ? (j0 + h - 2 * width - rows) * t.NI + i0 + width : -1;
  }
  DEV int place(int h) const {
    if (h < width) return h + 1;
    if (h < 2 * width) return (rows + 1) * stride + h - width + 1;
    if (h < 2 * width + rows) return (h - 2 * width + 1) * stride;
    return (h - 2 * width - rows + 1) * stride + width + 1;
  }
  template <typename Loader>
  DEV int source(const WideTeam& t, const Loader& load, int h) const {
    if (h < width) return (j0 > 0) ? topRows + (rt - 1) * t.NI + i0 + h : load.wake(i0 + h);
    if (h < 2 * width) return (rt + 1) * t.NI + i0 + h - width;
    if (h < 2 * width + rows) return rightCols + (ct - 1) * t.NJ + j0 + h - 2 * width;
    return leftCols + (ct + 1) * t.NJ + j0 + h - 2 * width - rows;
  }
  /// Where an own cell's w is published, -1: nowhere.
  DEV int toBelow(const WideTeam& t, int q, int lr) const {
    return (lr == 0 && (j0 > 0 || splitWake)) ? rt * t.NI + i0 + q : -1;
  }
  DEV int toAbove(const WideTeam& t, int q, int lr) const {
    return (lr == rows - 1 && j0 + rows < t.NJ) ? topRows + rt * t.NI + i0 + q : -1;
  }
  DEV int toSide(const WideTeam& t, int q, int lr) const {
    if (q == 0 && i0 > 0) return leftCols + ct * t.NJ + j0 + lr;
    return (q == width - 1 && i0 + width < t.NI) ? rightCols + ct * t.NJ + j0 + lr : -1;
  }
};

/// The border cells' start, and the tile's coefficients by place (south face
/// of the cell at a place in sN, west face in sE). U, sN, sE zero before.
template <typename Loader>
DEV bool wideCgLoadBorder(const WideTeam& t, const WideCgSystem& S, const Loader& load, const WideCgTile& a, double* U,
                          double* hr) {
  const int border = a.border();
  bool odd = false;
  for (int h = t.tid; h < border; h += t.T) {
    const int c = a.cell(t, load, h);
    if (c < 0) continue;
    const double D = S.D[c], rc = load.first(c, c % t.NI, c / t.NI), d = wideCgReciprocal(D);
    if (!isfinite(d)) odd = true;
    hr[h] = rc;
    hr[h + border] = 0.0;
    hr[h + 2 * border] = d;
    U[a.place(h)] = isfinite(d) ? rc * d : wideCgPrecondition(rc, D);
  }
  return odd;
}
template <typename Loader>
DEV void wideCgLoadCoefficients(const WideTeam& t, const Loader& load, const WideCgTile& a, double* sN, double* sE) {
  for (int m = t.tid; m < (a.rows + 1) * a.width; m += t.T) {
    const int lr = m / a.width, q = m - lr * a.width;
    sN[(lr + 1) * a.stride + q + 1] = load.north(a.i0 + q, a.j0 + lr);
  }
  for (int m = t.tid; m < a.rows * (a.width + 1); m += t.T) {
    const int lr = m / (a.width + 1), q = m - lr * (a.width + 1);
    sE[(lr + 1) * a.stride + q + 1] = load.east(a.i0 + q, a.j0 + lr);
  }
}

/// A unit's three sums within the warps; slot = its place in the batch.
DEV void unitPartial(WideTeam& t, int lt, int slot, const double (&acc)[3]) {
  const double v = warpSum3(acc[0], acc[1], acc[2]);
  const int lane = t.tid & 31;
  if (lane < 3) t.sh->unitPart[slot][lt >> 5][lane] = v;
}
/// The sums of units [first, last) of this CTA, all warps' parts stored.
DEV void unitPublish(WideTeam& t, const WideCgTile& a, ulonglong2* set, int first, int last, unsigned tag) {
  const int warps = min(t.T, kUnitThreads) >> 5;
  for (int m = t.tid; m < 3 * kSumCopies * (last - first); m += t.T) {
    const int unit = m / (3 * kSumCopies), copy = (m - 3 * kSumCopies * unit) / 3, k = m % 3;
    const int line = copy * a.unitCount + a.ct * a.z.unitRows + a.unit0 + first + unit;
    messageStore(set + a.sums + line * kSumLine + k, unitTotal(t, unit, k, warps), tag);
  }
}
/// The team's sums by groups of 32 units into t.sh->warpPart, by `warps` warps
/// from `warp0` on: a lane waits for one unit.
DEV void sumsCollect(WideTeam& t, const WideCgTile& a, const ulonglong2* set, unsigned tag, int warp0, int warps) {
  const int lane = t.tid & 31;
  for (int part = (t.tid >> 5) - warp0; part * 32 < a.unitCount; part += warps) {
    const int unit = part * 32 + lane;
    const int line = a.sums + ((t.rank % kSumCopies) * a.unitCount + unit) * kSumLine;
    const int from[3] = {(unit < a.unitCount) ? line : -1, (unit < a.unitCount) ? line + 1 : -1,
                         (unit < a.unitCount) ? line + 2 : -1};
    double v[3] = {0.0, 0.0, 0.0};
    messageWaitAll(t, set, from, tag, kFaultTeamWait, v);
    __syncwarp();
    const double total = warpSum3(v[0], v[1], v[2]);
    if (lane < 3) t.sh->warpPart[part][lane] = total;
  }
}

/// The CG's scalars. step() takes the sums of an exchange: the reference's stop
/// tests, then the next alpha and beta; false when the solve is over.
struct WideCgScalars {
  double gamma{0.0}, dAd{0.0}, alpha{0.0}, beta{0.0};
  double inverse{0.0};  // 1 / gamma, of a subnormal gamma 1 / (2^600 gamma)
  bool tiny{false};     // it is subnormal
  double initial{0.0}, final{0.0};
  int iterations{-1};  // updates done; -1 before the first exchange
  bool converged{false};

  DEV bool step(const WideTeam& t, int units, double tolerance, int cap) {
    double sum0 = 0.0, sum1 = 0.0;
    final = 0.0;
#pragma unroll
    for (int part = 0; part < kMaxUnits / 32; ++part) {
      if (part * 32 >= units) continue;
      sum0 += t.sh->warpPart[part][0];
      sum1 += t.sh->warpPart[part][1];
      final += t.sh->warpPart[part][2];
    }
    if (iterations < 0) {
      iterations = 0;
      initial = final;
      converged = final <= 0.0;
      if (converged) return false;
      dAd = sum1;
    } else {
      converged = final <= tolerance * initial;
      if (converged || !(fabs(gamma) > 0.0)) return false;
      beta = sum0 * inverse;
      if (tiny) beta *= 0x1p600;
      dAd = fma(-beta * beta, dAd, sum1);
    }
    if (!(fabs(dAd) > 0.0) || iterations >= cap) return false;
    gamma = sum0;
    alpha = gamma / dAd;
    tiny = fabs(gamma) < 0x1p-1022;
    inverse = 1.0 / (tiny ? gamma * 0x1p600 : gamma);
    ++iterations;
    return true;
  }
};

/// A border cell's r, s, 1/D in shared memory, and its next u: the owner's
/// expressions, so its bits.
template <typename Loader>
DEV void updateBorder(const WideTeam& t, const WideCgSystem& S, const Loader& load, const WideCgTile& a,
                      const WideCgScalars& z, double* hr, double* U, int h, int place, double hw, bool odd) {
  const int border = a.border();
  const double sc = fma(z.beta, hr[h + border], hw), rc = fma(-z.alpha, sc, hr[h]), d = hr[h + 2 * border];
  hr[h + border] = sc;
  hr[h] = rc;
  U[place] = (odd && !isfinite(d)) ? wideCgPrecondition(rc, S.D[a.cell(t, load, h)]) : rc * d;
}

/// The unrolled forms: K rows of each of `kRounds` units per thread. kSplit:
/// one unit per CTA, held by the first 256 threads; the others have the border
/// and the waiting.
template <int K, int kRounds, bool kSplit, typename Loader>
__device__ __noinline__ WideCgResult wideCgUnrolledTile(WideTeam& team, const WideCgSystem& system, const Loader& load) {
  // a function of its own, for its registers; copies, because what is read
  // through a reference is read from the stack again after every message
  WideTeam t = team;
  const WideCgSystem S = system;
  extern __shared__ double dyn[];
  constexpr int C = K * kRounds;
  constexpr bool kAll = kSplit || C <= 2;  // the coefficients and 1/D in registers
  constexpr bool kPx = kAll && C <= 3;     // p and x too
  constexpr bool kU = C <= 4;              // a copy of u as well
  // The tile is the same for every thread but for its place in it: with four
  // cells a thread and more it lies on chip, to leave its registers to the cells
  // (8 cells: 664 bytes of spills instead of 848; a batch of 768x192 solves 8.46
  // -> 7.59 ms). With two it stays in registers, which is 6 % faster there.
  __shared__ int words[(sizeof(WideCgTile) + 3) / 4];
  const WideCgTile own(t, false);
  const int aTeam = own.team, lt = own.lt, q = own.q, g = own.g;
  const bool working = own.working;
  if constexpr (C >= 4) {
    if (t.tid == 0) *reinterpret_cast<WideCgTile*>(words) = own;
    __syncthreads();
  }
  const WideCgTile& a = (C >= 4) ? *reinterpret_cast<const WideCgTile*>(words) : own;
  const int T = t.T, tid = t.tid, NI = t.NI, SW = a.stride;
  const int plane = static_cast<int>(wideCgPlane(a.z)), border = a.border();
  double* const U = dyn;
  double* const hr = dyn + plane;
  double* const sN = hr + 3 * wideCgBorder(a.z);
  double* const sE = sN + plane;
  // p, x, 1/D of cell k at k*T, (C + k)*T, (2C + k)*T
  double* const mine = (kAll ? hr + 3 * wideCgBorder(a.z) : sE + plane) + tid;
  const int teams = kSplit ? 1 : a.z.teams;
  for (int m = tid; m < plane; m += T) U[m] = 0.0;
  if constexpr (!kAll) {
    for (int m = tid; m < 2 * plane; m += T) sN[m] = 0.0;
    __syncthreads();
    wideCgLoadCoefficients(t, load, a, sN, sE);
  }
  __syncthreads();
  const bool oddBorder = wideCgLoadBorder(t, S, load, a, U, hr);
  // the thread's unit in round m, its first row there and how many it has
  auto unitOf = [&](int m) { return aTeam + m * teams; };
  auto rowOf = [&](int m) { return unitOf(m) * a.z.B + g * K; };
  auto rowsOf = [&](int m) {
    return (working && unitOf(m) < a.units) ? min(max(a.rows - rowOf(m), 0), K) : 0;
  };
  WideCgScalars z;
  // the border cells a thread keeps: three of every waiting thread (2 * 256 + 2 *
  // B cells at most), or two of every thread and the rest of a long border as
  // it comes
  constexpr int kHeld = kSplit ? 3 : 2;
  const int h0 = kSplit ? tid - kUnitThreads : tid, hStep = kSplit ? T - kUnitThreads : T;
  int from[kHeld], place[kHeld];
  double hw[kHeld];
  auto source = [&](int h) { return (h >= 0 && h < border && a.cell(t, load, h) >= 0) ? a.source(t, load, h) : -1; };
#pragma unroll
  for (int k = 0; k < kHeld; ++k) {
    from[k] = source((h0 >= 0) ? h0 + k * hStep : -1);
    place[k] = (from[k] >= 0) ? a.place(h0 + k * hStep) : 0;
    hw[k] = 0.0;
  }
  auto setOf = [&](unsigned tag) { return t.mem.messages + ((tag & 1u) ? a.set : 0); };

  if (kSplit && tid >= kUnitThreads) {
    // ---- the waiting half: the border's state in registers, and a unit's sums
    // per lane of the first warps ----
    const bool odd = __syncthreads_or(oddBorder);
    double br[kHeld], bs[kHeld], bd[kHeld];
#pragma unroll
    for (int k = 0; k < kHeld; ++k) {
      br[k] = (from[k] >= 0) ? hr[h0 + k * hStep] : 0.0;
      bd[k] = (from[k] >= 0) ? hr[h0 + k * hStep + 2 * border] : 0.0;
      bs[k] = 0.0;
    }
    const int line = (h0 < a.unitCount) ? a.sums + ((t.rank % kSumCopies) * a.unitCount + h0) * kSumLine : -1;
    int both[kHeld + 3];
#pragma unroll
    for (int k = 0; k < kHeld; ++k) both[k] = from[k];
#pragma unroll
    for (int k = 0; k < 3; ++k) both[kHeld + k] = (line >= 0) ? line + k : -1;
    const bool summing = (h0 & ~31) < a.unitCount;
    for (;;) {
      const unsigned tag = ++t.epoch;
      const ulonglong2* const set = setOf(tag);
      __syncthreads();  // the unit's sums of the warps
      if (summing) {
        double got[kHeld + 3] = {};
        messageWaitAll(t, set, both, tag, kFaultTeamWait, got);
        __syncwarp();
        const double total = warpSum3(got[kHeld], got[kHeld + 1], got[kHeld + 2]);
        if ((tid & 31) < 3) t.sh->warpPart[h0 >> 5][tid & 31] = total;
#pragma unroll
        for (int k = 0; k < kHeld; ++k) hw[k] = got[k];
      } else {
        messageWaitAll(t, set, from, tag, kFaultHaloWait, hw);
      }
      __syncthreads();  // the sums
      if (!z.step(t, a.unitCount, S.tolerance, S.cap)) break;
#pragma unroll
      for (int k = 0; k < kHeld; ++k) {
        if (from[k] < 0) continue;
        bs[k] = fma(z.beta, bs[k], hw[k]);
        br[k] = fma(-z.alpha, bs[k], br[k]);
        double next = br[k] * bd[k];
        if (odd && !isfinite(bd[k])) next = wideCgPrecondition(br[k], S.D[a.cell(t, load, h0 + k * hStep)]);
        U[place[k]] = next;
      }
      __syncthreads();  // u
    }
    team.epoch = t.epoch;
    team.barriers = t.barriers;
    return WideCgResult{z.iterations, z.initial, z.final, z.converged};
  }

  // ---- the thread's cells ----
  double r[C], w[C], s[C], u[kU ? C : 1];
  double p[kPx ? C : 1], x[kPx ? C : 1], di[kAll ? C : 1];
  double cS[kAll ? kRounds : 1], cN[kAll ? C : 1], cW[kAll ? C : 1], cE[kAll ? C : 1];
  int first[kRounds];  // the place of the round's first cell; the others follow down the column
  int south = -SW;     // where the very first cell's south neighbour is, from its place
  int below = -1, above = -1, side = -1, top = 0;
  unsigned oddCells = 0, have = 0;
#pragma unroll
  for (int m = 0; m < kRounds; ++m) {
    const int lr0 = rowOf(m), n = rowsOf(m);
    // rows that are missing (have) are computed like the others, from whatever
    // lies there, and their w is set to zero
    first[m] = ((n > 0) ? lr0 + 1 : 1) * SW + q % a.width + 1;
#pragma unroll
    for (int kk = 0; kk < K; ++kk) {
      const int k = m * K + kk;
      r[k] = w[k] = s[k] = 0.0;
      if constexpr (kU) u[k] = 0.0;
      double xk = 0.0, dk = 0.0;
      if constexpr (kAll) cN[k] = cW[k] = cE[k] = 0.0;
      if (kAll && kk == 0) cS[m] = 0.0;
      if (kk < n) {
        const int i = a.i0 + q, lr = lr0 + kk, j = a.j0 + lr, c = j * NI + i;
        const double D = S.D[c];
        have |= 1u << k;
        r[k] = load.first(c, i, j);
        xk = S.x[c];
        dk = wideCgReciprocal(D);
        if (!isfinite(dk)) oddCells |= 1u << k;
        const double u0 = isfinite(dk) ? r[k] * dk : wideCgPrecondition(r[k], D);
        if constexpr (kU) u[k] = u0;
        U[first[m] + kk * SW] = u0;
        if constexpr (kAll) {
          if (kk == 0) cS[m] = load.north(i, j);
          cN[k] = load.north(i, j + 1);
          cW[k] = load.east(i, j);
          cE[k] = load.east(i + 1, j);
        }
        if (lr == 0 && j == 0 && a.z.columnTiles == 1 && load.wake(i) >= 0) {
          south = SW + load.wake(i) + 1 - first[m];
        }
        if (lr == 0) below = a.toBelow(t, q, 0);
        if (lr == a.rows - 1) {
          above = a.toAbove(t, q, lr);
          top = k;
        }
        if (k == 0) side = a.toSide(t, q, lr);
      }
      if constexpr (kPx) {
        p[k] = 0.0;
        x[k] = xk;
      } else {
        mine[k * T] = 0.0;
        mine[(C + k) * T] = xk;
      }
      if constexpr (kAll) di[k] = dk;
      else mine[(2 * C + k) * T] = dk;
    }
  }
  const bool odd = __syncthreads_or(oddBorder || oddCells != 0);
  auto cellOf = [&](int k) { return (a.j0 + rowOf(k / K) + k % K) * NI + a.i0 + q; };
  for (;;) {
    // ---- w = A u down the columns, the units' sums ----
    const unsigned tag = ++t.epoch;
    ulonglong2* const set = setOf(tag);
    double edge = 0.0;  // the w the CTA above needs
#pragma unroll
    for (int m = 0; m < kRounds; ++m) {
      const double* const at = U + first[m];
      double us = (m == 0) ? at[south] : at[-SW], acc[3] = {0.0, 0.0, 0.0};
      double uc = at[0];
#pragma unroll
      for (int kk = 0; kk < K; ++kk) {
        const int k = m * K + kk;
        const double un = at[(kk + 1) * SW];
        double y = r[k];  // D u is r, unless D has no reciprocal
        if (odd && (oddCells & (1u << k))) y = S.D[cellOf(k)] * uc;
        if constexpr (kAll) {
          y = fma((kk == 0) ? cS[m] : cN[k - 1], us, y);
          y = fma(cN[k], un, y);
          y = fma(cW[k], at[kk * SW - 1], y);
          y = fma(cE[k], at[kk * SW + 1], y);
        } else {
          const double* const n = sN + first[m] + kk * SW;
          const double* const e = sE + first[m] + kk * SW;
          y = fma(n[0], us, y);
          y = fma(n[SW], un, y);
          y = fma(e[0], at[kk * SW - 1], y);
          y = fma(e[1], at[kk * SW + 1], y);
        }
        const bool there = (have >> k) & 1u;
        if (!there) y = 0.0;
        w[k] = y;
        if (k == top) edge = y;
        acc[0] = fma(r[k], there ? uc : 0.0, acc[0]);
        acc[1] = fma(y, uc, acc[1]);
        acc[2] += fabs(r[k]);
        us = uc;
        uc = un;
      }
      if (unitOf(m) < a.units) unitPartial(t, lt, unitOf(m), acc);
    }
    if (below >= 0) messageStore(set + below, w[0], tag);
    if (above >= 0) messageStore(set + above, edge, tag);
    if (side >= 0) {
#pragma unroll
      for (int k = 0; k < C; ++k) {
        if ((have >> k) & 1u) messageStore(set + side + (k / K) * teams * a.z.B + k % K, w[k], tag);
      }
    }
    __syncthreads();  // the units' sums of the warps
    unitPublish(t, a, set, 0, a.units, tag);
    if constexpr (!kSplit) {
      messageWaitAll(t, set, from, tag, kFaultHaloWait, hw);
      sumsCollect(t, a, set, tag, 0, T >> 5);
    }
    __syncthreads();  // the sums
    if (!z.step(t, a.unitCount, S.tolerance, S.cap)) break;
    // ---- p, s, x, r and the next u ----
    if constexpr (!kSplit) {
#pragma unroll
      for (int k = 0; k < kHeld; ++k) {
        if (from[k] >= 0) updateBorder(t, S, load, a, z, hr, U, h0 + k * hStep, place[k], hw[k], odd);
      }
      for (int h = h0 + kHeld * hStep; h < border; h += hStep) {
        const int at = source(h);
        if (at < 0) continue;
        updateBorder(t, S, load, a, z, hr, U, h, a.place(h), messageWait(t, set + at, tag, kFaultHaloWait), odd);
      }
    }
#pragma unroll
    for (int k = 0; k < C; ++k) {
      s[k] = fma(z.beta, s[k], w[k]);
      r[k] = fma(-z.alpha, s[k], r[k]);
      double* const place = U + first[k / K] + (k % K) * SW;
      const double before = kU ? u[kU ? k : 0] : *place;
      double next = r[k] * (kAll ? di[kAll ? k : 0] : mine[(2 * C + k) * T]);
      if (odd && (oddCells & (1u << k))) next = wideCgPrecondition(r[k], S.D[cellOf(k)]);
      if constexpr (kU) u[k] = next;
      if ((have >> k) & 1u) *place = next;
      if constexpr (kPx) {
        p[k] = fma(z.beta, p[k], before);
        x[k] = fma(z.alpha, p[k], x[k]);
      } else {
        const double pc = fma(z.beta, mine[k * T], before);
        mine[k * T] = pc;
        mine[(C + k) * T] = fma(z.alpha, pc, mine[(C + k) * T]);
      }
    }
    __syncthreads();  // u
  }
#pragma unroll
  for (int k = 0; k < C; ++k) {
    if ((have >> k) & 1u) S.x[cellOf(k)] = kPx ? x[kPx ? k : 0] : mine[(C + k) * T];
  }
  team.epoch = t.epoch;
  team.barriers = t.barriers;
  return WideCgResult{z.iterations, z.initial, z.final, z.converged};
}

/// The form for any shape: every array in memory, on chip as far as
/// `smemBytes` reach, the rest in the CTA's part of S.spill.
template <typename Loader>
__device__ __noinline__ WideCgResult wideCgAnyTile(WideTeam& team, const WideCgSystem& system, const Loader& load,
                                                   int smemBytes) {
  WideTeam t = team;
  const WideCgSystem S = system;
  extern __shared__ double dyn[];
  const WideCgTile a(t, S.wakeAnywhere);
  const int T = t.T, tid = t.tid, NI = t.NI, SW = a.stride, border = a.border();
  const long long plane = wideCgPlane(a.z), slots = static_cast<long long>(a.z.rounds) * a.z.K * a.z.passes * T;
  double* next = dyn;
  double* back = S.spill + S.spillStride * t.rank;
  long long left = smemBytes / 8;
  auto array = [&](long long n) {
    double* out;
    if (n <= left) {
      out = next;
      next += n;
      left -= n;
    } else {
      out = back;
      back += n;
    }
    return out;
  };
  double* const U = array(plane);
  double* const hr = array(3 * wideCgBorder(a.z));
  double* const r = array(slots) + tid;
  double* const w = array(slots) + tid;
  double* const s = array(slots) + tid;
  double* const p = array(slots) + tid;
  double* const x = array(slots) + tid;
  double* const di = array(slots) + tid;
  double* const sN = array(plane);
  double* const sE = array(plane);
  double* const hs = hr + border;
  double* const hd = hs + border;
  // f(slot, lr, q) for the thread's cells of its team's unit, rows first
  auto unitCells = [&](int unit, auto&& f) {
    if (!a.working) return;
    for (int kk = 0; kk < a.z.K; ++kk) {
      const int lr = unit * a.z.B + a.g * a.z.K + kk;
      if (lr >= a.rows) break;
      int slot = (unit / a.z.teams * a.z.K + kk) * a.z.passes * T;
      for (int q = a.q; q < a.width; q += a.z.G, slot += T) f(slot, lr, q);
    }
  };
  for (int m = tid; m < plane; m += T) U[m] = sN[m] = sE[m] = 0.0;
  __syncthreads();
  wideCgLoadCoefficients(t, load, a, sN, sE);
  bool odd = wideCgLoadBorder(t, S, load, a, U, hr);
  for (int unit = a.team; unit < a.units; unit += a.z.teams) {
    unitCells(unit, [&](int slot, int lr, int q) {
      const int i = a.i0 + q, j = a.j0 + lr, c = j * NI + i;
      const double D = S.D[c], rc = load.first(c, i, j), d = wideCgReciprocal(D);
      if (!isfinite(d)) odd = true;
      r[slot] = rc;
      w[slot] = s[slot] = p[slot] = 0.0;
      x[slot] = S.x[c];
      di[slot] = d;
      U[(lr + 1) * SW + q + 1] = isfinite(d) ? rc * d : wideCgPrecondition(rc, D);
    });
  }
  odd = __syncthreads_or(odd);
  WideCgScalars z;
  for (;;) {
    if (S.wakeAnywhere) {
      // the wake may couple to any cell: put u where every CTA can read it
      for (int unit = a.team; unit < a.units; unit += a.z.teams) {
        unitCells(unit, [&](int, int lr, int q) { S.u[(a.j0 + lr) * NI + a.i0 + q] = U[(lr + 1) * SW + q + 1]; });
      }
      wideBarrier(t);
    }
    ++t.epoch;
    const unsigned tag = t.epoch;
    ulonglong2* const set = t.mem.messages + ((tag & 1u) ? a.set : 0);
    for (int first = 0; first < max(a.units, 1); first += kUnitBatch) {
      const int last = min(first + kUnitBatch, a.units);
      for (int unit = first + a.team; unit < last; unit += a.z.teams) {
        double acc[3] = {0.0, 0.0, 0.0};
        unitCells(unit, [&](int slot, int lr, int q) {
          const int at = (lr + 1) * SW + q + 1;
          const double uc = U[at], rc = r[slot];
          double y = rc;  // D u is r, unless D has no reciprocal
          if (odd && !isfinite(di[slot])) y = S.D[(a.j0 + lr) * NI + a.i0 + q] * uc;
          double us = U[at - SW];
          if (a.j0 + lr == 0 && !a.splitWake) {
            const int k = load.wake(a.i0 + q);
            if (k >= 0) us = S.wakeAnywhere ? __ldcg(S.u + k) : U[SW + k + 1];
          }
          y = fma(sN[at], us, y);
          y = fma(sN[at + SW], U[at + SW], y);
          y = fma(sE[at], U[at - 1], y);
          y = fma(sE[at + 1], U[at + 1], y);
          w[slot] = y;
          const int below = a.toBelow(t, q, lr), above = a.toAbove(t, q, lr), side = a.toSide(t, q, lr);
          if (below >= 0) messageStore(set + below, y, tag);
          if (above >= 0) messageStore(set + above, y, tag);
          if (side >= 0) messageStore(set + side, y, tag);
          acc[0] = fma(rc, uc, acc[0]);
          acc[1] = fma(y, uc, acc[1]);
          acc[2] += fabs(rc);
        });
        __syncwarp();
        if (a.team < a.z.teams) unitPartial(t, a.lt, unit - first, acc);
      }
      __syncthreads();
      unitPublish(t, a, set, first, last, tag);
      __syncthreads();
    }
    sumsCollect(t, a, set, tag, 0, T >> 5);
    __syncthreads();
    if (!z.step(t, a.unitCount, S.tolerance, S.cap)) break;
    for (int h = tid; h < border; h += T) {
      const int c = a.cell(t, load, h);
      if (c < 0) continue;
      const double hw = messageWait(t, set + a.source(t, load, h), tag, kFaultHaloWait);
      const double sc = fma(z.beta, hs[h], hw), rc = fma(-z.alpha, sc, hr[h]), d = hd[h];
      hs[h] = sc;
      hr[h] = rc;
      U[a.place(h)] = isfinite(d) ? rc * d : wideCgPrecondition(rc, S.D[c]);
    }
    for (int unit = a.team; unit < a.units; unit += a.z.teams) {
      unitCells(unit, [&](int slot, int lr, int q) {
        const int at = (lr + 1) * SW + q + 1;
        const double sc = fma(z.beta, s[slot], w[slot]);
        const double rc = fma(-z.alpha, sc, r[slot]);
        const double pc = fma(z.beta, p[slot], U[at]);
        const double d = di[slot];
        s[slot] = sc;
        r[slot] = rc;
        p[slot] = pc;
        U[at] = (odd && !isfinite(d)) ? wideCgPrecondition(rc, S.D[(a.j0 + lr) * NI + a.i0 + q]) : rc * d;
        x[slot] = fma(z.alpha, pc, x[slot]);
      });
    }
    __syncthreads();
  }
  for (int unit = a.team; unit < a.units; unit += a.z.teams) {
    unitCells(unit, [&](int slot, int lr, int q) { S.x[(a.j0 + lr) * NI + a.i0 + q] = x[slot]; });
  }
  team.epoch = t.epoch;
  team.barriers = t.barriers;
  return WideCgResult{z.iterations, z.initial, z.final, z.converged};
}

/// The whole solve by every thread of the team, in the block's dynamic shared
/// memory of `smemBytes`; on return x is written (no barrier after it). The team is
/// whole rows of CTAs, one per column tile in each and no more rows than units (R is
/// columnTiles * RT: wideUsefulCtas, wideChooseCtas). A CTA without a unit would
/// publish nothing, so the others could overwrite the messages it waits for. `any`:
/// the form for any shape.
template <typename Loader>
DEV WideCgResult wideCg(WideTeam& t, const WideCgSystem& S, const Loader& load, int smemBytes, bool any) {
  const WideCgShape z = wideCgShape(t.NI, t.NJ, t.R, t.T);
  switch ((any || S.wakeAnywhere) ? 0 : wideCgForm(z, t.T, smemBytes)) {
    case 16: return wideCgUnrolledTile<2, 1, true>(t, S, load);
    case 24: return wideCgUnrolledTile<3, 1, true>(t, S, load);
    case 32: return wideCgUnrolledTile<4, 1, true>(t, S, load);
    case 17: return wideCgUnrolledTile<2, 1, false>(t, S, load);
    case 18: return wideCgUnrolledTile<2, 2, false>(t, S, load);
    case 20: return wideCgUnrolledTile<2, 4, false>(t, S, load);
    case 33: return wideCgUnrolledTile<4, 1, false>(t, S, load);
    case 34: return wideCgUnrolledTile<4, 2, false>(t, S, load);
    default: break;
  }
  return wideCgAnyTile(t, S, load, smemBytes);
}

}  // namespace cfdb
