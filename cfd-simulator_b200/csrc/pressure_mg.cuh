// pressure_mg.cuh - the mixed form's pressure-correction solve (included by
// simple_kernel.cu inside its anonymous namespace).
//
// The plain form runs the reference's Jacobi-PCG (LinearSystem.cpp:118-210)
// and, at its cap of 200 iterations, reduces the L1 residual of the p'
// system by only ~2.5x on a 384x96 C-grid (it would need ~1000 iterations
// for the reference's 1% target). The mixed form solves the same system to
// the same stopping rule (sum |r| <= tol * sum |r0|) with a stronger inner
// solver, at most `mgCap` iterations (the settings' inner_iterations):
//
//   outer (FP64):  x = 0, r = b;  repeat: inner solve A e = r in FP32,
//                  x += e, r = b - A x (FP64 rows), stop on the L1 rule.
//   inner (FP32):  flexible CG (Polak-Ribiere beta, dot products and norms
//                  accumulated in FP64) preconditioned by one multigrid
//                  V-cycle per iteration.
//   V-cycle:       2x2 aggregation with Galerkin rows, so every level is a
//                  five-point block with the wake-cut map carried over;
//                  red-black Gauss-Seidel (red then black going down, black
//                  then red coming up, so the cycle is symmetric).
//
// What bounds it is the number of steps that need the whole team, each a
// barrier through L2 (1.0 us) around a microsecond or two of work. So:
//   * the red half sweep of a level from a zero start is x = b / D and is
//     written by whatever phase produced b;
//   * a level's way down is one phase, its way up another. A thread has a 2x2
//     aggregate and forms the half sweep's values at its neighbours itself
//     (the same expressions, so the same bits) instead of waiting for them;
//   * the top's way up is one with the CG's dot products;
//   * the coarse levels (a few thousand cells) run on every CTA alike, from
//     its shared memory with __syncthreads only and the last few (64 cells or
//     fewer) on its warp 0 with __syncwarp: nobody waits for one CTA's result.

/// A level that the team shares, as the code sees it (all in global memory).
struct Lv {
  int NI, NJ;
  float *D, *S, *N, *W, *E, *inv, *x, *b;
  const int* wake;
};

/// A level in a CTA's shared memory, its cells apart by colour: cell (i, j) is
/// number k = j * half + i / 2 of colour (i + j) & 1 and lies at colour * n + k.
/// A half sweep's threads then read consecutive words (every other one of a row
/// is two to a bank), a row's coefficients come in one load, and all neighbours
/// of a cell are of the other colour at k, k +- 1 and k +- half.
struct SharedLv {
  int NI, NJ, half, n;
  unsigned perHalf;  // ceil(2^32 / half), for divisions by it
  float4* row;       // S, N, W, E
  float2* diag;      // D, 1 / D
  float *b, *x;
  int* wake;

  DEV int rowOf(int k) const { return (half > 1) ? static_cast<int>(__umulhi(static_cast<unsigned>(k), perHalf)) : k; }
  DEV int at(int i, int j) const { return ((i + j) & 1) * n + j * half + (i >> 1); }
};

/// A coarse level's values for the prolongation: by cell, or apart by colour.
struct CoarseValues {
  const float* x;
  int NI, half, n;  // n: 0 by cell
  DEV float operator()(int I, int J) const {
    return x[(n > 0) ? ((I + J) & 1) * n + J * half + (I >> 1) : J * NI + I];
  }
};

/// The cells [c0, c1) of a level that one worker set covers (c0 even), and a
/// thread's place in it: a CTA's share of the team's, all of a level for a CTA
/// or for one warp.
struct Span {
  int c0, c1, tid, T;
};

DEV Lv globalLevel(const MgLevel& M) {
  return Lv{M.NI, M.NJ, M.D, M.S, M.N, M.W, M.E, M.inv, M.x, M.b, M.wake};
}

/// The level in shared memory, from byte offset M.smem (32 bytes a cell), its
/// wake map from M.smemWake.
DEV SharedLv sharedLevel(const MgLevel& M) {
  extern __shared__ __align__(16) double dyn[];
  char* smem = reinterpret_cast<char*>(dyn);
  SharedLv v;
  v.NI = M.NI;
  v.NJ = M.NJ;
  v.half = (M.NI + 1) >> 1;
  v.n = v.half * M.NJ;
  v.perHalf = M.perHalf;
  v.row = reinterpret_cast<float4*>(smem + M.smem);
  v.diag = reinterpret_cast<float2*>(v.row + 2 * v.n);
  v.b = reinterpret_cast<float*>(v.diag + 2 * v.n);
  v.x = v.b + 2 * v.n;
  v.wake = reinterpret_cast<int*>(smem + M.smemWake);
  return v;
}

/// This CTA's share of n cells, in pieces of 64 so that no two CTAs write one
/// 128-byte line of a half sweep's values.
DEV Span shareOf(const WideTeam& t, int n) {
  const int pieces = (n + 63) / 64;
  return Span{64 * static_cast<int>(static_cast<long long>(pieces) * t.rank / t.R),
              min(64 * static_cast<int>(static_cast<long long>(pieces) * (t.rank + 1) / t.R), n), t.tid, t.T};
}
DEV Span shareOf(const Lv& L, const WideTeam& t) { return shareOf(t, L.NI * L.NJ); }
/// f(c, i, j) for every cell of the span.
template <typename F>
DEV void forCells(const Lv& L, const Span& s, F&& f) {
  for (int c = s.c0 + s.tid; c < s.c1; c += s.T) {
    const int j = c / L.NI;
    f(c, c - j * L.NI, j);
  }
}

/// Neighbour indices of cell (i, j) for branch-free row products: a missing
/// neighbour is replaced by the cell itself, whose coefficient on that side
/// is zero on every level (the fine rows are built that way and the Galerkin
/// sums only ever add existing couplings), so every load can be issued
/// unconditionally and together.
struct Nbrs {
  int s, n, w, e;
};
DEV Nbrs neighbours(const int* wake, int NI, int NJ, int c, int i, int j) {
  int a = c - NI;
  if (j == 0) a = wake[i];  // a load that the other rows must not wait for
  Nbrs q;
  q.s = (a >= 0) ? a : c;
  q.n = (j < NJ - 1) ? c + NI : c;
  q.w = (i > 0) ? c - 1 : c;
  q.e = (i < NI - 1) ? c + 1 : c;
  return q;
}

/// Off-diagonal part of row c applied to x (S, N, W, E).
DEV float offSum(const Lv& L, const float* x, int c, int i, int j) {
  const Nbrs q = neighbours(L.wake, L.NI, L.NJ, c, i, j);
  return L.S[c] * x[q.s] + L.N[c] * x[q.n] + L.W[c] * x[q.w] + L.E[c] * x[q.e];
}

/// The same with every neighbour's value corrected by its aggregate's value
/// on the next coarser level (piecewise-constant prolongation). The
/// aggregates follow from (i, j) directly; a missing neighbour (the cell
/// itself, zero coefficient) uses the cell's own aggregate.
DEV float offSumProlonged(const Lv& L, const CoarseValues& ec, int c, int i, int j) {
  const Nbrs q = neighbours(L.wake, L.NI, L.NJ, c, i, j);
  const int I = i >> 1, J = j >> 1;
  const float eS = (j > 0) ? ec(I, (j - 1) >> 1) : ec((q.s != c) ? (q.s >> 1) : I, J);
  const float eN = ec(I, (j < L.NJ - 1) ? (j + 1) >> 1 : J);
  const float eW = ec((i > 0) ? (i - 1) >> 1 : I, J);
  const float eE = ec((i < L.NI - 1) ? (i + 1) >> 1 : I, J);
  return L.S[c] * (L.x[q.s] + eS) + L.N[c] * (L.x[q.n] + eN) + L.W[c] * (L.x[q.w] + eW) + L.E[c] * (L.x[q.e] + eE);
}

/// Gauss-Seidel half sweep over the cells of one colour. The new values are
/// written through a pointer declared not to alias the one the neighbours
/// are read through (they never touch the same cells: a colour's neighbours
/// are all of the other colour), so consecutive cells' loads can overlap.
template <bool kProlonged>
DEV void sweepCells(const Lv& L, const Span& s, int colour, const CoarseValues& ec) {
  if ((L.NI & 1) != 0) {
    // the coarsest level may have an odd width: plain loop
    forCells(L, s, [&](int c, int i, int j) {
      if (((i + j) & 1) != colour) return;
      const float off = kProlonged ? offSumProlonged(L, ec, c, i, j) : offSum(L, L.x, c, i, j);
      L.x[c] = (L.b[c] - off) * L.inv[c];
    });
    return;
  }
  // cells (2m, 2m + 1) are one of each colour
  const int half = L.NI >> 1, last = s.c1 >> 1;
  auto cellOf = [&](int m, int& c, int& i, int& j) {
    j = m / half;
    i = 2 * (m - j * half) + ((colour + j) & 1);
    c = j * L.NI + i;
  };
  auto value = [&](int c, int i, int j) {
    const float off = kProlonged ? offSumProlonged(L, ec, c, i, j) : offSum(L, L.x, c, i, j);
    return (L.b[c] - off) * L.inv[c];
  };
  // two cells per step, both computed before either is stored, so their
  // loads overlap (a store to x could alias the other cell's loads)
  for (int m = (s.c0 >> 1) + s.tid; m < last; m += 2 * s.T) {
    int cA, iA, jA;
    cellOf(m, cA, iA, jA);
    const float vA = value(cA, iA, jA);
    const int mB = m + s.T;
    if (mB < last) {
      int cB, iB, jB;
      cellOf(mB, cB, iB, jB);
      const float vB = value(cB, iB, jB);
      L.x[cA] = vA;
      L.x[cB] = vB;
    } else {
      L.x[cA] = vA;
    }
  }
}

DEV void colourSweep(const Lv& L, const Span& s, int colour) { sweepCells<false>(L, s, colour, CoarseValues{}); }

/// The black half sweep that opens post-smoothing, with the coarse
/// correction ec added to the neighbours on the fly.
DEV void colourSweepProlonged(const Lv& L, const Span& s, const CoarseValues& ec) { sweepCells<true>(L, s, 1, ec); }

/// Sum of the fine residual b - A x over the aggregate of coarse cell (I, J).
DEV float aggregateResidual(const Lv& F, int I, int J) {
  float sum = 0.0f;
  for (int bj = 0; bj < 2; ++bj) {
    const int jf = 2 * J + bj;
    if (jf >= F.NJ) break;
#pragma unroll
    for (int ai = 0; ai < 2; ++ai) {
      const int fi = 2 * I + ai, f = jf * F.NI + fi;
      sum += F.b[f] - F.D[f] * F.x[f] - offSum(F, F.x, f, fi, jf);
    }
  }
  return sum;
}

/// Restrict the fine residual b - A x to the coarse right-hand side (sum over
/// each aggregate). With `start`, also begin the coarse level: red cells
/// b / D, black 0.
template <bool kStart>
DEV void restrictCells(const Lv& F, const Lv& C, const Span& s) {
  float* __restrict__ bw = C.b;
  float* __restrict__ xw = C.x;
#pragma unroll 2
  for (int cc = s.c0 + s.tid; cc < s.c1; cc += s.T) {
    const int J = cc / C.NI, I = cc - J * C.NI;
    const float val = aggregateResidual(F, I, J);
    bw[cc] = val;
    if (kStart) xw[cc] = (((I + J) & 1) == 0) ? val * C.inv[cc] : 0.0f;
  }
}

/// A five-point row.
struct Row5 {
  float D, S, N, W, E;
};
/// Galerkin row of coarse cell (I, J): P^T A P with P the 2x2 aggregation, from
/// the rows fine(i, j) of an NI x NJ level. Couplings inside an aggregate join
/// the diagonal; the others are summed per side. Row 0's S couplings cross the
/// wake cut to the partner aggregate.
template <typename Fine>
DEV Row5 galerkin(int NI, int NJ, const int* wake, int I, int J, Fine&& fine) {
  Row5 C{0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
  for (int bj = 0; bj < 2; ++bj) {
    const int jf = 2 * J + bj;
    if (jf >= NJ) break;
#pragma unroll
    for (int ai = 0; ai < 2; ++ai) {
      const int fi = 2 * I + ai;
      const Row5 f = fine(fi, jf);
      C.D += f.D;
      if (jf > 0) {
        if (bj == 1) C.D += f.S; else C.S += f.S;
      } else if (wake[fi] >= 0) {
        C.S += f.S;
      }
      if (jf < NJ - 1) {
        if (bj == 0) C.D += f.N; else C.N += f.N;
      }
      if (fi > 0) {
        if (ai == 1) C.D += f.W; else C.W += f.W;
      }
      if (fi < NI - 1) {
        if (ai == 0) C.D += f.E; else C.E += f.E;
      }
    }
  }
  return C;
}
DEV float inverse(float D) { return (D != 0.0f) ? 1.0f / D : 0.0f; }

// ---- one phase down, one phase up -----------------------------------------------

/// What a half sweep makes of black cell (i, j), from the red cells' x. Every load
/// is unconditional, so they overlap: a missing neighbour is the cell itself.
DEV float blackDown(const Lv& L, int c, int i, int j) { return (L.b[c] - offSum(L, L.x, c, i, j)) * L.inv[c]; }
/// The same with the red cells' x corrected from the coarse level.
DEV float blackUp(const Lv& L, const CoarseValues& ec, int c, int i, int j) {
  return (L.b[c] - offSumProlonged(L, ec, c, i, j)) * L.inv[c];
}

/// The black cells that aggregate (I, J) and its red cells' rows meet:
/// value(c, i, j) of each. Red are (2I, 2J) and (2I + 1, 2J + 1), black the other
/// two (`east`, `north`) and four around: below and west of the first red, above
/// and east of the second. Where there is none the first black cell's value
/// stands in (the red cell's coefficient on that side is zero).
struct Blacks {
  float east, north, below, west, above, right;
};
template <typename Value>
DEV Blacks blacksOf(const Lv& L, int I, int J, Value&& value) {
  const int i = 2 * I, j = 2 * J;
  const bool two = j + 1 < L.NJ;
  auto at = [&](bool there, int ib, int jb) {
    ib = there ? ib : i + 1;
    jb = there ? jb : j;
    return value(jb * L.NI + ib, ib, jb);
  };
  int iS = i, jS = j - 1;
  if (j == 0) {
    iS = L.wake[i];
    jS = 0;
  }
  Blacks k;
  k.east = at(true, i + 1, j);
  k.north = at(two, i, j + 1);
  k.below = at(iS >= 0, iS, jS);
  k.west = at(i > 0, i - 1, j);
  k.above = at(j + 2 < L.NJ, i + 1, j + 2);
  k.right = at(two && i + 2 < L.NI, i + 2, j + 1);
  return k;
}

/// A level's way down with one sweep: the black half sweep and the restriction
/// of its residual, from the red start. The black values are used and not kept
/// (the way up starts with that half sweep). kStart: begin the coarse level, red
/// cells b / D, black 0. 768x192 on 148 CTAs: 2.8 us and a barrier; as two
/// phases on 16 CTAs it took 6.4 and 6.7.
template <bool kStart>
DEV void levelDown(const Lv& F, const Lv& C, const Span& s) {
  float* __restrict__ bw = C.b;
  float* __restrict__ xw = C.x;
  for (int cc = s.c0 + s.tid; cc < s.c1; cc += s.T) {
    const int J = cc / C.NI, I = cc - J * C.NI;
    const int c0 = 2 * J * F.NI + 2 * I, c1 = c0 + F.NI;
    const Blacks k = blacksOf(F, I, J, [&](int c, int i, int j) { return blackDown(F, c, i, j); });
    auto residual = [&](int c, float x, float s_, float n, float w, float e) {
      return F.b[c] - F.D[c] * x - (F.S[c] * s_ + F.N[c] * n + F.W[c] * w + F.E[c] * e);
    };
    auto blackResidual = [&](int c, int i, int j, float x) {
      return F.b[c] - F.D[c] * x - offSum(F, F.x, c, i, j);
    };
    float sum = 0.0f;
    sum += residual(c0, F.x[c0], k.below, k.north, k.west, k.east);
    sum += blackResidual(c0 + 1, 2 * I + 1, 2 * J, k.east);
    if (2 * J + 1 < F.NJ) {
      sum += blackResidual(c1, 2 * I, 2 * J + 1, k.north);
      sum += residual(c1 + 1, F.x[c1 + 1], k.east, k.above, k.north, k.right);
    }
    bw[cc] = sum;
    if (kStart) xw[cc] = (((I + J) & 1) == 0) ? sum * C.inv[cc] : 0.0f;
  }
}

/// A level's way up with one sweep, for aggregate (I, J): the coarse correction
/// added, the black half sweep, the red one. F.x holds the red cells' values from
/// the way down; the new ones of the aggregate's cells go to y.
DEV void aggregateUp(const Lv& F, const CoarseValues& ec, int I, int J, float* __restrict__ y) {
  const int c0 = 2 * J * F.NI + 2 * I, c1 = c0 + F.NI;
  const Blacks k = blacksOf(F, I, J, [&](int c, int i, int j) { return blackUp(F, ec, c, i, j); });
  auto red = [&](int c, float s_, float n, float w, float e) {
    const float off = F.S[c] * s_ + F.N[c] * n + F.W[c] * w + F.E[c] * e;
    return (F.b[c] - off) * F.inv[c];
  };
  const float first = red(c0, k.below, k.north, k.west, k.east);
  if (2 * J + 1 < F.NJ) {
    const float second = red(c1 + 1, k.east, k.above, k.north, k.right);
    y[c1] = k.north;
    y[c1 + 1] = second;
  }
  y[c0] = first;
  y[c0 + 1] = k.east;
}

// ---- the coarse levels on one CTA -----------------------------------------------

/// A half sweep of colour `colour` by threads tid, tid + T, ...; `prolonged`: the
/// neighbours' values corrected from the coarser level C.
DEV void sharedSweep(const SharedLv& A, int colour, bool prolonged, const SharedLv& C, int tid, int T) {
  const float* const other = A.x + (1 - colour) * A.n;
  float* const own = A.x + colour * A.n;
#pragma unroll 1
  for (int k = tid; k < A.n; k += T) {
    const int j = A.rowOf(k), h = k - j * A.half, odd = (colour + j) & 1, i = 2 * h + odd;
    if (i >= A.NI) continue;
    const float4 row = A.row[colour * A.n + k];
    // a missing neighbour: any value, its coefficient is zero
    auto value = [&](bool there, int at, int I, int J) {
      float v = other[there ? at : k];
      if (prolonged) v += C.x[there ? C.at(I, J) : 0];
      return v;
    };
    const int I = i >> 1, J = j >> 1;
    int south = k - A.half, Is = I;
    if (j == 0) {
      const int a = A.wake[i];
      south = (a >= 0) ? a >> 1 : -1;
      Is = a >> 1;
    }
    const float vS = value(south >= 0, south, Is, (j > 0) ? (j - 1) >> 1 : 0);
    const float vN = value(j < A.NJ - 1, k + A.half, I, (j + 1) >> 1);
    const float vW = value(i > 0, k - 1 + odd, (i - 1) >> 1, J);
    const float vE = value(i < A.NI - 1, k + odd, (i + 1) >> 1, J);
    const float off = row.x * vS + row.y * vN + row.z * vW + row.w * vE;
    own[k] = (A.b[colour * A.n + k] - off) * A.diag[colour * A.n + k].y;
  }
}

/// Restrict the residual b - A x of level A to the right-hand side of level C,
/// and begin that: red cells b / D, black 0. Coarse cells in rows of
/// 2 * C.half places, so that neighbouring threads read neighbouring words.
DEV void sharedRestrict(const SharedLv& A, const SharedLv& C, int tid, int T) {
#pragma unroll 1
  for (int m = tid; m < A.half * C.NJ; m += T) {
    const int J = A.rowOf(m), I = m - J * A.half;  // C.NI is A.half
    const int k0 = 2 * J * A.half + I, k1 = k0 + A.half, i = 2 * I, j = 2 * J;
    const bool two = j + 1 < A.NJ, more = j + 2 < A.NJ, first = I == 0, last = i + 2 >= A.NI;
    const float* const red = A.x;
    const float* const black = A.x + A.n;
    int sR = k0 - A.half, sB = sR;  // south of the first red, of the first black
    if (j == 0) {
      const int aR = A.wake[i], aB = A.wake[i + 1];
      sR = (aR >= 0) ? aR >> 1 : -1;
      sB = (aB >= 0) ? aB >> 1 : -1;
    }
    // a missing neighbour: any value, its coefficient is zero
    auto pick = [&](const float* x, bool there, int at) { return x[there ? at : k0]; };
    auto residual = [&](int at, float x, float s_, float n, float w, float e) {
      const float4 row = A.row[at];
      return A.b[at] - A.diag[at].x * x - (row.x * s_ + row.y * n + row.z * w + row.w * e);
    };
    const float r0 = red[k0], b0 = black[k0];
    const float r1 = pick(red, two, k1), b1 = pick(black, two, k1);
    float sum = 0.0f;
    sum += residual(k0, r0, pick(black, sR >= 0, sR), b1,
                    pick(black, !first, k0 - 1), b0);
    sum += residual(A.n + k0, b0, pick(red, sB >= 0, sB), r1, r0,
                    pick(red, !last, k0 + 1));
    if (two) {
      sum += residual(A.n + k1, b1, r0, pick(red, more, k1 + A.half), pick(red, !first, k1 - 1), r1);
      sum += residual(k1, r1, b0, pick(black, more, k1 + A.half), b1, pick(black, !last, k1 + 1));
    }
    const int at = C.at(I, J);
    C.b[at] = sum;
    C.x[at] = (((I + J) & 1) == 0) ? sum * C.diag[at].y : 0.0f;
  }
}

DEV CoarseValues sharedValues(const SharedLv& C) { return CoarseValues{C.x, C.NI, C.half, C.n}; }

/// The V-cycle of the shared-memory levels, by every CTA alike: their
/// right-hand side is where the team restricted it (global memory); the result
/// stays in shared memory. 96x24 cells and the four levels below: 10 us; by
/// cell, with a division and eight loads of separate arrays a cell, 15.5 us. One
/// phase a level as above is slower here (384x96: 1.80 -> 1.97 ms a call).
DEV void sharedCycle(const Multigrid& G) {
  const int L = G.levels, m = G.distributed, w = G.warpFrom;
  const int tid = static_cast<int>(threadIdx.x);
  {
    const SharedLv C = sharedLevel(G.lv[m]);
    const float* bg = G.lv[m].b;
    for (int k = tid; k < 2 * C.n; k += static_cast<int>(blockDim.x)) {
      const int colour = (k >= C.n) ? 1 : 0, at = k - colour * C.n, j = C.rowOf(at);
      const int i = 2 * (at - j * C.half) + ((colour + j) & 1);
      if (i >= C.NI) continue;
      const float b = bg[j * C.NI + i];
      C.b[k] = b;
      C.x[k] = (colour == 0) ? b * C.diag[k].y : 0.0f;
    }
  }
  // one piece of code for every level: what a step costs is its latency, the
  // fetch of its instructions included
  auto meet = [&](int l) {
    if (l >= w) __syncwarp();
    else __syncthreads();
  };
#pragma unroll 1
  for (int l = m; l < L; ++l) {
    if (l == w) {
      __syncthreads();
      if (tid >= 32) break;
    }
    const SharedLv A = sharedLevel(G.lv[l]), C = sharedLevel(G.lv[min(l + 1, L - 1)]);
    const int T = (l >= w) ? 32 : static_cast<int>(blockDim.x);
    const int halves = 2 * ((l == L - 1) ? G.coarse : G.pre) - 1;
#pragma unroll 1
    for (int h = 0; h < halves; ++h) {
      meet(l);
      sharedSweep(A, 1 - (h & 1), false, C, tid, T);
    }
    if (l == L - 1) break;
    meet(l);
    sharedRestrict(A, C, tid, T);
  }
#pragma unroll 1
  for (int l = ((tid < 32) ? L - 1 : min(w, L - 1)) - 1; l >= m; --l) {
    const SharedLv A = sharedLevel(G.lv[l]), C = sharedLevel(G.lv[l + 1]);
    const int T = (l >= w) ? 32 : static_cast<int>(blockDim.x);
#pragma unroll 1
    for (int h = 0; h < 2 * G.post; ++h) {
      meet(l);
      sharedSweep(A, 1 - (h & 1), h == 0, C, tid, T);
    }
  }
  __syncthreads();
}

/// The shared-memory levels' rows, by every CTA alike, from the last level in
/// global memory. Ends with a barrier of the block.
DEV void sharedRows(const Multigrid& G) {
  const int tid = static_cast<int>(threadIdx.x), T = static_cast<int>(blockDim.x);
  for (int l = G.distributed; l < G.levels; ++l) {
    const SharedLv C = sharedLevel(G.lv[l]);
    for (int i = tid; i < C.NI; i += T) C.wake[i] = G.lv[l].wake[i];
    for (int k = tid; k < 2 * C.n; k += T) C.x[k] = 0.0f;  // the places without a cell stay so
  }
  __syncthreads();
  for (int l = G.distributed; l < G.levels; ++l) {
    const SharedLv C = sharedLevel(G.lv[l]);
    auto rows = [&](int NI, int NJ, const int* wake, auto&& fine) {
      for (int m = tid; m < C.NI * C.NJ; m += T) {
        const int J = m / C.NI, I = m - J * C.NI, at = C.at(I, J);
        const Row5 r = galerkin(NI, NJ, wake, I, J, fine);
        C.row[at] = make_float4(r.S, r.N, r.W, r.E);
        C.diag[at] = make_float2(r.D, inverse(r.D));
      }
    };
    if (l == G.distributed) {
      const Lv F = globalLevel(G.lv[l - 1]);
      rows(F.NI, F.NJ, F.wake, [&](int i, int j) {
        const int f = j * F.NI + i;
        return Row5{F.D[f], F.S[f], F.N[f], F.W[f], F.E[f]};
      });
    } else {
      const SharedLv F = sharedLevel(G.lv[l - 1]);
      rows(F.NI, F.NJ, F.wake, [&](int i, int j) {
        const float4 q = F.row[F.at(i, j)];
        return Row5{F.diag[F.at(i, j)].x, q.x, q.y, q.z, q.w};
      });
    }
    __syncthreads();
  }
}

/// What the way up of level l adds: level l + 1's result.
DEV CoarseValues coarseResult(const Multigrid& G, int l, bool phased) {
  const int c = l + 1;
  if (c >= G.distributed) return sharedValues(sharedLevel(G.lv[c]));
  return CoarseValues{(phased || G.post > 1 || c == G.levels - 1) ? G.lv[c].x : G.lv[c].y, G.lv[c].NI, 0, 0};
}

/// z = M r, one V-cycle, and sums of the caller: item(c, z, acc) for every
/// cell, with its new z. On entry (before any barrier) the fine level's red cells
/// of G.zs hold r / D and its black cells 0; z is written.
template <int K, typename Item>
DEV void vcycle(const Multigrid& G, WideTeam& t, const WideRange& aggregates, bool phased, float* z, double (&out)[K],
                Item&& item) {
  const int L = G.levels, Ld = G.distributed;
  auto view = [&](int l) {
    Lv v = globalLevel(G.lv[l]);
    if (l == 0) {
      v.x = G.zs;
      v.b = G.r;
    }
    return v;
  };
  for (int l = 0; l < Ld; ++l) {
    const Lv F = view(l);
    const Span s = shareOf(F, t);
    const bool coarsest = (l == L - 1);
    const int sweeps = coarsest ? G.coarse : G.pre;
    wideBarrier(t);
    const bool apart = phased || sweeps > 1;  // a phase per half sweep
    if (coarsest || apart) {
      colourSweep(F, s, 1);
      for (int k = 1; k < sweeps; ++k) {
        wideBarrier(t);
        colourSweep(F, s, 0);
        wideBarrier(t);
        colourSweep(F, s, 1);
      }
      if (coarsest) break;
      wideBarrier(t);
    }
    const Lv C = globalLevel(G.lv[l + 1]);
    const Span sc = shareOf(C, t);
    if (apart) {
      if (l + 1 < Ld) restrictCells<true>(F, C, sc);
      else restrictCells<false>(F, C, sc);
    } else {
      if (l + 1 < Ld) levelDown<true>(F, C, sc);
      else levelDown<false>(F, C, sc);
    }
  }
  if (Ld < L) {
    wideBarrier(t);
    sharedCycle(G);
  }
  for (int l = ((Ld < L) ? Ld : L - 1) - 1; l >= 0; --l) {
    const Lv F = view(l);
    const CoarseValues ec = coarseResult(G, l, phased);
    const int NIc = G.lv[l + 1].NI;
    if (l + 1 < Ld) wideBarrier(t);
    if (phased || G.post > 1) {
      for (int h = 0; h < 2 * G.post; ++h) {
        if (h > 0) wideBarrier(t);
        if (h == 0) colourSweepProlonged(F, shareOf(F, t), ec);
        else colourSweep(F, shareOf(F, t), (h & 1) ? 0 : 1);
      }
    } else if (l > 0) {
      const Span s = shareOf(t, NIc * G.lv[l + 1].NJ);
      for (int cc = s.c0 + s.tid; cc < s.c1; cc += s.T) {
        const int J = cc / NIc;
        aggregateUp(F, ec, cc - J * NIc, J, G.lv[l].y);
      }
    } else {
      wideItemSums(t, aggregates, out, [&](int cc, double (&acc)[K]) {
        const int J = cc / NIc, I = cc - J * NIc, c0 = 2 * J * F.NI + 2 * I;
        aggregateUp(F, ec, I, J, z);
        item(c0, z[c0], acc);
        item(c0 + 1, z[c0 + 1], acc);
        if (2 * J + 1 < F.NJ) {
          item(c0 + F.NI, z[c0 + F.NI], acc);
          item(c0 + F.NI + 1, z[c0 + F.NI + 1], acc);
        }
      });
      return;
    }
  }
  // several sweeps on the way up, or one level alone: z is where they left it
  wideBarrier(t);
  if (L == 1) {
    colourSweep(view(0), shareOf(view(0), t), 0);
    wideBarrier(t);
  }
  wideSums(t, out, [&](int c, int, int, double (&acc)[K]) {
    const float v = G.zs[c];
    z[c] = v;
    item(c, v, acc);
  });
}

/// The pressure-correction solve of the mixed form. On entry I.x = 0 and
/// I.r = I.pB; `initial` = sum |b|. Returns the inner iterations run (the
/// monitor's pressure iterations). `phased`: the V-cycle with a phase per half
/// sweep.
__device__ __noinline__ int pressureMixed(const Instance& I, WideTeam& team, double initial, bool phased) {
  // The multigrid descriptor is read at every phase: keep a copy on chip.
  __shared__ Multigrid mgs;
  WideTeam t = team;
  {
    const int* src = reinterpret_cast<const int*>(&I.mg);
    int* dst = reinterpret_cast<int*>(&mgs);
    for (int k = t.tid; k < static_cast<int>(sizeof(Multigrid) / sizeof(int)); k += t.T) dst[k] = src[k];
    __syncthreads();
  }
  const Multigrid& G = mgs;
  const int NI = I.NI, NJ = I.NJ;
  const WideRange aggregates = wideRange(t, (G.levels > 1) ? G.lv[1].NI * G.lv[1].NJ : t.N);

  // ---- set-up: the fine rows in FP32, then the Galerkin levels ----
  const Lv F0 = globalLevel(G.lv[0]);
  wideCells(t, [&](int c, int i, int j) {
    F0.D[c] = static_cast<float>(I.pD[c]);
    F0.S[c] = static_cast<float>((j > 0) ? I.pN[j * NI + i] : ((I.acrossJ0[i] >= 0) ? I.pN[i] : 0.0));
    F0.N[c] = static_cast<float>((j < NJ - 1) ? I.pN[(j + 1) * NI + i] : 0.0);
    F0.W[c] = static_cast<float>((i > 0) ? I.pE[j * (NI + 1) + i] : 0.0);
    F0.E[c] = static_cast<float>((i < NI - 1) ? I.pE[j * (NI + 1) + i + 1] : 0.0);
    F0.inv[c] = inverse(F0.D[c]);
  });
  wideBarrier(t);
  for (int l = 1; l < G.distributed; ++l) {
    const Lv F = globalLevel(G.lv[l - 1]), C = globalLevel(G.lv[l]);
    forCells(C, shareOf(C, t), [&](int c, int i, int j) {
      const Row5 r = galerkin(F.NI, F.NJ, F.wake, i, j, [&](int fi, int fj) {
        const int f = fj * F.NI + fi;
        return Row5{F.D[f], F.S[f], F.N[f], F.W[f], F.E[f]};
      });
      C.D[c] = r.D; C.S[c] = r.S; C.N[c] = r.N; C.W[c] = r.W; C.E[c] = r.E;
      C.inv[c] = inverse(r.D);
    });
    wideBarrier(t);
  }
  if (G.distributed < G.levels) sharedRows(G);

  const double tolAbs = I.cgTol * initial;
  float* r = G.r;
  float* q = G.q;
  float* e = G.e;
  int total = 0;
  for (int refine = 0; refine < 3 && total < I.mgCap; ++refine) {
    // ---- inner solve of A e = r in FP32 ----
    float* zc = G.z0;
    float* zp = G.z1;
    float* dc = G.d0;
    float* dn = G.d1;
    wideCells(t, [&](int c, int i, int j) {
      const float rc = static_cast<float>(I.r[c]);
      r[c] = rc;
      e[c] = 0.0f;
      G.zs[c] = (((i + j) & 1) == 0) ? rc * F0.inv[c] : 0.0f;
    });
    double v1[1];
    vcycle(G, t, aggregates, phased, zc, v1, [&](int c, float z, double (&acc)[1]) {
      acc[0] += static_cast<double>(r[c]) * static_cast<double>(z);
    });
    double rz = v1[0];
    double beta = 0.0;
    for (int it = 0; total < I.mgCap; ++it) {
      // q = A d' with d' = z + beta d, formed for each cell and its neighbours.
      const float fb = static_cast<float>(beta);
      auto dir = [&](int n) { return (it == 0) ? zc[n] : zc[n] + fb * dc[n]; };
      double dq[1];
      wideSums(t, dq, [&](int c, int i, int j, double (&acc)[1]) {
        const Nbrs nb = neighbours(F0.wake, NI, NJ, c, i, j);
        const float dv = dir(c);
        const float y = F0.D[c] * dv + F0.S[c] * dir(nb.s) + F0.N[c] * dir(nb.n) + F0.W[c] * dir(nb.w) +
                        F0.E[c] * dir(nb.e);
        dn[c] = dv;
        q[c] = y;
        acc[0] += static_cast<double>(dv) * static_cast<double>(y);
      });
      {
        float* tmp = dc;
        dc = dn;
        dn = tmp;
      }
      if (!(fabs(dq[0]) > 0.0) || !isfinite(dq[0])) break;
      const float alpha = static_cast<float>(rz / dq[0]);
      // e += alpha d, r -= alpha q, and the next V-cycle's red start z = r / D
      wideCells(t, [&](int c, int i, int j) {
        const float rv = r[c] - alpha * q[c], ev = e[c] + alpha * dc[c];
        const float inv = F0.inv[c];
        e[c] = ev;
        r[c] = rv;
        G.zs[c] = (((i + j) & 1) == 0) ? rv * inv : 0.0f;
      });
      ++total;
      // the V-cycle with r.z_new, r.z_old and sum |r|
      double v3[3];
      vcycle(G, t, aggregates, phased, zp, v3, [&](int c, float z, double (&acc)[3]) {
        const double rc = static_cast<double>(r[c]);
        acc[0] += rc * static_cast<double>(z);
        acc[1] += rc * static_cast<double>(zc[c]);
        acc[2] += fabs(rc);
      });
      if (v3[2] <= tolAbs) break;
      if (!(fabs(rz) > 0.0) || !isfinite(v3[0])) break;
      beta = (v3[0] - v3[1]) / rz;  // Polak-Ribiere: stays a CG for a varying preconditioner
      rz = v3[0];
      float* tmp = zc;
      zc = zp;
      zp = tmp;
    }
    // ---- outer refinement in FP64: x += e, r = b - A x ----
    wideCells(t, [&](int c, int, int) { I.x[c] += static_cast<double>(e[c]); });
    wideBarrier(t);
    double l1[1];
    wideSums(t, l1, [&](int c, int i, int j, double (&acc)[1]) {
      const double rc = I.pB[c] - pressureRow(I, c, i, j, I.x, I.x[c]);
      I.r[c] = rc;
      acc[0] += fabs(rc);
    });
    if (l1[0] <= tolAbs) break;
  }
  team.epoch = t.epoch;
  team.barriers = t.barriers;
  return total;
}
