// Per-track AMR split/merge (Grid::regrid, src/Dimensions/1d.cpp:484-728) with
// the problem module's refinement criterion (Hooks::check_cell_for_regrid, e.g.
// src/Initial/Tests/BM1D.cpp:277-319).
//
// The reference walks the active cells left to right and acts immediately:
// a split inserts a cell (the right half is examined next), a merge removes one
// (a left merge skips the next cell), and the criterion itself reads the live
// track (the outermost active cell and the shock index).  Decisions are
// therefore inherently sequential, but almost every cell is a no-op whose
// decision does not depend on earlier actions.  So:
//   A. all threads evaluate the criterion for every original cell in the
//      original context (bitmasks of split / merge / high-pressure cells); a
//      track where none acts is left as it is;
//   B. one thread replays the loop exactly.  For an untouched original cell the
//      precomputed decision is valid whenever its distance to the shock is the
//      same as in the original context (checked per cell); runs of valid no-op
//      cells are skipped a bitmask word at a time, so the replay costs
//      O(actions + cells/32).  New cells and cells near a moved shock are
//      evaluated in place.  The replay emits the new track as segments
//      (a run of original cells, or one new cell).  A merged cell is never
//      examined itself, so the replay only notes its two cells, and takes its
//      high-pressure mark to be theirs (where they differ, it is formed at
//      once; where a merged cell has to be formed during the replay and its mark
//      is not as assumed, the replay runs again as below);
//   C. all threads form the merged cells (a merged cell's victim may be a merged
//      cell: rounds) and compare their marks with the assumed ones; if one
//      differs, the replay runs again and forms each merged cell as it goes;
//   D. all threads expand the segments into the new track.
// Merged one by one inside the replay, the first regrids of a sweep took 10 of
// its 11 ms per step (thousands of merges per run, each a chain of loads, two
// state conversions and a pressure root on one thread).
#pragma once

#include "physics.cuh"
#include "types.cuh"

namespace gb {

struct RegridScratch {
  double *nprim;                    // [NQS][2N] new cells of run r at 2*off[r] + id
  double *nx, *ndx, *ndtl, *nrifx;  // [2N]
  int *nrif;                        // [2N] right interface: original index, or -1 (then nrifx)
  int *ncur, *nvic;                 // [2N] a merged cell's two cells: original index, or -(id+1)
  int *nstate;                      // [2N] the round that formed the cell, or kMergeLeft / kMergeRight
                                    // (these three share memory with tprim)
  int *seg_start, *seg_src;         // [4N] at 4*off[r]: output position; src >= 0 original, else -(id+1)
  double *tprim;                    // [NQS][N] compaction target (step D)
  double *tx, *tdx, *tdtl, *txI;    // [N]
  long long N;
};

constexpr int kMergeLeft = -1, kMergeRight = -2;  // merged cells still to be formed

// One cell's record: an original (data fetched lazily) or new.
template <class Cfg>
struct RCell {
  double prim[Cfg::NQ];
  double x, dx, dtl;
  double rifx;
  int orig;    // original index, or -1 for a new cell
  int rif;     // right interface: original index, or -1 (position in rifx)
  bool loaded;
};

template <class Cfg>
struct RegridView {
  static constexpr int NQ = Cfg::NQ;
  static constexpr int NQS = Cfg::NQ - 1;
  const double *prim;
  long long N;
  const double *x, *dx, *dtl, *xI;
  long long off;

  __device__ __forceinline__ static int q_of(int s) { return s < 3 ? s : s + 1; }

  __device__ void fetch(RCell<Cfg> &c) const {
    if (c.loaded) return;
    const long long g = off + c.orig;
#pragma unroll
    for (int s = 0; s < NQS; ++s) c.prim[q_of(s)] = prim[s * N + g];
    c.prim[UU2] = 0.;
    c.x = x[g];
    c.dx = dx[g];
    c.dtl = dtl[g];
    c.loaded = true;
  }
  __device__ RCell<Cfg> orig_cell(int k) const {
    RCell<Cfg> c;
    c.orig = k;
    c.rif = k;
    c.rifx = 0.;
    c.loaded = false;
    return c;
  }
};

__device__ __forceinline__ bool bit_of(const uint32_t *w, int k) { return (w[k >> 5] >> (k & 31)) & 1u; }

// first set bit at index >= from and < to, or to
__device__ __forceinline__ int next_set(const uint32_t *w, int from, int to) {
  if (from >= to) return to;
  int wi = from >> 5;
  uint32_t m = w[wi] & (0xffffffffu << (from & 31));
  const int wlast = (to - 1) >> 5;
  while (true) {
    if (m) {
      const int k = (wi << 5) + __ffs(m) - 1;
      return k < to ? k : to;
    }
    if (++wi > wlast) return to;
    m = w[wi];
  }
}

// highest set bit at index in [lo, hi], or -1
__device__ __forceinline__ int last_set(const uint32_t *w, int lo, int hi) {
  if (hi < lo) return -1;
  int wi = hi >> 5;
  uint32_t m = w[wi] & (0xffffffffu >> (31 - (hi & 31)));
  const int wlo = lo >> 5;
  while (true) {
    if (wi == wlo) m &= 0xffffffffu << (lo & 31);
    if (m) return (wi << 5) + 31 - __clz(m);
    if (--wi < wlo) return -1;
    m = w[wi];
  }
}

// Split cell c (between cL and cR) into A | B (Grid::split, 1d.cpp:560-662).
template <class Cfg>
__device__ void split_cells(const RCell<Cfg> &cL, const RCell<Cfg> &c, const RCell<Cfg> &cR, RCell<Cfg> &A,
                            RCell<Cfg> &B) {
  constexpr int NQ = Cfg::NQ;
  const double cenL = make_geom<Cfg>(cL.x, cL.dx).cen;
  const double cen = make_geom<Cfg>(c.x, c.dx).cen;
  const double cenR = make_geom<Cfg>(cR.x, cR.dx).cen;
  double gC[NQ];
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    double gL = (c.prim[q] - cL.prim[q]) / (cen - cenL);
    double gR = (cR.prim[q] - c.prim[q]) / (cenR - cen);
    double gN = (cR.prim[q] - cL.prim[q]) / (cenR - cenL);
    gL = minmod(gL, gN);
    gR = minmod(gR, gN);
    gC[q] = minmod(gL, gR);
  }
  const double x_old = c.x, dl_old = c.dx;
  A.x = x_old - dl_old / 4.;
  B.x = x_old + dl_old / 4.;
  A.dx = dl_old / 2.;
  B.dx = dl_old / 2.;
  const double xL = make_geom<Cfg>(A.x, A.dx).cen;
  const double xR = make_geom<Cfg>(B.x, B.dx).cen;
  const double xI = A.x + A.dx / 2.;
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    const double Sc = c.prim[q];
    A.prim[q] = Sc + gC[q] * (xL - xI);
    B.prim[q] = Sc + gC[q] * (xR - xI);
  }
  A.prim[UU2] = 0.;
  B.prim[UU2] = 0.;
  // the right half reuses the record of the old right neighbour (1d.cpp:577)
  A.dtl = c.dtl;
  B.dtl = cR.dtl;
  A.rif = -1;
  A.rifx = x_old;
  B.rif = c.rif;
  B.rifx = c.rifx;
  A.orig = B.orig = -1;
  A.loaded = B.loaded = true;
}

// Merge cell c with victim v (Grid::merge, 1d.cpp:665-728).
// (With the plain operators: a few lanes merge, and FlatOps' longer code costs
// more instruction fetches than its overlap gains, 1.91 against 1.79 ms per step
// of a sweep's first steps.)
template <class Cfg, class Hooks>
__device__ __forceinline__ void merge_cells(const Phys &ph, const RCell<Cfg> &c, const RCell<Cfg> &v, bool left,
                                            RCell<Cfg> &M, const double *par) {
  constexpr int NQ = Cfg::NQ;
  PlainOps ar;
  double cc[NQ], cv[NQ], cons[NQ];
  prim2cons<Cfg>(ar, ph, c.prim, cc);
  prim2cons<Cfg>(ar, ph, v.prim, cv);
  const double dV_loc = make_geom<Cfg>(ar, c.x, c.dx).dV;
  const double dV_vic = make_geom<Cfg>(ar, v.x, v.dx).dV;
  const auto by = ar.by(dV_loc + dV_vic);
#pragma unroll
  for (int q = 0; q < NQ; ++q) cons[q] = ar.quo0(cc[q] * dV_loc + cv[q] * dV_vic, by);
  if (left) M.x = ((v.x - v.dx / 2.) + (c.x + c.dx / 2.)) / 2.;
  else M.x = ((v.x + v.dx / 2.) + (c.x - c.dx / 2.)) / 2.;
  M.dx = c.dx + v.dx;
#pragma unroll
  for (int q = 0; q < NQ; ++q) M.prim[q] = c.prim[q];
  cons2prim<Cfg, Hooks>(ar, ph, cons, M.prim, nullptr, par);
  M.dtl = c.dtl;
  if (left) {
    M.rif = c.rif;
    M.rifx = c.rifx;
  } else {
    M.rif = v.rif;
    M.rifx = v.rifx;
  }
  M.orig = -1;
  M.loaded = true;
}

// The scratch records of run r's new cells (from 2*off).
template <class Cfg>
__device__ __forceinline__ void store_new_cell(const RegridScratch &S, long long gid, const RCell<Cfg> &c) {
#pragma unroll
  for (int s = 0; s < Cfg::NQ - 1; ++s) S.nprim[s * 2 * S.N + gid] = c.prim[s < 3 ? s : s + 1];
  S.nx[gid] = c.x;
  S.ndx[gid] = c.dx;
  S.ndtl[gid] = c.dtl;
  S.nrif[gid] = c.rif;
  S.nrifx[gid] = c.rifx;
}

// The whole record of cell d (an original, or formed new cell -(id+1)).
template <class Cfg>
__device__ __forceinline__ RCell<Cfg> whole_cell(const RegridView<Cfg> &V, const RegridScratch &S, long long noff,
                                                 int d) {
  RCell<Cfg> c;
  if (d >= 0) {
    c = V.orig_cell(d);
    V.fetch(c);
  } else {
    const long long gid = noff + (-d - 1);
#pragma unroll
    for (int s = 0; s < Cfg::NQ - 1; ++s) c.prim[s < 3 ? s : s + 1] = S.nprim[s * 2 * S.N + gid];
    c.prim[UU2] = 0.;
    c.x = S.nx[gid];
    c.dx = S.ndx[gid];
    c.dtl = S.ndtl[gid];
    c.rif = S.nrif[gid];
    c.rifx = S.nrifx[gid];
    c.orig = -1;
    c.loaded = true;
  }
  return c;
}

// Forms merged cell id from its two cells, the examined one and its victim (the
// cell on its left or right), and stores its record; returns its
// high-pressure mark.  Out of line: it is the regrid's, not the step's.
template <class Cfg, class Hooks>
__device__ __noinline__ bool form_merged(const Phys &ph, const RegridView<Cfg> &V, const RegridScratch &S,
                                         long long noff, int id, int cur, int vic, bool left, const double *par) {
  const RCell<Cfg> c = whole_cell(V, S, noff, cur), v = whole_cell(V, S, noff, vic);
  RCell<Cfg> M;
  merge_cells<Cfg, Hooks>(ph, c, v, left, M, par);
  store_new_cell(S, noff + id, M);
  return Hooks::regrid_marker(par, M.prim);
}

// A cell of the walk: what the decisions need of it.
struct WalkCell {
  int d;      // original index, or -(id+1)
  double dx;  // (of an original: once loaded)
  bool has_dx, hp;
};

// Bit words of one mark per cell of a track of capacity cap, and how many marks
// regrid_track keeps in shared memory (high-pressure, split, merge).
__host__ __device__ constexpr int regrid_words(int cap) { return (cap + 31) / 32; }
constexpr int kRegridMarks = 3;

// Regrid one track; returns the new ntrack.  Called by all threads of the CTA.
// words: kRegridMarks * regrid_words(cap) uint32 of shared memory.
//
// The criterion: Hooks::check_cell_for_regrid(par, dx, prim, i, iS, rOut) for
// the cell at live position i, where iS is the live position of the rightmost
// active cell marked by Hooks::regrid_marker (iLbnd+1 if none) and rOut the
// centre of the outermost active cell -- the two things BM1D.cpp:285-301 reads
// from the live track.  The criterion may depend on i - iS only through whether
// 0 < i - iS < Hooks::REGRID_WINDOW, so a cell's decision in the original track
// stays valid while that test gives the same answer as in the original track.
template <class Cfg, class Hooks, int BS>
__device__ int regrid_track(double *prim, long long N, double *x, double *dx, double *dtl, double *xI,
                            long long off, int n, int cap, const Phys &ph, const double *par,
                            const RegridScratch &S, uint32_t *words, unsigned long long &nsplit,
                            unsigned long long &nmerge) {
  constexpr int NQ = Cfg::NQ;
  constexpr int NQS = NQ - 1;
  const int ng = ph.ngst, iL = ng - 1, iR0 = n - ng;
  const int nw = regrid_words(cap);
  uint32_t *hpw = words, *spw = words + nw, *mgw = words + 2 * nw;
  __shared__ int s_hpmax, s_nnew, s_nseg, s_first, s_nid;
  const double rOut0 = x[off + iR0 - 1];
  auto load = [&](long long g, double *p) {
#pragma unroll
    for (int s = 0; s < NQS; ++s) p[s < 3 ? s : s + 1] = prim[s * N + g];
    p[UU2] = 0.;
  };

  // ---- A. high-pressure bits and the original shock index
  if (threadIdx.x == 0) s_hpmax = -1;
  for (int w = threadIdx.x; w < kRegridMarks * nw; w += BS) words[w] = 0u;
  __syncthreads();
  for (int base = 0; base < n; base += BS) {
    const int k = base + threadIdx.x;
    bool hp = false;
    if (k < n && k >= iL + 1 && k <= iR0 - 1) {
      double p[NQ];
      load(off + k, p);
      hp = Hooks::regrid_marker(par, p);
    }
    const uint32_t b = __ballot_sync(0xffffffffu, hp);
    if ((threadIdx.x & 31) == 0 && k < n) hpw[k >> 5] = b;
    if (hp) atomicMax(&s_hpmax, k);
  }
  __syncthreads();
  const int hpMax = s_hpmax;
  const double iS0 = hpMax >= 0 ? (double)hpMax : (double)(iL + 1);
  // decisions in the original context
  for (int base = 0; base < n; base += BS) {
    const int k = base + threadIdx.x;
    int a = SKIP;
    if (k < n && k >= iL + 1 && k <= iR0 - 1) {
      double p[NQ];
      load(off + k, p);
      a = Hooks::check_cell_for_regrid(par, dx[off + k], p, k, (int)iS0, rOut0);
    }
    const uint32_t bs = __ballot_sync(0xffffffffu, a == SPLIT);
    const uint32_t bm = __ballot_sync(0xffffffffu, a == MERGE);
    if ((threadIdx.x & 31) == 0 && k < n) {
      spw[k >> 5] = bs;
      mgw[k >> 5] = bm;
    }
  }
  __syncthreads();
  bool acts = false;
  for (int w = threadIdx.x; w < nw; w += BS) acts = acts || (spw[w] | mgw[w]) != 0u;
  if (!__syncthreads_or(acts)) return n;  // no cell acts, so none moves, so each decision stands

  const RegridView<Cfg> V{prim, N, x, dx, dtl, xI, off};
  const long long noff = 2 * off;
  unsigned long long walk_splits = 0, walk_merges = 0;

  // the mark of an original or of a split's half, assumed of a cell merged from it
  auto mark_of = [&](int d) {
    if (d >= 0) return bit_of(hpw, d);
    double p[NQ];
#pragma unroll
    for (int s = 0; s < NQS; ++s) p[s < 3 ? s : s + 1] = S.nprim[s * 2 * S.N + noff + (-d - 1)];
    p[UU2] = 0.;
    return Hooks::regrid_marker(par, p);
  };
  // ---- B. sequential replay (thread 0); eager: each merged cell formed at once.
  // False, and the replay is given up, where a merged cell that has to be formed
  // in it does not have the mark assumed of it.
  auto walk = [&](bool eager) -> bool {
    int *seg_start = S.seg_start + 4 * off;
    int *seg_src = S.seg_src + 4 * off;
    int nseg = 0, out = 0, nid = 0;
    int seg_next_orig = -2;  // original index that would extend the open segment
    int hp_final = -1;       // rightmost final position (> iL) holding a high-pressure cell
    int first_change = n;    // first output position that differs from the input
    walk_splits = walk_merges = 0;

    auto emit_orig_range = [&](int k0, int k1) {  // originals [k0, k1) at positions out..
      if (k1 <= k0) return;
      if (!(nseg > 0 && seg_next_orig == k0)) {
        seg_start[nseg] = out;
        seg_src[nseg] = k0;
        ++nseg;
      }
      if (out != k0 && first_change > out) first_change = out;
      const int h = last_set(hpw, k0, k1 - 1);
      if (h >= 0) hp_final = max(hp_final, out + (h - k0));
      out += k1 - k0;
      seg_next_orig = k1;
    };
    auto emit = [&](const WalkCell &c) {
      if (c.d >= 0) {
        emit_orig_range(c.d, c.d + 1);
        return;
      }
      seg_start[nseg] = out;
      seg_src[nseg] = c.d;
      ++nseg;
      seg_next_orig = -2;
      if (first_change > out) first_change = out;
      if (out > iL && c.hp) hp_final = max(hp_final, out);
      ++out;
    };
    auto orig = [&](int k) { return WalkCell{k, 0., false, bit_of(hpw, k)}; };
    auto width = [&](WalkCell &c) {
      if (!c.has_dx) {
        c.dx = dx[off + c.d];
        c.has_dx = true;
      }
      return c.dx;
    };
    // form new cell d if it waits (its victim first, and so on down); whether
    // the marks are as assumed
    auto form = [&](int d) -> bool {
      bool as_assumed = true;
      while (d < 0 && S.nstate[noff + (-d - 1)] < 0) {
        int t = d;
        for (int v; (v = S.nvic[noff + (-t - 1)]) < 0 && S.nstate[noff + (-v - 1)] < 0;) t = v;
        const long long gid = noff + (-t - 1);
        const int c = S.ncur[gid];
        if (form_merged<Cfg, Hooks>(ph, V, S, noff, -t - 1, c, S.nvic[gid], S.nstate[gid] == kMergeLeft, par) !=
            mark_of(c))
          as_assumed = false;
        S.nstate[gid] = 0;
      }
      return as_assumed;
    };
    auto add_new = [&](const RCell<Cfg> &c) {  // a half of a split cell
      const int id = nid++;
      store_new_cell(S, noff + id, c);
      S.nstate[noff + id] = 0;
      return WalkCell{-(id + 1), c.dx, true, Hooks::regrid_marker(par, c.prim)};
    };

    int ntrack = n, iR = iR0;
    emit_orig_range(0, iL);
    WalkCell prev = orig(iL), curc = orig(iL + 1);
    int k = iL + 2;
    int i = iL + 1;
    while (i <= iR - 1) {
      // current shock index (rightmost high-pressure cell among positions iL+1..iR-1)
      int iS;
      if (hpMax >= k) {
        iS = i + 1 + (hpMax - k);
      } else {
        iS = hp_final;
        if (i - 1 > iL && prev.hp) iS = max(iS, i - 1);
        if (curc.hp) iS = max(iS, i);
        if (iS < 0) iS = iL + 1;
      }
      int action;
      bool valid = false;
      if (curc.d >= 0) {
        const int dc = i - iS, d0 = curc.d - (int)iS0;
        const bool mc = 0 < dc && dc < Hooks::REGRID_WINDOW, m0 = 0 < d0 && d0 < Hooks::REGRID_WINDOW;
        if (mc == m0) {
          valid = true;
          action = bit_of(spw, curc.d) ? SPLIT : (bit_of(mgw, curc.d) ? MERGE : SKIP);
        }
      }
      if (!valid) {
        const RCell<Cfg> c = whole_cell(V, S, noff, curc.d);  // an original, or a split's half
        double rOut;
        if (iR - 1 == i) rOut = c.x;
        else rOut = x[off + k + (iR - 1 - (i + 1))];
        action = Hooks::check_cell_for_regrid(par, c.dx, c.prim, i, iS, rOut);
      } else if (action == SKIP) {
        // skip a run of original no-op cells whose distance to the shock
        // matches the original context (no action moves anything meanwhile)
        const int kc = curc.d;
        const int delta = i - kc;
        int lim = kc + (iR - i);  // positions i .. iR-1 can be examined
        const bool aligned = (hpMax >= k) || (iS - delta == (int)iS0);
        if (!aligned) {
          // stop before either shock window
          const int w0 = (int)iS0 + 1;
          if (w0 > kc) lim = min(lim, w0);
          else if ((int)iS0 + Hooks::REGRID_WINDOW - 1 > kc) lim = kc + 1;
          const int w1 = iS - delta + 1;
          if (w1 > kc) lim = min(lim, w1);
          else if (iS - delta + Hooks::REGRID_WINDOW - 1 > kc) lim = kc + 1;
        }
        // first original > kc whose precomputed action is not a no-op
        int m = kc + 1;
        if (m < lim) m = min(next_set(spw, m, lim), next_set(mgw, m, lim));
        if (m > lim) m = lim;
        const int J = m - kc;  // examined no-op positions i .. i+J-1
        if (J >= 2) {
          emit(prev);
          emit_orig_range(kc, m - 1);
          prev = orig(m - 1);
          curc = orig(m);
          k = m + 1;
          i += J;
          continue;
        }
      }

      if (action == SPLIT && ntrack < cap - 1) {
        if (!form(prev.d)) return false;
        RCell<Cfg> A, B;
        split_cells<Cfg>(whole_cell(V, S, noff, prev.d), whole_cell(V, S, noff, curc.d), whole_cell(V, S, noff, k), A,
                         B);
        emit(prev);
        prev = add_new(A);
        curc = add_new(B);
        ++ntrack;
        ++iR;
        ++walk_splits;
        ++i;
        continue;
      }
      if (action == MERGE && ntrack > 2 * ng + 2) {
        WalkCell nxt = orig(k);
        const bool left = (width(prev) < width(nxt) && i != ng) || i == iR - 1;
        WalkCell &vic = left ? prev : nxt;
        const int id = nid++;
        const long long gid = noff + id;
        S.ncur[gid] = curc.d;
        S.nvic[gid] = vic.d;
        S.nstate[gid] = left ? kMergeLeft : kMergeRight;
        WalkCell M{-(id + 1), width(curc) + width(vic), true, curc.hp};
        if (eager || curc.hp != vic.hp) {
          if (!form(vic.d)) return false;
          M.hp = form_merged<Cfg, Hooks>(ph, V, S, noff, id, curc.d, vic.d, left, par);
          S.nstate[gid] = 0;
        }
        if (left) {
          emit(M);
          prev = nxt;
        } else {
          emit(prev);
          prev = M;
        }
        curc = orig(k + 1);
        k += 2;
        --ntrack;
        --iR;
        ++walk_merges;
        ++i;
        continue;
      }
      // no action
      emit(prev);
      prev = curc;
      curc = orig(k);
      ++k;
      ++i;
    }
    emit(prev);
    emit(curc);
    emit_orig_range(k, n);
    s_nnew = out;
    s_nseg = nseg;
    s_first = first_change;
    s_nid = nid;
    return true;
  };
  for (bool eager = false;; eager = true) {
    bool differs = threadIdx.x == 0 && !walk(eager);
    if (__syncthreads_or(differs)) continue;
    if (eager) break;
    // ---- C. the merged cells, and whether their marks are as assumed
    const int nid = s_nid;
    for (int round = 1;; ++round) {
      bool waits = false;
      for (int id = threadIdx.x; id < nid; id += BS) {
        const long long gid = noff + id;
        if (S.nstate[gid] >= 0) continue;
        const int v = S.nvic[gid];
        const int vs = v < 0 ? S.nstate[noff + (-v - 1)] : 0;
        if (vs < 0 || vs >= round) {  // its victim is formed in this round or later
          waits = true;
          continue;
        }
        const int c = S.ncur[gid];
        if (form_merged<Cfg, Hooks>(ph, V, S, noff, id, c, v, S.nstate[gid] == kMergeLeft, par) != mark_of(c))
          differs = true;
        S.nstate[gid] = round;
      }
      if (!__syncthreads_or(waits)) break;
    }
    if (!__syncthreads_or(differs)) break;
  }
  nsplit += walk_splits;
  nmerge += walk_merges;
  const int nnew = s_nnew, nseg = s_nseg, first = s_first;
  if (first >= nnew && nnew == n) return n;  // nothing moved

  // ---- D. expand the segments into the new track (positions >= first)
  const int *seg_start = S.seg_start + 4 * off;
  const int *seg_src = S.seg_src + 4 * off;
  for (int p = first + threadIdx.x; p < nnew; p += BS) {
    int lo = 0, hi = nseg - 1;  // last segment with start <= p
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (seg_start[mid] <= p) lo = mid;
      else hi = mid - 1;
    }
    const int src = seg_src[lo];
    const long long gp = off + p;
    if (src >= 0) {
      const int kk = src + (p - seg_start[lo]);
      const long long gk = off + kk;
#pragma unroll
      for (int s = 0; s < NQS; ++s) S.tprim[s * S.N + gp] = prim[s * N + gk];
      S.tx[gp] = x[gk];
      S.tdx[gp] = dx[gk];
      S.tdtl[gp] = dtl[gk];
      if (p <= nnew - 2) S.txI[gp] = xI[gk];
    } else {
      const long long gid = noff + (-src - 1);
#pragma unroll
      for (int s = 0; s < NQS; ++s) S.tprim[s * S.N + gp] = S.nprim[s * 2 * S.N + gid];
      S.tx[gp] = S.nx[gid];
      S.tdx[gp] = S.ndx[gid];
      S.tdtl[gp] = S.ndtl[gid];
      if (p <= nnew - 2) {
        const int rif = S.nrif[gid];
        S.txI[gp] = rif >= 0 ? xI[off + rif] : S.nrifx[gid];
      }
    }
  }
  __syncthreads();
  for (int p = first + threadIdx.x; p < nnew; p += BS) {
    const long long gp = off + p;
#pragma unroll
    for (int s = 0; s < NQS; ++s) prim[s * N + gp] = S.tprim[s * S.N + gp];
    x[gp] = S.tx[gp];
    dx[gp] = S.tdx[gp];
    dtl[gp] = S.tdtl[gp];
    if (p <= nnew - 2) xI[gp] = S.txI[gp];
  }
  __syncthreads();
  return nnew;
}

}  // namespace gb
