// One team advances one run (one 1D track of cells) through whole RK3 steps: one
// CTA, or a cluster of CTAs where there are fewer runs than the GPU has room for.
//
// Per step (src/simu.cpp:79-105): [regrid] -> reset shocks -> ghosts ->
// stage-1 CFL candidates -> per-run dt (team min) -> stage-1 update ->
// ghosts -> stage-2 fluxes+update+RK combine -> ghosts -> stage-3 -> inject.
// With the Euler module (Timestep/euler.cpp:12-19) the step ends after the
// stage-1 update: inject, and no RK combine.
//
// Each CTA owns a segment of consecutive cells (alone, the whole track).  Each
// stage is one left-to-right sweep over the segment in chunks of CH = BS CPT
// cells (one interface and one cell per thread at a time).  A chunk stages the
// stencil (cells a-1 .. a+CH+1) in shared memory, computes the interfaces
// a .. a+CH-1 (PLM + HLLC at the contact-speed interface), then updates cells
// a .. a+CH-1 in place.  The old state of cell a+CH-1 and the results of
// interface a+CH-1 are carried to the next chunk, so the in-place update never
// feeds a neighbour's stencil.  The last three staged cells and the gradients
// between them move to the next chunk's first slots, so that staging and
// gradients take one pass of the threads each.  In a team, a segment's first
// chunk starts at the interface on its left, which its neighbour computes too
// (the same bits); the two cells beyond either end are read before any CTA
// updates (halo), and the CTAs wait for one another twice per stage.
// Measured us of the kernel per step, one B200, the same formulas: 12 tubes of
// 1,001 to 8,191 cells 1,305 with a CTA of 128 threads each and 80 with 8 of 512,
// one tube of 500 cells 90.6 and 46, one BM1D run of 2,000 initial cells 393 and
// 103.
// (A segment per warp, whose warps wait only twice per stage, is slower: 4,096
// tubes 3.97 against 3.58 ms per step, the BM1D sweep 1.82 against 1.38 ms.  The
// warps drift apart and no longer share the instruction cache.)
// Runs are independent (own dt, own regrid), so a team takes runs from a work
// queue and can advance each by many steps without any grid-wide
// synchronisation.
#pragma once

#include "gamma_problem.h"
#include "mlp.cuh"
#include "physics.cuh"
#include "regrid.cuh"

#include <type_traits>

#ifdef GB_SWEEP_NOINLINE
#define GB_SWEEP_ATTR __noinline__
#else
#define GB_SWEEP_ATTR __forceinline__
#endif

namespace gb {

// Device view of the pooled structure-of-arrays state.  Run r owns cells
// [off[r], off[r]+cap[r]) of every per-cell array.  Primitive slot q is stored
// at row (q < 3 ? q : q-1): slot 3 is identically zero in 1D.
struct Tracks {
  double *prim;     // [NQS][N]
  double *x, *dx;   // cell centre and width at step start
  double *dtl;      // Cell::dt_loc, carried between steps
  double *xI;       // interface i sits between cells i and i+1
  double *u0;       // [NQS][N] step-start cons * dV (stage combine)
  double *xI0;      // step-start interface positions
  double *fl1;      // [NQS][N] stage-1 interface fluxes (kept from the CFL pass)
  double *v1;       // stage-1 interface velocities
  double *sd, *pspec;
  uint8_t *shocked;
  long long N;      // row stride
  const long long *off;
  const int *cap;
  RunState *run;    // per-run scalars (ntrack, t, dt, it, status)
  const double *par;  // [nruns][gamma_problem::PARAM_WORDS] problem parameters
  RegridScratch rg;
  const float *mlp;  // learned cons2prim guess parameters (kernels built with GUESS only)
};

template <class Cfg>
struct Slots {
  static constexpr int NQS = Cfg::NQ - 1;
  __device__ __forceinline__ static constexpr int q_of(int s) { return s < 3 ? s : s + 1; }
};

struct StepStats {
  unsigned long long c2p_calls;
  unsigned long long c2p_iters;
  unsigned long long c2p_fallbacks;
  unsigned long long zone_updates;
  unsigned long long splits, merges;
  int c2p_max_iters;
  int status;
  unsigned long long c2p_guesses;  // cons2prim calls started from the learned guess
  unsigned long long c2p_poor;     // cons2prim calls whose warm start was poor (c2p_warm_start_poor)
  unsigned long long learned;      // launches of the step with the learned guess that ran
};


// The CTAs that advance one run (a cluster), and this one's rank.
struct Team {
  int ncta, rank;

  // every thread of the team: what any wrote before is seen by all after
  __device__ __forceinline__ void sync() const {
    if (ncta == 1) {
      __syncthreads();
    } else {
      asm volatile("barrier.cluster.arrive.release;" ::: "memory");
      asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    }
  }
};

// BS threads of each CTA of the team; each sweep chunk holds CPT cells per
// thread (CH = BS CPT), which a thread takes in turn.  Hooks: the problem module
// (include/gamma_problem.h), whose hooks run where the reference calls its
// own: userBoundaries in ghosts, userKinematics and userSourceTerms in the
// sweep, cons2prim_user in cons2prim, checkCellForRegrid in regrid_track.
template <class Cfg, class Hooks, int BS, bool GUESS = false, int CPT = 1>
struct TrackStep {
  static constexpr int NQ = Cfg::NQ;
  static constexpr int NQS = Cfg::NQ - 1;
  static constexpr int CH = BS * CPT;  // cells and interfaces per chunk
  static constexpr int NC = CH + 3;    // staged cells per chunk: a-1 .. a+CH+1

  struct Smem {
    // by cell (rows of NC; the carry between chunks treats them as one array)
    double cp[NQS][NC];  // staged primitives
    double cx[NC], cdx[NC], cen[NC];
    double gp[NQS][NC];  // gradient between slots k and k+1 (grad())
    // by interface (rows of CH+1; slot 0 = interface a-1)
    double fl[NQS][CH + 1];  // interface fluxes
    double lL[CH + 1], lR[CH + 1], v[CH + 1];
    double xnew[CH + 1], xcmb[CH + 1];
    // the segment's surroundings as the stage finds them: cells s-2, s-1, e,
    // e+1 and the interface on its left
    double hp[NQS][4], hx[4], hdx[4], hxI;
    double edge[4];  // x, dx of the track's left and right edge cells this stage
    double red[BS / 32], cta_min;
  };

  // --- helpers ------------------------------------------------------------

  __device__ __forceinline__ static double warp_min(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
  }
  // min over the team (order-free); every thread gets it
  __device__ static double team_min(Smem &sm, const Team &tm, double v) {
    v = warp_min(v);
    if ((threadIdx.x & 31) == 0) sm.red[threadIdx.x >> 5] = v;
    __syncthreads();
    double m = sm.red[0];
#pragma unroll
    for (int k = 1; k < BS / 32; ++k) m = fmin(m, sm.red[k]);
    if (tm.ncta > 1) {
      if (threadIdx.x == 0) sm.cta_min = m;
      tm.sync();
      const unsigned mine = (unsigned)__cvta_generic_to_shared(&sm.cta_min);
      for (int c = 0; c < tm.ncta; ++c) {
        unsigned theirs;
        double x;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(theirs) : "r"(mine), "r"(c));
        asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(x) : "r"(theirs) : "memory");
        m = fmin(m, x);
      }
    } else {
      __syncthreads();
    }
    return m;
  }

  // The segment [s, e) of the team's CTA c of nc: whole chunks as far as they
  // go.  A first chunk that starts at the interface on its left holds one cell
  // less.
  __device__ __forceinline__ static void segment(int n, int nc, int c, int &s, int &e) {
    const int k = (n + nc - 1 + nc * CH - 1) / (nc * CH);  // chunks per CTA
    s = min(n, c == 0 ? 0 : CH * k + (c - 1) * (CH * k - 1));
    e = min(n, CH * k + c * (CH * k - 1));
  }

  __device__ static void load_prim(const Tracks &T, long long g, double *p) {
#pragma unroll
    for (int s = 0; s < NQS; ++s) p[Slots<Cfg>::q_of(s)] = T.prim[s * T.N + g];
    p[UU2] = 0.;
  }
  __device__ static void store_prim(const Tracks &T, long long g, const double *p) {
#pragma unroll
    for (int s = 0; s < NQS; ++s) T.prim[s * T.N + g] = p[Slots<Cfg>::q_of(s)];
  }

  // Ghost cells and ghost interfaces (Grid::updateGhosts, 1d.cpp:217-246) and
  // the problem's boundary hook.  edge: geometry of the two edge cells.
  __device__ static void ghosts(const Tracks &T, const Phys &ph, const gamma_problem::HookArgs &A, long long off,
                                int n, const double *edge) {
    const int ng = ph.ngst, iL = ng - 1, iR = n - ng;
    const int tid = threadIdx.x;
    if (tid < 2 * ng) {
      const bool left = tid < ng;
      const int e = left ? iL + 1 : iR - 1;
      const int i = left ? tid : iR + (tid - ng);
      const long long ge = off + e, gi = off + i;
      double p[NQ];
      load_prim(T, ge, p);
      // the ghost's centre as updateGhosts shifts it (1d.cpp:221, 234)
      const double gx = left ? edge[0] - (iL - i + 1) * edge[1] : edge[2] + (i - iR + 1) * edge[3];
      Hooks::user_boundaries(A, i, gx, p);  // Grid::userBoundaries (1d.cpp:244)
      store_prim(T, gi, p);
      T.dtl[gi] = T.dtl[ge];
      if (Cfg::SHOCK) {
        T.sd[gi] = T.sd[ge];
        T.pspec[gi] = T.pspec[ge];
        T.shocked[gi] = T.shocked[ge];
      }
    }
    // ghost interfaces: left 0..iL-1 from iL+1; right iR..n-2 from iR-1
    if (tid >= 32 && tid < 32 + ng) {
      const int i = tid - 32;
      if (i <= iL - 1) T.xI[off + i] = T.xI[off + iL + 1] - (iL - i + 1) * edge[1];
      const int j = iR + i;
      if (j <= n - 2) T.xI[off + j] = T.xI[off + iR - 1] + (j - iR) * edge[3];
    }
  }

  // Geometry of cell i during the current stage.  Active cells: the step-start
  // arrays (stage 1) or the span of their interfaces (stages 2, 3: set by
  // Cell::move and CellGeomFromInterfacePos; xL: the left one's position where
  // it may no longer be read).  Ghosts: shifted copies of the edge cells
  // (updateGhosts).
  __device__ __forceinline__ static void cell_geom(const Tracks &T, const double *edge, long long off, int n, int ng,
                                                   int stage, int i, const double *xLp, double *gx, double *gdx) {
    const int iL = ng - 1, iR = n - ng;
    if (i <= iL) {
      *gx = edge[0] - (iL - i + 1) * edge[1];
      *gdx = edge[1];
    } else if (i >= iR) {
      *gx = edge[2] + (i - iR + 1) * edge[3];
      *gdx = edge[3];
    } else if (stage == 1) {
      *gx = T.x[off + i];
      *gdx = T.dx[off + i];
    } else {
      const double xL = xLp ? *xLp : T.xI[off + i - 1];
      const double xR = T.xI[off + i];
      *gx = (xR + xL) / 2.;
      *gdx = (xR - xL);
    }
  }

  // The surroundings of the CTA's segment, before any CTA updates.  Ghost
  // cells and interfaces are formed here as ghosts() forms them: they are being
  // written meanwhile.
  __device__ static void load_halo(const Tracks &T, const Phys &ph, const gamma_problem::HookArgs &A, Smem &sm,
                                   long long off, int n, int stage, int s, int e) {
    const int ng = ph.ngst, iL = ng - 1, iR = n - ng;
    const int k = threadIdx.x;
    if (k < 4 && s < e) {
      const int i = k < 2 ? s - 2 + k : e + k - 2;
      if (i >= 0 && i < n) {
        double gx, gdx, p[NQ];
        cell_geom(T, sm.edge, off, n, ng, stage, i, nullptr, &gx, &gdx);
        load_prim(T, off + min(max(i, iL + 1), iR - 1), p);
        if (i <= iL || i >= iR) Hooks::user_boundaries(A, i, gx, p);
#pragma unroll
        for (int q = 0; q < NQS; ++q) sm.hp[q][k] = p[Slots<Cfg>::q_of(q)];
        sm.hx[k] = gx;
        sm.hdx[k] = gdx;
      }
    }
    if (k == 4 && s > 0 && s < e) {
      const int i = s - 1;
      sm.hxI = i >= iR ? T.xI[off + iR - 1] + (i - iR) * sm.edge[3] : T.xI[off + i];
    }
  }

  // Reconstructed left/right states at interface i from staged cells
  // (Grid::reconstructStates, 1d.cpp:370-461).  c = slot of cell i.
  template <class Ar>
  __device__ __forceinline__ static void reconstruct(Ar &ar, const Smem &sm, const Phys &ph, int i, int n, int c,
                                                     double xI, FState<Cfg> &L, FState<Cfg> &R) {
    if (i == 0 || i == n - 2) {
#pragma unroll
      for (int s = 0; s < NQS; ++s) {
        L.prim[Slots<Cfg>::q_of(s)] = sm.cp[s][c];
        R.prim[Slots<Cfg>::q_of(s)] = sm.cp[s][c + 1];
      }
    } else {
      // cells i-1 .. i+2 (i+2 <= n-1 for every interior interface)
      const double cenL = sm.cen[c], cenR = sm.cen[c + 1];
      const double dL = xI - cenL, dR = xI - cenR;
#pragma unroll
      for (int s = 0; s < NQS; ++s) {
        const double qL = sm.cp[s][c], qR = sm.cp[s][c + 1];
        // grad() of 1d.cpp:262-274, formed once per cell pair in the sweep
        const double gN = sm.gp[s][c];
        double gL = sm.gp[s][c - 1];
        double gR = sm.gp[s][c + 1];
        gL = minmod(gL, gN);
        gR = minmod(gR, gN);
        L.prim[Slots<Cfg>::q_of(s)] = qL + gL * dL;
        R.prim[Slots<Cfg>::q_of(s)] = qR + gR * dR;
      }
    }
    L.prim[UU2] = 0.;
    R.prim[UU2] = 0.;
    fill_state<Cfg>(ar, ph, L);
    fill_state<Cfg>(ar, ph, R);
  }

  // What the solution of one interface gives: fluxes in the interface's frame
  // times its area, the outer wave speeds, its velocity, and the shock
  // detector's result into the cell on its left (pspec < 0: none).
  struct IfaceSol {
    double flux[NQ], lL, lR, v, Sd, pspec;
  };

  template <class Ar>
  __device__ __forceinline__ static void solve_interface(Ar &ar, const Smem &sm, const Phys &ph,
                                                         const gamma_problem::HookArgs &A, int i, int n, int c,
                                                         double xI, IfaceSol &s) {
    FState<Cfg> L, R;
    reconstruct(ar, sm, ph, i, n, c, xI, L, R);
    const Waves w = compute_lambda<Cfg>(ar, ph, L, R);
    s.v = ph.vi * w.lS;
    Hooks::user_kinematics(A, i, &s.v);  // Grid::userKinematics (1d.cpp:749)
    s.lL = w.lL;
    s.lR = w.lR;
#pragma unroll
    for (int q = 0; q < NQ; ++q) s.flux[q] = 0.;
    hllc_flux<Cfg>(ar, L, R, w, s.v, iface_area<Cfg>(xI), s.flux);
    s.Sd = -1.;
    s.pspec = -1.;
    if (Cfg::SHOCK) {
      double ps = 0.;
      if (compute_Sd<Cfg>(ar, ph, L, R, &s.Sd, &ps)) s.pspec = ps;
    }
  }

  // The hooks' arguments of run r, as step() forms them.
  __device__ __forceinline__ static gamma_problem::HookArgs hook_args(const Tracks &T, const Phys &ph, int r, int n) {
    const RunState &R = T.run[r];
    return gamma_problem::HookArgs{T.par + (size_t)r * gamma_problem::PARAM_WORDS, ph.gamma_ad, R.t, R.it, n,
                                   ph.ngst - 1, n - ph.ngst};
  }

  // Formulas formed again with the plain operators, where an operand left the
  // range of FlatOps: rare, hence out of line.  The interface's solution goes
  // through its shared slots (written by this lane only, before the warp's next
  // synchronisation).
  __device__ __noinline__ static void solve_interface_plain(Smem &sm, const Tracks &T, const Phys &ph, int r, int n,
                                                            int i, int c, double xI) {
    PlainOps ar;
    IfaceSol s;
    solve_interface(ar, sm, ph, hook_args(T, ph, r, n), i, n, c, xI, s);
#pragma unroll
    for (int k = 0; k < NQS; ++k) sm.fl[k][c] = s.flux[Slots<Cfg>::q_of(k)];
    sm.lL[c] = s.lL;
    sm.lR[c] = s.lR;
    sm.v[c] = s.v;
    sm.xnew[c] = s.Sd;
    sm.xcmb[c] = s.pspec;
  }
  __device__ __noinline__ static void pair_gradient_plain(Smem &sm, int k) {
    const double d = sm.cen[k + 1] - sm.cen[k];
    for (int s = 0; s < NQS; ++s) sm.gp[s][k] = qdiv(sm.cp[s][k + 1] - sm.cp[s][k], d);
  }
  __device__ __noinline__ static double centroid_plain(double x, double dx) { return make_geom<Cfg>(x, dx).cen; }

  // Cell::update (cell.cpp:102-127) up to cons2prim: cons per volume after the
  // stage, the primitives before it (the warm start) and the new geometry.
  template <class Ar>
  __device__ __forceinline__ static void advance_cell(Ar &ar, const Tracks &T, const Phys &ph,
                                                      const gamma_problem::HookArgs &A, const SynchConst &sc,
                                                      const Smem &sm, long long g, int tt, int stage, double dt,
                                                      double *cons, double *prim, Geom &G1) {
    const int c = tt + 1;
#pragma unroll
    for (int s = 0; s < NQS; ++s) prim[Slots<Cfg>::q_of(s)] = sm.cp[s][c];
    prim[UU2] = 0.;
    const Geom G0 = make_geom<Cfg>(ar, sm.cx[c], sm.cdx[c]);
    prim2cons<Cfg>(ar, ph, prim, cons);
#pragma unroll
    for (int q = 0; q < NQ; ++q) cons[q] *= G0.dV;
    if (stage == 1) {
#pragma unroll
      for (int s = 0; s < NQS; ++s) T.u0[s * T.N + g] = cons[Slots<Cfg>::q_of(s)];
    }
#pragma unroll
    for (int s = 0; s < NQS; ++s) {
      const int q = Slots<Cfg>::q_of(s);
      cons[q] += (sm.fl[s][tt] - sm.fl[s][tt + 1]) * dt;
    }
    if (Cfg::SPH) {  // Cell::sourceTerms, 1D (rel_sph.cpp:452-466)
      double p = prim[PPP];
      double r = G0.x, dr = G0.dx, dV = G0.dV;
      double r1 = r - dr / 2., r2 = r + dr / 2.;
      double rsq = ar.quo(r2 * r2 + r1 * r1 + r2 * r1, ar.by(3.));
      cons[SS1] += (2. * p) * ar.quo(r, ar.by(rsq)) * dV * dt;
    }
    if (Cfg::CYL) {  // Cell::sourceTerms of rel_cyl.cpp:358-364, r = G.x[r_]
      cons[SS1] += ar.quo(prim[PPP], ar.by(G0.x)) * G0.dV * dt;
    }
    Hooks::user_source_terms(A, G0.x, G0.dx, G0.dV, prim, cons, dt);  // Cell::userSourceTerms
    if (Cfg::SYNCH) {
      const double dg = radiative_source<Cfg>(ar, ph, sc, prim, G0.dV, dt);
      cons[GMX] += dg;
      cons[GMN] += dg;
    }
    G1 = geom_between<Cfg>(ar, sm.xnew[tt], sm.xnew[tt + 1]);
    per_volume(ar, cons, G1.dV);
  }

  // cons / dV
  template <class Ar>
  __device__ __forceinline__ static void per_volume(Ar &ar, double *cons, double dV) {
    if (Cfg::FAST) {
      const double rdV = ar.inv(dV);
#pragma unroll
      for (int q = 0; q < NQ; ++q) cons[q] *= rdV;
    } else {
      const auto by = ar.by(dV);
#pragma unroll
      for (int q = 0; q < NQ; ++q) cons[q] = q <= TAU ? ar.quo(cons[q], by) : ar.quo0(cons[q], by);
    }
  }

  // RK3 combine (rk3.cpp:27-55, 63-92)
  template <class Ar>
  __device__ __forceinline__ static void combine_cell(Ar &ar, const Tracks &T, const Smem &sm, long long g, int tt,
                                                      int stage, double dV1, double *cons) {
    const double w0 = stage == 2 ? 3. / 4. : 1. / 3.;
    const double w1 = stage == 2 ? 1. / 4. : 2. / 3.;
#pragma unroll
    for (int s = 0; s < NQS; ++s) {
      const int q = Slots<Cfg>::q_of(s);
      cons[q] = w0 * T.u0[s * T.N + g] + w1 * cons[q] * dV1;
    }
    per_volume(ar, cons, geom_between<Cfg>(ar, sm.xcmb[tt], sm.xcmb[tt + 1]).dV);
  }

  // The whole update of one cell, with the reference's warm starts; its
  // cons2prim statistics.
  template <class Ar>
  __device__ __forceinline__ static void update_cell(Ar &ar, const Tracks &T, const Phys &ph,
                                                     const gamma_problem::HookArgs &A, const SynchConst &sc,
                                                     const Smem &sm, long long g, int tt, int stage, double dt,
                                                     double *prim, C2PStats &c1, C2PStats &c2) {
    double cons[NQ];
    Geom G1;
    advance_cell(ar, T, ph, A, sc, sm, g, tt, stage, dt, cons, prim, G1);
    cons2prim<Cfg, Hooks>(ar, ph, cons, prim, &c1, A.par);
    if (stage > 1) {
      combine_cell(ar, T, sm, g, tt, stage, G1.dV, cons);
      cons2prim<Cfg, Hooks>(ar, ph, cons, prim, &c2, A.par);
    }
  }
  struct CellResult {
    double prim[NQS];
    C2PStats c1, c2;
  };
  __device__ __noinline__ static CellResult update_cell_plain(const Smem &sm, const Tracks &T, const Phys &ph, int r,
                                                              int n, long long g, int tt, int stage, double dt) {
    PlainOps ar;
    const gamma_problem::HookArgs A = hook_args(T, ph, r, n);
    SynchConst sc;
    Hooks::synchrotron_norm(A.par, &sc.Nalpha, &sc.Nmp, &sc.Nme);
    double prim[NQ];
    CellResult R{};
    update_cell(ar, T, ph, A, sc, sm, g, tt, stage, dt, prim, R.c1, R.c2);
#pragma unroll
    for (int s = 0; s < NQS; ++s) R.prim[s] = prim[Slots<Cfg>::q_of(s)];
    return R;
  }

  // Cell::update_dt, moving direction (cell.cpp:47-74).  Returns false on a
  // negative candidate (the reference's exit(30)).
  __device__ __forceinline__ static bool dt_candidate(double a, double lR_left, double v_right, double lL_right,
                                                      double v_left, double *cand) {
    const bool onL = lR_left > v_right, onR = lL_right < v_left;
    FlatOps ar;
    double dL = ar.quo(a, ar.by(onL ? lR_left - v_right : 1.));
    double dR = ar.quo(a, ar.by(onR ? v_left - lL_right : 1.));
    if (ar.bad()) {
      dL = a / (lR_left - v_right);
      dR = a / (v_left - lL_right);
    }
    *cand = fmin(onL ? dL : DT_INF, onR ? dR : DT_INF);
    return !(*cand < 0);
  }

  __device__ static void count_c2p(StepStats &st, const C2PStats &cs, int poor) {
    st.c2p_calls++;
    st.c2p_poor += poor;
    st.c2p_iters += cs.iters;
    st.c2p_fallbacks += cs.fallback;
    st.c2p_max_iters = max(st.c2p_max_iters, cs.iters);
  }

  // cons2prim of one cell, with the learned guess (GUESS): the search stops at
  // a poor warm start (C2PStats::deferred) and those cells search again from
  // the network's pressure (a non-finite or non-positive guess keeps the warm
  // one).  Every lane of the warp calls (upd = false: no cell); the network
  // runs only when a lane of the warp needs it, and the second search is the
  // out-of-line copy, so that the step's own loop stays as without the guess.
  __device__ static void cell_cons2prim(const mlp::InferSmem *inf, const Phys &ph, double *cons, double *prim,
                                        bool upd, StepStats &st, const double *par) {
    C2PStats cs;
    if (upd) cons2prim<Cfg, Hooks>(ph, cons, prim, &cs, par, GUESS);
    const int poor = upd ? cs.poor : 0;
    if (GUESS) {
      const bool need = upd && cs.deferred;
      if (__any_sync(0xffffffffu, need)) {
        const double pg = mlp::warp_guess_pressure(*inf, cons[DEN], cons[TAU], cons[SS1], need);
        if (need) {
          if (isfinite(pg) && pg > 0.) prim[PPP] = pg;
          cons2prim<Cfg, Hooks, true>(ph, cons, prim, &cs, par);
          st.c2p_guesses++;
        }
      }
    }
    if (upd) count_c2p(st, cs, poor);
  }

  // --- one stage sweep of the CTA's segment [s, e) ----------------------------
  // mode 0: stage-1 CFL candidates only (returns the thread's min dt_loc and
  //         resets dt_loc); mode 1: fluxes + update (+ RK combine for stage>1).
  __device__ GB_SWEEP_ATTR static double sweep(const Tracks &T, const Phys &ph, const gamma_problem::HookArgs &A,
                                               const SynchConst &sc, Smem &sm, int r, long long off, int n, int s,
                                               int e, int stage, int mode, double dt, StepStats &st,
                                               const mlp::InferSmem *inf) {
    const int tid = threadIdx.x;
    const int ng = ph.ngst, iL = ng - 1, iR = n - ng;
    // RK3 weights of the interface positions
    const double w0 = stage == 2 ? 3. / 4. : 1. / 3.;
    const double w1 = stage == 2 ? 1. / 4. : 2. / 3.;
    double run_min = DT_INF;
    // the step with the learned guess keeps the plain operators
    using Ops = typename std::conditional<GUESS, PlainOps, FlatOps>::type;
    const int a0 = s > 0 ? s - 1 : 0;
    const int last = min(n - 1, e + 1);  // last staged cell
    if (s >= e) return run_min;  // a short track leaves the last CTAs without cells

    for (int a = a0; a < e; a += CH) {
      // ---- stage cells a-1 .. a+CH+1 (slot k <-> cell a-1+k); slots 0..2 are
      // carried from the previous chunk
      for (int k = tid + (a > a0 ? 3 : 0); k < NC; k += BS) {
        const int i = a - 1 + k;
        if (i >= 0 && i <= last) {
          double gx, gdx;
          if (i < s || i >= e) {
            const int h = i < s ? i - s + 2 : i - e + 2;
#pragma unroll
            for (int q = 0; q < NQS; ++q) sm.cp[q][k] = sm.hp[q][h];
            gx = sm.hx[h];
            gdx = sm.hdx[h];
          } else {
            const long long g = off + i;
#pragma unroll
            for (int q = 0; q < NQS; ++q) sm.cp[q][k] = T.prim[q * T.N + g];
            // (the left interface of the segment's first cell is another CTA's)
            cell_geom(T, sm.edge, off, n, ng, stage, i, i == s && s > 0 ? &sm.hxI : nullptr, &gx, &gdx);
          }
          sm.cx[k] = gx;
          sm.cdx[k] = gdx;
          Ops ar;
          double cen = make_geom<Cfg>(ar, gx, gdx).cen;
          if (ar.bad()) cen = centroid_plain(gx, gdx);
          sm.cen[k] = cen;
        }
      }
      __syncthreads();
      if (!(mode == 1 && stage == 1)) {
        // grad() between staged cells k and k+1: (q[k+1] - q[k]) / (cen[k+1] - cen[k]),
        // each used by the three interfaces around it
        for (int k = tid + (a > a0 ? 2 : 0); k < NC - 1; k += BS) {
          if (a - 1 + k >= 0 && a + k <= last) {  // slots k and k+1 both hold cells
            const double d = sm.cen[k + 1] - sm.cen[k];
            // in the reference's order unless every formula may move (FAST_RIEMANN):
            // minmod of two equal slopes is 0 (1d.cpp:250-260), and a split's two
            // halves make such ties on purpose (their pair gradient is the split's)
            if (Cfg::FAST_RIEMANN) {
              const double rd = 1. / d;
#pragma unroll
              for (int q = 0; q < NQS; ++q) sm.gp[q][k] = (sm.cp[q][k + 1] - sm.cp[q][k]) * rd;
            } else {
              Ops ar;
              const auto by = ar.by(d);
#pragma unroll
              for (int q = 0; q < NQS; ++q) sm.gp[q][k] = ar.quo0(sm.cp[q][k + 1] - sm.cp[q][k], by);
              if (ar.bad()) pair_gradient_plain(sm, k);
            }
          }
        }
        __syncthreads();
      }

      // ---- interfaces i = a + tid + u BS
#pragma unroll 1
      for (int u = 0; u < CPT; ++u) {
      const int tt = tid + u * BS;
      const int i = a + tt;
      const bool has_if = i <= n - 2 && i < e;
      const bool own = i >= s;  // else the left neighbour keeps its results
      const int c = tt + 1;  // slot of cell i
      double myflux[NQ];
#pragma unroll
      for (int q = 0; q < NQ; ++q) myflux[q] = 0.;
      double my_lL = 0, my_lR = 0, my_v = 0, my_xnew = 0, my_xcmb = 0;
      if (has_if) {
        const long long gi = off + i;
        const double xI = own ? T.xI[gi] : sm.hxI;
        if (mode == 1 && stage == 1) {
          // stage-1 fluxes and velocities were solved by the CFL pass
          my_v = T.v1[gi];
#pragma unroll
          for (int s = 0; s < NQS; ++s) myflux[Slots<Cfg>::q_of(s)] = T.fl1[s * T.N + gi];
        } else {
          Ops ar;
          IfaceSol sol;
          solve_interface(ar, sm, ph, A, i, n, c, xI, sol);
          if (ar.bad()) {
            solve_interface_plain(sm, T, ph, r, n, i, c, xI);
#pragma unroll
            for (int k = 0; k < NQS; ++k) sol.flux[Slots<Cfg>::q_of(k)] = sm.fl[k][c];
            sol.lL = sm.lL[c];
            sol.lR = sm.lR[c];
            sol.v = sm.v[c];
            sol.Sd = sm.xnew[c];
            sol.pspec = sm.xcmb[c];
          }
          my_lL = sol.lL;
          my_lR = sol.lR;
          my_v = sol.v;
#pragma unroll
          for (int q = 0; q < NQ; ++q) myflux[q] = sol.flux[q];
          if (Cfg::SHOCK && own) {  // measureShock into cell i (radiation_sph.cpp:160-175)
            const double sd0 = fmax(T.sd[gi], sol.Sd);
            T.sd[gi] = sd0;
            if (sol.pspec > T.pspec[gi]) T.pspec[gi] = sol.pspec;
            if (stage == 1) T.shocked[gi] = sd0 > DETECT_SHOCK_THRESHOLD ? 1 : 0;  // detectShock
          }
          if (mode == 0 && own) {  // keep the stage-1 solution for the update pass
            T.v1[gi] = my_v;
#pragma unroll
            for (int s = 0; s < NQS; ++s) T.fl1[s * T.N + gi] = myflux[Slots<Cfg>::q_of(s)];
          }
        }
        if (mode == 1) {
          // Interface::move, then the RK combine of interface positions
          my_xnew = xI + dt * my_v;
          if (stage == 1) {
            if (own) T.xI0[gi] = xI;
            my_xcmb = my_xnew;
          } else if (i >= iL && i <= iR - 1) {
            my_xcmb = w0 * T.xI0[gi] + w1 * my_xnew;
          } else {
            my_xcmb = my_xnew;
          }
          if (own) T.xI[gi] = my_xcmb;
        }
      }
      // cell n-1 has no interface of its own; as for every cell, the shock
      // detector result of the last real interface is already in place.
      sm.lL[tt + 1] = my_lL;
      sm.lR[tt + 1] = my_lR;
      sm.v[tt + 1] = my_v;
      if (mode == 1) {
        sm.xnew[tt + 1] = my_xnew;
        sm.xcmb[tt + 1] = my_xcmb;
#pragma unroll
        for (int s = 0; s < NQS; ++s) sm.fl[s][tt + 1] = myflux[Slots<Cfg>::q_of(s)];
      }
      }
      __syncthreads();

      // ---- cells i = a + tid + u BS
#pragma unroll 1
      for (int u = 0; u < CPT; ++u) {
      const int tt = tid + u * BS;
      const int i = a + tt;
      const int c = tt + 1;
      const bool mine = i >= s && i < e;
      if (mine) {
        const long long g = off + i;
        if (i >= 1 && i <= n - 2 && (mode == 0 || stage > 1)) {
          double cand;
          if (!dt_candidate(sm.cdx[c], sm.lR[tt], sm.v[tt + 1], sm.lL[tt + 1], sm.v[tt], &cand)) {
            st.status = 30;
            cand = DT_INF;
          }
          const double d = fmin(T.dtl[g], cand);
          if (mode == 0) {
            run_min = fmin(run_min, d);
            T.dtl[g] = DT_INF;  // collect_dt resets (1d.cpp:785)
          } else {
            T.dtl[g] = d;
          }
        } else if (mode == 0) {
          run_min = fmin(run_min, T.dtl[g]);
          T.dtl[g] = DT_INF;
        }
      }

      if (mode == 1) {
        const bool upd = mine && i >= iL + 1 && i <= iR - 1;
        const long long g = off + i;
        double prim[NQ];
        if (GUESS) {
          // blocks under `upd`, so that the whole warp meets at each inference
          double cons[NQ];
          Geom G1;
          PlainOps ar;
          if (upd) advance_cell(ar, T, ph, A, sc, sm, g, tt, stage, dt, cons, prim, G1);
          cell_cons2prim(inf, ph, cons, prim, upd, st, A.par);
          if (stage > 1) {
            if (upd) combine_cell(ar, T, sm, g, tt, stage, G1.dV, cons);
            cell_cons2prim(inf, ph, cons, prim, upd, st, A.par);
          }
        } else if (upd) {
          Ops ar;
          C2PStats c1, c2;
          update_cell(ar, T, ph, A, sc, sm, g, tt, stage, dt, prim, c1, c2);
          if (ar.bad()) {
            const CellResult R = update_cell_plain(sm, T, ph, r, n, g, tt, stage, dt);
#pragma unroll
            for (int s = 0; s < NQS; ++s) prim[Slots<Cfg>::q_of(s)] = R.prim[s];
            c1 = R.c1;
            c2 = R.c2;
          }
          count_c2p(st, c1, c1.poor);
          if (stage > 1) count_c2p(st, c2, c2.poor);
        }
        if (upd) {
          if (Cfg::SYNCH && stage == (ph.euler ? 1 : 3)) {  // radiation_injectParticles, active cells
            inject_particles<Cfg>(ph, sc, prim, T.shocked[g] != 0, T.pspec[g]);
          }
          store_prim(T, g, prim);
        }
      }
      }
      __syncthreads();
      // ---- cells a+CH-1 .. a+CH+1, their gradients and interface a+CH-1 to
      // the next chunk's first slots
      if (a + CH < e) {
        constexpr int CELLS = 3 * (2 * NQS + 3), IFACES = NQS + 5;
        double *cell = &sm.cp[0][0], *iface = &sm.fl[0][0];
#pragma unroll
        for (int k = tid; k < CELLS + IFACES; k += BS) {
          if (k < CELLS) {
            double *row = cell + (k / 3) * NC + k % 3;
            row[0] = row[CH];
          } else {
            double *row = iface + (k - CELLS) * (CH + 1);
            row[0] = row[CH];
          }
        }
      }
      __syncthreads();
    }
    return run_min;
  }

  // Edge-cell geometry for the current stage
  __device__ static void edge_geom(const Tracks &T, Smem &sm, long long off, int n, int ng, int stage) {
    if (threadIdx.x < 2) {
      const long long g = off + (threadIdx.x == 0 ? ng : n - ng - 1);
      double gx, gdx;
      if (stage == 1) {
        gx = T.x[g];
        gdx = T.dx[g];
      } else {
        const double xL = T.xI[g - 1], xR = T.xI[g];
        gx = (xR + xL) / 2.;
        gdx = (xR - xL);
      }
      sm.edge[2 * threadIdx.x] = gx;
      sm.edge[2 * threadIdx.x + 1] = gdx;
    }
    __syncthreads();
  }

  // --- one full step of run r ---------------------------------------------
  // Starts and ends with the team in step (what one wrote, all see).
  __device__ static void step(const Tracks &T, const Phys &ph, Smem &sm, const Team &tm, uint32_t *words, int r,
                              StepStats &st, bool regrid_only, const mlp::InferSmem *inf) {
    const long long off = T.off[r];
    const double *par = T.par + (size_t)r * gamma_problem::PARAM_WORDS;
    SynchConst sc;
    Hooks::synchrotron_norm(par, &sc.Nalpha, &sc.Nmp, &sc.Nme);
    RunState &R = T.run[r];
    int n = R.ntrack;
    const int ng = ph.ngst;
    const int tid = tm.rank * BS + threadIdx.x, nth = tm.ncta * BS;  // place in the team
    const bool first = tm.rank == 0 && threadIdx.x == 0;

    if (Hooks::REGRID) {  // one CTA's work; its result reaches the others through R
      if (tm.rank == 0)
        n = regrid_track<Cfg, Hooks, BS>(T.prim, T.N, T.x, T.dx, T.dtl, T.xI, off, n, T.cap[r], ph, par, T.rg,
                                         words, st.splits, st.merges);
      if (tm.ncta > 1) {
        tm.sync();  // every CTA has read the old count
        if (first) R.ntrack = n;
        tm.sync();
        n = R.ntrack;
      } else {
        __syncthreads();
      }
    }
    const gamma_problem::HookArgs A{par, ph.gamma_ad, R.t, R.it, n, ng - 1, n - ng};
    if (regrid_only) {
      if (first) R.ntrack = n;
      tm.sync();
      return;
    }
    if (Cfg::SHOCK) {  // Cell::resetShock
      for (int i = tid; i < n; i += nth) {
        T.sd[off + i] = -1.;
        T.pspec[off + i] = 0.;
        T.shocked[off + i] = 0;
      }
      tm.sync();
    }

    // The sweeps of the step: the stage-1 CFL pass, which gives dt, the stage-1
    // update (the whole Grid::evolve of Timestep/euler.cpp), stage 2, stage 3.
    // One loop, so that the kernel holds one copy of the sweep's code: four
    // inlined copies overflow the instruction cache.  Before a stage's first
    // sweep every CTA reads its surroundings and one of them writes the ghosts;
    // nobody updates until all have.
    int s, e;
    segment(n, tm.ncta, tm.rank, s, e);
    double dt = 0.;
    const int npass = ph.euler ? 2 : 4;
#pragma unroll 1
    for (int pass = 0; pass < npass; ++pass) {
      const int stage = pass < 2 ? 1 : pass;
      if (pass != 1) {
        edge_geom(T, sm, off, n, ng, stage);
        if (tm.rank == 0) ghosts(T, ph, A, off, n, sm.edge);
        if (tm.ncta > 1) load_halo(T, ph, A, sm, off, n, stage, s, e);
        tm.sync();
      }
      const double m = sweep(T, ph, A, sc, sm, r, off, n, s, e, stage, pass > 0 ? 1 : 0, dt, st, inf);
      if (pass == 0) dt = ph.cfl * team_min(sm, tm, m);
      else tm.sync();
    }

    // step-end cell geometry.  RK3: ghosts 0 and n-1 keep the stage-3 ghost
    // copies, cells 1..n-2 span their interfaces (CellGeomFromInterfacePos).
    // Euler: only Cell::update moves cells (iL+1..iR-1); every ghost keeps
    // its stage-1 copy.
    const int iL = ng - 1, iR = n - ng;
    for (int i = tid; i < n; i += nth) {
      double gx, gdx;
      if (ph.euler ? (i <= iL || i >= iR) : (i == 0 || i == n - 1)) {
        if (i <= iL) {
          gx = sm.edge[0] - (iL - i + 1) * sm.edge[1];
          gdx = sm.edge[1];
        } else {
          gx = sm.edge[2] + (i - iR + 1) * sm.edge[3];
          gdx = sm.edge[3];
        }
      } else {
        const double xL = T.xI[off + i - 1], xR = T.xI[off + i];
        gx = (xR + xL) / 2.;
        gdx = (xR - xL);
      }
      T.x[off + i] = gx;
      T.dx[off + i] = gdx;
      // radiation_injectParticles on ghost cells (active cells did it in the sweep)
      if (Cfg::SYNCH && (i <= iL || i >= iR)) {
        double prim[NQ];
        load_prim(T, off + i, prim);
        inject_particles<Cfg>(ph, sc, prim, T.shocked[off + i] != 0, T.pspec[off + i]);
        store_prim(T, off + i, prim);
      }
    }
    if (st.status) R.status = st.status;  // any thread; every writer stores the same code
    if (first) {
      R.ntrack = n;
      R.dt = dt;
      R.t = R.t + dt;
      R.it = R.it + 1;
    }
    if (tm.rank == 0) st.zone_updates += (unsigned long long)(n - 2 * ng);
    tm.sync();
  }
};

// Dynamic shared memory: TrackStep::Smem, the regrid bit words (words_bytes),
// then, with GUESS, the tensor-core weights of the learned guess.
// gate (or nullptr): the launch returns at once unless *gate (k_guess_policy)
// chose this kernel, the one with (nonzero) or without (0) the learned guess.
template <class Cfg, class Hooks, int BS, bool GUESS = false, int CPT = 1, int MINB = Cfg::MIN_BLOCKS>
__global__ void __launch_bounds__(BS, MINB)
    track_step_kernel(const __grid_constant__ Tracks T, const __grid_constant__ Phys ph, int nsteps, const int *order,
                      int nruns, int *queue, StepStats *stats, int regrid_only, unsigned words_bytes, const int *gate) {
  if (gate && ((*gate != 0) != GUESS)) return;
  using TS = TrackStep<Cfg, Hooks, BS, GUESS, CPT>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  typename TS::Smem &sm = *reinterpret_cast<typename TS::Smem *>(smem_raw);
  uint32_t *words = reinterpret_cast<uint32_t *>(smem_raw + sizeof(typename TS::Smem));
  mlp::InferSmem *inf = nullptr;
  if (GUESS) {
    inf = reinterpret_cast<mlp::InferSmem *>(smem_raw + ((sizeof(typename TS::Smem) + words_bytes + 15u) & ~size_t(15)));
    mlp::load_infer_weights(T.mlp, *inf);
    __syncthreads();
  }
  StepStats st{};
  Team tm;
  asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(tm.ncta));
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(tm.rank));
  __shared__ int s_item;
  // one CTA per run: a queue; a cluster per run: every nteams-th run
  const int nteams = gridDim.x / tm.ncta;
  for (int item = blockIdx.x / tm.ncta;; item += nteams) {
    if (tm.ncta == 1) {
      if (threadIdx.x == 0) s_item = atomicAdd(queue, 1);
      __syncthreads();
      item = s_item;
      __syncthreads();
    }
    if (item >= nruns) break;
    const int r = order[item];
    for (int k = 0; k < nsteps; ++k) {
      // a run whose step failed stops (its status is the same to all: the step
      // before ended with the team in step)
      if (T.run[r].status != 0) break;
      TS::step(T, ph, sm, tm, words, r, st, regrid_only != 0, inf);
    }
    if (st.status) {  // this run's; the next one starts without it
      atomicMax(&stats->status, st.status);
      st.status = 0;
    }
  }
  // fold the per-thread statistics into the launch totals
  __syncthreads();
  if (st.c2p_guesses) atomicAdd(&stats->c2p_guesses, st.c2p_guesses);
  if (st.c2p_poor) atomicAdd(&stats->c2p_poor, st.c2p_poor);
  if (GUESS && blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(&stats->learned, 1ull);
  if (st.c2p_calls) {
    atomicAdd(&stats->c2p_calls, st.c2p_calls);
    atomicAdd(&stats->c2p_iters, st.c2p_iters);
    atomicAdd(&stats->c2p_fallbacks, st.c2p_fallbacks);
    atomicMax(&stats->c2p_max_iters, st.c2p_max_iters);
  }
  if (threadIdx.x == 0) {
    atomicAdd(&stats->zone_updates, st.zone_updates);
    if (st.splits) atomicAdd(&stats->splits, st.splits);
    if (st.merges) atomicAdd(&stats->merges, st.merges);
  }
}

}  // namespace gb
