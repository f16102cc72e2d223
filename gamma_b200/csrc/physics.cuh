// Device physics of the 1D moving-mesh relativistic hydro step (FP64).
//
// Each function restates one member of the GAMMA reference and keeps its
// floating-point operation order, so that with -fmad=false the only
// differences to the CPU reference come from libm (tanh, and pow other than
// the correctly rounded x^(3/4) of the shock detector) and from the pressure
// root finder (Newton-Raphson here, GSL Brent there).
//
// Variable slots follow src/environment.h:33-82.  Slot 3 (the theta momentum /
// 4-velocity) is identically zero in 1D: it is only ever multiplied by r
// (rel_sph.cpp:78,108,441) starting from zero, so it is neither stored nor
// computed here.
#pragma once

#include <cstdint>
#include <math.h>

#include "gamma_problem.h"

#ifndef GB_HD
#define GB_HD __device__ __forceinline__
#endif
// one out-of-line copy per kernel (see c2p_pressure)
#ifndef GB_HD_OUTLINE
#define GB_HD_OUTLINE __device__ __noinline__
#endif

#include "flat_ops.cuh"

namespace gb {

enum { RHO = 0, PPP = 1, UU1 = 2, UU2 = 3 };
enum { DEN = 0, TAU = 1, SS1 = 2, SS2 = 3 };
enum { TR1 = 4, GMN = 6, GMX = 7, GMD = 8, PSN = 9 };
enum { SKIP = 0, MERGE = 1, SPLIT = 2 };

// src/constants.h:6-28
constexpr double P_FLOOR = 1.e-10;
constexpr double PI_ = 3.14159265358979323846;
constexpr double MP = 1.6726219e-24;
constexpr double ME = 9.1093835e-28;
constexpr double C_LIGHT = 2.99792458e10;
constexpr double ALPHA_SYN = 1.29251816e-09;
constexpr double P_SPEC = 2.22;
constexpr double EPS_E = 0.1;
constexpr double EPS_B = 0.01;
constexpr double ZETA = 1.;
constexpr double GAMMA_MAX_INIT = 1.e8;
constexpr double DETECT_SHOCK_THRESHOLD = 0.01;
constexpr double DT_INF = 1.e15;

// ---------------------------------------------------------------------------
// Module selections (the reference's Makefile GEOMETRY/HYDRO/RADIATION slots and
// environment.h switches) as compile-time policies.

// Arithmetic form of the 1D step.
//   0: every formula in the reference's operation order, so a state, flux or
//      wave speed computed from the same inputs is bit for bit the reference's.
//   1: divisions by a shared denominator become one reciprocal and
//      multiplications (about half the FP64 instructions of the step); results
//      move at the ulp level, which the reference's own cold-gas conditioning
//      amplifies beyond the parity bars (lambda* from a near-cancelling
//      quadratic; f(p) of cons2prim cancelling to eps*E).
//   2 (default): the shared reciprocals of 1 everywhere except where the
//      reference's results hinge on exact values, which keep its order: the
//      wave speeds and the contact speed lambda*, the PLM pair gradients whose
//      minmod returns 0 on a tie (FAST_RIEMANN), and f(p) of the cons2prim
//      root search with the primitive recovery after it (FAST_ROOT).  It meets
//      every parity bar that 0 meets, with the same cell counts and regrid
//      decisions, and runs the tube step ~20% faster.
#ifndef GB_FAST_ARITH
#define GB_FAST_ARITH 2
#endif

// cartesian + rel_cart, ideal gas, no shock detection / synchrotron: NUM_Q = 6.
#ifndef GB_CART_MIN_BLOCKS
#define GB_CART_MIN_BLOCKS 6
#endif
struct CfgCart {
  static constexpr bool FAST = GB_FAST_ARITH != 0;
  static constexpr bool FAST_RIEMANN = GB_FAST_ARITH == 1;
  static constexpr bool FAST_ROOT = GB_FAST_ARITH == 1;
  static constexpr int MIN_BLOCKS = GB_CART_MIN_BLOCKS;  // 128-thread CTAs per SM (6: 80 registers)
  static constexpr int NQ = 6;
  static constexpr bool SPH = false;    // rel_sph hydro and spherical1D geometry
  static constexpr bool SHOCK = false;  // SHOCK_DETECTION_
  static constexpr bool SYNCH = false;  // LOCAL_SYNCHROTRON_
  static constexpr bool CYL = false;    // rel_cyl hydro (Hydro/rel_cyl.cpp)
};

// cartesian + rel_cyl (Hydro/rel_cyl.cpp, the HYDRO module whose GEOMETRY
// partner, Geometry/cylindrical.cpp, does not compile): rel_cart with the
// cylindrical source p/r on S_r, a root search only where |f| at the previous
// pressure exceeds 1e-13, and a zero velocity below |S| = 1e-14 (NUM_Q = 6).
struct CfgCyl : CfgCart {
  static constexpr bool CYL = true;
};

// spherical1D + rel_sph + radiation_sph: NUM_Q = 10.
#ifndef GB_SPH_MIN_BLOCKS
#define GB_SPH_MIN_BLOCKS 3
#endif
struct CfgSph {
  static constexpr bool FAST = GB_FAST_ARITH != 0;
  static constexpr bool FAST_RIEMANN = GB_FAST_ARITH == 1;
  static constexpr bool FAST_ROOT = GB_FAST_ARITH == 1;
  static constexpr int MIN_BLOCKS = GB_SPH_MIN_BLOCKS;
  static constexpr int NQ = 10;
  static constexpr bool SPH = true;
  static constexpr bool SHOCK = true;
  static constexpr bool SYNCH = true;
  static constexpr bool CYL = false;
};

// A module set with every formula in the reference's operation order, whatever
// GB_FAST_ARITH says: for results that must equal the reference's bit for bit
// (the text dump's conserved columns).
template <class Cfg>
struct RefOrder : Cfg {
  static constexpr bool FAST = false;
  static constexpr bool FAST_RIEMANN = false;
  static constexpr bool FAST_ROOT = false;
};

// Run-time constants shared by every run of a context.
struct Phys {
  double gamma_ad;  // GAMMA_
  double kgam;      // GAMMA_ / (GAMMA_ - 1), the enthalpy factor of the ideal EOS
  double rgm1;      // 1 / (GAMMA_ - 1)
  double cfl;       // CFL_
  double vi;        // VI
  int eos;          // 0 ideal, 1 Synge / Taub-Mathews (rel_sph.cpp:37-52)
  int ngst;
  int eos_ws;       // 1: each state's Gamma_eff in the wave speeds and the shock
                    // detector too (the reference uses GAMMA_ there)
  int euler;        // 1: Grid::evolve of Timestep/euler.cpp (one Grid::update),
                    // 0: the three SSP-RK3 stages of Timestep/rk3.cpp
};

template <class Cfg>
struct Prim {
  double v[Cfg::NQ];
};

// FluidState: primitive, conserved and physical flux of one state, with its
// Lorentz factor and 3-velocity cached (FluidState::lfac is called many times
// per interface in the reference).
template <class Cfg>
struct FState {
  double prim[Cfg::NQ];
  double cons[Cfg::NQ];
  double flux[Cfg::NQ];
  double lfac, v;
};

template <class Ar>
GB_HD double lfac_of(Ar &ar, double uu) {
  // fluid.cpp:10-22 takes u = sqrt(uu^2) and then sqrt(1 + u^2): the root of a
  // rounded square is the number itself, and where the square underflows
  // 1 + u^2 is 1
  return ar.root(1 + uu * uu);
}
GB_HD double lfac_of(double uu) {
  PlainOps ar;
  return lfac_of(ar, uu);
}

// The formulas below take their quotients and roots from an operator set Ar
// (flat_ops.cuh): PlainOps, the operators themselves, or FlatOps, the same
// results without branches.  The forms without `ar` use PlainOps.

// GAMMA_ - 1 as a divisor (its reciprocal comes from the host)
template <class Ar>
GB_HD typename Ar::By by_gm1(Ar &ar, const Phys &ph) {
  return ar.by_known(ph.gamma_ad - 1., ph.rgm1);
}

// FluidState::gamma (rel_sph.cpp:37-52)
template <class Ar>
GB_HD double eos_gamma(Ar &ar, const Phys &ph, double rho, double p) {
  const double G = ph.gamma_ad;
  if (ph.eos == 0) return G;
  double a = ar.quo(ar.quo(p, ar.by(rho)), by_gm1(ar, ph));
  double e_ratio = a + ar.root(a * a + 1.);
  return G - (G - 1.) / 2. * (1. - ar.inv(e_ratio * e_ratio));
}
GB_HD double eos_gamma(const Phys &ph, double rho, double p) {
  PlainOps ar;
  return eos_gamma(ar, ph, rho, p);
}

// 1/x to about 2^-22, for correction terms only
GB_HD double recip_approx(double x) {
#ifdef __CUDA_ARCH__
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  return r;
#else
  return 1. / x;
#endif
}

// x^(3/4) rounded to nearest: the isentrope rho1 (p/p1)^(1/GAMMA_) of the shock
// detector when 1/GAMMA_ is exactly 3/4 (GAMMA_ = 4/3), as the C library's pow
// returns it.  sqrt(x) and then x^(1/4) are carried as double-double pairs:
// the remainder of a correctly rounded square root, x - s^2, is exact as one
// FMA (Markstein 1990; Boldo & Daumas 2003), so sqrt(x) = s + (x - s^2)/(2s)
// to twice the precision, and Dekker's exact product (the FMA form) gives the
// pair s*q; it is rounded once.  The correction terms need ~20 bits, hence the
// approximate reciprocal.  Outside [2^-900, 2^900] (or NaN): pow itself.
template <class Ar>
GB_HD double pow_3_4(Ar &ar, double x) {
  if (!Ar::FLAT && !(x >= 0x1p-900 && x <= 0x1p900)) return pow(x, 0.75);  // FlatOps::root sees the range
  const double s = ar.root(x);
  const double sl = fma(-s, s, x) * 0.5 * recip_approx(s);  // sqrt(x) = s + sl
  const double q = ar.root(s);
  const double ql = (fma(-q, q, s) + sl) * 0.5 * recip_approx(q);  // sqrt(s + sl) = q + ql
  const double ph = s * q;
  const double lo = fma(s, q, -ph) + (s * ql + sl * q);
  return ph + lo;
}
GB_HD double pow_3_4(double x) {
  PlainOps ar;
  return pow_3_4(ar, x);
}

// (p/p1)^(1/GAMMA_) of the isentrope
template <class Ar>
GB_HD double isentrope_pow(Ar &ar, double x, double ginv) {
  return ginv == 0.75 ? pow_3_4(ar, x) : pow(x, ginv);
}

template <class Cfg, class Ar>
GB_HD double state_gamma(Ar &ar, const Phys &ph, const double *prim) {
  return Cfg::SPH ? eos_gamma(ar, ph, prim[RHO], prim[PPP]) : ph.gamma_ad;
}
template <class Cfg>
GB_HD double state_gamma(const Phys &ph, const double *prim) {
  PlainOps ar;
  return state_gamma<Cfg>(ar, ph, prim);
}

// a state's Gamma - 1 as a divisor
template <class Cfg, class Ar>
GB_HD typename Ar::By by_state_gm1(Ar &ar, const Phys &ph, double gma) {
  return Cfg::SPH && ph.eos != 0 ? ar.by(gma - 1.) : by_gm1(ar, ph);
}

// gamma/(gamma-1) of a state: cached for the ideal EOS
template <class Cfg, class Ar>
GB_HD double enth_k(Ar &ar, const Phys &ph, const double *prim) {
  if (Cfg::SPH && ph.eos != 0) {
    const double g = eos_gamma(ar, ph, prim[RHO], prim[PPP]);
    return ar.quo(g, ar.by(g - 1.));
  }
  return ph.kgam;
}

// prim2cons (rel_sph.cpp:55-82, rel_cart.cpp:37-64)
template <class Cfg, class Ar>
GB_HD void prim2cons(Ar &ar, const Phys &ph, const double *prim, double *cons) {
  double rho = prim[RHO];
  double p = prim[PPP];
  double uu = prim[UU1];
  double lfac = lfac_of(ar, uu);
  double h;
  if (Cfg::FAST) {
    h = 1. + ar.quo(enth_k<Cfg>(ar, ph, prim) * p, ar.by(rho));
  } else {
    const double gma = state_gamma<Cfg>(ar, ph, prim);
    h = 1. + ar.quo(ar.quo(p * gma, by_state_gm1<Cfg>(ar, ph, gma)), ar.by(rho));
  }
  double D = lfac * rho;
  double tau = D * h * lfac - p - D;
  double ss = D * h * uu;
  cons[DEN] = D;
  cons[TAU] = tau;
  cons[SS1] = ss;
  cons[SS2] = 0.;
#pragma unroll
  for (int t = TR1; t < Cfg::NQ; ++t) cons[t] = prim[t] * D;
}
template <class Cfg>
GB_HD void prim2cons(const Phys &ph, const double *prim, double *cons) {
  PlainOps ar;
  prim2cons<Cfg>(ar, ph, prim, cons);
}

// prim2cons + state2flux of a reconstructed or cell state in one pass
// (rel_sph.cpp:55-113): lfac and v = u/lfac are formed once.
template <class Cfg, class Ar>
GB_HD void state2flux(Ar &ar, const double *prim, const double *cons, double *flux);

template <class Cfg, class Ar>
GB_HD void fill_state(Ar &ar, const Phys &ph, FState<Cfg> &S) {
  if (!Cfg::FAST) {
    prim2cons<Cfg>(ar, ph, S.prim, S.cons);
    state2flux<Cfg>(ar, S.prim, S.cons, S.flux);
    S.lfac = lfac_of(ar, S.prim[UU1]);
    S.v = ar.quo0(S.prim[UU1], ar.by(S.lfac));
    return;
  }
  const double rho = S.prim[RHO], p = S.prim[PPP], uu = S.prim[UU1];
  const double lfac = ar.root(1. + uu * uu);
  const double v = ar.quo(uu, ar.by(lfac));
  const double h = 1. + ar.quo(enth_k<Cfg>(ar, ph, S.prim) * p, ar.by(rho));
  const double D = lfac * rho;
  const double Dh = D * h;
  S.lfac = lfac;
  S.v = v;
  S.cons[DEN] = D;
  S.cons[TAU] = Dh * lfac - p - D;
  S.cons[SS1] = Dh * uu;
  S.cons[SS2] = 0.;
  S.flux[DEN] = D * v;
  S.flux[SS1] = S.cons[SS1] * v + p;
  S.flux[SS2] = 0.;
  S.flux[TAU] = S.cons[SS1] - D * v;
#pragma unroll
  for (int t = TR1; t < Cfg::NQ; ++t) {
    S.cons[t] = S.prim[t] * D;
    S.flux[t] = S.cons[t] * v;
  }
}

// state2flux (rel_sph.cpp:85-113, rel_cart.cpp:67-95)
template <class Cfg, class Ar>
GB_HD void state2flux(Ar &ar, const double *prim, const double *cons, double *flux) {
  double p = prim[PPP];
  double uu = prim[UU1];
  const auto lfac = ar.by(lfac_of(ar, uu));
  double D = cons[DEN];
  double ss = cons[SS1];
  flux[DEN] = ar.quo0(D * uu, lfac);
  flux[SS1] = ar.quo0(ss * uu, lfac) + p;
  flux[SS2] = 0.;
  flux[TAU] = ss - flux[DEN];
#pragma unroll
  for (int t = TR1; t < Cfg::NQ; ++t) flux[t] = ar.quo0(cons[t] * uu, lfac);
}

// ---------------------------------------------------------------------------
// cons2prim: pressure root of f(p) (rel_sph.cpp:191-210 / rel_cart.cpp:108-123)
// by safeguarded Newton-Raphson on the same bracket and with the same
// no-solution semantics as the reference's Brent driver (rel_sph.cpp:243-286).

struct C2PStats {
  int iters;     // f evaluations after the bracket set-up
  int fallback;  // 1 if the iteration cap was hit (bisection-limited)
  int deferred;  // 1 if a deferring search stopped at a poor warm start (c2p_pressure_body)
  int poor;      // 1 if a search was needed and its warm start was poor (c2p_warm_start_poor)
};

// A warm start is poor where the first Newton correction from it, |f/f'|,
// exceeds this fraction of the pressure: worse than the learned guess's own
// starting error of a few per cent.  (A build may set another fraction with
// -DGB_GUESS_GATE=...)
#ifndef GB_GUESS_GATE
#define GB_GUESS_GATE 3e-2
#endif
constexpr double kGuessGate = GB_GUESS_GATE;

GB_HD bool c2p_warm_start_poor(double f, double df, double p) { return !(fabs(f) <= kGuessGate * fabs(df) * p); }

// f(p) = E + p - D lfac - k p lfac^2 with lfac = (1 - S^2/(E+p)^2)^(-1/2)
// (rel_sph.cpp:191-210 takes |1 - S^2/W^2|, rel_cart.cpp:108-123 does not).
// Returns f; with df != nullptr also df/dp and lfac^2.  For the Synge EOS the
// derivative of Gamma_eff is included through rho = D/lfac and a = p/rho/(G-1).
template <class Cfg>
GB_HD double c2p_f(const Phys &ph, double p, double D, double S2, double E, double *df = nullptr,
                   double *l2out = nullptr) {
  const double W = E + p;
  const double rW = 1. / W;
  const double x = S2 * rW * rW;
  const double arg = Cfg::SPH ? fabs(1. - x) : (1. - x);
  const double lfac = rsqrt(arg);
  const double l2 = lfac * lfac;
  double k, dk = 0.;
  if (Cfg::SPH && ph.eos != 0) {
    const double G = ph.gamma_ad;
    const double rho = D / lfac;
    const double a = p / rho / (G - 1.);
    const double sq = sqrt(a * a + 1.);
    const double e = a + sq;
    const double gma = G - (G - 1.) / 2. * (1. - 1. / (e * e));
    k = gma / (gma - 1.);
    if (df) {
      const double sgn = (1. - x) >= 0. ? 1. : -1.;
      const double dl = -sgn * lfac * l2 * x * rW;
      const double da = (lfac + p * dl) / (D * (G - 1.));
      const double dgma = -(G - 1.) / (e * e * e) * (da * (1. + a / sq));
      dk = -dgma / ((gma - 1.) * (gma - 1.));
    }
  } else {
    k = ph.kgam;
  }
  const double f = W - D * lfac - k * p * l2;
  if (df) {
    const double sgn = (1. - x) >= 0. ? 1. : -1.;
    const double dl = -sgn * lfac * l2 * x * rW;
    *df = 1. - D * dl - dk * p * l2 - k * (l2 + 2. * p * lfac * dl);
  }
  if (l2out) *l2out = l2;
  return f;
}

// f(p) with x = S^2/W^2, lfac and lfac^2 at p, and whether 1 - x was not
// negative there (else lfac is that of its magnitude).
struct C2PEval {
  double f, x, lfac, l2;
  bool inside;
};

// f in the reference's operation order (rel_sph.cpp:198-207, rel_cart.cpp:118-120).
template <class Cfg, class Ar>
GB_HD C2PEval c2p_f_ref(Ar &ar, const Phys &ph, double p, double D, double S, double E, bool p_may_be_zero = false) {
  C2PEval e;
  const double W = E + p;
  e.x = ar.quo0(S * S, ar.by(W * W));
  const double arg = Cfg::SPH ? fabs(1. - e.x) : (1. - e.x);
  const double lfac = ar.rroot(arg);
  const bool ideal = !Cfg::SPH || ph.eos == 0;
  const double gma = ideal ? ph.gamma_ad : eos_gamma(ar, ph, ar.quo(D, ar.by(lfac)), p);
  const auto gm1 = ideal ? by_gm1(ar, ph) : ar.by(gma - 1.);
  // p = 0 at the bracket's lower end p_lo
  const double kp = gma * p * lfac * lfac;
  e.f = (E + p - D * lfac - (p_may_be_zero ? ar.quo0(kp, gm1) : ar.quo(kp, gm1)));
  e.l2 = lfac * lfac;
  e.lfac = lfac;
  e.inside = arg >= 0.;
  return e;
}

// df/dp at p, after c2p_f_ref there
template <class Cfg, class Ar>
GB_HD double c2p_slope_ref(Ar &ar, const Phys &ph, double p, double D, double S, double E, const C2PEval &e) {
  if (Cfg::SPH && ph.eos != 0) {  // Gamma_eff(p) terms: take them from the derivative form
    double dfast;
    c2p_f<Cfg>(ph, p, D, S * S, E, &dfast);
    return dfast;
  }
  // d lfac/dp = -lfac^3 x / W with the same lfac and x as f
  const double sgn = (1. - e.x) >= 0. ? 1. : -1.;
  const double dl = ar.quo0(-sgn * e.lfac * e.l2 * e.x, ar.by(E + p));
  // kgam is GAMMA_/(GAMMA_-1) rounded once on the host: gma/(gma-1) exactly
  return 1. - D * dl - ph.kgam * (e.l2 + 2. * p * e.lfac * dl);
}

// What the root search returns: the pressure the reference would go on with
// (the starting one where it finds none) and the Lorentz factor
// 1/sqrt(|1 - S^2/(E+p)^2|) there when the search evaluated f at it (the same
// rounding as f's), else -1; then its statistics (C2PStats).
struct C2PRoot {
  double p, lfac;
  C2PStats st;
};

// Pressure root of the cons2prim driver (rel_sph.cpp:243-286): the bracket,
// its no-solution tests and the warm start pCand are the reference's; the
// Brent search is replaced by safeguarded Newton-Raphson.
//
// defer: where a search is needed and the warm start is poor
// (c2p_warm_start_poor), stop before it and set st.deferred; the caller then
// starts the search again from a better pressure (the learned guess).
//
// With FlatOps the result counts only if !ar.bad(); the loops stop early where
// it is set.
template <class Cfg, class Ar>
GB_HD C2PRoot c2p_pressure_body(Ar &ar, const Phys &ph, double D, double S, double S2, double E, double pCand,
                                bool defer) {
  auto feval = [&](double p, bool p_may_be_zero = false) -> C2PEval {
    if (!Cfg::FAST_ROOT) return c2p_f_ref<Cfg>(ar, ph, p, D, S, E, p_may_be_zero);
    C2PEval e;
    e.f = c2p_f<Cfg>(ph, p, D, S2, E, nullptr, &e.l2);
    e.x = 0.;
    e.lfac = sqrt(e.l2);
    e.inside = false;
    return e;
  };
  auto slope = [&](double p, const C2PEval &e) -> double {
    if (!Cfg::FAST_ROOT) return c2p_slope_ref<Cfg>(ar, ph, p, D, S, E, e);
    double df;
    c2p_f<Cfg>(ph, p, D, S2, E, &df);
    return df;
  };
  C2PRoot R;
  R.st = C2PStats{0, 0, 0, 0};
  // f at the warm start: the search starts there when it lies in the bracket
  C2PEval e0 = feval(pCand);
  R.p = pCand;
  R.lfac = e0.inside ? e0.lfac : -1.;
  // rel_cyl.cpp:161 searches only where |f| exceeds 1e-13 (rel_sph, rel_cart: 0)
  if (fabs(e0.f) > (Cfg::CYL ? 1.e-13 : 0.)) {
    double df = slope(pCand, e0);
    R.st.poor = c2p_warm_start_poor(e0.f, df, pCand);
    if (defer && R.st.poor) {
      R.st.deferred = 1;
      return R;
    }
    double p_lo = fmax(0., (1. + 1e-13) * S - E);
    // No solution where f(p_lo) < 0.  At p_lo = 0, f = E - D lfac with
    // lfac^2 = E^2 / (E^2 - S^2): certainly not negative, whatever its rounding
    // (lfac carries eps E^2 / (E^2 - S^2)), where D^2 stays that much below
    // E^2 - S^2, as it does unless the gas is colder than p/rho ~ 1e-14 lfac^2;
    // then f need not be formed (2 quotients and 2 roots of every search).  (The
    // squares must not lose digits to underflow.)
    bool find_p = true;
    const bool surely = p_lo == 0. && E * E >= 0x1p-900 && D * D <= (E - S) * (E + S) - 0x1p-47 * (E * E);
    if (!surely && feval(p_lo, true).f < 0) find_p = false;
    double p_hi;
    if (e0.f < 0) {
      p_hi = 1. * pCand;
    } else {
      p_hi = pCand;
      // the reference grows p_hi without bound (a zero guess would never end);
      // 400 decades reach infinity, where f is NaN and the loop stops anyway.
      // Its first test re-evaluates f(pCand), which is e0.f.
      for (int g = 0; g < 400 && (g == 0 ? e0.f : feval(p_hi).f) > 0; ++g) {
        p_hi *= 10;
        if (Ar::FLAT && ar.bad()) break;
      }
    }
    if (p_hi < p_lo) find_p = false;
    if (find_p) {
      // f(lo) >= 0 >= f(hi).  The warm start tightens one side.
      double lo = p_lo, hi = p_hi;
      if (e0.f > 0.) lo = fmax(lo, pCand);
      double p = fmin(fmax(pCand, lo), hi);
      if (!(p == pCand)) {
        e0 = feval(p);
        df = slope(p, e0);
      }
      const int MAXIT = 100;
      const double eps = 2.220446049250313e-16;
      int iters;
      for (iters = 1; iters <= MAXIT; ++iters) {
        // Rounding noise of f: E, p, D lfac and k p lfac^2 cancel, and lfac
        // itself carries eps*lfac^2 relative error from 1 - S^2/W^2.  Below
        // this level the sign of f is noise and p is as good as it gets.
        // (lfac is sqrt(l2): the root of a rounded square is exact.)
        const double noise =
            eps * (E + p + D * e0.lfac * (1. + e0.l2) + 4. * p * e0.l2 * (1. + 2. * e0.l2));
        if (e0.f == 0. || fabs(e0.f) <= noise) break;
        if (iters > 1) df = slope(p, e0);
        double pn = p - ar.quo(e0.f, ar.by(df));
        if (!(pn > lo && pn < hi)) {
          // Newton left the bracket: bisect, geometrically once lo > 0
          pn = lo > 0. ? sqrt(lo) * sqrt(hi) : 0.5 * (lo + hi);
          if (!(pn > lo && pn < hi)) pn = 0.5 * (lo + hi);
        }
        e0 = feval(pn);
        if (e0.f > 0.) lo = pn;
        else if (e0.f < 0.) hi = pn;
        const double step = fabs(pn - p);
        p = pn;
        if (e0.f == 0. || step <= 1.e-14 * pn || (hi - lo) <= 1.e-14 * hi) break;
        if (Ar::FLAT && ar.bad()) break;
      }
      R.st.iters = iters;
      if (iters > MAXIT) R.st.fallback = 1;
      R.p = p;
      R.lfac = e0.inside ? e0.lfac : -1.;
    }
  }
  return R;
}

template <class Cfg>
GB_HD_OUTLINE C2PRoot c2p_pressure_outline(const Phys &ph, double D, double S, double S2, double E, double pCand,
                                           bool defer) {
  PlainOps ar;
  return c2p_pressure_body<Cfg>(ar, ph, D, S, S2, E, pCand, defer);
}

// The step with the learned guess, and formulas formed again with PlainOps,
// call the cartesian search from one out-of-line copy: inlined at every call
// site of the fused step kernel it crowds the instruction cache.  OUTLINE
// forces the out-of-line copy (a second, rarely taken call site).  FlatOps
// searches are inline: a call would end their straight-line code.
template <class Cfg, bool OUTLINE, class Ar>
GB_HD C2PRoot c2p_pressure(Ar &ar, const Phys &ph, double D, double S, double S2, double E, double pCand,
                           bool defer = false) {
  if (Ar::FLAT || !OUTLINE) return c2p_pressure_body<Cfg>(ar, ph, D, S, S2, E, pCand, defer);
  return c2p_pressure_outline<Cfg>(ph, D, S, S2, E, pCand, defer);
}

// What cons2prim's root search is given: D, E = D + tau, S and S^2 of the
// momentum, and the starting pressure (the previous one, floored in rel_sph).
struct C2PInput {
  double D, E, ss, S2, S, pCand;
};

template <class Cfg, class Ar>
GB_HD C2PInput c2p_input(Ar &ar, const double *cons, const double *prim) {
  C2PInput in;
  in.D = cons[DEN];
  const double tau = cons[TAU];
  in.E = in.D + tau;
  in.ss = cons[SS1];
  double S2 = 0.;
  S2 += in.ss * in.ss;
  in.S2 = S2;
  in.S = Cfg::FAST_ROOT ? fabs(in.ss) : ar.root_of_square(in.ss, S2);  // sqrt(S2)
  in.pCand = Cfg::SPH ? fmax(1.e-13, prim[PPP]) : prim[PPP];
  return in;
}

// FluidState::cons2prim (rel_sph.cpp:213-320; rel_cart.cpp:125-229).
// On entry prim holds the previous primitives (pressure warm start); on exit
// prim holds the recovered primitives and cons is rewritten by prim2cons.
// Hooks::cons2prim_user (the problem module's FluidState::cons2prim_user,
// rel_sph.cpp:304) sees rho, p and u before the pressure floor; par is the
// run's parameter words.
// defer (with st): where the warm start is poor the search stops before it
// (st->deferred, c2p_pressure_body) and prim and cons are left as they were,
// for a second call from a better starting pressure.  OUTLINE: the search's
// out-of-line copy (c2p_pressure).
template <class Cfg, class Hooks = gamma_problem::Problem, bool OUTLINE = !Cfg::SPH, class Ar>
GB_HD void cons2prim(Ar &ar, const Phys &ph, double *cons, double *prim, C2PStats *st, const double *par = nullptr,
                     bool defer = false) {
  const C2PInput in = c2p_input<Cfg>(ar, cons, prim);
  const double D = in.D, E = in.E, ss = in.ss, S2 = in.S2, S = in.S;
  const C2PRoot root = c2p_pressure<Cfg, OUTLINE>(ar, ph, D, S, S2, E, in.pCand, defer);
  if (st) *st = root.st;
  if (defer && root.st.deferred) return;

  const double lf_root = root.lfac;
  double p = root.p;
  double rho, uu;
  if (Cfg::FAST_ROOT) {  // lfac = W/sqrt(W^2-S^2), rho = D/lfac, u = lfac v S_i/S with v = S/W
    const double rW = 1. / (E + p);
    const double v2 = S2 * rW * rW;
    const double s1 = sqrt(fabs(1. - v2));  // 1/lfac
    rho = D * s1;
    uu = (fabs(S) == 0.) ? 0. : (ss * rW) / s1;
  } else {  // rel_sph.cpp:288-302
    // lfac = 1/sqrt(|1 - S2/(E+p)^2|): the root search's last f evaluation
    // formed the same quotient from S*S, which is S2 whenever S*S == S2
    double lfac = lf_root;
    if (!(lfac > 0. && S * S == S2)) {
      double Ep2 = (E + p) * (E + p);
      double v2 = ar.quo0(S2, ar.by(Ep2));
      lfac = ar.rroot(fabs(1. - v2));
    }
    rho = ar.quo(D, ar.by(lfac));
    if (Cfg::CYL ? fabs(S) < 1.e-14 : fabs(S) == 0.) {  // rel_cyl.cpp:207
      uu = 0;
    } else {
      double v = ar.root(1. - ar.inv(lfac * lfac));
      // ss/S is exactly +-1 when S == |ss|
      uu = lfac * v * (fabs(ss) == S ? (ss > 0. ? 1. : -1.) : ss / S);
    }
  }
  Hooks::cons2prim_user(par, &rho, &p, &uu);
  if (Cfg::SPH) p = fmax(p, P_FLOOR);
  prim[PPP] = p;
  prim[RHO] = rho;
  prim[UU1] = uu;
  prim[UU2] = 0.;
  if (Cfg::FAST) {
    const double rD = ar.inv(D);
#pragma unroll
    for (int t = TR1; t < Cfg::NQ; ++t) prim[t] = cons[t] * rD;
  } else {
    const auto byD = ar.by(D);
#pragma unroll
    for (int t = TR1; t < Cfg::NQ; ++t) prim[t] = ar.quo0(cons[t], byD);
  }
  prim2cons<Cfg>(ar, ph, prim, cons);
}
template <class Cfg, class Hooks = gamma_problem::Problem, bool OUTLINE = !Cfg::SPH>
GB_HD void cons2prim(const Phys &ph, double *cons, double *prim, C2PStats *st, const double *par = nullptr,
                     bool defer = false) {
  PlainOps ar;
  cons2prim<Cfg, Hooks, OUTLINE>(ar, ph, cons, prim, st, par, defer);
}

#ifdef __CUDACC__
// State k of a batch (cons, prim: [NQ rows][n] in the reference's slot order),
// from its own pressure or, if positive, from p0.
template <class Cfg, class Ar>
GB_HD bool cons2prim_at_ops(const Phys &ph, double *cons, double *prim, int n, int k, int *iters, double p0) {
  constexpr int NQ = Cfg::NQ;
  Ar ar;
  double c[NQ], p[NQ];
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    c[q] = cons[(long long)q * n + k];
    p[q] = prim[(long long)q * n + k];
  }
  if (p0 > 0.) p[PPP] = p0;
  C2PStats st;
  cons2prim<Cfg, gamma_problem::Problem, false>(ar, ph, c, p, &st);
  if (ar.bad()) return false;  // nothing written yet
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    cons[(long long)q * n + k] = c[q];
    prim[(long long)q * n + k] = p[q];
  }
  if (iters) iters[k] = st.iters;
  return true;
}
template <class Cfg>
GB_HD_OUTLINE void cons2prim_at_plain(const Phys &ph, double *cons, double *prim, int n, int k, int *iters, double p0) {
  cons2prim_at_ops<Cfg, PlainOps>(ph, cons, prim, n, k, iters, p0);
}
template <class Cfg>
GB_HD void cons2prim_at(const Phys &ph, double *cons, double *prim, int n, int k, int *iters, double p0) {
  if (!cons2prim_at_ops<Cfg, FlatOps>(ph, cons, prim, n, k, iters, p0))
    cons2prim_at_plain<Cfg>(ph, cons, prim, n, k, iters, p0);
}
#endif  // __CUDACC__

// ---------------------------------------------------------------------------
// Riemann problem at a moving interface

struct Waves {
  double lL, lS, lR;
};

// Interface::wavespeedEstimates + computeLambda (rel_sph.cpp:322-394;
// rel_cart.cpp:260-302 switches to the linear root when |FhllE| < 1e-15).
template <class Cfg, class Ar>
GB_HD Waves compute_lambda_ref(Ar &ar, const Phys &ph, const FState<Cfg> &L, const FState<Cfg> &R) {
  const bool ws = Cfg::SPH && ph.eos_ws;
  const double GL = ws ? eos_gamma(ar, ph, L.prim[RHO], L.prim[PPP]) : ph.gamma_ad;
  const double GR = ws ? eos_gamma(ar, ph, R.prim[RHO], R.prim[PPP]) : ph.gamma_ad;
  Waves w;
  double lfacL = L.lfac;
  double lfacR = R.lfac;
  double vL = L.v;
  double vR = R.v;
  const auto gm1L = ws ? ar.by(GL - 1.) : by_gm1(ar, ph), gm1R = ws ? ar.by(GR - 1.) : by_gm1(ar, ph);
  double cSL = ar.root(ar.quo(GL * L.prim[PPP], ar.by(L.prim[RHO] + ar.quo(L.prim[PPP] * GL, gm1L))));
  double cSR = ar.root(ar.quo(GR * R.prim[PPP], ar.by(R.prim[RHO] + ar.quo(R.prim[PPP] * GR, gm1R))));
  double sgSL = ar.quo(cSL * cSL, ar.by(lfacL * lfacL * (1. - cSL * cSL)));
  double sgSR = ar.quo(cSR * cSR, ar.by(lfacR * lfacR * (1. - cSR * cSR)));
  const double rtL = ar.root(sgSL * (1. - vL * vL + sgSL)), rtR = ar.root(sgSR * (1. - vR * vR + sgSR));
  const auto nL = ar.by(1. + sgSL), nR = ar.by(1. + sgSR);
  double l1, l2;
  l1 = ar.quo(vR - rtR, nR);
  l2 = ar.quo(vL - rtL, nL);
  w.lL = fmin(l1, l2);
  l1 = ar.quo(vR + rtR, nR);
  l2 = ar.quo(vL + rtL, nL);
  w.lR = fmax(l1, l2);

  const double lL = w.lL, lR = w.lR;
  double mmL = L.cons[SS1];
  double mmR = R.cons[SS1];
  double pL = L.prim[PPP];
  double pR = R.prim[PPP];
  double EL = L.cons[TAU] + L.cons[DEN];
  double ER = R.cons[TAU] + R.cons[DEN];
  double AL = lL * EL - mmL;
  double AR = lR * ER - mmR;
  double BL = mmL * (lL - vL) - pL;
  double BR = mmR * (lR - vR) - pR;
  const auto dl = ar.by(lR - lL);
  double FhllE = ar.quo0(lL * AR - lR * AL, dl);
  double Ehll = ar.quo(AR - AL, dl);
  double Fhllm = ar.quo(lL * BR - lR * BL, dl);
  double mhll = ar.quo0(BR - BL, dl);
  bool linear = Cfg::SPH ? (fabs(FhllE) == 0) : (fabs(FhllE) < 1.e-15);
  if (linear) {
    w.lS = ar.quo0(mhll, ar.by(Ehll + Fhllm));
  } else {
    // pow(x, 2.) of the C library is the correctly rounded square: x*x
    const double ef = Ehll + Fhllm;
    double delta = ef * ef - 4. * FhllE * mhll;
    w.lS = ar.quo((Ehll + Fhllm) - ar.root(delta), ar.by(2. * FhllE));
  }
  return w;
}

template <class Cfg, class Ar>
GB_HD Waves compute_lambda(Ar &ar, const Phys &ph, const FState<Cfg> &L, const FState<Cfg> &R) {
  if (!Cfg::FAST_RIEMANN || ph.eos_ws) return compute_lambda_ref<Cfg>(ar, ph, L, R);
  const double G = ph.gamma_ad;
  const double kg = ph.kgam;
  Waves w;
  const double vL = L.v, vR = R.v;
  // relativistic sound speed (uses GAMMA_ in the reference for either EOS)
  const double cs2L = G * L.prim[PPP] / (L.prim[RHO] + L.prim[PPP] * kg);
  const double cs2R = G * R.prim[PPP] / (R.prim[RHO] + R.prim[PPP] * kg);
  const double sgSL = cs2L / (L.lfac * L.lfac * (1. - cs2L));
  const double sgSR = cs2R / (R.lfac * R.lfac * (1. - cs2R));
  const double qL = sqrt(sgSL * (1. - vL * vL + sgSL));
  const double qR = sqrt(sgSR * (1. - vR * vR + sgSR));
  const double rL = 1. / (1. + sgSL), rR = 1. / (1. + sgSR);
  w.lL = fmin((vR - qR) * rR, (vL - qL) * rL);
  w.lR = fmax((vR + qR) * rR, (vL + qL) * rL);

  const double lL = w.lL, lR = w.lR;
  const double mmL = L.cons[SS1], mmR = R.cons[SS1];
  const double pL = L.prim[PPP], pR = R.prim[PPP];
  const double EL = L.cons[TAU] + L.cons[DEN];
  const double ER = R.cons[TAU] + R.cons[DEN];
  const double AL = lL * EL - mmL;
  const double AR = lR * ER - mmR;
  const double BL = mmL * (lL - vL) - pL;
  const double BR = mmR * (lR - vR) - pR;
  const double rd = 1. / (lR - lL);
  const double FhllE = (lL * AR - lR * AL) * rd;
  const double Ehll = (AR - AL) * rd;
  const double Fhllm = (lL * BR - lR * BL) * rd;
  const double mhll = (BR - BL) * rd;
  const bool linear = Cfg::SPH ? (fabs(FhllE) == 0) : (fabs(FhllE) < 1.e-15);
  const double eh = Ehll + Fhllm;
  if (linear) {
    w.lS = mhll / eh;
  } else {
    const double delta = eh * eh - 4. * FhllE * mhll;
    w.lS = (eh - sqrt(delta)) / (2. * FhllE);
  }
  return w;
}

// HLLC flux F - vU in the frame of an interface moving at v, times dA
// (hllc.cpp:12-39 with starState rel_sph.cpp:397-450).  The four branch tests
// are independent ifs in the reference and stay so.
template <class Cfg, class Ar>
GB_HD void hllc_flux(Ar &ar, const FState<Cfg> &L, const FState<Cfg> &R, const Waves &w, double v, double dA,
                     double *flux) {
  const double lS = w.lS;
  auto star = [&](const FState<Cfg> &Sin, double lbda, double *out_cons) {
    const double m = Sin.cons[SS1];
    const double vv = Sin.v;
    const double p = Sin.prim[PPP];
    const double D = Sin.cons[DEN];
    const double E = Sin.cons[TAU] + Sin.cons[DEN];
    const double A = lbda * E - m;
    const double B = m * (lbda - vv) - p;
    const double pS = ar.quo(A * lS - B, ar.by(1. - lbda * lS));
    double k;
    if (Cfg::FAST) {
      const double rk = ar.inv(lbda - lS);
      k = (lbda - vv) * rk;
      out_cons[SS1] = (m * (lbda - vv) + pS - p) * rk;
      out_cons[TAU] = (E * (lbda - vv) + pS * lS - p * vv) * rk - D * k;
    } else {  // rel_sph.cpp:433-442
      const auto dl = ar.by(lbda - lS);
      k = ar.quo(lbda - vv, dl);
      out_cons[SS1] = ar.quo(m * (lbda - vv) + pS - p, dl);
      out_cons[TAU] = ar.quo(E * (lbda - vv) + pS * lS - p * vv, dl) - D * k;
    }
    out_cons[DEN] = D * k;
    out_cons[SS2] = 0.;
#pragma unroll
    for (int t = TR1; t < Cfg::NQ; ++t) out_cons[t] = Sin.cons[t] * k;
  };
  if (v < w.lL) {
#pragma unroll
    for (int q = 0; q < Cfg::NQ; ++q) flux[q] = L.flux[q] - v * L.cons[q];
  }
  if (w.lL <= v && v < lS) {
    double sc[Cfg::NQ];
    star(L, w.lL, sc);
#pragma unroll
    for (int q = 0; q < Cfg::NQ; ++q) flux[q] = L.flux[q] + w.lL * (sc[q] - L.cons[q]) - v * sc[q];
  }
  if (lS <= v && v < w.lR) {
    double sc[Cfg::NQ];
    star(R, w.lR, sc);
#pragma unroll
    for (int q = 0; q < Cfg::NQ; ++q) flux[q] = R.flux[q] + w.lR * (sc[q] - R.cons[q]) - v * sc[q];
  }
  if (w.lR <= v) {
#pragma unroll
    for (int q = 0; q < Cfg::NQ; ++q) flux[q] = R.flux[q] - v * R.cons[q];
  }
#pragma unroll
  for (int q = 0; q < Cfg::NQ; ++q) flux[q] *= dA;
}

// ---------------------------------------------------------------------------
// Shock detector (radiation_sph.cpp:41-158), forward direction.  Returns false
// (and leaves *pspec alone) where the reference returns -1 early.
template <class Cfg, class Ar>
GB_HD bool compute_Sd(Ar &ar, const Phys &ph, const FState<Cfg> &S1, const FState<Cfg> &S2, double *Sd,
                      double *pspec) {
  // with eos_ws, the upstream state's Gamma_eff throughout
  const double G = (Cfg::SPH && ph.eos_ws) ? eos_gamma(ar, ph, S1.prim[RHO], S1.prim[PPP]) : ph.gamma_ad;
  const int n_evals = 10;
  const double chi = 0.5;
  double p1 = S1.prim[PPP];
  double p2 = S2.prim[PPP];
  const auto by_p1 = ar.by(p1);
  if (fabs(ar.quo0(p1 - p2, by_p1)) < 1.e-10 || p1 < p2) {
    *Sd = -1;
    return false;
  }
  double delta_p = p2 - p1;
  double dp = ar.quo(delta_p, ar.by((double)n_evals));
  double rho1 = S1.prim[RHO];
  double rho2 = S2.prim[RHO];
  const auto bgm1 = Cfg::SPH && ph.eos_ws ? ar.by(G - 1.) : by_gm1(ar, ph);
  double h1 = 1 + ar.quo(ar.quo(p1 * G, bgm1), ar.by(rho1));
  const auto by_rho2 = ar.by(rho2);
  double h2 = 1 + ar.quo(ar.quo(p2 * G, bgm1), by_rho2);
  double lfac2 = S2.lfac;
  double vx1 = S1.v;
  double vx2 = S2.v;
  double v12 = ar.quo(vx1 - vx2, ar.by(1 - vx1 * vx2));
  double A1 = h1 * 0.;
  double I = 0;
  const double ginv = ar.inv(G);
#pragma unroll 2
  for (int ip = 0; ip < n_evals; ++ip) {
    double p = p1 + (ip + .5) * dp;
    double rho = rho1 * isentrope_pow(ar, ar.quo(p, by_p1), ginv);
    const double pg = ar.quo(p * G, bgm1);
    double h = 1 + ar.quo(pg, ar.by(rho));
    double cs = ar.root(ar.quo(G * p, ar.by(rho + pg)));
    // with A1 = 0 (1D: no transverse velocity) the root is sqrt(h*h) = h exactly
    // (h >= 1, and sqrt of a rounded square is the number itself)
    const double num = A1 == 0. ? h : ar.root(h * h + A1 * A1 * (1. - cs * cs));
    double dI = ar.quo(num, ar.by((h * h + A1 * A1) * rho * cs)) * dp;
    I += dI;
  }
  double vSR = tanh(I);
  double rho22 = rho2 * rho2;
  double lfac22 = lfac2 * lfac2;
  double vx22 = vx2 * vx2;
  double g = G;
  double gm1 = (g - 1.);
  double gm12 = gm1 * gm1;
  double Da = ar.quo(4. * g * p1 * ((g - 1) * p2 + p1), ar.by(gm12 * (p1 - p2) * (p1 - p2)));
  double Db = ar.quo(h2 * (p2 - p1), by_rho2) - h2 * h2;
  double Dd = 1. - Da * Db;
  // the root of a negative number is NaN, and so is then all that follows
  if (!(Dd >= 0.)) {
    *Sd = nan("");
    *pspec = P_SPEC;
    return true;
  }
  double h3 = ar.quo((ar.root(Dd) - 1) * gm1 * (p1 - p2), ar.by(2 * (gm1 * p2 + p1)));
  double J232a = ar.quo(-g, bgm1) * (p1 - p2);
  double J232b = ar.quo(h3 * (h3 - 1), by_p1) - ar.quo(h2 * (h2 - 1), ar.by(p2));
  double J232 = ar.quo(J232a, ar.by(J232b));
  if (!(J232 >= 0.)) {
    *Sd = nan("");
    *pspec = P_SPEC;
    return true;
  }
  double J23 = ar.root(J232);
  double Vsa = rho22 * lfac22 * vx2 + fabs(J23) * ar.root(J232 + rho22 * lfac22 * (1. - vx22));
  double Vsb = rho22 * lfac22 + J232;
  double Vs = ar.quo(Vsa, ar.by(Vsb));
  double v2Sa = (p1 - p2) * (1. - vx2 * Vs);
  double v2Sb = (Vs - vx2) * (h2 * rho2 * lfac22 * (1. - vx22) + p1 - p2);
  double v2S = ar.quo(v2Sa, ar.by(v2Sb));
  double vlim = vSR + chi * (v2S - vSR);
  *Sd = v12 - vlim;
  *pspec = P_SPEC;  // spectral_p with VARIABLE_PSPEC_ disabled
  return true;
}

// ---------------------------------------------------------------------------
// Local synchrotron tracers (radiation_sph.cpp:196-300)

struct SynchConst {
  double Nalpha, Nmp, Nme;
};

template <class Cfg>
GB_HD double gammae2trac(double gme, const double *prim) {
  double lfac = lfac_of(prim[UU1]);
  double rho = prim[RHO];
  if (gme != 0.) return (lfac * pow(rho, 4. / 3.) / gme);
  return 0;
}

template <class Cfg>
GB_HD double gamma_min_init(const Phys &ph, const SynchConst &sc, const double *prim) {
  double rho = prim[RHO];
  double p = prim[PPP];
  double psyn = prim[PSN];
  double gma = state_gamma<Cfg>(ph, prim);
  double h = 1. + p * gma / (gma - 1.) / rho;
  double eps = rho * (h - 1.) / gma;
  double ee = EPS_E * eps;
  double ne = ZETA * rho / sc.Nmp;
  double lfac_av = ee / (ne * sc.Nme);
  return (psyn - 2.) / (psyn - 1.) * lfac_av;
}

// Cell::radiation_injectParticles
template <class Cfg>
GB_HD void inject_particles(const Phys &ph, const SynchConst &sc, double *prim, bool shocked, double pspec) {
  double lfac = lfac_of(prim[UU1]);
  double rho = prim[RHO];
  if (shocked) {
    if (pspec > prim[PSN] || isnan(prim[PSN])) prim[PSN] = pspec;
    prim[GMX] = gammae2trac<Cfg>(GAMMA_MAX_INIT, prim) / (lfac * rho);
    prim[GMN] = gammae2trac<Cfg>(gamma_min_init<Cfg>(ph, sc, prim), prim) / (lfac * rho);
  }
  if (isnan(prim[GMX]) || isnan(prim[GMN])) {  // lim only where it is used
    const double lim = lfac * pow(rho, 4. / 3.) / (lfac * rho);
    if (isnan(prim[GMX])) prim[GMX] = lim;
    if (isnan(prim[GMN])) prim[GMN] = lim;
  }
}

// Cell::radiativeSourceTerms: returns the increment of cons[GMX] and cons[GMN]
template <class Cfg, class Ar>
GB_HD double radiative_source(Ar &ar, const Phys &ph, const SynchConst &sc, const double *prim, double dV,
                              double dt) {
  double rho = prim[RHO];
  double p = prim[PPP];
  double gma = state_gamma<Cfg>(ar, ph, prim);
  double h = 1 + ar.quo(ar.quo(p * gma, by_state_gm1<Cfg>(ar, ph, gma)), ar.by(rho));
  double eps = ar.quo(rho * (h - 1.), ar.by(gma));
  double eB = EPS_B * eps;
  double B = ar.root(8. * PI_ * eB);
  return sc.Nalpha * pow(rho, 4. / 3.) * B * B * dV * dt;
}
template <class Cfg>
GB_HD double radiative_source(const Phys &ph, const SynchConst &sc, const double *prim, double dV, double dt) {
  PlainOps ar;
  return radiative_source<Cfg>(ar, ph, sc, prim, dV, dt);
}

// ---------------------------------------------------------------------------
// Geometry (spherical1D.cpp:12-76, cartesian.cpp:11-43)

struct Geom {
  double x, dx, dV, dl, cen;
};

template <class Cfg, class Ar>
GB_HD Geom make_geom(Ar &ar, double x, double dx) {
  Geom g;
  g.x = x;
  g.dx = dx;
  g.dl = dx;
  if (Cfg::SPH) {
    double r = x, dr = dx;
    g.dV = 4. * PI_ * r * r * dr;
    double r2 = r * r;
    double dr2 = dr * dr;
    g.cen = ar.quo(3. * r * (r2 + dr2), ar.by(3 * r2 + dr2));
  } else {
    g.dV = 1. * dx;
    g.cen = x;
  }
  return g;
}
template <class Cfg>
GB_HD Geom make_geom(double x, double dx) {
  PlainOps ar;
  return make_geom<Cfg>(ar, x, dx);
}

// Cell::move: geometry between two interfaces
template <class Cfg, class Ar>
GB_HD Geom geom_between(Ar &ar, double xL, double xR) {
  return make_geom<Cfg>(ar, (xR + xL) / 2., (xR - xL));
}

template <class Cfg>
GB_HD double iface_area(double x) {
  if (Cfg::SPH) {
    double r = x;
    return 4. * PI_ * r * r;
  }
  return 1.;
}

GB_HD double minmod(double a, double b) {
  if (fabs(a) < fabs(b) && a * b > 0) return a;
  if (fabs(b) < fabs(a) && a * b > 0) return b;
  return 0;
}

}  // namespace gb
