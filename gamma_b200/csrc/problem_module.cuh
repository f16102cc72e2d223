// Problem modules: what one module .cu file instantiates and registers.
//
// A module (include/gamma_problem.h) is a struct of hooks plus the module set
// it runs with.  GAMMA_PROBLEM_MODULE(name, Hooks, modules, id) at the end of
// its file instantiates the 1D step kernel for it in every launch shape of the
// autotuner (tune.h), without and with the learned cons2prim guess, and adds an entry
// to the library's registry (gamma_api.cu), through which the C ABI configures
// and launches it.  The set-up hooks run on the host (initial_state below).
#pragma once

#include <cuda_runtime.h>

#include "gamma_gpu.h"
#include "gamma_problem.h"
#include "smem_limit.h"
#include "track_step.cuh"
#include "tune.h"

namespace gb {

// One launch: the kernel (its shape in tune.h), grid, shared memory and CTAs per
// run (a cluster).
struct LaunchShape {
  int kernel = 0;
  int grid = 0;  // 0: not configured yet
  size_t smem = 0;
  int cluster = 1;
};

// CTAs per run for a CTA of `threads`: runs that leave SMs idle are spread over
// clusters of up to 8 CTAs (the portable size), as many as there are SMs for
// and cells to work on.
inline int team_size(int nsm, int nruns, int cells, int threads) {
  int c = 1;
  while (c < 8 && 2LL * c * nruns <= nsm && c * threads < cells) c *= 2;
  return c;
}

// The shape behind variant 0 on nsm SMs.  The runs of a batch differ in length
// and each runs at its CTA's pace, so a batch that does not fill the GPU wants
// more threads per run, and one that does wants small CTAs (their chunk barriers
// stall fewer warps).  Measured us per step with 128, 256, 512 threads per run
// (tubes of 1,001 to 8,191 cells; settled BM1D runs of 1,000 to 8,000 initial
// cells), clusters by team_size:
//   runs   tubes                 BM1D
//     20    341   206   137      201   177   160
//     72    646   392   256      302   236   256
//    200   1302   770   494      511   398   429
//    440   1606   927   684      728   696   718
//    900   1881  1105  1403     1516  1283  1348
//   4096 (256 to 8,192 cells)  3507  3618  4720
inline int default_shape(int nsm, int nruns, int cells) {
  const int most = nruns <= 3LL * nsm ? 512 : (nruns <= 16LL * nsm ? 256 : 128);
  int c = 1;
  while (c < 8 && 2LL * c * nruns <= nsm) c *= 2;
  int threads = 128;
  while (threads < most && c * threads < cells) threads *= 2;  // no more than the cells of a run
  return tune::shape_of(threads);
}

struct ProblemEntry {
  const char *name;
  int id;       // a fixed id (the built-in GAMMA_PROBLEM_* values), or -1
  int modules;  // gamma_problem::MODULES_*
  bool regrid;  // Hooks::REGRID
  // launch shape v of the step kernel, without or with the learned guess, for
  // nruns runs of about `cells` cells (max_cap sizes the regrid's bit words)
  cudaError_t (*configure)(int v, bool guess, int nruns, int cells, int max_cap, LaunchShape *shape);
  // gate: nullptr, or the step kernels' choice (track_step_kernel)
  cudaError_t (*launch)(bool guess, const LaunchShape &shape, cudaStream_t s, const Tracks &T, const Phys &ph,
                        int nsteps, const int *order, int nruns, int *queue, StepStats *stats, int regrid_only,
                        int max_cap, const int *gate);
  // Simu::initialise of one run on the host (prim [NQ][cap])
  int (*initial_state)(const Phys &ph, const double *par, int cap, int *ntrack, double *t, double *prim, double *x,
                       double *dx, double *xI, double *dt_loc);
};

// The registry (gamma_api.cu).  Entries register from static initialisers.
int register_problem(ProblemEntry *e);
const ProblemEntry *find_problem(int id);
int problem_id(const char *name);

template <int M>
struct ModuleCfg;
template <>
struct ModuleCfg<gamma_problem::MODULES_CARTESIAN> {
  using type = CfgCart;
};
template <>
struct ModuleCfg<gamma_problem::MODULES_SPHERICAL1D> {
  using type = CfgSph;
};
template <>
struct ModuleCfg<gamma_problem::MODULES_CARTESIAN_REL_CYL> {
  using type = CfgCyl;
};

// Shared memory of one launch: TrackStep::Smem, the regrid bit words (modules
// with a refinement criterion only), then the learned guess's weights.
template <class Hooks>
__host__ __device__ constexpr unsigned module_words_bytes(int max_cap) {
  return Hooks::REGRID ? 4u * kRegridMarks * (unsigned)regrid_words(max_cap) : 0u;
}

template <class C, class Hooks, int V, bool GUESS>
struct ModuleKernel {
  static constexpr int BS = tune::kShapes[V].threads;
  static constexpr int CPT = tune::kShapes[V].cells_per_thread;
  static constexpr int MINB = tune::min_blocks(C::MIN_BLOCKS, BS);
  static constexpr auto fn = track_step_kernel<C, Hooks, BS, GUESS, CPT, MINB>;
  static size_t smem(int max_cap) {
    size_t b = sizeof(typename TrackStep<C, Hooks, BS, GUESS, CPT>::Smem) + module_words_bytes<Hooks>(max_cap);
    if (GUESS) b = ((b + 15u) & ~size_t(15)) + sizeof(mlp::InferSmem);
    return b;
  }
  // whether a CTA's shared memory holds it with the regrid words of max_cap cells
  static bool fits(int dev, int max_cap) {
    int most = 0;
    cudaFuncAttributes a{};
    return cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) == cudaSuccess &&
           cudaFuncGetAttributes(&a, (const void *)fn) == cudaSuccess &&
           smem(max_cap) + a.sharedSizeBytes <= (size_t)most;
  }
  static cudaError_t configure(int nruns, int cells, int max_cap, LaunchShape *L) {
    L->smem = smem(max_cap);
    cudaError_t e = raise_smem_limit((const void *)fn, L->smem);
    if (e != cudaSuccess) return e;
    int dev = 0, nsm = 0, occ = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    L->kernel = V;
    L->cluster = team_size(nsm, nruns, cells, BS * CPT);
    for (; L->cluster > 1; L->cluster /= 2) {
      cudaLaunchAttribute at;
      cudaLaunchConfig_t c = config(*L, &at, L->cluster, nullptr);
      int nc = 0;
      if ((e = cudaOccupancyMaxActiveClusters(&nc, fn, &c)) != cudaSuccess) return e;
      if (nc < 1) continue;
      L->grid = L->cluster * (nruns < nc ? nruns : nc);
      return cudaSuccess;
    }
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, BS, L->smem)) != cudaSuccess) return e;
    if (occ < 1) occ = 1;
    L->grid = nruns < nsm * occ ? nruns : nsm * occ;
    return cudaSuccess;
  }
  static cudaLaunchConfig_t config(const LaunchShape &L, cudaLaunchAttribute *at, int grid, cudaStream_t s) {
    at->id = cudaLaunchAttributeClusterDimension;
    at->val.clusterDim.x = L.cluster;
    at->val.clusterDim.y = at->val.clusterDim.z = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(grid);
    c.blockDim = dim3(BS);
    c.dynamicSmemBytes = L.smem;
    c.stream = s;
    c.attrs = at;
    c.numAttrs = L.cluster > 1 ? 1 : 0;
    return c;
  }
  static cudaError_t launch(const LaunchShape &L, cudaStream_t s, const Tracks &T, const Phys &ph, int nsteps,
                            const int *order, int nruns, int *queue, StepStats *stats, int regrid_only, int max_cap,
                            const int *gate) {
    cudaLaunchAttribute at;
    const cudaLaunchConfig_t c = config(L, &at, L.grid, s);
    return cudaLaunchKernelEx(&c, fn, T, ph, nsteps, order, nruns, queue, stats, regrid_only,
                              module_words_bytes<Hooks>(max_cap), gate);
  }
};

#define GB_MODULE_SHAPES(X) X(0) X(1) X(2) X(3) X(4) X(5) X(6) X(7)
static_assert(tune::kVariants == 8, "GB_MODULE_SHAPES lists every launch shape");

template <class C, class Hooks>
bool module_fits(int v, bool guess, int dev, int max_cap) {
  switch (v) {
#define GB_CASE(k)                                                            \
  case k:                                                                     \
    return guess ? ModuleKernel<C, Hooks, k, true>::fits(dev, max_cap) \
                 : ModuleKernel<C, Hooks, k, false>::fits(dev, max_cap);
    GB_MODULE_SHAPES(GB_CASE)
#undef GB_CASE
  }
  return false;
}

template <class C, class Hooks>
cudaError_t module_configure(int v, bool guess, int nruns, int cells, int max_cap, LaunchShape *L) {
  if (v == 0) {
    int dev = 0, nsm = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    v = default_shape(nsm, nruns, cells);
    // A long track's regrid words leave a large CTA no room (512 threads of the
    // spherical step take 144 KB, 128 take 37 KB): the largest that fits.
    while (v != 0 && !module_fits<C, Hooks>(v, guess, dev, max_cap)) v = tune::shape_of(tune::kShapes[v].threads / 2);
  }
  switch (v) {
#define GB_CASE(k)                                                                       \
  case k:                                                                                \
    return guess ? ModuleKernel<C, Hooks, k, true>::configure(nruns, cells, max_cap, L)      \
                 : ModuleKernel<C, Hooks, k, false>::configure(nruns, cells, max_cap, L);
    GB_MODULE_SHAPES(GB_CASE)
#undef GB_CASE
  }
  return cudaErrorInvalidValue;
}

template <class C, class Hooks>
cudaError_t module_launch(bool guess, const LaunchShape &L, cudaStream_t s, const Tracks &T, const Phys &ph,
                          int nsteps, const int *order, int nruns, int *queue, StepStats *stats, int regrid_only,
                          int max_cap, const int *gate) {
  switch (L.kernel) {
#define GB_CASE(k)                                                                                              \
  case k:                                                                                                       \
    return guess ? ModuleKernel<C, Hooks, k, true>::launch(L, s, T, ph, nsteps, order, nruns, queue, stats,     \
                                                           regrid_only, max_cap, gate)                          \
                 : ModuleKernel<C, Hooks, k, false>::launch(L, s, T, ph, nsteps, order, nruns, queue, stats,    \
                                                            regrid_only, max_cap, gate);
    GB_MODULE_SHAPES(GB_CASE)
#undef GB_CASE
  }
  return cudaErrorInvalidValue;
}

// Simu::initialise for one run, on the host (src/simu.cpp:24-38 with
// src/Dimensions/1d.cpp:53-81, 217-246, 844-856, 931-951 and
// radiation_sph.cpp:246-260): loadParams, initialGeometry and initialValues of
// the module on the active cells, FluidState's default state (rho = p = 1)
// elsewhere, prepForRun's v2u and interface positions, radiation_initGammas,
// then the first updateGhosts with the module's userBoundaries.
template <class C, class Hooks>
int module_initial_state(const Phys &ph, const double *par, int cap, int *ntrack, double *t, double *prim, double *x,
                         double *dx, double *xI, double *dt_loc) {
  constexpr int NQ = C::NQ;
  const gamma_problem::Setup s = Hooks::load_params(par);
  const int ng = ph.ngst;
  const int n = s.ncell + 2 * ng;
  if (s.ncell < 3 || s.nmax < s.ncell) return GAMMA_ERR_INVALID;
  if (s.nmax + 2 * ng > cap) return GAMMA_ERR_CAPACITY;
  for (int i = 0; i < cap; ++i) {
    for (int q = 0; q < NQ; ++q) prim[(size_t)q * cap + i] = (q == RHO || q == PPP) ? 1. : 0.;
    x[i] = dx[i] = xI[i] = 0.;
    dt_loc[i] = DT_INF;
  }
  const int iL = ng - 1, iR = n - ng;
  const gamma_problem::HookArgs a{par, ph.gamma_ad, s.tini, 0, n, iL, iR};
  for (int i = 0; i < s.ncell; ++i) Hooks::initial_geometry(a, i, s.ncell, &x[ng + i], &dx[ng + i]);
  for (int i = 0; i < s.ncell; ++i) {
    double c[NQ];
    for (int q = 0; q < NQ; ++q) c[q] = (q == RHO || q == PPP) ? 1. : 0.;
    Hooks::initial_values(a, x[ng + i], dx[ng + i], c);
    for (int q = 0; q < NQ; ++q) prim[(size_t)q * cap + ng + i] = c[q];
  }
  // v2u (1d.cpp:931-951)
  for (int i = 0; i < n; ++i) {
    double v = 0.;
    const double vv = prim[(size_t)UU1 * cap + i];
    v += vv * vv;
    v = sqrt(v);
    const double lfac = 1. / sqrt(1. - v * v);
    prim[(size_t)UU1 * cap + i] *= lfac;
  }
  // interfaceGeomFromCellPos (1d.cpp:844-856)
  for (int i = 0; i < n - 1; ++i) xI[i] = i != iL ? x[i] + dx[i] / 2. : x[i + 1] - dx[i + 1] / 2.;
  if (C::SYNCH) {  // radiation_initGammas on every cell
    for (int i = 0; i < n; ++i) {
      const double lfac = gamma_problem::lorentz_factor(prim[(size_t)UU1 * cap + i]);
      const double rho = prim[(size_t)RHO * cap + i];
      const double lim = lfac * pow(rho, 4. / 3.);
      for (int q : {GMX, GMN}) {
        double &g = prim[(size_t)q * cap + i];
        if (g > lim / (lfac * rho) || g <= 0.) g = lim / (lfac * rho);
      }
    }
  }
  // updateGhosts (1d.cpp:217-246), then userBoundaries
  for (int i = 0; i <= iL; ++i) {
    for (int q = 0; q < NQ; ++q) prim[(size_t)q * cap + i] = prim[(size_t)q * cap + iL + 1];
    x[i] = x[iL + 1] - (iL - i + 1) * dx[iL + 1];
    dx[i] = dx[iL + 1];
  }
  for (int i = 0; i <= iL - 1; ++i) xI[i] = xI[iL + 1] - (iL - i + 1) * dx[iL + 1];
  for (int i = iR; i < n; ++i) {
    for (int q = 0; q < NQ; ++q) prim[(size_t)q * cap + i] = prim[(size_t)q * cap + iR - 1];
    x[i] = x[iR - 1] + (i - iR + 1) * dx[iR - 1];
    dx[i] = dx[iR - 1];
  }
  for (int i = iR; i < n - 1; ++i) xI[i] = xI[iR - 1] + (i - iR) * dx[iR - 1];
  for (int i = 0; i < n; ++i) {
    if (i > iL && i < iR) continue;
    double c[NQ];
    for (int q = 0; q < NQ; ++q) c[q] = prim[(size_t)q * cap + i];
    Hooks::user_boundaries(a, i, x[i], c);
    for (int q = 0; q < NQ; ++q) prim[(size_t)q * cap + i] = c[q];
  }
  *ntrack = n;
  *t = s.tini;
  return GAMMA_OK;
}

template <class Hooks, int MODULES>
ProblemEntry make_problem_entry(const char *name, int id) {
  using C = typename ModuleCfg<MODULES>::type;
  return ProblemEntry{name, id, MODULES, Hooks::REGRID, &module_configure<C, Hooks>, &module_launch<C, Hooks>,
                      &module_initial_state<C, Hooks>};
}

}  // namespace gb

// Registers module Hooks (module set MODULES) under NAME.  ID: a fixed id, or -1
// for the next free one (gamma_gpu_problem_id looks modules up by name).
#define GAMMA_PROBLEM_MODULE(NAME, HOOKS, MODULES, ID)                                               \
  namespace {                                                                                        \
  gb::ProblemEntry gb_problem_entry_ = gb::make_problem_entry<HOOKS, MODULES>(NAME, ID);            \
  const int gb_problem_registered_ = gb::register_problem(&gb_problem_entry_);                       \
  }
