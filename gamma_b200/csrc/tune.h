// Launch-shape variants of the 1D step kernel for the autotuner
// (gamma_gpu_autotune).  Variant 0 is the default: 128 threads per run, one
// cell per thread per sweep chunk, or, in a batch that does not fill the GPU
// that way, one of the larger CTAs (default_shape in problem_module.cuh).
// Variants 1.. fix the threads per CTA and the cells each thread takes per
// chunk.  In any of them a run may be spread over a cluster of CTAs (team_size
// there).  Every problem module instantiates all of them
// (problem_module.cuh).  The arithmetic of every cell is the same in all of
// them, so they give identical results; only the speed differs.
#pragma once

namespace gb {
namespace tune {

constexpr int kVariants = 8;  // variant 0 included

struct Shape {
  int threads, cells_per_thread;
};

// threads per run and cells per thread of each variant
constexpr Shape kShapes[kVariants] = {{128, 1}, {64, 1}, {256, 1}, {128, 2}, {64, 2}, {128, 4}, {512, 1}, {256, 2}};

// the variant of this many threads with one cell each (0 where there is none)
constexpr int shape_of(int threads) {
  for (int v = 0; v < kVariants; ++v)
    if (kShapes[v].threads == threads && kShapes[v].cells_per_thread == 1) return v;
  return 0;
}

// The register cap of each variant keeps the default's resident warps per SM,
// with at least two CTAs of 256 threads: a run's chunk barriers then stall
// half an SM, not all of it (the spherical step, 3 x 128 by default, would
// otherwise get one 256-thread CTA of 232 registers; with two of 128 the BM1D
// sweep runs 8.7% faster, at the same bits).
constexpr int min_blocks(int default_blocks, int threads) {
  const int b = default_blocks * 128 / threads;
  return threads == 256 && b < 2 ? 2 : (b > 0 ? b : 1);
}

}  // namespace tune
}  // namespace gb
