// Training side of the learned cons2prim guess: parameter initialisation,
// training pairs, FP32 forward/backward and Adam.  Included by one translation
// unit only (its kernels are not templates).
#pragma once

#include "mlp.cuh"
#include "tiles.h"

namespace gb {
namespace mlp {

// ---------------------------------------------------------------------------
// Parameter initialisation: uniform(-sqrt(6/(fan_in+fan_out)), +...) weights
// (Glorot), zero biases, from a counter-based hash of (seed, index).

__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
  // splitmix64 finaliser (Steele, Lea, Flood 2014)
  z += 0x9e3779b97f4a7c15ull;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}
__device__ __forceinline__ double uniform01(unsigned long long seed, unsigned long long k, int j) {
  return (double)(mix64(seed ^ mix64(8 * k + j)) >> 11) * (1.0 / 9007199254740992.0);
}

__global__ void init_kernel(float *P, unsigned long long seed) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < NPARAM; i += gridDim.x * blockDim.x) {
    float lim = 0.f;
    if (i < OFF_B1) lim = sqrtf(6.f / (3 + H));
    else if (i >= OFF_W2 && i < OFF_B2) lim = sqrtf(6.f / (H + H));
    else if (i >= OFF_W3 && i < OFF_B3) lim = sqrtf(6.f / (H + 2));
    P[i] = lim * (float)(2. * uniform01(seed, i, 0) - 1.);
  }
}

// ---------------------------------------------------------------------------
// Training pairs from primitive states [NQ rows][n] (the first n pairs) and
// uniform draws (the next nu): ln lfac ~ U(0, ln 1e3), log10 p/rho ~ U(-10, 3),
// log10 rho ~ U(-6, 6), direction of motion +-1 with equal probability.
template <class Cfg>
__global__ void pairs_kernel(Phys ph, const double *prim, long long n, long long nu, unsigned long long seed,
                             float *x, float *y) {
  constexpr int NQ = Cfg::NQ;
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n + nu;
       k += (long long)gridDim.x * blockDim.x) {
    double pr[NQ], cs[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) pr[q] = 0.;
    if (k < n) {
#pragma unroll
      for (int q = 0; q < NQ; ++q) pr[q] = prim[q * n + k];
      pr[UU2] = 0.;
    } else {
      const unsigned long long kk = k - n;
      const double lg = exp(uniform01(seed, kk, 0) * log(1e3));
      const double pr_rho = pow(10., -10. + 13. * uniform01(seed, kk, 1));
      const double rho = pow(10., -6. + 12. * uniform01(seed, kk, 2));
      const double sgn = uniform01(seed, kk, 3) < 0.5 ? -1. : 1.;
      pr[RHO] = rho;
      pr[PPP] = rho * pr_rho;
      pr[UU1] = sgn * sqrt(fmax(lg * lg - 1., 0.));
      pr[TR1] = 1.;
    }
    prim2cons<Cfg>(ph, pr, cs);
    float f[3], t[2];
    features(cs[DEN], cs[TAU], cs[SS1], f);
    targets(cs[DEN], pr[PPP], lfac_of(pr[UU1]), t);
    x[3 * k + 0] = f[0];
    x[3 * k + 1] = f[1];
    x[3 * k + 2] = f[2];
    y[2 * k + 0] = t[0];
    y[2 * k + 1] = t[1];
  }
}

// ---------------------------------------------------------------------------
// Training: loss = sum over a mini-batch and both outputs of (out - y)^2 / (2 m).
// Sample j of the mini-batch is pair (perm_mul * (start + j) + perm_add) mod
// n_total, a bijection when gcd(perm_mul, n_total) = 1 (the host checks).
//
// A block takes tiles of 64 samples through the forward and backward pass as
// 64 x 64 x 64 products in FP32 from shared memory, 4 x 4 outputs per thread:
// z2 = h1 W2^T, dL/dh1 = d2 W2 and dL/dW2 = d2^T h1.  Thread (tx, ty) of 16 x 16
// holds rows ty + 16 i and columns tx + 16 j; every operand is kept with the
// summed index last (so W2, h1 and d2 also transposed), rows padded to 68 floats:
// a quarter warp's 16-byte loads of consecutive rows then touch all 32 banks.
// The block's gradient goes to its own row of partial sums, which adam_kernel
// adds up in a fixed order, so that training repeats bit for bit.  The loss, the
// mean of up to millions of squares, is summed in 64 bits from a thread's eight
// of a tile on.
// A mini-batch of 8,192 is 128 tiles, one per SM; the products are 0.8 MFLOP of
// FMA per tile, ~3 us of the SM's FP32 rate, which bounds it (a sample per thread
// with its activations in local memory took 128 us per mini-batch; now 11 us).

constexpr int TILE = 64;              // samples per tile
constexpr int TRAIN_THREADS = 256;
constexpr int LD = H + 4;             // padded row
constexpr int NPART = NPARAM + 2;     // a block's partial sums: gradient, then the squared errors (a double)
static_assert(NPARAM % 2 == 0, "every row's double is 8-byte aligned");

struct TrainSmem {
  float W2[H][LD], W2T[H][LD];        // [o][i] and [i][o]
  float h1[TILE][LD], h1T[H][LD];     // [sample][unit] and [unit][sample]
  float d2[TILE][LD], d2T[H][LD];     // dL/dz2, likewise
  float x[TILE][4], y[TILE][2];
  float W1[H][3], b1[H], b2[H], W3[2][H], b3[2];
  float red[TRAIN_THREADS / 32][28][16];
  float red3[TRAIN_THREADS / 32][2];
  double redl[TRAIN_THREADS / 32];
};

// The kernels of a training run follow one another in a stream, each launched
// while the one before still runs (programmatic stream serialization): a kernel
// lets the next one be launched as it starts, does what needs no results of the
// one before, and waits for those here.
__device__ __forceinline__ void launch_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// acc[i][j] += sum_k A[ty + 16 i][k] B[tx + 16 j][k]
__device__ __forceinline__ void tile_product(const float (*A)[LD], const float (*B)[LD], int tx, int ty,
                                             float acc[4][4]) {
#pragma unroll 4
  for (int k = 0; k < H; k += 4) {
    float4 a[4], b[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      a[i] = *reinterpret_cast<const float4 *>(&A[ty + 16 * i][k]);
      b[i] = *reinterpret_cast<const float4 *>(&B[tx + 16 * i][k]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        acc[i][j] = fmaf(a[i].x, b[j].x, acc[i][j]);
        acc[i][j] = fmaf(a[i].y, b[j].y, acc[i][j]);
        acc[i][j] = fmaf(a[i].z, b[j].z, acc[i][j]);
        acc[i][j] = fmaf(a[i].w, b[j].w, acc[i][j]);
      }
  }
}

// part != nullptr: the block's sums go to part[blockIdx.x][NPART]; else they are
// added to grad and loss (zeroed by the caller).
__global__ void __launch_bounds__(TRAIN_THREADS, 1)
    grad_kernel(const float *Pg, const float *x, const float *y, long long n_total, long long perm_mul,
                long long perm_add, long long start, int m, float *part, float *grad, float *loss) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  TrainSmem &sm = *reinterpret_cast<TrainSmem *>(smem_raw);
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  launch_next();
  // sample s of the block's tile at base: its pair (zeros past the mini-batch)
  auto load_pair = [&](long long base, int s) {
    const long long j = base + s;
    float xi[3] = {0.f, 0.f, 0.f}, yi[2] = {0.f, 0.f};
    if (j < m) {
      const long long k = (long long)(((unsigned long long)perm_mul * (unsigned long long)(start + j) +
                                       (unsigned long long)perm_add) % (unsigned long long)n_total);
#pragma unroll
      for (int c = 0; c < 3; ++c) xi[c] = x[3 * k + c];
      yi[0] = y[2 * k];
      yi[1] = y[2 * k + 1];
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) sm.x[s][c] = xi[c];
    sm.y[s][0] = yi[0];
    sm.y[s][1] = yi[1];
  };
  Tiles tile(m, TILE, blockIdx.x, gridDim.x);
  if (tid < TILE) load_pair(tile.base, tid);
  wait_previous();  // the parameters
#pragma unroll
  for (int k = tid; k < H * H; k += TRAIN_THREADS) {
    const float w = Pg[OFF_W2 + k];
    sm.W2[k / H][k % H] = w;
    sm.W2T[k % H][k / H] = w;
  }
  for (int k = tid; k < 3 * H; k += TRAIN_THREADS) sm.W1[k / 3][k % 3] = Pg[OFF_W1 + k];
  if (tid < H) {
    sm.b1[tid] = Pg[OFF_B1 + tid];
    sm.b2[tid] = Pg[OFF_B2 + tid];
  }
  if (tid < 2 * H) sm.W3[tid / H][tid % H] = Pg[OFF_W3 + tid];
  if (tid < 2) sm.b3[tid] = Pg[OFF_B3 + tid];

  // gradients of this thread: W2[ty + 16 i][tx + 16 j]; summed over its rows'
  // samples, of unit tx + 16 j: b1, b2, W1[.][3], W3[2][.]; b3, and the loss
  float gW2[4][4] = {}, gb1[4] = {}, gb2[4] = {}, gW1[4][3] = {}, gW3[2][4] = {}, gb3[2] = {0.f, 0.f};
  double lsum = 0.;
  const float inv_m = 1.f / (float)m;

  for (bool first = true; tile.more(); tile.next(), first = false) {
    if (!first) {
      __syncthreads();  // the tile before is done with
      if (tid < TILE) load_pair(tile.base, tid);
    }
    __syncthreads();
    float ds1[4][4], z2[4][4];  // silu'(z1), z2
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int s = ty + 16 * i, o = tx + 16 * j;
        const float z = sm.b1[o] + sm.W1[o][0] * sm.x[s][0] + sm.W1[o][1] * sm.x[s][1] + sm.W1[o][2] * sm.x[s][2];
        const float sg = 1.f / (1.f + __expf(-z)), h = z * sg;
        ds1[i][j] = sg + h * (1.f - sg);
        sm.h1[s][o] = h;
        sm.h1T[o][s] = h;
        z2[i][j] = sm.b2[o];
      }
    __syncthreads();
    tile_product(sm.h1, sm.W2, tx, ty, z2);
    // output layer: sums over the 16 threads of a row
    float out[4][2], sg2[4][4], sq = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      out[i][0] = out[i][1] = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        sg2[i][j] = 1.f / (1.f + __expf(-z2[i][j]));
        z2[i][j] *= sg2[i][j];  // h2 from here on
        out[i][0] += sm.W3[0][tx + 16 * j] * z2[i][j];
        out[i][1] += sm.W3[1][tx + 16 * j] * z2[i][j];
      }
#pragma unroll
      for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int d = 8; d > 0; d >>= 1) out[i][q] += __shfl_xor_sync(0xffffffffu, out[i][q], d);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int s = ty + 16 * i;
      float dout[2];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const float e = tile.base + s < m ? out[i][q] + sm.b3[q] - sm.y[s][q] : 0.f;
        dout[q] = e * inv_m;
        if (tx == 0) {
          sq += e * e;
          gb3[q] += dout[q];
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int o = tx + 16 * j;
        const float h2 = z2[i][j];
        gW3[0][j] += dout[0] * h2;
        gW3[1][j] += dout[1] * h2;
        // dL/dz2 = (W3^T dout) * silu'(z2)
        const float d =
            (sm.W3[0][o] * dout[0] + sm.W3[1][o] * dout[1]) * (sg2[i][j] + h2 * (1.f - sg2[i][j]));
        gb2[j] += d;
        sm.d2[s][o] = d;
        sm.d2T[o][s] = d;
      }
    }
    lsum += sq;
    __syncthreads();
    tile_product(sm.d2T, sm.h1T, tx, ty, gW2);
    // dL/dz1 = (W2^T dL/dz2) * silu'(z1)
    float d1[4][4] = {};
    tile_product(sm.d2, sm.W2T, tx, ty, d1);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float d = d1[i][j] * ds1[i][j];
        gb1[j] += d;
#pragma unroll
        for (int c = 0; c < 3; ++c) gW1[j][c] += d * sm.x[ty + 16 * i][c];
      }
  }
  // sums over the threads of a unit: two rows of a warp, then the warps
  float v[28];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    v[j] = gb1[j];
    v[4 + j] = gb2[j];
    v[8 + j] = gW3[0][j];
    v[12 + j] = gW3[1][j];
#pragma unroll
    for (int c = 0; c < 3; ++c) v[16 + 3 * j + c] = gW1[j][c];
  }
#pragma unroll
  for (int k = 0; k < 28; ++k) {
    v[k] += __shfl_xor_sync(0xffffffffu, v[k], 16);
    if ((tid & 31) < 16) sm.red[tid >> 5][k][tx] = v[k];
  }
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    gb3[k] += __shfl_xor_sync(0xffffffffu, gb3[k], 16);
    if ((tid & 31) == 0) sm.red3[tid >> 5][k] = gb3[k];
  }
  lsum += __shfl_xor_sync(0xffffffffu, lsum, 16);
  if ((tid & 31) == 0) sm.redl[tid >> 5] = lsum;
  __syncthreads();
  float *row = part ? part + (size_t)blockIdx.x * NPART : nullptr;
  auto give = [&](int g, float s) {
    if (row) row[g] = s;
    else atomicAdd(&grad[g], s);
  };
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) give(OFF_W2 + (ty + 16 * i) * H + tx + 16 * j, gW2[i][j]);
  for (int k = tid; k < 28 * 16; k += TRAIN_THREADS) {
    const int q = k / 16, t = k % 16;
    float s = 0.f;
#pragma unroll
    for (int u = 0; u < TRAIN_THREADS / 32; ++u) s += sm.red[u][q][t];
    int g;
    if (q < 4) g = OFF_B1 + t + 16 * q;
    else if (q < 8) g = OFF_B2 + t + 16 * (q - 4);
    else if (q < 16) g = OFF_W3 + (q >= 12 ? H : 0) + t + 16 * (q & 3);
    else g = OFF_W1 + 3 * (t + 16 * ((q - 16) / 3)) + (q - 16) % 3;
    give(g, s);
  }
  if (tid < 2) {
    float s = 0.f;
#pragma unroll
    for (int u = 0; u < TRAIN_THREADS / 32; ++u) s += sm.red3[u][tid];
    give(OFF_B3 + tid, s);
  }
  if (tid == 2) {
    double s = 0.;
#pragma unroll
    for (int u = 0; u < TRAIN_THREADS / 32; ++u) s += sm.redl[u];
    if (row) *reinterpret_cast<double *>(row + NPARAM) = s;
    else if (loss) atomicAdd(loss, (float)(0.5 * s / (double)m));
  }
}

// The gradient from nb blocks' partial sums, then Adam (Kingma & Ba 2015); the
// mini-batch's loss, inv_2m = 1 / (2 m) times its squared errors, is added to
// *loss.  c1 = 1 - b1, c2 = 1 - b2 and the bias corrections bc1 = 1 - b1^t,
// bc2 = 1 - b2^t come from the host, each rounded once from 64 bits: formed in 32
// bits, 1 - 0.999 is off by 1.3e-5 of itself and the products b2^t by as much in
// the first steps, the same way in every training.
// The moments move by c (g - m) for the same reason: b2 itself, in 32 bits, is
// 1.3e-8 off, 1.3e-5 of its distance from 1.  (The epochs' losses against 64 bits,
// 700 to 150,007 pairs in batches of 64 to 150,007: off by 2e-7 to 1.4e-6 with the
// constants formed in 32 bits, by up to 1.3e-7 so.)
// Eight threads per parameter, one of every eight blocks' sums each; the last block
// takes the loss (in a parameter's block, its loads would follow theirs: 3% of an
// epoch's time).
constexpr int ADAM_PARAMS = 32;  // parameters per block of 256 threads
constexpr int ADAM_BLOCKS = (NPARAM + ADAM_PARAMS - 1) / ADAM_PARAMS + 1;
__global__ void __launch_bounds__(256) adam_kernel(float *P, const float *part, int nb, float *m, float *v, float lr,
                                                   float c1, float c2, float eps, float bc1, float bc2,
                                                   double inv_2m, double *loss) {
  __shared__ float red[8][ADAM_PARAMS];
  __shared__ double redl[8];
  const int t = threadIdx.x & 31, k = threadIdx.x >> 5;
  const int i = blockIdx.x * ADAM_PARAMS + t;
  launch_next();
  wait_previous();
  if (blockIdx.x == ADAM_BLOCKS - 1) {
    double s = 0.;
    for (int b = threadIdx.x; b < nb; b += 256)
      s += *reinterpret_cast<const double *>(part + (size_t)b * NPART + NPARAM);
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
    if (t == 0) redl[k] = s;
    __syncthreads();
    if (threadIdx.x != 0) return;
#pragma unroll
    for (int u = 1; u < 8; ++u) s += redl[u];
    *loss += s * inv_2m;
    return;
  }
  float s = 0.f;
  if (i < NPARAM) {
#pragma unroll 8
    for (int b = k; b < nb; b += 8) s += part[(size_t)b * NPART + i];
  }
  red[k][t] = s;
  __syncthreads();
  if (k != 0 || i >= NPARAM) return;
  float g = red[0][t];
#pragma unroll
  for (int u = 1; u < 8; ++u) g += red[u][t];
  const float mi = m[i] + c1 * (g - m[i]);
  const float vi = v[i] + c2 * (g * g - v[i]);
  m[i] = mi;
  v[i] = vi;
  P[i] -= lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
}

// FP32 forward of n samples (x [n][3] -> out [n][2])
__global__ void forward_kernel(const float *P, const float *x, long long n, float *out) {
  __shared__ float sP[NPARAM];
  for (int i = threadIdx.x; i < NPARAM; i += blockDim.x) sP[i] = P[i];
  __syncthreads();
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
    const float xi[3] = {x[3 * k], x[3 * k + 1], x[3 * k + 2]};
    float o[2];
    forward(sP, xi, o);
    out[2 * k] = o[0];
    out[2 * k + 1] = o[1];
  }
}

}  // namespace mlp
}  // namespace gb
