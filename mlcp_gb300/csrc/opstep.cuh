// One mode step of the ALS-fitted Hamiltonian applications from its normal
// equations and right-hand side on, for a CTA of 512 threads that holds one
// vector: shared by the one-CTA form (opals.cu) and the grid form
// (opals_grid.cu), so that both run the same operations in the same order.
#pragma once

#include "dword.cuh"
#include "dwsolve.cuh"

namespace mlcp {

namespace {

constexpr int kStepThreads = 512;
constexpr int kSumThreads = 256;  // threads (the first ones) whose partial sums make a sum's order
constexpr int kSumWarps = kSumThreads / 32;

struct StepSmem {
  dw* X;      // [R][npmax] solution (column-major, ld R)
  dw* b0;     // [R][npmax] right-hand side
  dw* res;    // [R][npmax] refinement residual
  dw* BB;     // [R][R] normal equations
  float* gi;  // [R][R] FP32 inverse of BB (its place is twice that)
  dw* cf;     // [R] weights of F
  dw* red;    // [kSumWarps] reduction scratch
  dw* dinv;   // [R] LDL^T reciprocal pivots
  dw* u;      // [R] LDL^T scratch column
  dw* misc;   // [2] penalty, norm
  float* rred;  // [4] refinement scratch
  float* prow;  // [2][72] pivot rows of the inverse
  dwsolve::ColScratch cs;
  int* flags;  // [4] [1] non-positive pivot seen, [2] inverse usable, [3] solved
};

// Carves the shared memory (null base: sizes only); returns the bytes.
__host__ __device__ inline size_t step_carve(StepSmem& s, unsigned char* base, int R, int npm) {
  size_t o = 0;
  auto take = [&](size_t bytes) -> unsigned char* {
    const size_t r = o;
    o += (bytes + 15) / 16 * 16;
    return base ? base + r : nullptr;
  };
  const size_t Rn = (size_t)R * npm, RR = (size_t)R * R;
  s.X = (dw*)take(sizeof(dw) * Rn);
  s.b0 = (dw*)take(sizeof(dw) * Rn);
  s.res = (dw*)take(sizeof(dw) * Rn);
  s.BB = (dw*)take(sizeof(dw) * RR);
  s.gi = (float*)take(sizeof(float) * 2 * RR);
  s.cf = (dw*)take(sizeof(dw) * R);
  s.red = (dw*)take(sizeof(dw) * kSumWarps);
  s.dinv = (dw*)take(sizeof(dw) * R);
  s.u = (dw*)take(sizeof(dw) * R);
  s.misc = (dw*)take(sizeof(dw) * 2);
  s.rred = (float*)take(sizeof(float) * 4);
  s.prow = (float*)take(sizeof(float) * 2 * 72);
  s.cs.conv = (float*)take(sizeof(float) * 64);
  s.cs.rmax = (float*)take(sizeof(float) * 16 * 32);
  s.cs.rsum = (dw*)take(sizeof(dw) * 16 * 32);
  s.flags = (int*)take(sizeof(int) * 4);
  return o;
}

// Entry (i, i2) of prod_{d != j} G_d + pen I (G: the Grams of F, [D][R][R]);
// rows and columns beyond the vector's rank rv are the identity.
__device__ __forceinline__ dw normal_equation(const dw* G, int D, int j, int i, int i2, int R, int rv, dw pen) {
  const int RR = R * R, e = i + i2 * R;
  dw bb = dw_make(1.f);
  for (int d = 0; d < D; ++d)
    if (d != j) bb = dw_mul(bb, G[(size_t)d * RR + e]);
  if (i == i2) bb = dw_add(bb, pen);
  if (i >= rv || i2 >= rv) bb = dw_make(i == i2 ? 1.f : 0.f);
  return bb;
}

// X = BB^-1 b0 with unit rows, their norms to cf; ends with a block barrier.
// (Norms by 128 threads: their partial sums depend on how many share a row.)
__device__ inline void step_solve(const StepSmem& s, int R, int nj) {
  bool gj_ok = s.flags[2] != 0;
  const float* inv = s.gi;
  bool solved = false;
  const int nsw = dwsolve::solve_cols_warps(R, nj);
  if (gj_ok && R <= 32 && nj <= 16 && nsw <= kSumWarps) {
    if (threadIdx.x < nsw * 32) {
      const bool ok = dwsolve::solve_cols_any(s.BB, R, s.b0, s.X, nj, inv, s.cf, s.cs);
      if (threadIdx.x == 0) s.flags[3] = ok;
    }
    __syncthreads();
    solved = s.flags[3] != 0;
    gj_ok = false;  // not converged: straight to the LDL^T
  }
  if (!solved) {
    if (!(gj_ok && dwsolve::refine_any<kStepThreads>(s.BB, R, s.b0, s.X, nj, inv, s.res, s.rred))) {
      if (threadIdx.x < dwsolve::kSolverThreads) {
        for (int e = threadIdx.x; e < R * nj; e += dwsolve::kSolverThreads) s.X[e] = s.b0[e];
        const int bad = dwsolve::dw_ldlt(s.BB, R, s.dinv, s.u);
        dwsolve::dw_ldlt_solve(s.BB, R, s.dinv, s.X, nj);
        if (threadIdx.x == 0 && bad) s.flags[1] = 1;
      }
      __syncthreads();
    }
    if (threadIdx.x < dwsolve::kSolverThreads) dwsolve::dw_normalise_rows(s.X, R, nj, s.cf);
    __syncthreads();
  }
}

// In-place POW applies (H - E) once per mode step, so within a sweep the
// weights grow (or shrink) by about ||H - E|| per step: a 12-mode quartic
// force field in cm^-1 passes the FP32 exponent range after nine steps, and a
// 400-term random Hamiltonian over 24 modes overflows the squared row norms
// (weights above 1.8e19).  The end-of-sweep renormalisation divides out any
// common factor, so after each step the weights are multiplied by the power
// of two that brings the largest into [0.5, 1): exact, and the solve is linear
// in the weights, so the sweep's result is unchanged.  Warp 0 only; each lane
// rescales the entries it read.
__device__ inline void rescale_weights_warp(dw* cf, int R) {
  float m = 0.f;
  for (int i = threadIdx.x; i < R; i += 32) m = fmaxf(m, fabsf(cf[i].hi));
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (!(m > 0.f && m <= 3.4028235e38f)) return;  // zero, or non-finite (reported by the next solve)
  int e;
  frexpf(m, &e);
  for (int i = threadIdx.x; i < R; i += 32) cf[i] = dw_make(ldexpf(cf[i].hi, -e), ldexpf(cf[i].lo, -e));
}

// The new weights (warp 0; no other thread reads them before the next
// barrier): none beyond the vector's rank, rescaled in POW, FP64 to fc.
__device__ inline void step_weights(const StepSmem& s, int R, int rv, bool pow_mode, double* fc) {
  if (threadIdx.x >= 32) return;
  for (int i = rv + threadIdx.x; i < R; i += 32) s.cf[i] = dw_make(0.f);
  __syncwarp();
  if (pow_mode) rescale_weights_warp(s.cf, R);
  for (int i = threadIdx.x; i < R; i += 32) fc[i] = dw_to_double(s.cf[i]);
}

// The new factor: FP64 (row stride nD), double-word (row stride ldf), and its Gram.
__device__ inline void step_factor(const StepSmem& s, int R, int nj, double* fb, int nD, dw* f, int ldf, dw* G) {
  for (int e = threadIdx.x; e < R * nj; e += kStepThreads) {
    const int i = e / nj, m = e % nj;
    const dw x = s.X[i + m * R];
    fb[(size_t)i * nD + m] = dw_to_double(x);
    f[(size_t)i * ldf + m] = x;
  }
  for (int e = threadIdx.x; e < R * R; e += kStepThreads) {
    const int i = e % R, i2 = e / R;
    if (i > i2) continue;
    dw_acc acc = acc_zero();
    for (int m = 0; m < nj; ++m) acc_fma(acc, s.X[i + m * R], s.X[i2 + m * R]);
    const dw g = acc_value(acc);
    G[i + i2 * R] = g;
    G[i2 + i * R] = g;
  }
}

// Sum over the first kSumThreads threads; thread 0 gets the result (fixed order).
__device__ inline dw step_block_sum(dw v, dw* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int o = 16; o > 0; o >>= 1) v = dw_add(v, dwsolve::dw_shfl_xor(v, o));
  __syncthreads();
  if (lane == 0 && warp < kSumWarps) red[warp] = v;
  __syncthreads();
  dw s = dw_make(0.f);
  if (threadIdx.x == 0)
    for (int w = 0; w < kSumWarps; ++w) s = dw_add(s, red[w]);
  return s;
}

// Weight renormalisation after a POW sweep (src/intertw_mvp.cu:491-494).
__device__ inline void step_renormalise(const StepSmem& s, int R, int D, const dw* G, double* fc) {
  dw part = dw_make(0.f);
  for (int e = threadIdx.x; e < R * R && threadIdx.x < kSumThreads; e += kSumThreads) {
    dw prod = dw_mul(s.cf[e % R], s.cf[e / R]);
    for (int d = 0; d < D; ++d) prod = dw_mul(prod, G[(size_t)d * R * R + e]);
    part = dw_add(part, prod);
  }
  const dw tot = step_block_sum(part, s.red);
  if (threadIdx.x == 0) s.misc[1] = dw_sqrt(dw_abs(tot));
  __syncthreads();
  const dw q = s.misc[1];
  for (int i = threadIdx.x; i < R; i += kStepThreads) {
    s.cf[i] = dw_div(s.cf[i], q);
    fc[i] = dw_to_double(s.cf[i]);
  }
  __syncthreads();
}

}  // namespace

}  // namespace mlcp
