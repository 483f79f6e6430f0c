// Vector updates of the intertwined cycle over the whole GPU (larger blocks; upd.cu
// has the form for smaller ones and the choice between them).
//
// Reference: VectorUpdates / UPDATES_ALS (src/intertw_lcv.cu:209-304) with
// lcv_build_linear_system(gs = false) (:75-127).  Every vector i of the block
// is replaced by the rank-R ALS fit, started from Q_i itself, of the linear
// combination sum_k U(k,i) Q_k of the block's old vectors (U: the
// eigenvectors of the Rayleigh-Ritz problem), nals sweeps over the modes,
// then its weights are divided by its norm.  Mode step k:
//   b(i',n)   = sum_{l,r} U(l,i) c_{l,r} Q_{l,r}^k(n) prod_{d!=k} <Q_{l,r}^d, F_i'^d>
//   BB(i',i") = prod_{d!=k} <F_i'^d, F_i"^d> + pen delta,  pen = 1e-10 max c(Q_i)
//   F^k = rows of BB^-1 b, normalised (the norms become the weights).
// The penalty is the reference's FP64-build rule (src/als.cu:248-267): a
// nearly converged block makes these normal equations ill-conditioned up to
// the penalty, so b is formed in double-word arithmetic (about 48 bits), as
// are the Grams and the solve; FP32 right-hand sides are not accurate enough
// for that rule.
//
// GB300 layout: the vectors are fitted independently, so a mode step of all of
// them is three launches over the whole GPU:
//   upd_rhs_kernel      the right-hand sides: a CTA per vector, rows i' and range
//                       of the B R block terms lr; the products over d != k of 32
//                       terms at a time go through shared memory into the
//                       contraction with their mode-k factors (12-16 sums a thread);
//   upd_solve_kernel    a CTA per vector: the ranges summed in order, the solve, the
//                       new factor and its Gram (opstep.cuh);
//   upd_overlap_kernel  the overlaps <Q_lr^k, F_i'^k> of every block term with every
//                       vector's new factor: one matrix product of the two factor lists.
// The block's factors are converted once to a double-word, mode-major copy (the
// mode-k slice of all B R terms is one contiguous run); since F starts from Q, the
// first overlaps are that copy's with itself.
//
// What bounds it: the compensated multiply-add (13 FP32 instructions), 2 B^2 R^2 n of them per
// mode step, and reading the overlaps of the other modes once
// per step (72 MB each for 100 vectors of rank 30).  100 such vectors on a 6 x 48 node, one sweep, take
// 4.2 ms (70 ms with a CTA per vector, operands through L2); two sweeps of 40 of rank 16 on
// 3 x 30 take 0.33 ms (0.70 ms with a cluster of three CTAs per vector).  A step of small
// blocks is its three launches and the solve, 20 us or more.
#include <algorithm>

#include "common.cuh"
#include "dword.cuh"
#include "dwsolve.cuh"
#include "intertwine.cuh"
#include "opstep.cuh"

namespace mlcp {

namespace {

constexpr int kRhsThreads = 128;
constexpr int kChunk = 32;     // block terms of one stage of the right-hand side
constexpr int kTile = 64;      // rows and columns of an overlap tile
constexpr int kOvThreads = 256;
constexpr int kRhsCtas = 608;  // CTAs the right-hand side is split into: four for every SM

// Scratch (dw).
struct UpdScratch {
  dw *gram;  // [D][B R][B R]: <Q_lr^d, F_i'^d> at row i R + i', column lr
  dw *fg;    // [B][D][R R] Grams of F
  dw *w;     // [B][B R] target weights U(l,i) c_lr
  dw *fk;    // [B R][n_k] the mode's new factors
  dw *part;  // [ranges][B][R npmax] parts of the right-hand sides (i + m R)
  dw *pen;   // [B]
};
// Most ranges times vectors of a right-hand side.
__host__ __device__ inline size_t upd_parts(int B) { return (size_t)kRhsCtas + B; }
__host__ __device__ inline size_t upd_scratch(int B, int R, int D, int npm, dw* base, UpdScratch* s) {
  size_t o = 0;
  auto take = [&](size_t n) -> dw* {
    dw* r = base ? base + o : nullptr;
    o += (n + 1) / 2 * 2;
    return r;
  };
  const size_t BR = (size_t)B * R;
  s->gram = take((size_t)D * BR * BR);
  s->fg = take((size_t)B * D * R * R);
  s->w = take(BR * B);
  s->fk = take(BR * npm);
  s->part = take(upd_parts(B) * R * npm);
  s->pen = take(B);
  return o;
}

// Target weights and penalties.
__global__ void upd_weights_kernel(UpdParams p) {
  const int BR = p.B * p.R;
  UpdScratch s;
  upd_scratch(p.B, p.R, p.D, p.npmax, p.work, &s);
  const long long nw = (long long)BR * p.B;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < nw + p.B;
       e += (long long)gridDim.x * blockDim.x) {
    if (e < nw) {
      const int i = (int)(e / BR), lr = (int)(e - (long long)i * BR);
      s.w[e] = dw_from_double(p.U[lr / p.R + (size_t)i * p.B] * p.qc[lr]);
    } else {
      const int i = (int)(e - nw);
      const double* c = p.qc + (size_t)i * p.R;
      double pen = c[0];
      for (int r = 1; r < p.R; ++r) pen = c[r] > pen ? c[r] : pen;
      s.pen[i] = dw_from_double(pen * p.pen_factor);
    }
  }
}

// Overlaps of mode d0 + blockIdx.z: a 64 x 64 tile of F's terms (rows; the block's own
// with `first`, when the Grams of F are its diagonal blocks) and the block's.  Both
// operands whole in shared memory, transposed; 16 sums a thread.
__global__ void __launch_bounds__(kOvThreads) upd_overlap_kernel(UpdParams p, int d0, int first) {
  constexpr int ld = kTile + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  UpdScratch s;
  upd_scratch(p.B, p.R, p.D, p.npmax, p.work, &s);
  const int d = d0 + blockIdx.z, n = p.nbas[d], R = p.R, BR = p.B * R, c0 = blockIdx.x * kTile, r0 = blockIdx.y * kTile;
  dw* fs = reinterpret_cast<dw*>(smem_raw);
  dw* qs = fs + (size_t)n * ld;
  const dw* q = p.qdw + (size_t)p.off[d] * BR;
  const dw* f = first ? q : s.fk;
  for (int e = threadIdx.x; e < kTile * n; e += kOvThreads) {
    const int t = e / n, m = e - t * n;
    fs[m * ld + t] = r0 + t < BR ? f[(size_t)r0 * n + e] : dw_make(0.f);
    qs[m * ld + t] = c0 + t < BR ? q[(size_t)c0 * n + e] : dw_make(0.f);
  }
  __syncthreads();
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  dw_acc acc[4][4];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[a][b] = acc_zero();
  for (int m = 0; m < n; ++m) {
    dw y[4];
#pragma unroll
    for (int b = 0; b < 4; ++b) y[b] = qs[m * ld + tx + 16 * b];
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const dw x = fs[m * ld + ty + 16 * a];
#pragma unroll
      for (int b = 0; b < 4; ++b) acc_fma(acc[a][b], x, y[b]);
    }
  }
  dw* G = s.gram + (size_t)d * BR * BR;
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int r = r0 + ty + 16 * a, c = c0 + tx + 16 * b;
      if (r >= BR || c >= BR) continue;
      const dw v = acc_value(acc[a][b]);
      G[(size_t)r * BR + c] = v;
      if (first && r / R == c / R) s.fg[((size_t)(r / R) * p.D + d) * R * R + r % R + c % R * R] = v;
    }
}

// Right-hand side of mode k: vector blockIdx.z, rows 8 A blockIdx.y .., block terms of range
// blockIdx.x (`per` of them); all n_k <= 16 NC columns.
template <int A, int NC>
__global__ void __launch_bounds__(kRhsThreads) upd_rhs_kernel(UpdParams p, int k, int per) {
  constexpr int TR = 8 * A, ldw = TR + 1, NP = kChunk * TR / kRhsThreads;  // NP products a thread
  __shared__ dw ws[kChunk * ldw];
  __shared__ dw zs[kChunk * 16 * NC];
  UpdScratch s;
  upd_scratch(p.B, p.R, p.D, p.npmax, p.work, &s);
  const int R = p.R, D = p.D, BR = p.B * R, n = p.nbas[k], i = blockIdx.z, i0 = blockIdx.y * TR;
  const int lr1 = min(BR, (int)(blockIdx.x + 1) * per);
  const int lane = threadIdx.x % 32, wq = threadIdx.x / 32, tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  const dw* q = p.qdw + (size_t)p.off[k] * BR;
  const dw* w = s.w + (size_t)i * BR;
  const dw* g = s.gram + ((size_t)i * R + i0 + wq) * BR + lane;
  dw_acc acc[A][NC];
#pragma unroll
  for (int a = 0; a < A; ++a)
#pragma unroll
    for (int b = 0; b < NC; ++b) acc[a][b] = acc_zero();
  for (int c0 = blockIdx.x * per; c0 < lr1; c0 += kChunk) {
    const int cn = min(kChunk, lr1 - c0);
    __syncthreads();
    for (int e = threadIdx.x; e < cn * n; e += kRhsThreads)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(zs + e)),
                   "l"(q + (size_t)c0 * n + e)
                   : "memory");
    {
      const bool term = lane < cn;
      const dw w0 = term ? w[c0 + lane] : dw_make(0.f);
      dw pr[NP];
#pragma unroll
      for (int u = 0; u < NP; ++u) pr[u] = term && i0 + wq + 4 * u < R ? w0 : dw_make(0.f);
      for (int d = 0; d < D; ++d) {
        if (d == k) continue;
        const dw* gd = g + (size_t)d * BR * BR + c0;
        dw v[NP];
#pragma unroll
        for (int u = 0; u < NP; ++u)
          v[u] = term && i0 + wq + 4 * u < R ? gd[(size_t)(4 * u) * BR] : dw_make(0.f);
#pragma unroll
        for (int u = 0; u < NP; ++u) pr[u] = dw_mul(pr[u], v[u]);
      }
#pragma unroll
      for (int u = 0; u < NP; ++u) ws[lane * ldw + wq + 4 * u] = pr[u];
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    for (int c = 0; c < cn; ++c) {
      dw z[NC];
#pragma unroll
      for (int b = 0; b < NC; ++b) z[b] = zs[c * n + tx + 16 * b];
#pragma unroll
      for (int a = 0; a < A; ++a) {
        const dw x = ws[c * ldw + ty + 8 * a];
#pragma unroll
        for (int b = 0; b < NC; ++b) acc_fma(acc[a][b], x, z[b]);
      }
    }
  }
  dw* part = s.part + ((size_t)blockIdx.x * p.B + i) * R * p.npmax;
#pragma unroll
  for (int a = 0; a < A; ++a)
#pragma unroll
    for (int b = 0; b < NC; ++b) {
      const int ip = i0 + ty + 8 * a, m = tx + 16 * b;
      if (ip < R && m < n) part[ip + m * R] = acc_value(acc[a][b]);
    }
}

// The solve of mode k for vector blockIdx.x; `last`: its weights are divided by its norm too
// (src/intertw_lcv.cu:269-273).
__global__ void __launch_bounds__(kStepThreads, 1) upd_solve_kernel(UpdParams p, int k, int nrange, int last) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  StepSmem m;
  step_carve(m, smem_raw, p.R, p.npmax);
  UpdScratch s;
  upd_scratch(p.B, p.R, p.D, p.npmax, p.work, &s);
  const int i = blockIdx.x, R = p.R, RR = R * R, D = p.D, n = p.nbas[k], rv = p.rank_v ? p.rank_v[i] : R;
  const size_t vec = (size_t)R * p.npmax;
  dw* G = s.fg + (size_t)i * D * RR;
  for (int e = threadIdx.x; e < RR; e += kStepThreads) m.BB[e] = normal_equation(G, D, k, e % R, e / R, R, rv, s.pen[i]);
  if (threadIdx.x == 0) {
    m.flags[1] = 0;
    m.flags[2] = 1;
  }
  const dw* part = s.part + i * vec;
  for (int e = threadIdx.x; e < R * n; e += kStepThreads) {
    dw_acc acc = acc_zero();
    for (int r = 0; r < nrange; ++r) acc_add(acc, part[(size_t)r * p.B * vec + e]);
    m.b0[e] = e % R >= rv ? dw_make(e / R == 0 ? 1.f : 0.f) : acc_value(acc);  // ragged padding decoupled
  }
  __syncthreads();
  if (threadIdx.x < 32 * dwsolve::invert_warps(R)) dwsolve::invert_any(m.BB, R, m.gi, m.prow, m.flags + 2);
  __syncthreads();
  step_solve(m, R, n);
  double* fc = p.qnc + (size_t)i * R;
  step_weights(m, R, rv, false, fc);
  step_factor(m, R, n, p.qn + (size_t)i * R * p.nD + p.off[k], p.nD, s.fk + (size_t)i * R * n, n, G + (size_t)k * RR);
  __syncthreads();
  if (last) step_renormalise(m, R, D, G, fc);
  if (threadIdx.x == 0 && m.flags[1]) atomicOr(&p.status[i], 1);
}

template <int A>
void rhs_launch(const UpdParams& p, int k, int n, dim3 grid, int per, cudaStream_t st) {
  switch ((n + 15) / 16) {
    case 1: upd_rhs_kernel<A, 1><<<grid, kRhsThreads, 0, st>>>(p, k, per); break;
    case 2: upd_rhs_kernel<A, 2><<<grid, kRhsThreads, 0, st>>>(p, k, per); break;
    case 3: upd_rhs_kernel<A, 3><<<grid, kRhsThreads, 0, st>>>(p, k, per); break;
    default: upd_rhs_kernel<A, 4><<<grid, kRhsThreads, 0, st>>>(p, k, per);
  }
}

}  // namespace

size_t upd_grid_dw(int B, int R, int D, int npm) {
  UpdScratch s;
  return upd_scratch(B, R, D, npm, nullptr, &s);
}

int upd_grid_launch(const UpdParams& p, cudaStream_t st) {
  const int R = p.R, BR = p.B * R;
  const long long n = (long long)BR * p.B + p.B;
  upd_weights_kernel<<<(int)std::min<long long>((n + 255) / 256, 4096), 256, 0, st>>>(p);
  MLCP_CUDA_TRY(cudaGetLastError());
  StepSmem m;
  const size_t s_solve = step_carve(m, nullptr, R, p.npmax);
  const size_t s_ov = sizeof(dw) * 2 * (size_t)p.npmax * (kTile + 1);
  MLCP_CUDA_TRY(cudaFuncSetAttribute(upd_solve_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s_solve));
  MLCP_CUDA_TRY(cudaFuncSetAttribute(upd_overlap_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s_ov));
  const int tiles = (BR + kTile - 1) / kTile;
  if (p.D > 1) {  // mode 0 is solved before its overlaps are used
    upd_overlap_kernel<<<dim3(tiles, tiles, p.D - 1), kOvThreads, s_ov, st>>>(p, 1, 1);
    MLCP_CUDA_TRY(cudaGetLastError());
  }
  // ranges of the block terms: whole chunks, about four CTAs for every SM
  const int rows = R <= 16 ? 1 : (R + 31) / 32, chunks = (BR + kChunk - 1) / kChunk;
  const int want = std::max(1, std::min(chunks, kRhsCtas / (p.B * rows)));
  const int per = (chunks + want - 1) / want * kChunk, nrange = (BR + per - 1) / per;
  for (int sw = 0; sw < p.nals; ++sw)
    for (int k = 0; k < p.D; ++k) {
      const dim3 grid(nrange, rows, p.B);
      if (R <= 16) rhs_launch<2>(p, k, p.h_off[k + 1] - p.h_off[k], grid, per, st);
      else rhs_launch<4>(p, k, p.h_off[k + 1] - p.h_off[k], grid, per, st);
      MLCP_CUDA_TRY(cudaGetLastError());
      const bool last = sw == p.nals - 1 && k == p.D - 1;
      upd_solve_kernel<<<p.B, kStepThreads, s_solve, st>>>(p, k, nrange, last ? 1 : 0);
      MLCP_CUDA_TRY(cudaGetLastError());
      if (!last) {
        upd_overlap_kernel<<<dim3(tiles, tiles, 1), kOvThreads, s_ov, st>>>(p, k, 0);
        MLCP_CUDA_TRY(cudaGetLastError());
      }
    }
  return kOk;
}

}  // namespace mlcp
