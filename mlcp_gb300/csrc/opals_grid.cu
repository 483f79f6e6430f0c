// ALS-fitted Hamiltonian applications over the whole GPU: the algorithm of
// opals.cu (POW_ALS and PRODHV_ALS; see there for the definitions and the
// precision) as a few launches per mode step instead of one CTA per vector,
// for blocks whose work per step is more than launches cost.
//
// A mode step j is
//   og_products_kernel   W_u(r,i) c_r for every operator u of mode j (the
//                        term products of opals.cu times the weight) and the
//                        normal equations;
//   og_rhs_kernel        b(i,n) = sum_u sum_r W_u(r,i) c_r Z_u(r,n);
//   og_solve_kernel      one CTA per vector: the solve, the new factor, its
//                        Gram, at the end of a POW sweep the renormalisation;
//   og_operators_kernel  Z_u = h_u F_j (POW) and M_u = Z_u F_j^T.
// Z of every mode is kept from step to step: POW needs h_u F_j of the factor
// that the previous sweep left, PRODHV h_u Fo_j throughout, so nothing is
// applied twice (opals.cu's CTA applied every operator again for each right-
// hand side).
//
// Each entry is the same chain of the same double-word operations in the same
// order as in the one-CTA form, so both forms give the same bits; only who
// computes an entry differs.
//
// What bounds it: the compensated multiply-add (13 FP32 instructions), about
// 3.1e12 a second over 152 SMs; the three contractions run 12-16
// accumulators a thread on operands in shared memory, and the term products
// are bound by reading M once per step.  On a 6 x 48 node (400 terms, 100
// vectors, rank 30) a POW sweep and a PRODHV sweep took 260 and 198 ms with
// one CTA per vector (256 threads, operands through L2) and take 23 ms
// together.
#include <algorithm>

#include "common.cuh"
#include "dword.cuh"
#include "dwsolve.cuh"
#include "intertwine.cuh"
#include "opstep.cuh"

namespace mlcp {

namespace {

constexpr int kOpThreads = 128;
constexpr int kChunkK = 32;         // rows of one right-hand-side stage

__device__ __forceinline__ uint32_t og_saddr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void og_cp8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(og_saddr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void og_cp16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(og_saddr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void og_cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void og_cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Scratch of the grid form, per vector.
struct OgScratch {
  dw *f, *bb, *b0, *cf, *cfo, *pen;
};
__host__ __device__ inline size_t og_carve(const OpTable& t, int nvec, dw* base, OgScratch* s) {
  size_t o = 0;
  auto take = [&](size_t n) -> dw* {
    dw* r = base ? base + o : nullptr;
    o += (n + 1) / 2 * 2;  // 16-byte boundaries
    return r;
  };
  s->f = take((size_t)nvec * t.R * t.nDp);       // [R][nDp] factors
  s->bb = take((size_t)nvec * t.R * t.R);        // normal equations
  s->b0 = take((size_t)nvec * t.R * t.npmax);    // right-hand side (column-major, ld R)
  s->cf = take((size_t)nvec * t.R);              // weights of F
  s->cfo = take((size_t)nvec * t.R);             // weights of Fo
  s->pen = take(nvec);
  return o;
}

// F (= Fo) in double-word, weights, penalty, Grams of F.  One CTA per vector.
__global__ void __launch_bounds__(kStepThreads) og_setup_kernel(OpAlsParams p) {
  const OpTable& t = p.ops;
  const int v = blockIdx.x, R = t.R, D = t.D, nD = p.nD, RR = R * R;
  OgScratch s;
  og_carve(t, p.nvec, p.gscr, &s);
  const double* fob = p.fo_base + (size_t)v * R * nD;
  const double* foc = p.fo_coef + (size_t)v * R;
  dw* f = s.f + (size_t)v * R * t.nDp;
  if (p.mode != 0) {
    double* fb = p.f_base + (size_t)v * R * nD;
    double* fc = p.f_coef + (size_t)v * R;
    for (int e = threadIdx.x; e < R * nD; e += blockDim.x) fb[e] = fob[e];
    for (int e = threadIdx.x; e < R; e += blockDim.x) fc[e] = foc[e];
  }
  for (int e = threadIdx.x; e < R * t.nDp; e += blockDim.x) {
    const int r = e / t.nDp, q = e % t.nDp;
    int d = 0;
    while (d + 1 < D && t.offp[d + 1] <= q) ++d;
    const int k = q - t.offp[d];
    f[e] = dw_from_double((k < t.nbas[d]) ? fob[(size_t)r * nD + t.off[d] + k] : 0.0);
  }
  for (int e = threadIdx.x; e < R; e += blockDim.x)
    s.cf[(size_t)v * R + e] = s.cfo[(size_t)v * R + e] = dw_from_double(foc[e]);
  if (threadIdx.x == 0) {
    double pen = foc[0];
    for (int i = 1; i < R; ++i) pen = foc[i] > pen ? foc[i] : pen;
    s.pen[v] = dw_from_double(pen * p.pen_factor);
  }
  dw* G = reinterpret_cast<dw*>(p.g64) + (size_t)v * D * RR;
  for (int e = threadIdx.x; e < D * RR; e += blockDim.x) {
    const int d = e / RR, ee = e - d * RR, i = ee % R, i2 = ee / R, o = t.off[d];
    double acc = 0.0;
    for (int q = 0; q < t.nbas[d]; ++q) acc += fob[(size_t)i * nD + o + q] * fob[(size_t)i2 * nD + o + q];
    G[e] = dw_from_double(acc);
  }
}

// Term products of mode j times the weights, and the normal equations: one
// thread per (operator, entry), vector blockIdx.y.
__global__ void __launch_bounds__(kOpThreads) og_products_kernel(OpAlsParams p, int j) {
  const OpTable& t = p.ops;
  const int v = blockIdx.y, R = t.R, RR = R * R, D = t.D, nu = t.uoff[j + 1] - t.uoff[j];
  const int item = blockIdx.x * kOpThreads + threadIdx.x;
  if (item >= (nu + 1) * RR) return;
  const int u = item / RR, e = item - u * RR;
  OgScratch s;
  og_carve(t, p.nvec, p.gscr, &s);
  if (u == nu) {
    const dw* G = reinterpret_cast<const dw*>(p.g64) + (size_t)v * D * RR;
    s.bb[(size_t)v * RR + e] = normal_equation(G, D, j, e % R, e / R, R, p.rank_v ? p.rank_v[v] : R, s.pen[v]);
    return;
  }
  const dw* __restrict__ M = p.mscr + (size_t)v * t.utot * RR + e;
  const int* __restrict__ ord = t.order + (size_t)j * t.T;
  const int q0 = t.gstart[(size_t)j * (t.umax + 1) + u], q1 = t.gstart[(size_t)j * (t.umax + 1) + u + 1];
  dw_acc acc = acc_zero();
  for (int q = q0; q < q1; q += 4) {
    dw pr[4];
    const int* sl[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int term = ord[min(q + k, q1 - 1)];
      pr[k] = t.alphadw[term];
      sl[k] = t.slot + (size_t)term * D;
    }
    for (int d = 0; d < D; ++d) {
      if (d == j) continue;
#pragma unroll
      for (int k = 0; k < 4; ++k) pr[k] = dw_mul(pr[k], M[(size_t)sl[k][d] * RR]);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (q + k < q1) acc_add(acc, pr[k]);
  }
  if (u == 0 && p.ishift != 0) {
    dw prod = dw_from_double(-(p.eshift_v ? p.eshift_v[v] : p.eshift));
    for (int d = 0; d < D; ++d)
      if (d != j) prod = dw_mul(prod, M[(size_t)t.uoff[d] * RR]);
    acc_add(acc, prod);
  }
  const dw c = (p.mode == 0 ? s.cf : s.cfo)[(size_t)v * R + e / R];
  p.wscr[(size_t)v * t.umax * RR + item] = dw_mul(acc_value(acc), c);
}

// b(i,n) = sum over k = (u, r) of W[k][i] Z[k][n]: a tile of 8 A rows i x 16
// columns n per CTA, the rows k staged in shared memory two chunks deep.
// Every entry is one chain over k.
template <int A>
__global__ void __launch_bounds__(kOpThreads) og_rhs_kernel(OpAlsParams p, int j) {
  constexpr int TI = 8 * A, TN = 16;
  __shared__ __align__(16) dw ws[2][kChunkK][TI];
  __shared__ __align__(16) dw zs[2][kChunkK][TN];
  const OpTable& t = p.ops;
  const int v = blockIdx.z, R = t.R, npm = t.npmax, nj = t.nbas[j], K = (t.uoff[j + 1] - t.uoff[j]) * R;
  const int n0 = blockIdx.x * TN, i0 = blockIdx.y * TI;
  const dw* W = p.wscr + (size_t)v * t.umax * R * R + i0;
  const dw* Z = p.zscr + ((size_t)v * t.utot + t.uoff[j]) * R * npm + n0;
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  auto stage = [&](int k0, int b) {
#pragma unroll
    for (int e = threadIdx.x; e < kChunkK * TI; e += kOpThreads) {
      const int k = e / TI, i = e % TI;
      if (k0 + k < K && i0 + i < R) og_cp8(&ws[b][k][i], W + (size_t)(k0 + k) * R + i);
    }
#pragma unroll
    for (int e = threadIdx.x; e < kChunkK * TN; e += kOpThreads) {
      const int k = e / TN, n = e % TN;
      if (k0 + k < K && n0 + n < nj) og_cp8(&zs[b][k][n], Z + (size_t)(k0 + k) * npm + n);
    }
    og_cp_commit();
  };
  // entries outside the matrices stay zero (they feed results never stored)
  for (int e = threadIdx.x; e < 2 * kChunkK * TI; e += kOpThreads) (&ws[0][0][0])[e] = dw_make(0.f);
  for (int e = threadIdx.x; e < 2 * kChunkK * TN; e += kOpThreads) (&zs[0][0][0])[e] = dw_make(0.f);
  __syncthreads();
  dw_acc acc[A];
#pragma unroll
  for (int a = 0; a < A; ++a) acc[a] = acc_zero();
  stage(0, 0);
  for (int k0 = 0, b = 0; k0 < K; k0 += kChunkK, b ^= 1) {
    if (k0 + kChunkK < K) {
      stage(k0 + kChunkK, b ^ 1);
      og_cp_wait<1>();
    } else {
      og_cp_wait<0>();
    }
    __syncthreads();
    const int kn = min(kChunkK, K - k0);
#pragma unroll 4
    for (int k = 0; k < kn; ++k) {
      const dw z = zs[b][k][tx];
#pragma unroll
      for (int a = 0; a < A; ++a) acc_fma(acc[a], ws[b][k][ty + 8 * a], z);
    }
    __syncthreads();
  }
  OgScratch s;
  og_carve(t, p.nvec, p.gscr, &s);
  const int n = n0 + tx, rv = p.rank_v ? p.rank_v[v] : R;
  if (n >= nj) return;
#pragma unroll
  for (int a = 0; a < A; ++a) {
    const int i = i0 + ty + 8 * a;
    if (i >= R) continue;
    const dw b = acc_value(acc[a]);
    s.b0[(size_t)v * R * npm + i + n * R] =
        i >= rv ? dw_make(n == 0 ? 1.f : 0.f) : (p.ishift < 0 ? dw_neg(b) : b);  // ragged padding decoupled
  }
}

// The solve of mode j and what follows from the new factor; one CTA per vector.
__global__ void __launch_bounds__(kStepThreads, 1) og_solve_kernel(OpAlsParams p, int j) {
  const OpTable& t = p.ops;
  const int v = blockIdx.x, R = t.R, RR = R * R, npm = t.npmax, nD = p.nD, nj = t.nbas[j], opj = t.offp[j];
  extern __shared__ __align__(16) unsigned char smem_raw[];
  StepSmem m;
  step_carve(m, smem_raw, R, npm);
  OgScratch s;
  og_carve(t, p.nvec, p.gscr, &s);
  for (int e = threadIdx.x; e < RR; e += kStepThreads) m.BB[e] = s.bb[(size_t)v * RR + e];
  for (int e = threadIdx.x; e < R * nj; e += kStepThreads) m.b0[e] = s.b0[(size_t)v * R * npm + e];
  if (threadIdx.x == 0) {
    m.flags[1] = 0;
    m.flags[2] = 1;
  }
  __syncthreads();
  if (threadIdx.x < 32 * dwsolve::invert_warps(R)) dwsolve::invert_any(m.BB, R, m.gi, m.prow, m.flags + 2);
  __syncthreads();
  step_solve(m, R, nj);
  const int rv = p.rank_v ? p.rank_v[v] : R;
  dw* cf = s.cf + (size_t)v * R;
  double* fc = p.f_coef + (size_t)v * R;
  double* fb = p.f_base + (size_t)v * R * nD;
  dw* G = reinterpret_cast<dw*>(p.g64) + (size_t)v * t.D * RR;
  step_weights(m, R, rv, p.mode == 0, fc);
  step_factor(m, R, nj, fb + t.off[j], nD, s.f + (size_t)v * R * t.nDp + opj, t.nDp, G + (size_t)j * RR);
  __syncthreads();
  if (p.mode == 0 && j == t.D - 1) step_renormalise(m, R, t.D, G, fc);
  for (int i = threadIdx.x; i < R; i += kStepThreads) cf[i] = m.cf[i];
  if (threadIdx.x == 0 && m.flags[1]) atomicOr(&p.status[v], 1);
}

// Z_u = h_u F_j (apply) or Z_u as stored, and M_u(r,i) = <Z_u(r,:), F_j(i,:)>
// for the operators u of mode j in chunk blockIdx.x, vector blockIdx.y.
// Thread (ty, tx) holds rows ty + 8 a and columns tx + 16 c.  A 8: two
// passes of four (ranks above 32).
template <int A, int NC>
__global__ void __launch_bounds__(kOpThreads) og_operators_kernel(OpAlsParams p, int j, int per, int apply) {
  constexpr int AP = A < 4 ? A : 4, IC = A / 2 < 1 ? 1 : A / 2;  // rows of one pass, columns of 16 for R entries
  const OpTable& t = p.ops;
  const int v = blockIdx.y, R = t.R, RR = R * R, npm = t.npmax, n = t.nbas[j];
  const int u0 = blockIdx.x * per, u1 = min(u0 + per, t.uoff[j + 1] - t.uoff[j]);
  constexpr int ldr = 8 * A;  // rows padded to the tile
  extern __shared__ __align__(16) unsigned char smem_raw[];
  dw* fs = reinterpret_cast<dw*>(smem_raw);  // [n][ldr]: F transposed
  dw* zs = fs + (size_t)n * ldr;             // [n][ldr]: Z_u transposed
  dw* hs = zs + (size_t)n * ldr;             // [2][n][16 NC]: h_u (symmetric)
  constexpr int ldh = 16 * NC;
  OgScratch s;
  og_carve(t, p.nvec, p.gscr, &s);
  const dw* f = s.f + (size_t)v * R * t.nDp + t.offp[j];
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  for (int e = threadIdx.x; e < n * ldr; e += kOpThreads) {
    const int r = e / n, m = e - r * n;
    fs[m * ldr + r] = r < R ? f[(size_t)r * t.nDp + m] : dw_make(0.f);
    zs[m * ldr + r] = dw_make(0.f);
  }
  auto fetch = [&](int u, int b) {
    if (apply && u < u1 && !t.ident[t.uoff[j] + u]) {
      const dw* h = t.hdw + (size_t)(t.uoff[j] + u) * npm * npm;
      dw* d = hs + (size_t)b * n * ldh;
      const int half = (n + 1) / 2;  // 16-byte pairs of a row (rows are padded to a multiple of four entries)
      for (int e = threadIdx.x; e < n * half; e += kOpThreads) {
        const int k = e / half, q = e - k * half;
        og_cp16(d + k * ldh + 2 * q, h + (size_t)k * npm + 2 * q);
      }
    }
    og_cp_commit();
  };
  fetch(u0, 0);
  for (int u = u0, b = 0; u < u1; ++u, b ^= 1) {
    const int g = t.uoff[j] + u;
    dw* Z = p.zscr + ((size_t)v * t.utot + g) * R * npm;
    fetch(u + 1, b ^ 1);
    og_cp_wait<1>();
    __syncthreads();  // h_u and, the first time, F have landed; the previous M is done with zs
    if (!apply) {
      for (int e = threadIdx.x; e < R * n; e += kOpThreads) {
        const int r = e / n, m = e - r * n;
        zs[m * ldr + r] = Z[(size_t)r * npm + m];
      }
    } else if (t.ident[g]) {
      for (int e = threadIdx.x; e < R * n; e += kOpThreads) {
        const int r = e / n, m = e - r * n;
        const dw x = fs[m * ldr + r];
        zs[m * ldr + r] = x;
        Z[(size_t)r * npm + m] = x;
      }
    } else {
      const dw* h = hs + (size_t)b * n * ldh;
#pragma unroll
      for (int a0 = 0; a0 < A; a0 += AP) {
        dw_acc acc[AP][NC];
#pragma unroll
        for (int a = 0; a < AP; ++a)
#pragma unroll
          for (int c = 0; c < NC; ++c) acc[a][c] = acc_zero();
        for (int k = 0; k < n; ++k) {
          dw hv[NC];
#pragma unroll
          for (int c = 0; c < NC; ++c) hv[c] = h[k * ldh + tx + 16 * c];
#pragma unroll
          for (int a = 0; a < AP; ++a) {
            const dw x = fs[k * ldr + ty + 8 * (a0 + a)];
#pragma unroll
            for (int c = 0; c < NC; ++c) acc_fma(acc[a][c], hv[c], x);
          }
        }
#pragma unroll
        for (int a = 0; a < AP; ++a)
#pragma unroll
          for (int c = 0; c < NC; ++c) {
            const int r = ty + 8 * (a0 + a), m = tx + 16 * c;
            if (r >= R || m >= n) continue;
            const dw z = acc_value(acc[a][c]);
            zs[m * ldr + r] = z;
            Z[(size_t)r * npm + m] = z;
          }
      }
    }
    __syncthreads();
    dw* M = p.mscr + ((size_t)v * t.utot + g) * RR;
#pragma unroll
    for (int a0 = 0; a0 < A; a0 += AP) {
      dw_acc acc[AP][IC];
#pragma unroll
      for (int a = 0; a < AP; ++a)
#pragma unroll
        for (int c = 0; c < IC; ++c) acc[a][c] = acc_zero();
      for (int m = 0; m < n; ++m) {
        dw fv[IC];
#pragma unroll
        for (int c = 0; c < IC; ++c) fv[c] = fs[m * ldr + tx + 16 * c];
#pragma unroll
        for (int a = 0; a < AP; ++a) {
          const dw z = zs[m * ldr + ty + 8 * (a0 + a)];
#pragma unroll
          for (int c = 0; c < IC; ++c) acc_fma(acc[a][c], z, fv[c]);
        }
      }
#pragma unroll
      for (int a = 0; a < AP; ++a)
#pragma unroll
        for (int c = 0; c < IC; ++c) {
          const int r = ty + 8 * (a0 + a), i = tx + 16 * c;
          if (r < R && i < R) M[r * R + i] = acc_value(acc[a][c]);
        }
    }
  }
}

template <int A, int NC>
int operators_launch(const OpAlsParams& p, int j, int nu, int n, int nsm, bool apply, cudaStream_t st) {
  const size_t smem = sizeof(dw) * ((size_t)2 * n * 8 * A + (size_t)2 * n * 16 * NC);
  MLCP_CUDA_TRY(cudaFuncSetAttribute(og_operators_kernel<A, NC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)smem));
  // operators per CTA: about eight CTAs for every SM, so that a CTA's set-up
  // (its vector's factor) is shared by several operators where there are many
  const int chunks = std::max(1, std::min(nu, (8 * nsm + p.nvec - 1) / p.nvec)), per = (nu + chunks - 1) / chunks;
  og_operators_kernel<A, NC><<<dim3((nu + per - 1) / per, p.nvec), kOpThreads, smem, st>>>(p, j, per, apply ? 1 : 0);
  MLCP_CUDA_TRY(cudaGetLastError());
  return kOk;
}

template <int A>
int operators_launch_n(const OpAlsParams& p, int j, int nu, int n, int nsm, bool apply, cudaStream_t st) {
  switch ((n + 15) / 16) {
    case 1: return operators_launch<A, 1>(p, j, nu, n, nsm, apply, st);
    case 2: return operators_launch<A, 2>(p, j, nu, n, nsm, apply, st);
    case 3: return operators_launch<A, 3>(p, j, nu, n, nsm, apply, st);
    default: return operators_launch<A, 4>(p, j, nu, n, nsm, apply, st);
  }
}

int operators_any(const OpAlsParams& p, int j, int nu, int n, int nsm, bool apply, cudaStream_t st) {
  const int R = p.ops.R;
  if (R <= 16) return operators_launch_n<2>(p, j, nu, n, nsm, apply, st);
  if (R <= 32) return operators_launch_n<4>(p, j, nu, n, nsm, apply, st);
  return operators_launch_n<8>(p, j, nu, n, nsm, apply, st);
}

}  // namespace

size_t opals_grid_dw(const OpTable& t, int nvec) {
  OgScratch s;
  return og_carve(t, nvec, nullptr, &s);
}

int opals_grid_launch(const OpAlsParams& p, cudaStream_t st) {
  const OpTable& t = p.ops;
  const int R = t.R, RR = R * R, D = t.D;
  int dev = 0, nsm = 0;
  MLCP_CUDA_TRY(cudaGetDevice(&dev));
  MLCP_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  StepSmem m;
  const size_t ssm = step_carve(m, nullptr, R, t.npmax);
  MLCP_CUDA_TRY(cudaFuncSetAttribute(og_solve_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ssm));
  og_setup_kernel<<<p.nvec, kStepThreads, 0, st>>>(p);
  MLCP_CUDA_TRY(cudaGetLastError());
  for (int d = 0; d < D; ++d)
    if (int rc = operators_any(p, d, t.h_uoff[d + 1] - t.h_uoff[d], t.h_nbas[d], nsm, true, st)) return rc;
  for (int sw = 0; sw < p.nsweeps; ++sw)
    for (int j = 0; j < D; ++j) {
      const int nu = t.h_uoff[j + 1] - t.h_uoff[j], nj = t.h_nbas[j];
      og_products_kernel<<<dim3((unsigned)(((size_t)(nu + 1) * RR + kOpThreads - 1) / kOpThreads), p.nvec), kOpThreads,
                           0, st>>>(p, j);
      MLCP_CUDA_TRY(cudaGetLastError());
      if (R <= 16) og_rhs_kernel<2><<<dim3((nj + 15) / 16, 1, p.nvec), kOpThreads, 0, st>>>(p, j);
      else og_rhs_kernel<4><<<dim3((nj + 15) / 16, (R + 31) / 32, p.nvec), kOpThreads, 0, st>>>(p, j);
      MLCP_CUDA_TRY(cudaGetLastError());
      og_solve_kernel<<<p.nvec, kStepThreads, ssm, st>>>(p, j);
      MLCP_CUDA_TRY(cudaGetLastError());
      if (sw + 1 < p.nsweeps || j + 1 < D)  // the last factor's products are not needed
        if (int rc = operators_any(p, j, nu, nj, nsm, p.mode == 0, st)) return rc;
    }
  return kOk;
}

}  // namespace mlcp
