// Double-word dense kernels for one small n x n symmetric positive definite
// system (the normal equations of every fit), run by a team of warps (threads 0
// .. 127 of the block unless a function says otherwise) that synchronise on
// named barrier 1.  Matrices are column-major with leading dimension n.
#pragma once

#include <cfloat>

#include "dword.cuh"

namespace mlcp {
namespace dwsolve {

constexpr int kSolverWarps = 4;
constexpr int kSolverThreads = kSolverWarps * 32;

// Barrier among the solver warps only (named barrier 1): threads 0 .. NT-1 of
// the block.
template <int NT>
__device__ __forceinline__ void team_sync() {
  asm volatile("bar.sync 1, %0;" ::"n"(NT) : "memory");
}
__device__ __forceinline__ void solver_sync() { team_sync<kSolverThreads>(); }

// In-place LDL^T of the symmetric A (lower triangle): afterwards A(i,j) =
// L(i,j) for i > j and dinv[j] = 1/D(j).  The next pivot is formed first so
// its reciprocal overlaps the rest of the trailing update.  Returns the
// 1-based index of the first non-positive pivot (replaced by its magnitude
// plus a tiny amount, as the FP64 Cholesky fallback of the reference would
// fail there) or 0.  u is scratch of n entries.
__device__ inline int dw_ldlt(dw* A, int n, dw* dinv, dw* u) {
  const int t = threadIdx.x, lane = t & 31, wq = t >> 5;
  int bad = 0;
  dw d0 = A[0];
  if (!(d0.hi > 0.f)) {
    bad = 1;
    d0 = dw_make(fabsf(d0.hi) + 1e-30f);
  }
  dw inv = dw_rcp(d0);
  for (int j = 0; j < n; ++j) {
    const int m = n - j - 1;
    for (int r = t; r < m; r += kSolverThreads) {
      const dw a = A[j + 1 + r + j * n];
      u[j + 1 + r] = a;
      A[j + 1 + r + j * n] = dw_mul(a, inv);
    }
    if (t == 0) dinv[j] = inv;
    solver_sync();
    if (m == 0) break;
    dw next = dw_fms(A[j + 1 + j * n], u[j + 1], A[(j + 1) * (n + 1)]);
    if (!(next.hi > 0.f)) {
      if (!bad) bad = j + 2;
      next = dw_make(fabsf(next.hi) + 1e-30f);
    }
    const dw inv_next = dw_rcp(next);
    // trailing update: row i = j+1+ri (lane), columns j+1+cc <= i (warp-strided)
    for (int ri = lane; ri < m; ri += 32) {
      if (ri == 0) continue;  // (j+1, j+1) is `next`
      const int i = j + 1 + ri;
      const dw l = A[i + j * n];
      for (int cc = wq; cc <= ri; cc += kSolverWarps) {
        const int col = j + 1 + cc;
        A[i + col * n] = dw_fms(l, u[col], A[i + col * n]);
      }
    }
    if (t == 0) A[(j + 1) * (n + 1)] = next;
    inv = inv_next;
    solver_sync();
  }
  return bad;
}

// Solve L D L^T X = B in place for nrhs columns (B column-major, ld n).
__device__ inline void dw_ldlt_solve(const dw* A, int n, const dw* dinv, dw* B, int nrhs) {
  const int t = threadIdx.x;
  for (int j = 0; j < n - 1; ++j) {
    const int m = n - j - 1;
    for (int e = t; e < m * nrhs; e += kSolverThreads) {
      const int col = e / m, i = j + 1 + (e - col * m);
      B[i + col * n] = dw_fms(A[i + j * n], B[j + col * n], B[i + col * n]);
    }
    solver_sync();
  }
  for (int e = t; e < n * nrhs; e += kSolverThreads) {
    const int col = e / n, i = e - col * n;
    B[i + col * n] = dw_mul(B[i + col * n], dinv[i]);
  }
  solver_sync();
  for (int j = n - 1; j > 0; --j) {
    for (int e = t; e < j * nrhs; e += kSolverThreads) {
      const int col = e / j, i = e - col * j;
      B[i + col * n] = dw_fms(A[j + i * n], B[j + col * n], B[i + col * n]);
    }
    solver_sync();
  }
}

__device__ __forceinline__ dw dw_shfl_xor(dw v, int o) {
  return dw{__shfl_xor_sync(0xffffffffu, v.hi, o), __shfl_xor_sync(0xffffffffu, v.lo, o)};
}

// The rows of X (nr of them, column-major, ld nr, n columns) scaled to unit norm, as the
// reference's normonebase (src/modvecvec.cu:225-262: max-scaled 2-norm; a zero row gives
// NaN), by threads 0 .. NT-1, G lanes of one warp per row (G the largest power of two
// <= 32 with G nr <= NT); norms to nrm[i].  The lanes of a row combine
// their maxima and sums of squares by butterflies, so all of them hold the
// same norm.  Ends without a barrier.
template <int NT = kSolverThreads>
__device__ inline void dw_normalise_rows(dw* X, int nr, int n, dw* nrm) {
  int G = 32;
  while (G > 1 && G * nr > NT) G >>= 1;
  const int t = threadIdx.x, row = t / G, sub = t - row * G;
  const bool live = row < nr;
  dw* x = X + (live ? row : 0);
  dw largest = dw_make(0.f);
  for (int q = sub; q < n; q += G) {
    const dw a = dw_abs(x[q * nr]);
    if (dw_gt(a, largest)) largest = a;
  }
  for (int o = G / 2; o > 0; o >>= 1) {
    const dw b = dw_shfl_xor(largest, o);
    if (dw_gt(b, largest)) largest = b;
  }
  const bool zero = !(largest.hi > 0.f);
  const dw il = dw_rcp(zero ? dw_make(1.f) : largest);
  dw acc = dw_make(0.f);
  for (int q = sub; q < n; q += G) {
    const dw y = dw_mul(x[q * nr], il);
    acc = dw_fma(y, y, acc);
  }
  for (int o = G / 2; o > 0; o >>= 1) acc = dw_add(acc, dw_shfl_xor(acc, o));
  if (!live) return;
  if (zero) {  // NaN, as the reference's zero-row norm
    const float nan = __int_as_float(0x7fffffff);
    for (int q = sub; q < n; q += G) x[q * nr] = dw_make(nan);
    if (sub == 0) nrm[row] = dw_make(nan);
    return;
  }
  const dw r = dw_mul(largest, dw_sqrt(acc));
  const dw inv = dw_rcp(r);
  for (int q = sub; q < n; q += G) x[q * nr] = dw_mul(x[q * nr], inv);
  if (sub == 0) nrm[row] = r;
}

// Walk over the entries e = tid, tid + NT, ... of a matrix with n rows
// (column-major), tracking (row, column) = (e mod n, e div n) without dividing.
struct Walk {
  int i, j, di, dj, n;
};
template <int NT = kSolverThreads>
__device__ __forceinline__ Walk walk_start(int t, int n) {
  return Walk{t % n, t / n, NT % n, NT / n, n};
}
__device__ __forceinline__ void walk_next(Walk& w) {
  w.i += w.di;
  w.j += w.dj;
  if (w.i >= w.n) {
    w.i -= w.n;
    w.j += 1;
  }
}

// Entries a solver thread handles per batch (operands loaded before any store).
constexpr int kSolveBatch = 4;

// FP32 Gauss-Jordan inverse of the symmetric positive definite n x n matrix
// given by the high parts of A (column-major), without pivoting (its pivots
// are the positive Schur-complement diagonals).  Two buffers alternate so each
// elimination step reads the previous one and needs one barrier; a thread
// loads the operands of up to four entries before it stores any (a store
// would otherwise order every later shared-memory load behind it).  Returns
// the buffer holding the inverse; *ok is false when a pivot is not positive.
__device__ inline const float* gj_inverse(const dw* A, int n, float* gi, bool* ok) {
  const int t = threadIdx.x, nn = n * n;
  for (int e = t; e < nn; e += kSolverThreads) gi[e] = A[e].hi;
  solver_sync();
  int cur = 0;
  bool good = true;
  // (row, column) of the first batch of entries, fixed for all steps
  int i0[kSolveBatch], j0[kSolveBatch];
  Walk w_later = walk_start(t, n);  // walk state at the second batch
#pragma unroll
  for (int q = 0; q < kSolveBatch; ++q) {
    i0[q] = w_later.i;
    j0[q] = w_later.j;
    walk_next(w_later);
  }
  for (int k = 0; k < n; ++k) {
    const float* s = gi + cur * nn;
    float* d = gi + (cur ^ 1) * nn;
    const float piv = s[k + k * n];
    good = good && piv > 0.f;
    float pk = f_rcp_approx(piv);
    pk = pk * fmaf(-piv, pk, 2.0f);
    Walk w = w_later;
    for (int e0 = t; e0 < nn; e0 += kSolveBatch * kSolverThreads) {
      float a[kSolveBatch], b[kSolveBatch], x[kSolveBatch];
      int ii[kSolveBatch], jj[kSolveBatch];
      const bool first = e0 == t;
#pragma unroll
      for (int q = 0; q < kSolveBatch; ++q) {
        ii[q] = first ? i0[q] : w.i;
        jj[q] = first ? j0[q] : w.j;
        if (!first) walk_next(w);
        if (e0 + q * kSolverThreads < nn) {
          a[q] = s[ii[q] + k * n];
          b[q] = s[k + jj[q] * n];
          x[q] = s[e0 + q * kSolverThreads];
        }
      }
#pragma unroll
      for (int q = 0; q < kSolveBatch; ++q) {
        const int e = e0 + q * kSolverThreads;
        if (e >= nn) continue;
        const float ta = a[q] * pk;
        float v = fmaf(-ta, b[q], x[q]);
        if (ii[q] == k) v = (jj[q] == k) ? pk : b[q] * pk;
        else if (jj[q] == k) v = -ta;
        d[e] = v;
      }
    }
    cur ^= 1;
    solver_sync();
  }
  *ok = good;
  return gi + cur * nn;
}

// The same FP32 Gauss-Jordan inverse for n <= N <= 32 by one warp, in
// registers: lane j holds column j, and each elimination step broadcasts the
// pivot column from its lane by shuffles, so no step touches shared memory or
// waits at a barrier.  Writes the inverse to inv (column-major, ld n) and
// returns whether every pivot was positive.  All 32 lanes must call it.
template <int N>
__device__ inline bool gj_inverse_warp_n(const dw* A, int n, float* inv) {
  const int lane = threadIdx.x & 31;
  const bool col = lane < n;
  float a[N];
#pragma unroll
  for (int i = 0; i < N; ++i) a[i] = (col && i < n) ? A[i + lane * n].hi : 0.f;
  bool good = true;
#pragma unroll
  for (int k = 0; k < N; ++k) {
    if (k >= n) break;
    const float piv = __shfl_sync(0xffffffffu, a[k], k);
    good = good && piv > 0.f;
    float pk = f_rcp_approx(piv);
    pk = pk * fmaf(-piv, pk, 2.0f);
    const float rk = a[k] * pk;  // row k of this column, scaled
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const float cik = __shfl_sync(0xffffffffu, a[i], k);  // column k, before the step
      if (i == k) a[i] = (lane == k) ? pk : rk;
      else a[i] = (lane == k) ? -cik * pk : fmaf(-cik, rk, a[i]);
    }
  }
  if (col)
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (i < n) inv[i + lane * n] = a[i];
  return good;
}

// The same for n <= 16 with the rows split over the half-warps: lane (h, j)
// holds rows 8 h .. 8 h + 7 of column j, so that a step costs half the
// instructions (it is bound by one warp's issue); the same operations on
// every entry, so the same bits as gj_inverse_warp_n<16>.
__device__ inline bool gj_inverse_half(const dw* A, int n, float* inv) {
  const int lane = threadIdx.x & 31, j = lane & 15, h = lane >> 4;
  float a[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) a[q] = (j < n && 8 * h + q < n) ? A[8 * h + q + j * n].hi : 0.f;
  bool good = true;
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    if (k >= n) break;
    const int kh = k >> 3, kq = k & 7;  // row k: register kq of half kh
    const float piv = __shfl_sync(0xffffffffu, a[kq], 16 * kh + k);
    good = good && piv > 0.f;
    float pk = f_rcp_approx(piv);
    pk = pk * fmaf(-piv, pk, 2.0f);
    const float rk = __shfl_sync(0xffffffffu, a[kq], 16 * kh + j) * pk;  // row k of this column, scaled
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const float ci = __shfl_sync(0xffffffffu, a[q], 16 * h + k);  // column k, before the step
      const float v = j == k ? -ci * pk : fmaf(-ci, rk, a[q]);
      a[q] = q == kq && h == kh ? (j == k ? pk : rk) : v;
    }
  }
  if (j < n)
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (8 * h + q < n) inv[8 * h + q + j * n] = a[q];
  return good;
}

// Register Gauss-Jordan for n <= 32, by the calling warp.
__device__ inline bool gj_inverse_warp(const dw* A, int n, float* inv) {
  if (n <= 8) return gj_inverse_warp_n<8>(A, n, inv);
  if (n <= 16) return gj_inverse_half(A, n, inv);
  return gj_inverse_warp_n<32>(A, n, inv);
}

// The FP32 inverses above by NW warps (threads 0 .. 32 NW - 1, named barrier
// 1) in registers: warp w holds rows w, w + NW, ... (ROWS of them), lane l
// columns l and, when COLS is 2, l + 32.  A step's pivot row goes through
// shared memory (row: [2][72] floats, two buffers so that a step needs one
// barrier); a row's own multiplier is a shuffle from the pivot column's lane.
// kColumn picks whose rounding is kept: the pivot column scaled first, as in
// gj_inverse, or the pivot row, as in gj_inverse_warp; entries are then the
// same bits as there.  What it replaces is bound by latency: one warp takes
// ~15 cycles per row and step (15.7 k cycles for n = 32), four warps through
// two shared-memory matrices ~1600 cycles per step (100 k for n = 64); this
// takes ~210 per step with four warps (8.3 k for n = 32) and ~500 with eight (33 k for
// n = 64).  Writes inv (column-major, ld n); *flag (set by the caller before a barrier) becomes 0
// when a pivot is not positive.  Ends without a barrier.
template <int NW, int ROWS, int COLS, bool kColumn>
__device__ inline void team_inverse(const dw* A, int n, float* inv, float* row, int* flag) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  float a[ROWS][COLS];
#pragma unroll
  for (int q = 0; q < ROWS; ++q)
#pragma unroll
    for (int c = 0; c < COLS; ++c) {
      const int i = w + NW * q, j = lane + 32 * c;
      a[q][c] = i < n && j < n ? A[i + j * n].hi : 0.f;
    }
  float* buf = row;
#pragma unroll
  for (int q = 0; q < ROWS; ++q) {
    for (int wk = 0; wk < NW; ++wk) {
      const int k = NW * q + wk;
      if (k >= n) break;
      const int kl = k & 31, kc = k >> 5;
      if (w == wk) {
        const float piv = __shfl_sync(0xffffffffu, COLS > 1 && kc ? a[q][COLS - 1] : a[q][0], kl);
        if (!(piv > 0.f) && lane == 0) *flag = 0;
        float pk = f_rcp_approx(piv);
        pk = pk * fmaf(-piv, pk, 2.0f);
#pragma unroll
        for (int c = 0; c < COLS; ++c) {
          const float rk = a[q][c] * pk;
          buf[lane + 32 * c] = kColumn ? a[q][c] : rk;
          a[q][c] = lane + 32 * c == k ? pk : rk;
        }
        if (lane == 0) buf[64] = pk;
      }
      team_sync<32 * NW>();
      float r[COLS];
#pragma unroll
      for (int c = 0; c < COLS; ++c) r[c] = buf[lane + 32 * c];
      const float pk = buf[64];
#pragma unroll
      for (int p = 0; p < ROWS; ++p) {
        const float ci = __shfl_sync(0xffffffffu, COLS > 1 && kc ? a[p][COLS - 1] : a[p][0], kl);
        if (p == q && w == wk) continue;
        const float cp = ci * pk;
#pragma unroll
        for (int c = 0; c < COLS; ++c)
          a[p][c] = lane + 32 * c == k ? -cp : fmaf(kColumn ? -cp : -ci, r[c], a[p][c]);
      }
      buf = buf == row ? row + 72 : row;
    }
  }
#pragma unroll
  for (int q = 0; q < ROWS; ++q)
#pragma unroll
    for (int c = 0; c < COLS; ++c) {
      const int i = w + NW * q, j = lane + 32 * c;
      if (i < n && j < n) inv[i + j * n] = a[q][c];
    }
}

// Warps that invert an n x n matrix (n <= 64) beside other work.
__host__ __device__ constexpr int invert_warps(int n) { return n <= 16 ? 1 : n <= 32 ? 4 : 8; }

// The inverse by threads 0 .. 32 invert_warps(n) - 1; row: [2][72] floats.
// *flag must be 1 on entry (ordered before the call); 0 on return when a pivot
// was not positive.
__device__ inline void invert_any(const dw* A, int n, float* inv, float* row, int* flag) {
  if (n <= 16) {
    const bool good = gj_inverse_warp(A, n, inv);
    if (threadIdx.x == 0 && !good) *flag = 0;
  } else if (n <= 32) {
    team_inverse<4, 8, 1, false>(A, n, inv, row, flag);
  } else {
    team_inverse<8, 8, 2, true>(A, n, inv, row, flag);
  }
}

// Refinement rounds before falling back to the double-word LDL^T.
constexpr int kRefineMax = 4;

// X = A^-1 B (A n x n double-word, B and X n x nrhs, ld n) by iterative
// refinement preconditioned with the FP32 inverse: X = inv B, then
// X += inv (B - A X) with the residual formed in double-word, until the last
// correction is below 1e-10 of max |X| (or the first is below 1e-5, which
// bounds the remaining error by 1e-10).  Returns whether that happened within
// kRefineMax rounds.  Each thread computes up to four entries in registers
// before storing them.  Threads 0 .. NT-1; every entry is the same chain
// whatever NT (128 where other warps work beside it, the whole block where
// they would wait: 30 x 48 entries take ~12 us with 128 threads and ~4 with 512).
template <int NT = kSolverThreads>
__device__ inline bool refine_solve(const dw* A, int n, const dw* B, dw* X, int nrhs, const float* inv, dw* R, float* red) {
  const int t = threadIdx.x, nr = n * nrhs;
  // X = inv * B
  {
    Walk w = walk_start<NT>(t, n);
    for (int e0 = t; e0 < nr; e0 += kSolveBatch * NT) {
      int ii[kSolveBatch], jj[kSolveBatch];
      float acc[kSolveBatch];
#pragma unroll
      for (int q = 0; q < kSolveBatch; ++q) {
        ii[q] = w.i;
        jj[q] = w.j;
        acc[q] = 0.f;
        walk_next(w);
      }
      for (int j = 0; j < n; ++j)
#pragma unroll
        for (int q = 0; q < kSolveBatch; ++q)
          if (e0 + q * NT < nr) acc[q] = fmaf(inv[ii[q] + j * n], B[j + jj[q] * n].hi, acc[q]);
#pragma unroll
      for (int q = 0; q < kSolveBatch; ++q)
        if (e0 + q * NT < nr) X[e0 + q * NT] = dw_make(acc[q]);
    }
  }
  bool ok = false;
  for (int round = 0; round < kRefineMax && !ok; ++round) {
    float* rd = red + 2 * (round & 1);
    if (t == 0) rd[0] = rd[1] = 0.f;
    team_sync<NT>();
    // R = B - A X, compensated accumulation (two entries per thread)
    {
      Walk w = walk_start<NT>(t, n);
      for (int e0 = t; e0 < nr; e0 += 2 * NT) {
        int ii[2], jj[2];
        dw_acc acc[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          ii[q] = w.i;
          jj[q] = w.j;
          acc[q] = acc_zero();
          if (e0 + q * NT < nr) acc_add(acc[q], B[e0 + q * NT]);
          walk_next(w);
        }
        const bool two = e0 + NT < nr;
        for (int j = 0; j < n; ++j) {
          acc_fma(acc[0], dw_neg(A[ii[0] + j * n]), X[j + jj[0] * n]);
          if (two) acc_fma(acc[1], dw_neg(A[ii[1] + j * n]), X[j + jj[1] * n]);
        }
        R[e0] = acc_value(acc[0]);
        if (two) R[e0 + NT] = acc_value(acc[1]);
      }
    }
    team_sync<NT>();
    // X += inv * R
    float mdx = 0.f, mx = 0.f;
    {
      Walk w = walk_start<NT>(t, n);
      for (int e0 = t; e0 < nr; e0 += kSolveBatch * NT) {
        int ii[kSolveBatch], jj[kSolveBatch];
        float acc[kSolveBatch];
        dw xv[kSolveBatch];
#pragma unroll
        for (int q = 0; q < kSolveBatch; ++q) {
          ii[q] = w.i;
          jj[q] = w.j;
          acc[q] = 0.f;
          if (e0 + q * NT < nr) xv[q] = X[e0 + q * NT];
          walk_next(w);
        }
        for (int j = 0; j < n; ++j)
#pragma unroll
          for (int q = 0; q < kSolveBatch; ++q)
            if (e0 + q * NT < nr) acc[q] = fmaf(inv[ii[q] + j * n], R[j + jj[q] * n].hi, acc[q]);
#pragma unroll
        for (int q = 0; q < kSolveBatch; ++q) {
          if (e0 + q * NT >= nr) continue;
          const dw xn = dw_add_f(xv[q], acc[q]);
          X[e0 + q * NT] = xn;
          mdx = fmaxf(mdx, (fabsf(acc[q]) <= FLT_MAX) ? fabsf(acc[q]) : INFINITY);
          mx = fmaxf(mx, fabsf(xn.hi));
        }
      }
    }
    // non-negative floats order like their bit patterns
    atomicMax(reinterpret_cast<int*>(rd), __float_as_int(mdx));
    atomicMax(reinterpret_cast<int*>(rd + 1), __float_as_int(mx));
    team_sync<NT>();
    // converged when the correction just applied is negligible, or when the
    // contraction it shows (rho ~ |dX|/|X|) leaves an error of rho^2 |X| <=
    // 1e-10 |X| (refinement converges linearly with rate rho), far below the
    // FP32 rounding of the right-hand side
    ok = rd[0] <= 1e-10f * rd[1] || (round == 0 && rd[0] <= 1e-5f * rd[1]);
  }
  return ok;
}


// refine_solve with the entries of a thread fixed at compile time: NQ of them
// (NT NQ >= n nrhs), the right-hand sides in registers, the products over j
// unrolled by four so that their shared-memory loads are in flight together.
// Every entry is the same chain as in refine_solve, and the maxima that
// decide convergence are the same numbers: the same bits.  Rh: [n nrhs]
// floats (the corrections read the residuals' high parts only).
template <int NT, int NQ>
__device__ inline bool refine_solve_q(const dw* __restrict__ A, int n, const dw* __restrict__ B, dw* X, int nrhs,
                                      const float* __restrict__ inv, float* Rh, float* red) {
  const int t = threadIdx.x, nr = n * nrhs;
  int i[NQ], mo[NQ];  // row, offset of the column
  dw b[NQ], x[NQ];
  {
    Walk w = walk_start<NT>(t, n);
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const bool live = t + q * NT < nr;
      i[q] = live ? w.i : 0;
      mo[q] = live ? w.j * n : 0;
      walk_next(w);
      b[q] = B[live ? t + q * NT : 0];
    }
  }
  // acc[q] = sum_j inv(i, j) v(j), v the high parts of column mo[q] of a dw
  // matrix (stride 2 floats) or a float matrix (stride 1)
  auto apply = [&](const float* v, int stride, float(&acc)[NQ]) {
#pragma unroll
    for (int q = 0; q < NQ; ++q) acc[q] = 0.f;
    int j = 0;
    for (; j + 4 <= n; j += 4)
#pragma unroll
      for (int q = 0; q < NQ; ++q)
#pragma unroll
        for (int u = 0; u < 4; ++u) acc[q] = fmaf(inv[i[q] + (j + u) * n], v[(j + u + mo[q]) * stride], acc[q]);
    for (; j < n; ++j)
#pragma unroll
      for (int q = 0; q < NQ; ++q) acc[q] = fmaf(inv[i[q] + j * n], v[(j + mo[q]) * stride], acc[q]);
  };
  {
    float acc[NQ];
    apply(reinterpret_cast<const float*>(B), 2, acc);
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      x[q] = dw_make(acc[q]);
      if (t + q * NT < nr) X[t + q * NT] = x[q];
    }
  }
  bool ok = false;
  for (int round = 0; round < kRefineMax && !ok; ++round) {
    float* rd = red + 2 * (round & 1);
    if (t == 0) rd[0] = rd[1] = 0.f;
    team_sync<NT>();
    {  // residuals B - A X, compensated
      dw_acc acc[NQ];
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        acc[q] = acc_zero();
        acc_add(acc[q], b[q]);
      }
      int j = 0;
      for (; j + 4 <= n; j += 4)
#pragma unroll
        for (int q = 0; q < NQ; ++q)
#pragma unroll
          for (int u = 0; u < 4; ++u) acc_fma(acc[q], dw_neg(A[i[q] + (j + u) * n]), X[j + u + mo[q]]);
      for (; j < n; ++j)
#pragma unroll
        for (int q = 0; q < NQ; ++q) acc_fma(acc[q], dw_neg(A[i[q] + j * n]), X[j + mo[q]]);
#pragma unroll
      for (int q = 0; q < NQ; ++q)
        if (t + q * NT < nr) Rh[t + q * NT] = acc_value(acc[q]).hi;
    }
    team_sync<NT>();
    float d[NQ], mdx = 0.f, mx = 0.f;
    apply(Rh, 1, d);
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      if (t + q * NT >= nr) continue;
      x[q] = dw_add_f(x[q], d[q]);
      X[t + q * NT] = x[q];
      mdx = fmaxf(mdx, (fabsf(d[q]) <= FLT_MAX) ? fabsf(d[q]) : INFINITY);
      mx = fmaxf(mx, fabsf(x[q].hi));
    }
    // non-negative floats order like their bit patterns
    const int wd = __reduce_max_sync(0xffffffffu, __float_as_int(mdx)),
              wx = __reduce_max_sync(0xffffffffu, __float_as_int(mx));
    if ((t & 31) == 0) {
      atomicMax(reinterpret_cast<int*>(rd), wd);
      atomicMax(reinterpret_cast<int*>(rd + 1), wx);
    }
    team_sync<NT>();
    // the convergence rule of refine_solve
    ok = rd[0] <= 1e-10f * rd[1] || (round == 0 && rd[0] <= 1e-5f * rd[1]);
  }
  return ok;
}

// refine_solve by threads 0 .. NT-1 for n, nrhs <= 64 (res: [n nrhs] dw).  234 solves of
// 16 x 30 entries on the chain of a Gram-Schmidt took 0.6 ms less with refine_solve_q
// than with refine_solve<512>, whose entries are found at run time with an atomic per
// thread; the ALS cluster kernel's solve of 20 x 12 entries by 128 threads takes 7.8 k
// cycles and took 16.3 k.
template <int NT>
__device__ inline bool refine_any(const dw* A, int n, const dw* B, dw* X, int nrhs, const float* inv, dw* res,
                                  float* red) {
  const int nr = n * nrhs;
  float* Rh = reinterpret_cast<float*>(res);
  if (nr <= NT) return refine_solve_q<NT, 1>(A, n, B, X, nrhs, inv, Rh, red);
  if (nr <= 2 * NT) return refine_solve_q<NT, 2>(A, n, B, X, nrhs, inv, Rh, red);
  if (nr <= 4 * NT) return refine_solve_q<NT, 4>(A, n, B, X, nrhs, inv, Rh, red);
  if (nr <= 8 * NT) return refine_solve_q<NT, 8>(A, n, B, X, nrhs, inv, Rh, red);
  return refine_solve<NT>(A, n, B, X, nrhs, inv, res, red);
}

__device__ __forceinline__ dw dw_shfl(dw v, int src) {
  return dw{__shfl_sync(0xffffffffu, v.hi, src), __shfl_sync(0xffffffffu, v.lo, src)};
}

// Shared-memory scratch of solve_cols.
struct ColScratch {
  float* conv;  // [2][32] convergence partials per warp (two rounds in flight)
  float* rmax;  // [16][32] row maxima per warp
  dw* rsum;     // [16][32] row sums of squares per warp
};

// X = A^-1 B for n <= N rows and nrhs <= 16 columns by the first
// solve_cols_warps(n, nrhs) warps of the block, synchronising on named
// barrier 3: the iterative refinement of refine_solve with the rows of the
// FP32 inverse (symmetric, so row i = column i) and of A held in registers
// and the vectors exchanged by shuffles, so that a product costs n shuffles
// and multiply-adds per lane and a round one barrier.  A warp holds H = 32/S
// columns of S >= N lanes each (column m = H w + h; lane h S + i: row i).
// When it converges, the rows of X are normalised as dw_normalise_rows does
// (norms to nrm) and it returns true; otherwise it returns false with X
// untouched.
template <int N, int S>
__device__ inline bool solve_cols(const dw* A, int n, const dw* B, dw* X, int nrhs, const float* inv, dw* nrm,
                                  const ColScratch& s) {
  constexpr int H = 32 / S;
  static_assert(N <= S && S * H == 32, "column layout");
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, h = lane / S, i = lane - h * S, src = h * S;
  const int m = H * w + h, nw = (nrhs + H - 1) / H, nthr = nw * 32;
  const bool row = m < nrhs && i < n;
  float iv[N];
  dw ar[N <= 16 ? N : 1];
#pragma unroll
  for (int j = 0; j < N; ++j) {
    iv[j] = (row && j < n) ? inv[i + j * n] : 0.f;
    if constexpr (N <= 16) ar[j] = (row && j < n) ? A[i + j * n] : dw_make(0.f);
  }
  const dw b = row ? B[i + m * n] : dw_make(0.f);
  float x0 = 0.f;
#pragma unroll
  for (int j = 0; j < N; ++j) x0 = fmaf(iv[j], __shfl_sync(0xffffffffu, b.hi, src + j), x0);
  dw x = dw_make(x0);
  bool ok = false;
  for (int round = 0; round < kRefineMax && !ok; ++round) {
    // r = b - A x (compensated), then the FP32 correction inv r
    dw_acc acc = acc_zero();
    acc_add(acc, b);
#pragma unroll
    for (int j = 0; j < N; ++j) {
      const dw xj = dw_shfl(x, src + j);
      dw aij;
      if constexpr (N <= 16) aij = ar[j];
      else aij = (row && j < n) ? A[i + j * n] : dw_make(0.f);
      acc_fma(acc, dw_neg(aij), xj);
    }
    const dw r = acc_value(acc);
    float d = 0.f;
#pragma unroll
    for (int j = 0; j < N; ++j) d = fmaf(iv[j], __shfl_sync(0xffffffffu, r.hi, src + j), d);
    if (row) x = dw_add_f(x, d);
    float mdx = row ? ((fabsf(d) <= FLT_MAX) ? fabsf(d) : INFINITY) : 0.f;
    float mx = row ? fabsf(x.hi) : 0.f;
    for (int o = 16; o > 0; o >>= 1) {
      mdx = fmaxf(mdx, __shfl_xor_sync(0xffffffffu, mdx, o));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    float* cv = s.conv + (round & 1) * 32;
    if (lane == 0) {
      cv[w] = mdx;
      cv[16 + w] = mx;
    }
    asm volatile("bar.sync 3, %0;" ::"r"(nthr) : "memory");
    float gd = 0.f, gx = 0.f;
    for (int q = 0; q < nw; ++q) {
      gd = fmaxf(gd, cv[q]);
      gx = fmaxf(gx, cv[16 + q]);
    }
    // the convergence rule of refine_solve
    ok = gd <= 1e-10f * gx || (round == 0 && gd <= 1e-5f * gx);
  }
  if (!ok) return false;
  // rows: scale by the largest |x|, sum the squares over the columns
  const int slot = (m < 16 ? m : 15) * 32 + i;
  if (m < nrhs) s.rmax[slot] = fabsf(x.hi);
  asm volatile("bar.sync 3, %0;" ::"r"(nthr) : "memory");
  float big = 0.f;
  for (int q = 0; q < nrhs; ++q) big = fmaxf(big, s.rmax[q * 32 + i]);
  const bool zero = !(big > 0.f);
  const dw il = dw_rcp(dw_make(zero ? 1.f : big));
  const dw y = dw_mul(x, il);
  if (m < nrhs) s.rsum[slot] = dw_mul(y, y);
  asm volatile("bar.sync 3, %0;" ::"r"(nthr) : "memory");
  dw_acc sq = acc_zero();
  for (int q = 0; q < nrhs; ++q) acc_add(sq, s.rsum[q * 32 + i]);
  if (!row) return true;
  if (zero) {  // NaN, as the reference's zero-row norm
    const float nan = __int_as_float(0x7fffffff);
    X[i + m * n] = dw_make(nan);
    if (m == 0) nrm[i] = dw_make(nan);
    return true;
  }
  const dw r = dw_mul(dw_make(big), dw_sqrt(acc_value(sq)));
  X[i + m * n] = dw_mul(x, dw_rcp(r));
  if (m == 0) nrm[i] = r;
  return true;
}

// Warps used by solve_cols_any for an n-row system with nrhs columns.
__host__ __device__ inline int solve_cols_warps(int n, int nrhs) { return n <= 16 ? (nrhs + 1) / 2 : nrhs; }

// solve_cols for n <= 32 (two columns per warp when n <= 16).
__device__ inline bool solve_cols_any(const dw* A, int n, const dw* B, dw* X, int nrhs, const float* inv, dw* nrm,
                                      const ColScratch& s) {
  if (n <= 16) return solve_cols<16, 16>(A, n, B, X, nrhs, inv, nrm, s);
  return solve_cols<32, 32>(A, n, B, X, nrhs, inv, nrm, s);
}

// The sum of two compensated accumulations.
__device__ __forceinline__ dw_acc acc_merge(dw_acc a, dw_acc b) {
  const dw t = two_sum(a.s, b.s);
  return dw_acc{t.hi, f_add(f_add(a.c, b.c), t.lo)};
}

// ---------------------------------------------------------------------------
// Systems of up to 16 rows by a dense double-word inverse
// ---------------------------------------------------------------------------
constexpr int kRowRank = 16;

// Sum over `lanes` (a power of two) neighbouring lanes, in all of them: compensated
// pairs merged without normalising in between (half the chain of dw_add).
template <int lanes>
__device__ __forceinline__ dw lane_sum(dw v) {
  dw_acc a{v.hi, v.lo};
#pragma unroll
  for (int o = lanes / 2; o > 0; o >>= 1)
    a = acc_merge(a, dw_acc{__shfl_xor_sync(0xffffffffu, a.s, o), __shfl_xor_sync(0xffffffffu, a.c, o)});
  return acc_value(a);
}

// One correction of correct_inverse: *big = n max |I - Iv A| before it; none when that is
// above `most`.
template <int RT, bool kFirst>
__device__ __forceinline__ bool correct_round(const dw* A, int n_, const float* gi, dw* Iv, float* Ef, float* emax,
                                              float most, float* big) {
  constexpr int NE = kRowRank * kRowRank / kSolverThreads;
  const int n = RT ? RT : n_, nn = n * n, t = threadIdx.x, lane = t & 31;
  int i[NE], k[NE];
  dw_acc acc[NE];
#pragma unroll
  for (int q = 0; q < NE; ++q) {
    const int p = t + q * kSolverThreads, pl = p < nn ? p : 0;
    k[q] = (unsigned)pl / (unsigned)n;
    i[q] = pl - k[q] * n;
    acc[q] = dw_acc{i[q] == k[q] ? 1.f : 0.f, 0.f};
  }
#pragma unroll 4
  for (int l = 0; l < n; ++l)
#pragma unroll
    for (int q = 0; q < NE; ++q) {
      const dw v = kFirst ? dw_make(-gi[i[q] + l * n]) : dw_neg(Iv[i[q] + l * n]);
      acc_fma(acc[q], v, A[l + k[q] * n]);
    }
  int mx = 0;  // non-negative floats order like their bit patterns, NaN above all
#pragma unroll
  for (int q = 0; q < NE; ++q) {
    const float ev = acc_value(acc[q]).hi;
    if (t + q * kSolverThreads < nn) Ef[i[q] + k[q] * n] = ev;
    mx = max(mx, __float_as_int(fabsf(ev)));
  }
  mx = __reduce_max_sync(0xffffffffu, mx);
  if (lane == 0) emax[t >> 5] = __int_as_float(mx);
  solver_sync();
  *big = n * __int_as_float(__reduce_max_sync(0xffffffffu, __float_as_int(emax[lane & (kSolverWarps - 1)])));
  if (!(*big <= most)) return false;
  float d[NE] = {};
#pragma unroll 4
  for (int l = 0; l < n; ++l)
#pragma unroll
    for (int q = 0; q < NE; ++q) d[q] = fmaf(Ef[i[q] + l * n], kFirst ? gi[l + k[q] * n] : Iv[l + k[q] * n].hi, d[q]);
  dw v[NE];
#pragma unroll
  for (int q = 0; q < NE; ++q) v[q] = dw_add_f(kFirst ? dw_make(gi[i[q] + k[q] * n]) : Iv[i[q] + k[q] * n], d[q]);
  if (!kFirst) solver_sync();
#pragma unroll
  for (int q = 0; q < NE; ++q)
    if (t + q * kSolverThreads < nn) Iv[i[q] + k[q] * n] = v[q];
  return true;
}

// Iv = A^-1 in double-word (threads 0 .. 127, n <= 16; RT: n when known at compile
// time, else 0): the FP32 inverse gi corrected by Iv += (I - Iv A) Iv (Schulz's iteration, the
// residual in double-word).  The first correction squares the residual; the product of a
// correction is FP32, so each later one shrinks it by about the first one's size e0 (the
// FP32 rounding of gi times the condition of A).  Corrections end when the residual e before
// the last has e e0 <= 1e-10, which is then about what it leaves; false when kCorrections do
// not suffice, when the residual does not shrink, or when e0 is above kCorrectable.  The left
// residual is taken so that a solution Iv b has an error of (residual)^2 |x| and (rounding)
// cond |x|.  Ef: [n n], emax: [4] floats.  Ends without a barrier.
//
// kCorrectable is where these solutions stay as good as those of refine_solve or, where that
// gives up, of the LDL^T (random systems of 8 and 16 rows with unit diagonal, condition 1e4 to
// 3e5: errors up to 7e-10 of the solution, at most 2.7 times theirs; 8 times with 2e-2), and it
// takes as many systems as refine_solve.  With 3e-3 and two corrections most of those of
// condition 3e4 went to the LDL^T: 28.6 k cycles for 16 rows against 5.9 k with three
// corrections and 6.8 to 8.5 k with the right-hand sides refined.
constexpr int kCorrections = 5;
constexpr float kCorrectable = 1.5e-2f;  // n max |I - gi A| up to which the corrections are tried
template <int RT>
__device__ inline bool correct_inverse(const dw* A, int n, const float* gi, dw* Iv, float* Ef, float* emax) {
  float first;
  if (!correct_round<RT, true>(A, n, gi, Iv, Ef, emax, kCorrectable, &first)) return false;
  float big = first;
  for (int round = 1; first * big > 1e-10f; ++round) {
    if (round == kCorrections) return false;
    solver_sync();
    if (!correct_round<RT, false>(A, n, gi, Iv, Ef, emax, 0.25f * big, &big)) return false;
  }
  return true;
}

// A row of X = Iv B by one warp: iv points at the row (entries ld apart), B is [n][nj].
// NC columns per lane, or (NC = 0, nj <= 16) one column with its sum split over the
// half-warps; columns beyond nj are 0.  Without `solved` the row is read from xr (entries
// ld apart) instead.
template <int RT, int NC>
__device__ __forceinline__ void row_product(const dw* iv, int ld, const dw* B, int nj, bool solved, const dw* xr, dw* x) {
  constexpr bool split = NC == 0;
  const int lane = threadIdx.x & 31, h = split ? lane >> 4 : 0, m0 = split ? lane & 15 : lane;
#pragma unroll
  for (int q = 0; q < (split ? 1 : NC); ++q) {
    const int m = m0 + 32 * q, ml = m < nj ? m : 0;
    if (solved) {
      dw_acc acc = acc_zero();
#pragma unroll
      for (int u = 0; u < (split ? kRowRank / 2 : kRowRank); ++u) {
        const int k = h * (kRowRank / 2) + u;
        if (RT == kRowRank || k < ld) acc_fma(acc, iv[k * ld], B[k * nj + ml]);
      }
      if (split)
        acc = acc_merge(acc, dw_acc{__shfl_xor_sync(0xffffffffu, acc.s, 16), __shfl_xor_sync(0xffffffffu, acc.c, 16)});
      x[q] = m < nj ? acc_value(acc) : dw_make(0.f);
    } else {
      x[q] = m < nj ? xr[m * ld] : dw_make(0.f);
    }
  }
}

// The row (as row_product leaves it) scaled to unit norm, its norm to *nrm.  Scaled by a
// power of two first, as normonebase scales by the largest entry; a zero row gives
// NaN, as there.
template <int NC>
__device__ __forceinline__ void row_normalise(dw* x, dw* nrm) {
  constexpr int N = NC == 0 ? 1 : NC;
  float big = 0.f;
#pragma unroll
  for (int q = 0; q < N; ++q) big = fmaxf(big, fabsf(x[q].hi));
  const int bits = __reduce_max_sync(0xffffffffu, __float_as_int(big)), ex = bits >> 23;
  const bool scaled = ex > 0 && ex < 254;
  const float sc = scaled ? __int_as_float((254 - ex) << 23) : 1.f, back = scaled ? __int_as_float(ex << 23) : 1.f;
  dw_acc sq = acc_zero();
#pragma unroll
  for (int q = 0; q < N; ++q) {
    x[q] = dw_make(x[q].hi * sc, x[q].lo * sc);
    acc_fma(sq, x[q], x[q]);
  }
  const dw sum = NC == 0 ? lane_sum<16>(acc_value(sq)) : lane_sum<32>(acc_value(sq));
  dw r = dw_sqrt(sum), rcp = dw_rcp(r);
  if (!(bits > 0 && sum.hi > 0.f)) r = rcp = dw_make(__int_as_float(0x7fffffff));
#pragma unroll
  for (int q = 0; q < N; ++q) x[q] = dw_mul(x[q], rcp);
  *nrm = dw_make(r.hi * back, r.lo * back);
}

}  // namespace dwsolve
}  // namespace mlcp
