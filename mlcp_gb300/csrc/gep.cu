// Block Rayleigh-Ritz step of the intertwined cycle (reference
// GenEigvalProblem, src/intertw_mvp.cu:589-654, and solve_geneigval,
// src/linalg.cu:22-69, cusolverDnDsygvd with itype 1, jobz V, lower).
//
//  * gep_inner_kernel: A(i,j) = <Q_j, (HQ)_i>, S(i,j) = <Q_j, Q_i> for j <= i,
//    full CP inner products in FP64 (one CTA per pair).
//  * gep_solve_launch: the generalised eigenproblem as a short sequence of
//    phases over a workspace in global memory (L2-resident: 160 vectors at
//    most).  S = L L^T and C = L^-1 A L^-T in FP64; eigenvectors of C by
//    parallel cyclic Jacobi in FP32, then refined in FP64 by iterations of
//    matrix products (Ogita and Aishima, Japan J. Indust. Appl. Math. 35
//    (2018) 1007-1035): with G = V^T V and S = V^T C V,
//      lambda_i = S_ii / G_ii,  m = (lambda_i + lambda_j) / 2,
//      E_ij = (S_ij - m G_ij) / (lambda_j - lambda_i) - G_ij / 2,  E_ii = (1 - G_ii) / 2,
//      V <- V + V E,
//    which squares the error of V each time.  The quotient is antisymmetric to the
//    last bit, so nearly equal levels cannot cost orthogonality through its rounding.  Pairs
//    whose quotient would pass a bound (1e-3, 1e-5, 1e-8 in the three iterations) are
//    rotated apart first, by FP64 Jacobi rotations of those pairs alone: a level close to
//    another on the scale of the FP32 error in the first iteration, on the scale of the
//    couplings of second order through third levels, which the iteration before
//    has left, in the others.  Rotations are orthogonal whatever their angle, so after
//    the last iteration V is off by the square of 1e-8.  A pair above the bound whose coupling
//    is below 2^-51 of the largest level is left as it is: that is rounding.  On shells
//    of equal levels split by 1e-6 to 1e-14, on several scales at once, residuals and
//    orthogonality end at a few eps (with one separation at 1e-3, in the first
//    iteration only, they ended at 1e-11).  The FP64 stage
//    matters: the vector updates combine the block with the eigenvectors,
//    and for nearly degenerate states (the benchmark block has relative gaps
//    of 4e-5) FP32 eigenvectors are off by ~1e-7 / gap, which moved the
//    updated vectors by 1e-5 against the reference's FP64 sygvd.  X = L^-T V
//    with unit columns of V.  Eigenpairs are returned in ascending order, each
//    eigenvector with its largest-magnitude entry positive.
//
// What bounds it: FP64 issues one warp instruction per SM in 17-19 cycles, so
// FP64 work has to be spread over the SMs and kept to matrix products; the
// sequential parts (Cholesky, the Jacobi rounds) are chains of barriers.  One
// CTA that did everything in global memory, with FP64 Jacobi sweeps (and
// 16-way bank conflicts in the FP32 ones), took 36.0 ms for 144 vectors and
// 1.36 ms for 40; the phases take 1.6 ms and 0.32 ms.  Of the 1.6 ms the FP32
// Jacobi rounds are 0.78, the Cholesky 0.28, the three triangular solves 0.22,
// the rotation replay 0.10 and the matrix products (eleven launches) 0.17; the three
// separations are launches of 2 us while there is nothing to separate.  Clustered levels pay for
// theirs: 40 levels in shells split by 1e-6 to 1e-12 0.6 to 1.9 ms more (2.1 to 2.6 ms in all when
// FP64 sweeps rotated every pair, 1.2 to 2.5 now), 144 levels of two ladders split by 1e-5 to 1e-9
// 7 to 11 ms more (74 to 84 in all then, 10 to 15 now).
#include <algorithm>
#include <cfloat>

#include "common.cuh"
#include "intertwine.cuh"

namespace mlcp {

namespace {
constexpr int kPairThreads = 128;
constexpr int kPairTile = 32, kPairLd = kPairTile + 1;
constexpr int kMaxBasisPair = 64;  // basis sizes of a cycle
}

// One CTA per pair (i, j <= i): 8 NA x 16 NB tiles of (r, s), a mode's factors of the tile
// staged in shared memory (transposed), NA NB entries of both products a thread (rows
// r0 + ty + 8 a, columns s0 + tx + 16 b).  FP64-bound then: 100 vectors of rank 30 on
// 6 x 48 take 5.1 ms (9.5 with an entry at a time from global memory; 4.9 at the
// FP64 pipe's rate), 40 of rank 16 on 3 x 30 88 us (83; 70).
template <int NA, int NB>
__global__ void __launch_bounds__(kPairThreads) gep_inner_kernel(GepParams p) {
  // pair index -> (i, j), j <= i
  const int e = blockIdx.x;
  int i = (int)((sqrt(8.0 * e + 1.0) - 1.0) / 2.0);
  while ((i + 1) * (i + 2) / 2 <= e) ++i;
  while (i * (i + 1) / 2 > e) --i;
  const int j = e - i * (i + 1) / 2;
  const int R = p.R, D = p.D, nD = p.nD;
  const double* qj = p.q_base + (size_t)j * R * nD;
  const double* qjc = p.q_coef + (size_t)j * R;
  const double* qi = p.q_base + (size_t)i * R * nD;
  const double* qic = p.q_coef + (size_t)i * R;
  const double* hi = p.hq_base + (size_t)i * R * nD;
  const double* hic = p.hq_coef + (size_t)i * R;
  constexpr int TR = 8 * NA, TS = 16 * NB;
  extern __shared__ double gi_sm[];
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  double accA = 0.0, accS = 0.0;
  for (int r0 = 0; r0 < R; r0 += TR)
    for (int s0 = 0; s0 < R; s0 += TS) {
      double pa[NA][NB], ps[NA][NB];
#pragma unroll
      for (int a = 0; a < NA; ++a)
#pragma unroll
        for (int b = 0; b < NB; ++b) {
          const int r = r0 + ty + 8 * a, s = s0 + tx + 16 * b;
          const bool live = r < R && s < R;
          pa[a][b] = live ? qjc[r] * hic[s] : 0.0;
          ps[a][b] = live ? qjc[r] * qic[s] : 0.0;
        }
      int o = 0;
      for (int d = 0; d < D; ++d) {
        const int n = p.nbas[d];
        double *X = gi_sm, *H = X + n * kPairLd, *Q = H + n * kPairLd;
        __syncthreads();
        for (int e2 = threadIdx.x; e2 < (TR > TS ? TR : TS) * n; e2 += kPairThreads) {
          const int t = e2 / n, q = e2 - t * n;
          const bool lr = t < TR && r0 + t < R, ls = t < TS && s0 + t < R;
          X[q * kPairLd + t] = lr ? qj[(size_t)(r0 + t) * nD + o + q] : 0.0;
          H[q * kPairLd + t] = ls ? hi[(size_t)(s0 + t) * nD + o + q] : 0.0;
          Q[q * kPairLd + t] = ls ? qi[(size_t)(s0 + t) * nD + o + q] : 0.0;
        }
        __syncthreads();
        double ta[NA][NB] = {}, ts[NA][NB] = {};
        for (int q = 0; q < n; ++q) {
          double h[NB], y[NB];
#pragma unroll
          for (int b = 0; b < NB; ++b) {
            h[b] = H[q * kPairLd + tx + 16 * b];
            y[b] = Q[q * kPairLd + tx + 16 * b];
          }
#pragma unroll
          for (int a = 0; a < NA; ++a) {
            const double x = X[q * kPairLd + ty + 8 * a];
#pragma unroll
            for (int b = 0; b < NB; ++b) {
              ta[a][b] = fma(x, h[b], ta[a][b]);
              ts[a][b] = fma(x, y[b], ts[a][b]);
            }
          }
        }
#pragma unroll
        for (int a = 0; a < NA; ++a)
#pragma unroll
          for (int b = 0; b < NB; ++b) {
            pa[a][b] *= ta[a][b];
            ps[a][b] *= ts[a][b];
          }
        o += n;
      }
#pragma unroll
      for (int a = 0; a < NA; ++a)
#pragma unroll
        for (int b = 0; b < NB; ++b) {
          accA += pa[a][b];
          accS += ps[a][b];
        }
    }
  __shared__ double ra[kPairThreads], rs_[kPairThreads];
  ra[threadIdx.x] = accA;
  rs_[threadIdx.x] = accS;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) {
      ra[threadIdx.x] += ra[threadIdx.x + w];
      rs_[threadIdx.x] += rs_[threadIdx.x + w];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    p.A[i + (size_t)j * p.nbloc] = ra[0];
    p.S[i + (size_t)j * p.nbloc] = rs_[0];
  }
}

namespace {

constexpr int kMaxB = 160;          // vectors of a block (shared memory of the Cholesky phase)
constexpr int kMaxQ = kMaxB / 32;   // rows per lane of a warp-held column
constexpr int kJacobiSweeps = 30;
constexpr int kVRows = 4;           // rows of V per CTA of the rotation replay
constexpr int kReplay = 8;          // rounds of rotations loaded together
constexpr int kIterations = 3;      // of the refinement
constexpr int kSeparateSweeps = 40;
// Pairs whose quotient is above this are separated by rotations first.
__host__ __device__ constexpr double unsafe_bound(int iteration) {
  return iteration == 0 ? 1.0e-3 : iteration == 1 ? 1.0e-5 : 1.0e-8;
}

// Workspace of the phases (doubles): L, L^T, C, W, V, V', G, S, E [B][B];
// invd [B]; the FP32 Jacobi's rotations; counters.
struct GepWork {
  double *L, *LT, *C, *W, *V, *V2, *G, *S, *E, *invd;
  double* floor;  // [1] couplings that are rounding: 2^-51 of the largest level
  float2* rot;  // [sweeps][Bp - 1][Bp / 2] (c, s)
  int* cnt;     // [0] Jacobi sweeps, [1] unsafe pairs seen in this iteration
};

__host__ __device__ inline int gep_pad(int B) { return (B + 1) / 2 * 2; }

__host__ __device__ inline size_t gep_carve(int B, double* base, GepWork* w) {
  const size_t bb = (size_t)B * B, Bp = gep_pad(B);
  size_t o = 0;
  auto take = [&](size_t n) -> double* {
    double* r = base ? base + o : nullptr;
    o += n;
    return r;
  };
  w->L = take(bb);
  w->LT = take(bb);
  w->C = take(bb);
  w->W = take(bb);
  w->V = take(bb);
  w->V2 = take(bb);
  w->G = take(bb);
  w->S = take(bb);
  w->E = take(bb);
  w->invd = take(B);
  w->floor = take(1);
  w->rot = reinterpret_cast<float2*>(take((size_t)kJacobiSweeps * (Bp - 1) * (Bp / 2)));
  w->cnt = reinterpret_cast<int*>(take(1));
  return o;
}

// Pair k of round `round` of the round-robin schedule over Bp (even)
// indices: (Bp-1, round) for k = 0, else ((round+k), (round-k)) mod Bp-1,
// smaller index first.
__device__ __forceinline__ void robin_pair(int Bp, int round, int k, int* a, int* b) {
  const int m = Bp - 1;
  int x, y;
  if (k == 0) {
    x = m;
    y = round;
  } else {
    x = round + k;
    if (x >= m) x -= m;
    y = round - k;
    if (y < 0) y += m;
  }
  *a = min(x, y);
  *b = max(x, y);
}

// Rotation (c, s) zeroing the (p,q) entry of a symmetric 2x2 block.
__device__ __forceinline__ void jacobi_rotation(float app, float aqq, float apq, float* c, float* s) {
  if (apq == 0.f) {
    *c = 1.f;
    *s = 0.f;
    return;
  }
  const float theta = (aqq - app) / (2.f * apq);
  const float t = copysignf(1.f, theta) / (fabsf(theta) + sqrtf(theta * theta + 1.f));
  *c = rsqrtf(t * t + 1.f);
  *s = t * *c;
}

// ---- Phases.  Each is run by CTA `cta` of `ncta`; a phase boundary is a
// kernel boundary, or a block barrier when one CTA runs them all. ----

// S = L L^T (lower triangle of S), one CTA, L in shared memory.  Warp 0 forms
// the next pivot (FP64 square root and division, ~1300 cycles) while the
// other warps run the trailing update.
__device__ void phase_cholesky(const GepParams& p, const GepWork& w, unsigned char* smem) {
  const int B = p.nbloc, tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
  double* L = reinterpret_cast<double*>(smem);  // [B][B] column-major
  double* inv_s = L + (size_t)B * B;            // [B]
  __shared__ int info;
  for (int e = tid; e < B * B; e += nt) {
    const int r = e % B, c = e / B;
    L[e] = (r >= c) ? p.S[e] : 0.0;
  }
  if (tid == 0) info = 0;
  if (tid < 2) w.cnt[tid] = 0;
  __syncthreads();
  auto pivot = [&](int j, double d) {
    if (!(d > 0.0)) {
      info = j + 1;
      d = fabs(d) + 1e-300;
    }
    const double l = sqrt(d);
    L[j + (size_t)j * B] = l;
    inv_s[j] = 1.0 / l;
  };
  if (tid == 0) pivot(0, L[0]);
  __syncthreads();
  for (int j = 0; j < B; ++j) {
    const double inv = inv_s[j];
    for (int i = j + 1 + tid; i < B; i += nt) L[i + (size_t)j * B] *= inv;
    __syncthreads();
    if (j + 1 < B) {
      if (warp == 0) {
        if (lane == 0) {
          const double x = L[j + 1 + (size_t)j * B];
          pivot(j + 1, fma(-x, x, L[j + 1 + (size_t)(j + 1) * B]));
        }
      } else {
        for (int c = j + warp; c < B; c += nw - 1) {
          const double x = L[c + (size_t)j * B];
          for (int i = c + lane; i < B; i += 32)
            if (i != j + 1) L[i + (size_t)c * B] = fma(-L[i + (size_t)j * B], x, L[i + (size_t)c * B]);
        }
      }
    }
    __syncthreads();
  }
  for (int e = tid; e < B * B; e += nt) {
    const int r = e % B, c = e / B;
    w.L[e] = L[e];
    w.LT[e] = L[c + (size_t)r * B];
  }
  for (int i = tid; i < B; i += nt) w.invd[i] = inv_s[i];
  if (tid == 0 && info) atomicOr(p.status, 2);
}

// One column of L^-1 X, held by a warp: lane `lane` has rows lane + 32 q.
__device__ __forceinline__ void warp_forward(const double* L, const double* invd, int B, double (&x)[kMaxQ],
                                             int lane) {
  double l[kMaxQ];
#pragma unroll
  for (int q = 0; q < kMaxQ; ++q) l[q] = lane + 32 * q < B ? L[lane + 32 * q] : 0.0;
#pragma unroll
  for (int q = 0; q < kMaxQ; ++q) {
    for (int jj = 0; jj < 32; ++jj) {
      const int j = 32 * q + jj;
      if (j >= B) break;
      double cur[kMaxQ];  // column j of L; the next column is fetched while it is used
#pragma unroll
      for (int q2 = 0; q2 < kMaxQ; ++q2) cur[q2] = l[q2];
      if (j + 1 < B)
#pragma unroll
        for (int q2 = q; q2 < kMaxQ; ++q2)
          if (lane + 32 * q2 < B) l[q2] = L[lane + 32 * q2 + (size_t)(j + 1) * B];
      const double v = __shfl_sync(0xffffffffu, x[q], jj) * invd[j];
      if (lane == jj) x[q] = v;
#pragma unroll
      for (int q2 = q; q2 < kMaxQ; ++q2)
        if (lane + 32 * q2 > j) x[q2] = fma(-cur[q2], v, x[q2]);
    }
  }
}

// W = L^-1 A (second = false, A from its lower triangle), then C = W L^-T as
// the columns of L^-1 W^T (second = true); one warp per column.
__device__ void phase_reduce(const GepParams& p, const GepWork& w, bool second, int cta, int ncta) {
  const int B = p.nbloc, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (int c = cta * nw + (threadIdx.x >> 5); c < B; c += ncta * nw) {
    double x[kMaxQ];
#pragma unroll
    for (int q = 0; q < kMaxQ; ++q) {
      const int r = lane + 32 * q;
      x[q] = 0.0;
      if (r < B) x[q] = second ? w.W[c + (size_t)r * B] : (r >= c ? p.A[r + (size_t)c * B] : p.A[c + (size_t)r * B]);
    }
    warp_forward(w.L, w.invd, B, x, lane);
    double* out = (second ? w.C : w.W) + (size_t)c * B;
#pragma unroll
    for (int q = 0; q < kMaxQ; ++q)
      if (lane + 32 * q < B) out[lane + 32 * q] = x[q];
  }
}

// FP32 cyclic Jacobi on C, one CTA, C in shared memory.  The rotations go to
// w.rot; the eigenvectors are formed afterwards by phase_replay, whose rows
// are independent.  A round updates every 2 x 2 block (pair k, pair l) of the
// upper half and mirrors it, each block owned by one thread, with an odd
// leading dimension so that neither access conflicts.
__device__ void phase_jacobi(const GepParams& p, const GepWork& w, unsigned char* smem) {
  const int B = p.nbloc, Bp = gep_pad(B), ld = Bp + 1, np = Bp / 2, tri = np * (np + 1) / 2;
  const int tid = threadIdx.x, nt = blockDim.x;
  float* C = reinterpret_cast<float*>(smem);  // [Bp][ld]
  float* rc = C + (size_t)Bp * ld;            // [np] cosines, then [np] sines
  float* rs = rc + np;
  int* pa = reinterpret_cast<int*>(rs + np);  // [np] pair members
  int* pb = pa + np;
  __shared__ float red[2][32];
  __shared__ int big[32];
  // scaled by the power of two that brings the largest entry to about one: FP32 then holds the
  // entries and the sums of their squares whatever the unit of H, and the rotations, which
  // are free of the scale, keep their bits.  (High words: they order like the magnitudes, and
  // the FP64 pipe is left alone.)
  int most = 0;
  for (int e = tid; e < B * B; e += nt) most = max(most, __double2hiint(w.C[e]) & 0x7fffffff);
  most = __reduce_max_sync(0xffffffffu, most);
  if (tid % 32 == 0) big[tid / 32] = most;
  __syncthreads();
  for (int q = 0; q < nt / 32; ++q) most = max(most, big[q]);
  const int ex = most >> 20;  // biased exponent; 2047: not finite, 0: zero (or nearly)
  const bool scaled = ex > 0 && ex < 2047;
  const double half = scaled ? ldexp(0.5, 1023 - max(ex, 24)) : 0.5, unit = scaled ? ldexp(1.0, max(ex, 24) - 1023) : 1.0;
  for (int e = tid; e < Bp * Bp; e += nt) {
    const int r = e % Bp, c = e / Bp;
    C[r + (size_t)c * ld] =
        r < B && c < B ? (float)(half * (w.C[r + (size_t)c * B] + w.C[c + (size_t)r * B])) : 0.f;
  }
  // the blocks of this thread, the same in every round (pairs k <= l)
  constexpr int kItems = 4;
  int ik[kItems], il[kItems];
#pragma unroll
  for (int q = 0; q < kItems; ++q) {
    const int e = tid + q * nt;
    ik[q] = -1;
    il[q] = 0;
    if (e < tri) {
      int l = (int)((sqrtf(8.f * e + 1.f) - 1.f) * 0.5f);
      while ((l + 1) * (l + 2) / 2 <= e) ++l;
      while (l * (l + 1) / 2 > e) --l;
      il[q] = l;
      ik[q] = e - l * (l + 1) / 2;
    }
  }
  __syncthreads();
  int sweep = 0;
  for (; sweep < kJacobiSweeps; ++sweep) {
    // until the off-diagonal mass is 1e-12 of the diagonal's
    float off = 0.f, dia = 0.f;
    for (int e = tid; e < Bp * Bp; e += nt) {
      const int r = e % Bp, c = e / Bp;
      const float v = C[r + (size_t)c * ld];
      if (r == c) dia = fmaf(v, v, dia); else off = fmaf(v, v, off);
    }
    for (int o = 16; o > 0; o >>= 1) {
      off += __shfl_xor_sync(0xffffffffu, off, o);
      dia += __shfl_xor_sync(0xffffffffu, dia, o);
    }
    __syncthreads();
    if (tid % 32 == 0) {
      red[0][tid / 32] = off;
      red[1][tid / 32] = dia;
    }
    __syncthreads();
    float offt = 0.f, diat = 0.f;
    for (int q = 0; q < nt / 32; ++q) {
      offt += red[0][q];
      diat += red[1][q];
    }
    if (offt <= 1e-12f * diat || offt == 0.f) break;
    for (int round = 0; round < Bp - 1; ++round) {
      for (int k = tid; k < np; k += nt) {
        int a, b;
        robin_pair(Bp, round, k, &a, &b);
        float c, s;
        jacobi_rotation(C[a + (size_t)a * ld], C[b + (size_t)b * ld], C[a + (size_t)b * ld], &c, &s);
        pa[k] = a;
        pb[k] = b;
        rc[k] = c;
        rs[k] = s;
        w.rot[((size_t)sweep * (Bp - 1) + round) * np + k] = make_float2(c, s);
      }
      __syncthreads();
#pragma unroll
      for (int q = 0; q < kItems; ++q) {
        const int k = ik[q], l = il[q];
        if (k < 0) continue;
        const int ak = pa[k], bk = pb[k], al = pa[l], bl = pb[l];
        const float ck = rc[k], sk = rs[k], cl = rc[l], sl = rs[l];
        const float x00 = C[ak + (size_t)al * ld], x01 = C[ak + (size_t)bl * ld], x10 = C[bk + (size_t)al * ld],
                    x11 = C[bk + (size_t)bl * ld];
        const float y00 = ck * x00 - sk * x10, y10 = sk * x00 + ck * x10;  // rows: J_k^T
        const float y01 = ck * x01 - sk * x11, y11 = sk * x01 + ck * x11;
        const float z00 = cl * y00 - sl * y01, z01 = sl * y00 + cl * y01;  // columns: J_l
        const float z10 = cl * y10 - sl * y11, z11 = sl * y10 + cl * y11;
        C[ak + (size_t)al * ld] = z00;
        C[bk + (size_t)bl * ld] = z11;
        if (k == l) {
          C[ak + (size_t)bl * ld] = 0.f;
          C[bk + (size_t)al * ld] = 0.f;
        } else {
          C[ak + (size_t)bl * ld] = z01;
          C[bk + (size_t)al * ld] = z10;
          C[al + (size_t)ak * ld] = z00;
          C[bl + (size_t)ak * ld] = z01;
          C[al + (size_t)bk * ld] = z10;
          C[bl + (size_t)bk * ld] = z11;
        }
      }
      __syncthreads();
    }
  }
  float top = 0.f;
  for (int i = tid; i < B; i += nt) top = fmaxf(top, fabsf(C[i + (size_t)i * ld]));
  for (int o = 16; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
  __syncthreads();
  if (tid % 32 == 0) red[0][tid / 32] = top;
  __syncthreads();
  if (tid == 0) {
    for (int q = 1; q < nt / 32; ++q) top = fmaxf(top, red[0][q]);
    *w.floor = (double)top * unit * (2.0 * DBL_EPSILON);
    w.cnt[0] = sweep;
  }
}

// V = the product of the recorded rotations, kVRows rows per CTA in shared
// memory, one (row, pair) per thread; rotations of kReplay rounds are loaded
// together.
__device__ void phase_replay(const GepParams& p, const GepWork& w, unsigned char* smem, int cta, int ncta) {
  const int B = p.nbloc, Bp = gep_pad(B), np = Bp / 2, tid = threadIdx.x, nt = blockDim.x;
  float* V = reinterpret_cast<float*>(smem);  // [kVRows][Bp]
  const int rounds = w.cnt[0] * (Bp - 1), k = tid % np, r = tid / np;
  for (int r0 = cta * kVRows; r0 < B; r0 += ncta * kVRows) {
    for (int e = tid; e < kVRows * Bp; e += nt) V[e] = (e % Bp == r0 + e / Bp) ? 1.f : 0.f;
    __syncthreads();
    for (int base = 0; base < rounds; base += kReplay) {
      float2 cs[kReplay];
#pragma unroll
      for (int u = 0; u < kReplay; ++u)
        cs[u] = r < kVRows && base + u < rounds ? w.rot[(size_t)(base + u) * np + k] : make_float2(1.f, 0.f);
#pragma unroll
      for (int u = 0; u < kReplay; ++u) {
        if (base + u >= rounds) break;
        if (r < kVRows) {
          int a, b;
          robin_pair(Bp, (base + u) % (Bp - 1), k, &a, &b);
          const float va = V[r * Bp + a], vb = V[r * Bp + b];
          V[r * Bp + a] = cs[u].x * va - cs[u].y * vb;
          V[r * Bp + b] = cs[u].y * va + cs[u].x * vb;
        }
        __syncthreads();
      }
    }
    for (int e = tid; e < kVRows * B; e += nt) {
      const int c = e / kVRows, q = e % kVRows;
      if (r0 + q < B) w.V[r0 + q + (size_t)c * B] = (double)V[q * Bp + c];
    }
    __syncthreads();
  }
}

// out = f(op(X) Y), FP64, 8 x 8 tiles of a 64-thread CTA, k in chunks of 32
// through shared memory.  op: transpose when `tx`.
//   kPlain: the product;  kNewton: 1.5 Y' - 0.5 (product), Y' = X (so X (3 I - G) / 2);
//   kAdd: X + product.
enum : int { kPlain = 0, kNewton = 1, kAdd = 2 };
constexpr int kTile = 8, kChunk = 32;

__device__ void phase_product(const double* X, const double* Y, double* out, int B, bool tx, int form, int cta,
                              int ncta, unsigned char* smem) {
  double(*xs)[kChunk + 1] = reinterpret_cast<double(*)[kChunk + 1]>(smem);  // [row of op(X)][k]
  double(*ys)[kChunk + 1] = xs + kTile;                                      // [column of Y][k]
  const int t = threadIdx.x, nb = (B + kTile - 1) / kTile, r = t % kTile, c = t / kTile;
  for (int tile = cta; tile < nb * nb; tile += ncta) {
    const int r0 = tile % nb * kTile, c0 = tile / nb * kTile;
    double acc = 0.0;
    for (int k0 = 0; k0 < B; k0 += kChunk) {
#pragma unroll
      for (int u = 0; u < kTile * kChunk / 64; ++u) {
        const int e = t + 64 * u;
        // along the contiguous index of each operand: k (X^T, Y) or the row (X)
        const int i = tx ? e / kChunk : e % kTile, k = tx ? e % kChunk : e / kTile;
        xs[i][k] = r0 + i < B && k0 + k < B
                       ? (tx ? X[k0 + k + (size_t)(r0 + i) * B] : X[r0 + i + (size_t)(k0 + k) * B])
                       : 0.0;
        ys[e / kChunk][e % kChunk] = c0 + e / kChunk < B && k0 + e % kChunk < B
                                         ? Y[k0 + e % kChunk + (size_t)(c0 + e / kChunk) * B]
                                         : 0.0;
      }
      __syncthreads();
      const int kn = min(kChunk, B - k0);
      for (int k = 0; k < kn; ++k) acc = fma(xs[r][k], ys[c][k], acc);
      __syncthreads();
    }
    const int row = r0 + r, col = c0 + c;
    if (row < B && col < B) {
      const size_t e = row + (size_t)col * B;
      out[e] = form == kPlain ? acc : form == kNewton ? 1.5 * X[e] - 0.5 * acc : X[e] + acc;
    }
  }
}

// The coupling of levels i and j in the metric G, S_ij - (lambda_i + lambda_j) / 2 G_ij.
__device__ __forceinline__ double coupling(double sij, double sji, double gij, double li, double lj) {
  return 0.5 * (sij + sji) - 0.5 * (li + lj) * gij;
}

// E_ij of one iteration from the coupling and the levels; *unsafe: the pair wants a rotation.
__device__ __forceinline__ double correction(double num, double gap, double gij, double bound, double floor, bool* unsafe) {
  double x = -0.5 * gij;
  *unsafe = false;
  if (fabs(num) <= bound * fabs(gap) && gap != 0.0) x += num / gap;
  else if (fabs(num) > floor) *unsafe = true;
  return x;
}

// E of iteration `it`; records in cnt[1] that there are pairs to be separated.
__device__ void phase_correction(const GepWork& w, int B, int it, int cta, int ncta) {
  const double bound = unsafe_bound(it), floor = *w.floor;
  for (int e = cta * blockDim.x + threadIdx.x; e < B * B; e += ncta * blockDim.x) {
    const int i = e % B, j = e / B;
    const double g = w.G[e];
    if (i == j) {
      w.E[e] = 0.5 * (1.0 - g);
      continue;
    }
    const double li = w.S[i + (size_t)i * B] / w.G[i + (size_t)i * B], lj = w.S[j + (size_t)j * B] / w.G[j + (size_t)j * B];
    bool unsafe;
    w.E[e] = correction(coupling(w.S[e], w.S[j + (size_t)i * B], g, li, lj), lj - li, g, bound, floor, &unsafe);
    if (unsafe) w.cnt[1] = 1;
  }
}

// The separation of unsafe pairs (one CTA; nothing to do unless cnt[1]): cyclic Jacobi
// sweeps in FP64 that rotate only those pairs, S and the levels in shared memory, G and V
// in global memory, until no pair is unsafe; then E from the rotated S and G.  A sweep
// looks at every pair first and visits only the rounds that hold an unsafe one.
__device__ void phase_separate(const GepWork& w, int B, int it, unsigned char* smem) {
  const bool any = w.cnt[1] != 0;
  __syncthreads();  // read by all before it is cleared
  if (!any) return;
  const int Bp = gep_pad(B), np = Bp / 2, m = Bp - 1, tid = threadIdx.x, nt = blockDim.x;
  const double bound = unsafe_bound(it), floor = *w.floor;
  double* S = reinterpret_cast<double*>(smem);  // [B][B]
  double* lev = S + (size_t)B * B;              // [B] the levels S_ii / G_ii
  double* rc = lev + B;                         // [np] cosines, then [np] sines
  double* rs = rc + np;
  int* round_hit = reinterpret_cast<int*>(rs + np);  // [Bp] rounds with an unsafe pair
  for (int e = tid; e < B * B; e += nt) {
    const int i = e % B, j = e / B;
    S[e] = 0.5 * (w.S[e] + w.S[j + (size_t)i * B]);
  }
  __syncthreads();
  for (int i = tid; i < B; i += nt) lev[i] = S[i + (size_t)i * B] / w.G[i + (size_t)i * B];
  for (int sweep = 0; sweep < kSeparateSweeps; ++sweep) {
    for (int r = tid; r < Bp; r += nt) round_hit[r] = 0;
    __syncthreads();
    bool mine = false;
    for (int e = tid; e < B * B; e += nt) {
      const int i = e % B, j = e / B;
      if (i >= j) continue;
      bool unsafe;
      correction(coupling(S[e], S[e], w.G[e], lev[i], lev[j]), lev[j] - lev[i], w.G[e], bound, floor, &unsafe);
      if (!unsafe) continue;
      mine = true;
      // the round of robin_pair that holds (i, j): j = m meets i in round i, else the
      // round's double is i + j modulo the odd m
      const int sum = i + j;
      round_hit[j == m ? i : (sum % 2 ? sum + m : sum) / 2 % m] = 1;
    }
    if (!__syncthreads_or(mine)) break;
    for (int round = 0; round < m; ++round) {
      if (!round_hit[round]) continue;
      for (int k = tid; k < np; k += nt) {
        int a, b;
        robin_pair(Bp, round, k, &a, &b);
        double c = 1.0, s = 0.0;
        if (b < B) {  // index Bp - 1 = B is padding when B is odd
          const size_t ab = a + (size_t)b * B;
          const double num = coupling(S[ab], S[ab], w.G[ab], lev[a], lev[b]), gap = lev[b] - lev[a];
          bool unsafe;
          correction(num, gap, w.G[ab], bound, floor, &unsafe);
          if (unsafe) {
            const double theta = gap / (2.0 * num);
            const double t = copysign(1.0, theta) / (fabs(theta) + sqrt(theta * theta + 1.0));
            c = 1.0 / sqrt(t * t + 1.0);
            s = t * c;
          }
        }
        rc[k] = c;
        rs[k] = s;
      }
      __syncthreads();
      auto rotate = [&](double* x, double* y, int k) {
        const double c = rc[k], s = rs[k], xa = *x, xb = *y;
        *x = c * xa - s * xb;
        *y = s * xa + c * xb;
      };
      for (int e = tid; e < np * B; e += nt) {  // rows: S <- J^T S, G <- J^T G
        const int k = e / B, col = e % B;
        if (rs[k] == 0.0) continue;
        int a, b;
        robin_pair(Bp, round, k, &a, &b);
        rotate(S + a + (size_t)col * B, S + b + (size_t)col * B, k);
        rotate(w.G + a + (size_t)col * B, w.G + b + (size_t)col * B, k);
      }
      __syncthreads();
      for (int e = tid; e < np * B; e += nt) {  // columns: S <- S J, G <- G J, V <- V J
        const int k = e / B, row = e % B;
        if (rs[k] == 0.0) continue;
        int a, b;
        robin_pair(Bp, round, k, &a, &b);
        rotate(S + row + (size_t)a * B, S + row + (size_t)b * B, k);
        rotate(w.G + row + (size_t)a * B, w.G + row + (size_t)b * B, k);
        rotate(w.V + row + (size_t)a * B, w.V + row + (size_t)b * B, k);
      }
      __syncthreads();
      for (int k = tid; k < np; k += nt) {
        if (rs[k] == 0.0) continue;
        int a, b;
        robin_pair(Bp, round, k, &a, &b);
        lev[a] = S[a + (size_t)a * B] / w.G[a + (size_t)a * B];
        lev[b] = S[b + (size_t)b * B] / w.G[b + (size_t)b * B];
      }
      __syncthreads();
    }
  }
  for (int e = tid; e < B * B; e += nt) {
    const int i = e % B, j = e / B, f = j + i * B;
    const double g = 0.5 * (w.G[e] + w.G[f]);  // equal in (i, j) and (j, i), as S is below: E's antisymmetry
    if (i == j) {
      w.E[e] = 0.5 * (1.0 - g);
      w.S[e] = S[e];  // the levels of phase_finish
      continue;
    }
    bool unsafe;
    w.E[e] = correction(coupling(S[e], S[f], g, lev[i], lev[j]), lev[j] - lev[i], g, bound, floor, &unsafe);
  }
  if (tid == 0) w.cnt[1] = 0;
}

// X = L^-T V with unit columns of V; eigenvalues; ascending order; signs.  One
// warp per column.
__device__ void phase_finish(const GepParams& p, const GepWork& w, int cta, int ncta) {
  const int B = p.nbloc, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (int c = cta * nw + (threadIdx.x >> 5); c < B; c += ncta * nw) {
    const double lam = w.S[c + (size_t)c * B] / w.G[c + (size_t)c * B];
    int pos = 0;  // place of this eigenvalue, ties by column, NaN last: every place is taken once
    for (int k = lane; k < B; k += 32) {
      const double o = w.S[k + (size_t)k * B] / w.G[k + (size_t)k * B];
      const bool same = o == lam || (isnan(o) && isnan(lam));
      pos += o < lam || (!isnan(o) && isnan(lam)) || (same && k < c);
    }
    for (int o = 16; o > 0; o >>= 1) pos += __shfl_xor_sync(0xffffffffu, pos, o);
    double x[kMaxQ], den = 0.0;
#pragma unroll
    for (int q = 0; q < kMaxQ; ++q) {
      x[q] = lane + 32 * q < B ? w.V[lane + 32 * q + (size_t)c * B] : 0.0;
      den = fma(x[q], x[q], den);
    }
    for (int o = 16; o > 0; o >>= 1) den += __shfl_xor_sync(0xffffffffu, den, o);
    const double sc = 1.0 / sqrt(den);
#pragma unroll
    for (int q = 0; q < kMaxQ; ++q) x[q] *= sc;
    // back substitution: row j of L is column j of L^T
#pragma unroll
    for (int q = kMaxQ - 1; q >= 0; --q) {
      for (int jj = 31; jj >= 0; --jj) {
        const int j = 32 * q + jj;
        if (j >= B) continue;
        double l[kMaxQ];
#pragma unroll
        for (int q2 = 0; q2 <= q; ++q2) l[q2] = lane + 32 * q2 < j ? w.LT[lane + 32 * q2 + (size_t)j * B] : 0.0;
        const double v = __shfl_sync(0xffffffffu, x[q], jj) * w.invd[j];
        if (lane == jj) x[q] = v;
#pragma unroll
        for (int q2 = 0; q2 <= q; ++q2) x[q2] = fma(-l[q2], v, x[q2]);
      }
    }
    double amax = -1.0, at = 0.0;  // the first largest magnitude and its value
    int imax = 0;
#pragma unroll
    for (int q = 0; q < kMaxQ; ++q)
      if (lane + 32 * q < B && fabs(x[q]) > amax) {
        amax = fabs(x[q]);
        at = x[q];
        imax = lane + 32 * q;
      }
    for (int o = 16; o > 0; o >>= 1) {
      const double a2 = __shfl_xor_sync(0xffffffffu, amax, o), t2 = __shfl_xor_sync(0xffffffffu, at, o);
      const int i2 = __shfl_xor_sync(0xffffffffu, imax, o);
      if (a2 > amax || (a2 == amax && i2 < imax)) {
        amax = a2;
        at = t2;
        imax = i2;
      }
    }
    const double sg = at < 0.0 ? -1.0 : 1.0;
#pragma unroll
    for (int q = 0; q < kMaxQ; ++q)
      if (lane + 32 * q < B) p.U[lane + 32 * q + (size_t)pos * B] = sg * x[q];
    if (lane == 0) p.eigv[pos] = lam;
  }
}

// The refinement iterations, in order: G = V^T V and W = C V; S = V^T W; E; the
// separation where E asks for it; V' = V + V E.  V and V' alternate, starting
// from V2 after the Newton step.
enum Phase : int {
  kCholesky, kReduce1, kReduce2, kJacobi, kReplayV, kGram0, kNewtonV, kGramApply, kProject, kCorrect, kSeparate,
  kUpdate, kFinish
};

__device__ void run_phase(const GepParams& p, const GepWork& w, int ph, int it, unsigned char* smem, int cta, int ncta) {
  const int B = p.nbloc, nb = (B + kTile - 1) / kTile;
  switch (ph) {
    case kCholesky: phase_cholesky(p, w, smem); break;
    case kReduce1: phase_reduce(p, w, false, cta, ncta); break;
    case kReduce2: phase_reduce(p, w, true, cta, ncta); break;
    case kJacobi: phase_jacobi(p, w, smem); break;
    case kReplayV: phase_replay(p, w, smem, cta, ncta); break;
    case kGram0: phase_product(w.V, w.V, w.G, B, true, kPlain, cta, ncta, smem); break;
    case kNewtonV: phase_product(w.V, w.G, w.V2, B, false, kNewton, cta, ncta, smem); break;
    case kGramApply:  // two products of V over twice the tiles
      if (ncta == 1 || cta < nb * nb) phase_product(w.V, w.V, w.G, B, true, kPlain, cta, ncta == 1 ? 1 : nb * nb, smem);
      if (ncta == 1 || cta >= nb * nb)
        phase_product(w.C, w.V, w.W, B, false, kPlain, ncta == 1 ? 0 : cta - nb * nb, ncta == 1 ? 1 : nb * nb, smem);
      break;
    case kProject: phase_product(w.V, w.W, w.S, B, true, kPlain, cta, ncta, smem); break;
    case kCorrect: phase_correction(w, B, it, cta, ncta); break;
    case kSeparate: phase_separate(w, B, it, smem); break;
    case kUpdate: phase_product(w.V, w.E, w.V2, B, false, kAdd, cta, ncta, smem); break;
    case kFinish: phase_finish(p, w, cta, ncta); break;
  }
}

// The sequence of phases; `swap` after a phase exchanges V and V'; `it` the iteration.
struct Step {
  Phase phase;
  bool swap;
  int it;
};
constexpr int kBefore = 7, kPerIteration = 5;  // steps before the iterations, and of each
constexpr int kNumSteps = kBefore + kPerIteration * kIterations + 1;
__host__ __device__ inline Step step_at(int q) {
  constexpr Phase before[kBefore] = {kCholesky, kReduce1, kReduce2, kJacobi, kReplayV, kGram0, kNewtonV};
  constexpr Phase each[kPerIteration] = {kGramApply, kProject, kCorrect, kSeparate, kUpdate};
  if (q < kBefore) return Step{before[q], before[q] == kNewtonV, 0};
  if (q == kNumSteps - 1) return Step{kFinish, false, 0};
  const Phase ph = each[(q - kBefore) % kPerIteration];
  return Step{ph, ph == kUpdate, (q - kBefore) / kPerIteration};
}

__device__ inline void swap_v(GepWork& w) {
  double* t = w.V;
  w.V = w.V2;
  w.V2 = t;
}

}  // namespace

// One phase per launch (swapped: V and V' exchanged; it: the iteration).
template <int kPhase>
__global__ void __launch_bounds__(1024) gep_phase_kernel(GepParams p, int swapped, int it) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  GepWork w;
  gep_carve(p.nbloc, p.work, &w);
  if (swapped) swap_v(w);
  run_phase(p, w, kPhase, it, smem_raw, blockIdx.x, gridDim.x);
}

// Every phase in one CTA of 64 threads, for blocks so small that the
// launches would cost more than the work.
__global__ void __launch_bounds__(64) gep_small_kernel(GepParams p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  GepWork w;
  gep_carve(p.nbloc, p.work, &w);
  for (int q = 0; q < kNumSteps; ++q) {
    const Step st = step_at(q);
    run_phase(p, w, st.phase, st.it, smem_raw, 0, 1);
    __syncthreads();
    if (st.swap) swap_v(w);
  }
}

size_t gep_work_doubles(int nbloc) {
  GepWork w;
  return nbloc > kMaxB ? 0 : gep_carve(nbloc, nullptr, &w);  // (larger blocks never get here)
}

int gep_launch(const GepParams& p, cudaStream_t st) {
  const int B = p.nbloc;
  const int npairs = B * (B + 1) / 2;
  // tiles as even as 32 x 32 allows: no more than a tile's rounding is computed for nothing
  const int tiles = (p.R + kPairTile - 1) / kPairTile, side = (p.R + tiles - 1) / tiles;
  void (*kern)(GepParams) = side <= 8    ? gep_inner_kernel<1, 1>
                            : side <= 16 ? gep_inner_kernel<2, 1>
                            : side <= 24 ? gep_inner_kernel<3, 2>
                                         : gep_inner_kernel<4, 2>;
  const size_t smem = sizeof(double) * 3 * (size_t)kPairLd * kMaxBasisPair;
  MLCP_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  kern<<<npairs, kPairThreads, smem, st>>>(p);
  MLCP_CUDA_TRY(cudaGetLastError());
  return gep_solve_launch(p, st);
}

namespace {

template <int kPhase>
int launch_phase(const GepParams& p, int swapped, int grid, int threads, size_t smem, cudaStream_t st, int it = 0) {
  if (smem > 48 * 1024)
    MLCP_CUDA_TRY(
        cudaFuncSetAttribute(gep_phase_kernel<kPhase>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  gep_phase_kernel<kPhase><<<grid, threads, smem, st>>>(p, swapped, it);
  MLCP_CUDA_TRY(cudaGetLastError());
  return kOk;
}

// Blocks of at most this many vectors run in gep_small_kernel: a whole
// diagonalizecpp_ call with it takes 160 us for 4 vectors, 214 for 8, 382 for
// 12 and 458 for 16; with one launch per phase about 290 us at each of these
// sizes (297 for 17).
constexpr int kSmallBlock = 8;

}  // namespace

int gep_solve_launch(const GepParams& p, cudaStream_t st) {
  const int B = p.nbloc, Bp = gep_pad(B), np = Bp / 2, nb = (B + kTile - 1) / kTile;
  const size_t s_chol = sizeof(double) * ((size_t)B * B + Bp), s_prod = sizeof(double) * 2 * kTile * (kChunk + 1),
               s_jac = sizeof(float) * ((size_t)Bp * (Bp + 1) + 4 * np), s_rep = sizeof(float) * kVRows * Bp,
               s_sep = sizeof(double) * ((size_t)B * B + B + 2 * np) + sizeof(int) * Bp;
  if (B <= kSmallBlock) {
    const size_t smem = std::max(std::max(std::max(s_chol, s_prod), std::max(s_jac, s_rep)), s_sep);
    gep_small_kernel<<<1, 64, smem, st>>>(p);
    MLCP_CUDA_TRY(cudaGetLastError());
    return kOk;
  }
  int swapped = 0, rc = kOk;
  for (int q = 0; q < kNumSteps && rc == kOk; ++q) {
    const Step step = step_at(q);
    switch (step.phase) {
      case kCholesky: rc = launch_phase<kCholesky>(p, swapped, 1, 1024, s_chol, st); break;
      case kReduce1: rc = launch_phase<kReduce1>(p, swapped, B, 32, 0, st); break;
      case kReduce2: rc = launch_phase<kReduce2>(p, swapped, B, 32, 0, st); break;
      case kJacobi: rc = launch_phase<kJacobi>(p, swapped, 1, 1024, s_jac, st); break;
      case kReplayV:
        rc = launch_phase<kReplayV>(p, swapped, (B + kVRows - 1) / kVRows, round_up(kVRows * np, 32), s_rep, st);
        break;
      case kGram0: rc = launch_phase<kGram0>(p, swapped, nb * nb, 64, s_prod, st); break;
      case kNewtonV: rc = launch_phase<kNewtonV>(p, swapped, nb * nb, 64, s_prod, st); break;
      case kGramApply: rc = launch_phase<kGramApply>(p, swapped, 2 * nb * nb, 64, s_prod, st); break;
      case kProject: rc = launch_phase<kProject>(p, swapped, nb * nb, 64, s_prod, st); break;
      case kCorrect: rc = launch_phase<kCorrect>(p, swapped, (B * B + 127) / 128, 128, 0, st, step.it); break;
      case kSeparate: rc = launch_phase<kSeparate>(p, swapped, 1, 1024, s_sep, st, step.it); break;
      case kUpdate: rc = launch_phase<kUpdate>(p, swapped, nb * nb, 64, s_prod, st); break;
      case kFinish: rc = launch_phase<kFinish>(p, swapped, B, 32, 0, st); break;
    }
    if (step.swap) swapped ^= 1;
  }
  return rc;
}

// ---------------------------------------------------------------------------
// Weight normalisation: coef /= sqrt(|<F,F>|) for each rank-R vector.
// ---------------------------------------------------------------------------

__global__ void normalize_coefs_kernel(int R, int D, int nD, const int* nbas, const double* base, double* coef) {
  const int v = blockIdx.x;
  const double* b = base + (size_t)v * R * nD;
  double* c = coef + (size_t)v * R;
  double acc = 0.0;
  for (int e = threadIdx.x; e < R * R; e += blockDim.x) {
    const int i = e % R, k = e / R;
    double prod = c[i] * c[k];
    int o = 0;
    for (int d = 0; d < D; ++d) {
      double t = 0.0;
      for (int q = 0; q < nbas[d]; ++q) t += b[(size_t)i * nD + o + q] * b[(size_t)k * nD + o + q];
      prod *= t;
      o += nbas[d];
    }
    acc += prod;
  }
  __shared__ double red[256];
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  const double q = sqrt(fabs(red[0]));
  __syncthreads();
  for (int i = threadIdx.x; i < R; i += blockDim.x) c[i] /= q;
}

int normalize_coefs_launch(int nvec, int R, int D, int nD, const int* nbas, const double* base, double* coef,
                           cudaStream_t st) {
  normalize_coefs_kernel<<<nvec, 256, 0, st>>>(R, D, nD, nbas, base, coef);
  MLCP_CUDA_TRY(cudaGetLastError());
  return kOk;
}

}  // namespace mlcp
