// ALS-guided Gram-Schmidt over a block of CP vectors (reference GramSchmidt,
// src/intertw_lcv.cu:131-205, with lcv_build_linear_system :77-127).
//
// Vector iv (iv >= 1) is fitted, mode by mode, to
//   F - sum_{k<iv} <Q_k, F> Q_k,
// where F is its current iterate and the coefficients <Q_k, F> are
// recomputed at every mode step (gramsumoverrow + sumarray in the reference).
// The pairwise per-mode overlaps P_k,d(r,i) = <Q_k,r^d, F_i^d> are kept and
// only the mode just solved is refreshed, so a mode step costs
// O(iv R^2 (D + 2n)) instead of rebuilding every product over all modes.
//
// Precision.  Once power iteration has made the block's vectors nearly
// parallel, the target F - sum_k <Q_k,F> Q_k is a small difference of large
// terms, and FP32 contractions lose it to cancellation; the reference runs
// this stage in FP64.  GB300 issues FP64 at a small fraction of its FP32
// rate, so everything here runs in double-word arithmetic (dword.cuh: about
// 48-bit significands on the FP32 pipes).  The R x R normal equations are
// solved by an FP32 Gauss-Jordan inverse with double-word iterative
// refinement, falling back to a double-word LDL^T (dwsolve.cuh).
//
// GB300 layout: the loop over vectors is sequential, but within a mode step
// the work over the earlier vectors k is independent.  For ranks up to 16 one
// thread-block cluster of up to 16 CTAs runs the whole orthogonalisation in one
// launch; CTA `rank` owns the earlier vectors k = rank (mod cluster) and keeps
// their factors, weights and overlaps resident in its shared memory (blocks
// that do not fit and larger ranks take the grid form, gs_grid.cu).  Each CTA
// forms its vectors' part of the right-hand side and stores it into every peer
// through distributed shared memory; every CTA then runs the same small solve
// on the same data, so each holds the identical new factor and nothing is
// broadcast back.
//
// What bounds it is the latency of a mode step's chain, so the step is arranged
// to keep that short:
//   - the new factor X of mode j is solved a row per warp, its norm taken there;
//   - its Gram gives the next normal equations BB; warp 0 inverts BB in FP32 as
//     soon as eight warps have written it, while the other fifteen refresh the
//     overlaps (with the next mode's products, and the coefficients <Q_k, F> from
//     those), form the right-hand side and exchange it;
//   - the FP32 inverse is then corrected once (more often if need be) by
//     Inv += (I - Inv BB) Inv with the residual in double-word (Schulz's
//     iteration), which leaves one product per right-hand side to the solve
//     instead of refinement rounds on it.  The left residual is used: the error of
//     X is then of the size (residual)^2 |X| and (rounding) cond |X|, as for
//     the refinement;
//   - the weights enter every step linearly, so they are rescaled by a power of
//     two only (exact) and divided by |F| once per vector.
// A mode step of rank 16 and 10 basis functions (6 modes) takes 5.7 us in a block of 40 vectors
// and 7.3 us in one of 100 (8.4 and 10.7 us with the weights normalised, the solve refined per
// right-hand side and the parts fetched from the peers); its issue slots alone, at the ~19
// of a double-word term with its two loads, are about 2 us.  Ranks above 16 have solves and inverses
// too long for one CTA: a step of rank 24, two modes of 24, takes 23.4 us in the grid
// form and took 42.5 here; rank 30 and 8 vectors, six modes of 8, 13.3 and 23.5.
#include <cooperative_groups.h>

#include <algorithm>
#include <cstdlib>
#include <map>
#include <mutex>
#include <string>
#include <tuple>
#include <vector>

#include "common.cuh"
#include "dword.cuh"
#include "dwsolve.cuh"
#include "fastdiv.cuh"
#include "intertwine.cuh"

namespace cg = cooperative_groups;

namespace mlcp {

namespace {

constexpr int kGsThreads = 512;
constexpr int kGsWarps = kGsThreads / 32;
constexpr int kGsInvert = dwsolve::kSolverThreads;        // warps 0..3: the inverse
constexpr int kGsWorkers = kGsThreads - kGsInvert;         // warps 4..15: the right-hand side
constexpr int kGsWorkerWarps = kGsWorkers / 32;
constexpr int kGsRank = dwsolve::kRowRank;  // ranks of this form: a row of the solve per warp
static_assert(kGsRank <= kGsWarps && 2 * kGsRank * kGsRank <= kGsThreads, "rows and entry halves of a step");

struct GsDims {
  int R, D, nD, npm, nkmax, cl, level;
};

struct GsArrays {
  dw *qf, *qc;    // [nkmax][R][ld] owned vectors' factors; [nkmax][R] their weights
  // Overlaps (index r*R+i).  P [nkmax][D][R*R]: before step j the products over d' >= d of
  // the old overlaps for d > j, the new overlaps of mode d for d < j; lead [nkmax][R*R]: c_k,r
  // times the product of those over d < j; psn [nkmax][R*R]: c_k,r times the product over d != j.
  dw *P, *lead, *psn;
  dw *fb;         // [R][ld] vector being fitted
  dw *g, *glead;  // [D][R*R], [R*R]: its Grams in the same way, without weights
  dw *fcs, *fg;   // [R] its weights; [R*R] c_r times its Grams' products over d != j
  dw *BB, *gpart; // [R*R] normal equations; [nkmax][ceil(R*R/32)] parts of <Q_k, F>
  dw *bs;         // [cl][R n, even] parts of the right-hand side received
  dw *Iv, *b0, *X;  // [R*R] inverse (column-major); [R][n] right-hand side; [i + m R] solution
  dw *dinv, *u, *red;
  float *gi, *Ef, *emax;  // [R*R] FP32 inverse and residual; [warps] largest residuals
  int *nb, *off, *flags;  // flags: [0] inverse usable, [1] non-positive pivot in the fallback
  FastDiv* fdn;  // [D] divisors n
};

// Row stride of the factors: odd, so that a warp reads different rows from different banks.
__host__ __device__ inline int gs_ld(int nD) { return nD | 1; }

// 32-entry chunks of an R x R matrix (at most 8).
__host__ __device__ inline int gs_chunks(int R) { return (R * R + 31) / 32; }

// Assigns the arrays (null base: sizes only) and returns the bytes.
// `level` 1 leaves P to global memory.
__host__ __device__ inline size_t gs_carve(const GsDims& m, GsArrays* a, unsigned char* sbase) {
  const int R = m.R, nkm = m.nkmax;
  const size_t RR = (size_t)R * R, Rn = (size_t)R * m.npm;
  size_t so = 0;
  auto take_s = [&](size_t bytes) -> unsigned char* {
    const size_t r = so;
    so += (bytes + 15) / 16 * 16;
    return sbase ? sbase + r : nullptr;
  };
  auto take = [&](size_t n) -> dw* { return (dw*)take_s(sizeof(dw) * n); };
  a->qf = take((size_t)nkm * R * gs_ld(m.nD));
  a->qc = take((size_t)nkm * R);
  if (m.level < 1) a->P = take((size_t)nkm * m.D * RR);
  a->lead = take((size_t)nkm * RR);
  a->psn = take((size_t)nkm * RR);
  a->fb = take((size_t)R * gs_ld(m.nD));
  a->g = take((size_t)m.D * RR);
  a->glead = take(RR);
  a->fcs = take(R);
  a->fg = take(RR);
  a->BB = take(RR);
  a->gpart = take((size_t)nkm * gs_chunks(R));
  a->bs = take((size_t)m.cl * ((Rn + 1) / 2 * 2));
  a->Iv = take(RR);
  a->b0 = take(Rn);
  a->X = take(Rn);
  a->dinv = take(R);
  a->u = take(R);
  a->red = take(kGsWarps);
  a->gi = (float*)take_s(sizeof(float) * RR);
  a->Ef = (float*)take_s(sizeof(float) * RR);
  a->emax = (float*)take_s(sizeof(float) * kGsWarps);
  a->nb = (int*)take_s(sizeof(int) * (m.D + 1));
  a->off = (int*)take_s(sizeof(int) * (m.D + 1));
  a->flags = (int*)take_s(sizeof(int) * 2);
  a->fdn = (FastDiv*)take_s(sizeof(FastDiv) * m.D);
  return so;
}

__device__ __forceinline__ void cl_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cl_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// Sum over the block; every thread gets the same value (dw_add is
// commutative, so the butterflies agree across lanes and warps).
__device__ dw block_sum(dw v, dw* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int o = 16; o > 0; o >>= 1) v = dw_add(v, dwsolve::dw_shfl_xor(v, o));
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  dw s = red[lane & (kGsWarps - 1)];
  for (int o = kGsWarps / 2; o > 0; o >>= 1) s = dw_add(s, dwsolve::dw_shfl_xor(s, o));
  return s;
}

// RT: the rank when it is known at compile time (16), else 0: index splits and
// strides of a step are then immediates (a step is bound by instruction issue).
template <int RT>
struct Gs {
  GsArrays a;
  int R_, D, nD, ld, CL, rank, tid, lane, warp;
  int rv;  // rank of the vector being fitted (ragged blocks; R otherwise)
  dw pen;
  FastDiv fdr;
  __device__ __forceinline__ int R() const { return RT ? RT : R_; }
  __device__ __forceinline__ int RR() const { return R() * R(); }
  __device__ __forceinline__ int chunks() const { return gs_chunks(R()); }
  // e = r R + i
  __device__ __forceinline__ void split(int e, int* r, int* i) const {
    if (RT) {
      *r = (unsigned)e / (RT ? RT : 1);
      *i = (unsigned)e % (RT ? RT : 1);
    } else {
      fdr.divmod((unsigned)e, r, i);
    }
  }
};

// Ragged ranks: rows and columns >= rv of the normal equations are the
// identity, so the padded terms stay decoupled from the fit.
template <int RT>
__device__ __forceinline__ dw normal_entry(const Gs<RT>& c, int i, int i2, dw v) {
  if (i >= c.rv || i2 >= c.rv) return dw_make(i == i2 ? 1.f : 0.f);
  return i == i2 ? dw_add(v, c.pen) : v;
}

// The vector iv as the working copy: factors, weights, penalty.
template <int RT>
__device__ void load_vector(Gs<RT>& c, const GsParams& p, int iv) {
  const int R = c.R();
  const double* fb = p.base + (size_t)iv * R * c.nD;
#pragma unroll 1
  for (int e = c.tid; e < R * c.nD; e += kGsThreads) c.a.fb[e / c.nD * c.ld + e % c.nD] = dw_from_double(fb[e]);
  if (c.tid < R) c.a.fcs[c.tid] = dw_from_double(p.coef[(size_t)iv * R + c.tid]);
  __syncthreads();
  dw pen = c.a.fcs[0];
#pragma unroll 1
  for (int i = 1; i < R; ++i)
    if (dw_gt(c.a.fcs[i], pen)) pen = c.a.fcs[i];
  c.pen = dw_mul(pen, dw_from_double(1.0e-10));  // FP64-build rule of the reference for this stage
}

// sum_m x[m sx] y[m sy], m < (N ? N : n)
template <int N = 0>
__device__ __forceinline__ dw dot(const dw* x, int sx, const dw* y, int sy, int n) {
  dw_acc acc = acc_zero();
  if (N) {
#pragma unroll
    for (int m = 0; m < N; ++m) acc_fma(acc, x[m * sx], y[m * sy]);
  } else {
#pragma unroll 4
    for (int m = 0; m < n; ++m) acc_fma(acc, x[m * sx], y[m * sy]);
  }
  return acc_value(acc);
}

// The share of 32 lanes in <Q_k, F>, to gpart.
template <int RT>
__device__ __forceinline__ void put_coefficient(const Gs<RT>& c, int kl, int ch, dw contrib) {
  const dw s = dwsolve::lane_sum<32>(contrib);
  if (c.lane == 0) c.a.gpart[kl * c.chunks() + ch] = s;
}

// The products over d' >= d of the overlaps (Grams) v[d stride], into v[d stride] for
// d >= 1; returns the product over d >= 1 (times `tail`, the value of mode D - 1).
__device__ __forceinline__ dw suffix_products(dw* v, size_t stride, int D, dw tail) {
  v[(D - 1) * stride] = tail;
#pragma unroll 1
  for (int d = D - 2; d > 0; --d) {
    tail = dw_mul(tail, v[d * stride]);
    v[d * stride] = tail;
  }
  return tail;
}

// A vector begins: its Grams and the owned vectors' overlaps with it, every
// mode, and what the first step (mode 0) needs of them.
template <int RT>
__device__ void vector_start(const Gs<RT>& c, int nk, bool fit) {
  const int R = c.R(), RR = c.RR(), D = c.D, ld = c.ld, nch = c.chunks();
#pragma unroll 1
  for (int q = c.warp; q < (nk + 1) * nch; q += kGsWarps) {
    const int s = q / nch, ch = q - s * nch, ee = 32 * ch + c.lane;
    const bool self = s == 0;  // the Grams first
    const int kl = s - 1;
    dw contrib = dw_make(0.f);
    if (ee < RR) {
      int r, i;
      c.split(ee, &r, &i);
      const dw *x = (self ? c.a.fb : c.a.qf + (size_t)kl * R * ld) + (size_t)r * ld, *y = c.a.fb + (size_t)i * ld;
      dw* v = (self ? c.a.g : c.a.P + (size_t)kl * D * RR) + ee;
      dw tail = dw_make(1.f);
#pragma unroll 1
      for (int d = 0; d < D; ++d) {
        const int o = c.a.off[d];
        tail = dot(x + o, 1, y + o, 1, c.a.nb[d]);
        v[(size_t)d * RR] = tail;
      }
      tail = suffix_products(v, RR, D, tail);
      const dw all = dw_mul(tail, v[0]);
      if (self) {
        c.a.glead[ee] = fit ? dw_make(1.f) : all;
        c.a.BB[ee] = normal_entry(c, i, r, tail);
        c.a.fg[ee] = dw_mul(c.a.fcs[r], tail);
      } else {
        const dw w = c.a.qc[kl * R + r];
        c.a.lead[(size_t)kl * RR + ee] = w;
        c.a.psn[(size_t)kl * RR + ee] = dw_mul(tail, w);
        contrib = dw_mul(dw_mul(all, w), c.a.fcs[i]);
      }
    }
    if (!self) put_coefficient(c, kl, ch, contrib);
  }
  __syncthreads();
}

// The finished vector: weights divided by sqrt(<F,F>), FP64 output (a share of each
// CTA), and the owner's resident copy when later vectors use it.
template <int RT>
__device__ void finish_vector(const Gs<RT>& c, const GsParams& p, int iv, bool factors) {
  const int R = c.R(), nD = c.nD;
  dw part = dw_make(0.f);
  if (c.tid < c.RR()) {
    int r, i;
    c.split(c.tid, &r, &i);
    part = dw_mul(dw_mul(c.a.fcs[r], c.a.fcs[i]), c.a.glead[c.tid]);
  }
  const dw q = dw_sqrt(dw_abs(block_sum(part, c.a.red)));
  const bool own = iv < p.nbloc - 1 && iv % c.CL == c.rank;
  const int kl = iv / c.CL;
  if (c.tid < R) {
    const dw x = dw_div(c.a.fcs[c.tid], q);
    if (own) c.a.qc[(size_t)kl * R + c.tid] = x;
    if (c.rank == 0) p.coef[(size_t)iv * R + c.tid] = dw_to_double(x);
  }
  if (own)
#pragma unroll 1
    for (int e = c.tid; e < R * c.ld; e += kGsThreads) c.a.qf[(size_t)kl * R * c.ld + e] = c.a.fb[e];
  if (factors)
#pragma unroll 1
    for (int e = c.rank * kGsThreads + c.tid; e < R * nD; e += c.CL * kGsThreads)
      p.base[(size_t)iv * R * nD + e] = dw_to_double(c.a.fb[e / nD * c.ld + e % nD]);
  __syncthreads();
}

// This CTA's part of the right-hand side of mode j (warps 4..15): sources s < nk,
//   -<Q_k, F> sum_r Q_k,r^j(m) psn_k(r,i),
// and, in the CTA that will own the fitted vector, sum_r F_r^j(m) fg(r,i), stored into
// every CTA of the cluster (entry i n + m).  Four lanes have two entries, two of them an
// entry's sums over r in halves; each stores the pair into a quarter of the CTAs.
template <int RT>
__device__ void step_rhs(const Gs<RT>& c, int j, int nk, bool self) {
  const int R = c.R(), RR = c.RR(), nj = c.a.nb[j], offj = c.a.off[j], Rn = R * nj, nch = c.chunks();
  const int nsrc = nk + (self ? 1 : 0), np = (Rn + 1) / 2, h = c.lane & 1;
  const int half = RT ? RT / 2 : (R + 1) / 2, r0 = h * half, nr = RT ? RT / 2 : min(R, r0 + half) - r0;
  const FastDiv fdn = c.a.fdn[j];
#pragma unroll 1
  for (int e0 = 0;; e0 += kGsWorkers / 2) {
    const int ew = e0 + 16 * (c.warp - kGsInvert / 32), e = ew + (c.lane >> 1);
    const bool none = ew >= Rn || nsrc == 0;
    dw v = dw_make(0.f);
    if (!none) {
      int i, m;
      fdn.divmod((unsigned)(e < Rn ? e : 0), &i, &m);
      const dw* A = c.a.qf + (size_t)r0 * c.ld + offj + m;
      const dw* M = c.a.psn + r0 * R + i;
      dw_acc tot = acc_zero();
      dw co = dw_make(0.f);
#pragma unroll 1
      for (int s = 0; s < nsrc; ++s) {
        if ((s & 3) == 0) {  // the coefficients of four sources, eight lanes each
          const int sk = s + (c.lane >> 3), q = c.lane & 7;
          co = sk < nk && q < nch ? c.a.gpart[sk * nch + q] : dw_make(0.f);
          co = dwsolve::lane_sum<8>(co);
          co = sk < nk ? dw_neg(co) : dw_make(1.f);
        }
        if (s == nk) {
          A = c.a.fb + (size_t)r0 * c.ld + offj + m;
          M = c.a.fg + r0 * R + i;
        }
        acc_fma(tot, dwsolve::dw_shfl(co, (s & 3) * 8), dot<RT / 2>(A, c.ld, M, R, nr));
        A += (size_t)R * c.ld;
        M += RR;
      }
      v = acc_value(
          dwsolve::acc_merge(tot, dw_acc{__shfl_xor_sync(0xffffffffu, tot.s, 1), __shfl_xor_sync(0xffffffffu, tot.c, 1)}));
    }
    if (e0 == 0) cl_wait();  // every CTA has read the parts of the step before
    if (none) return;
    const dw o = dwsolve::dw_shfl_xor(v, 2);
    const bool second = (c.lane & 2) != 0;
    const dw v0 = second ? o : v, v1 = second ? v : o;
    if (e < 2 * np) {
      const uint32_t local = (uint32_t)__cvta_generic_to_shared(c.a.bs + 2 * ((size_t)c.rank * np + (e >> 1)));
#pragma unroll 1
      for (int r = c.lane & 3; r < c.CL; r += 4) {
        uint32_t remote;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(r));
        asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(remote), "f"(v0.hi), "f"(v0.lo), "f"(v1.hi),
                     "f"(v1.lo)
                     : "memory");
      }
    }
  }
}

// After the exchange (every thread): the parts of the first nown CTAs in order, two lanes
// per entry, scaled by the power of two that brings the largest weight into
// [1, 2) (the weights enter linearly and are normalised at the vector's end).
template <int RT>
__device__ void step_gather(const Gs<RT>& c, int j, int nown) {
  const int Rn = c.R() * c.a.nb[j], ld = (Rn + 1) / 2 * 2, h = c.tid & 1;
  const float f = c.lane < c.R() ? fabsf(c.a.fcs[c.lane].hi) : 0.f;
  const int ex = __reduce_max_sync(0xffffffffu, __float_as_int(f)) >> 23;
  const float scale = ex > 0 && ex < 254 ? __int_as_float((254 - ex) << 23) : 1.f;
#pragma unroll 1
  for (int e0 = 0; e0 < Rn; e0 += kGsThreads / 2) {
    const int e = e0 + (c.tid >> 1);
    if (e0 + 16 * c.warp >= Rn) break;
    dw_acc acc = acc_zero();
    const dw* v = c.a.bs + h * ld + (e < Rn ? e : 0);
#pragma unroll 4
    for (int r = h; r < nown; r += 2, v += 2 * ld) acc_add(acc, *v);
    acc = dwsolve::acc_merge(acc, dw_acc{__shfl_xor_sync(0xffffffffu, acc.s, 1), __shfl_xor_sync(0xffffffffu, acc.c, 1)});
    const dw b = acc_value(acc);
    if (e < Rn && h == 0) c.a.b0[e] = dw_make(b.hi * scale, b.lo * scale);
  }
}

// The inverse of the normal equations (warps 0..3; FP32 by warp 0): flags[0].
template <int RT>
__device__ void step_inverse(const Gs<RT>& c) {
  if (c.warp == 0) {
    const bool good = dwsolve::gj_inverse_warp(c.a.BB, c.R(), c.a.gi);
    if (c.lane == 0) c.a.flags[0] = good;
    __syncwarp();
  }
  dwsolve::solver_sync();
  const bool ok = c.a.flags[0] != 0 && dwsolve::correct_inverse<RT>(c.a.BB, c.R(), c.a.gi, c.a.Iv, c.a.Ef, c.a.emax);
  dwsolve::solver_sync();
  if (c.tid == 0) c.a.flags[0] = ok;
}

// Row `warp` of the solution X = Iv b0 (of X itself after the fallback).
template <int RT, int NC>
__device__ void solve_row(const Gs<RT>& c, int j, bool solved) {
  const int R = c.R(), nj = c.a.nb[j], i = c.warp;
  dw x[NC ? NC : 1], nrm;
  dwsolve::row_product<RT, NC>(c.a.Iv + i, R, c.a.b0, nj, solved, c.a.X + i, x);
  dwsolve::row_normalise<NC>(x, &nrm);
  const bool pad = i >= c.rv;  // ragged: the first unit vector, without weight
#pragma unroll
  for (int q = 0; q < (NC ? NC : 1); ++q) {
    const int m = (NC ? c.lane : c.lane & 15) + 32 * q;
    const dw y = pad ? dw_make(m == 0 ? 1.f : 0.f) : x[q];
    if (m < nj && (NC || c.lane < 16)) {
      c.a.X[i + m * R] = y;
      c.a.fb[(size_t)i * c.ld + c.a.off[j] + m] = y;
    }
  }
  if (c.lane == 0) c.a.fcs[i] = pad ? dw_make(0.f) : nrm;
}

// LDL^T in double-word (threads 0 .. 127); out of line: a step's own code has to stay in the
// instruction cache.
__device__ __noinline__ void fallback_solve(dw* A, int n, dw* dinv, dw* u, dw* X, int nrhs, int* bad_flag) {
  const int bad = dwsolve::dw_ldlt(A, n, dinv, u);
  dwsolve::dw_ldlt_solve(A, n, dinv, X, nrhs);
  if (threadIdx.x == 0 && bad) *bad_flag = 1;
}

// The solve of mode j (every thread).
template <int RT>
__device__ void step_solve(const Gs<RT>& c, int j) {
  const int R = c.R(), nj = c.a.nb[j];
  const bool solved = c.a.flags[0] != 0;
  if (!solved) {  // the FP32 inverse is no use: LDL^T in double-word
    __syncthreads();
    if (c.tid < dwsolve::kSolverThreads) {
#pragma unroll 1
      for (int e = c.tid; e < R * nj; e += dwsolve::kSolverThreads) c.a.X[e] = c.a.b0[e % R * nj + e / R];
      fallback_solve(c.a.BB, R, c.a.dinv, c.a.u, c.a.X, nj, c.a.flags + 1);
    }
    __syncthreads();
  }
  if (c.warp < R) {
    if (nj <= 16) solve_row<RT, 0>(c, j, solved);
    else if (nj <= 32) solve_row<RT, 1>(c, j, solved);
    else solve_row<RT, 2>(c, j, solved);
  }
  __syncthreads();
}

// The Gram of mode j from the new factor (every thread, two per entry) and, with
// `more`, the next step's (mode jn) normal equations and self matrix.
template <int RT>
__device__ void update_gram(const Gs<RT>& c, int j, int jn, bool more) {
  const int R = c.R(), RR = c.RR(), ee = c.tid >> 1, h = c.tid & 1, nj = c.a.nb[j], half = (nj + 1) / 2;
  if (16 * c.warp >= RR) return;
  const bool live = ee < RR;
  int i2, i;
  c.split(live ? ee : 0, &i2, &i);
  const int m0 = h * half, nm = h ? nj - half : half;
  dw_acc acc = acc_zero();
  const dw *x = c.a.X + i + m0 * R, *y = c.a.X + i2 + m0 * R;
#pragma unroll 4
  for (int m = 0; m < nm; ++m) acc_fma(acc, x[m * R], y[m * R]);
  const dw s = acc_value(
      dwsolve::acc_merge(acc, dw_acc{__shfl_xor_sync(0xffffffffu, acc.s, 1), __shfl_xor_sync(0xffffffffu, acc.c, 1)}));
  if (!live || h) return;
  dw* v = c.a.g + ee;
  dw lead = dw_mul(c.a.glead[ee], s), gn;
  if (!more) {
    c.a.glead[ee] = lead;
    return;
  }
  if (jn > 0) {
    v[(size_t)j * RR] = s;
    gn = jn + 1 < c.D ? dw_mul(lead, v[(size_t)(jn + 1) * RR]) : lead;
  } else {
    gn = suffix_products(v, RR, c.D, s);
    lead = dw_make(1.f);
  }
  c.a.glead[ee] = lead;
  c.a.BB[ee] = normal_entry(c, i, i2, gn);
  c.a.fg[ee] = dw_mul(c.a.fcs[i2], gn);
}

// The owned overlaps of mode j, the next step's products over d != jn and the
// coefficients' parts (warps 4..15).
template <int RT>
__device__ void update_overlaps(const Gs<RT>& c, int j, int jn, int nk) {
  const int R = c.R(), RR = c.RR(), nj = c.a.nb[j], offj = c.a.off[j], nch = c.chunks();
#pragma unroll 1
  for (int q = c.warp - kGsInvert / 32; q < nk * nch; q += kGsWorkerWarps) {
    const int kl = q / nch, ch = q - kl * nch, ee = 32 * ch + c.lane;
    dw contrib = dw_make(0.f);
    if (ee < RR) {
      int r, i;
      c.split(ee, &r, &i);
      dw* v = c.a.P + (size_t)kl * c.D * RR + ee;
      const size_t le = (size_t)kl * RR + ee;
      // (loads that may be from global memory before the products)
      const dw ahead1 = v[(size_t)jn * RR], ahead2 = jn + 1 < c.D ? v[(size_t)(jn + 1) * RR] : dw_make(1.f),
               lead0 = c.a.lead[le];
      const dw s = dot(c.a.qf + ((size_t)kl * R + r) * c.ld + offj, 1, c.a.X + i, R, nj);
      dw prod, next;  // products over d != jn and over all d
      if (jn > 0) {
        const dw lead = dw_mul(lead0, s);
        v[(size_t)j * RR] = s;
        c.a.lead[le] = lead;
        prod = jn + 1 < c.D ? dw_mul(lead, ahead2) : lead;
        next = dw_mul(lead, ahead1);
      } else {
        const dw w = c.a.qc[kl * R + r];
        c.a.lead[le] = w;
        prod = dw_mul(suffix_products(v, RR, c.D, s), w);
        next = dw_mul(prod, ahead1);
      }
      c.a.psn[le] = prod;
      contrib = dw_mul(next, c.a.fcs[i]);
    }
    put_coefficient(c, kl, ch, contrib);
  }
}

}  // namespace

template <int RT>
__global__ void __launch_bounds__(kGsThreads, 1) gs_kernel(GsParams p) {
  cg::cluster_group cluster = cg::this_cluster();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Gs<RT> c;
  c.CL = (int)cluster.num_blocks();
  c.rank = (int)cluster.block_rank();
  c.R_ = p.R;
  c.fdr = FastDiv((unsigned)p.R);
  c.D = p.D;
  c.nD = p.nD;
  c.ld = gs_ld(p.nD);
  c.tid = threadIdx.x;
  c.lane = c.tid & 31;
  c.warp = c.tid >> 5;
  c.rv = p.R;
  gs_carve(GsDims{p.R, p.D, p.nD, p.npmax, p.nkmax, c.CL, p.level}, &c.a, smem_raw);
  if (p.level) c.a.P = reinterpret_cast<dw*>(p.work) + (size_t)c.rank * p.nkmax * p.D * p.R * p.R;
#pragma unroll 1
  for (int d = c.tid; d <= c.D; d += kGsThreads) {
    c.a.nb[d] = d < c.D ? p.nbas[d] : 0;
    c.a.off[d] = p.off[d];
    if (d < c.D) {
      c.a.fdn[d] = FastDiv((unsigned)p.nbas[d]);
    }
  }
  if (c.tid == 0) {
    c.a.flags[0] = 1;
    c.a.flags[1] = 0;
  }
  // the cluster barrier is used twice per step: parts stored, parts read; this
  // first arrival also says that the CTA runs
  cl_arrive();
  __syncthreads();

  load_vector(c, p, 0);
  vector_start(c, 0, false);
  finish_vector(c, p, 0, false);

#pragma unroll 1
  for (int iv = 1; iv < p.nbloc && p.nals > 0; ++iv) {
    c.rv = p.rank_v ? p.rank_v[iv] : p.R;
    load_vector(c, p, iv);
    const int nk = (iv - c.rank + c.CL - 1) / c.CL;  // owned k = rank, rank + CL, ... < iv
    vector_start(c, nk, true);
#pragma unroll 1
    for (int it = 0; it < p.nals; ++it) {
#pragma unroll 1
      for (int j = 0; j < c.D; ++j) {
        const bool more = it + 1 < p.nals || j + 1 < c.D;  // another step of this vector follows
        const int jn = j + 1 < c.D ? j + 1 : 0;
        if (c.tid < kGsInvert) {
          cl_wait();
          cl_arrive();
          step_inverse(c);
        } else {
          step_rhs(c, j, nk, iv % c.CL == c.rank);
          cl_arrive();
        }
        cl_wait();
        step_gather(c, j, min(c.CL, iv + 1));
        __syncthreads();
        cl_arrive();
        step_solve(c, j);
        update_gram(c, j, jn, more);
        if (!more) break;
        // the inverse starts with the complete BB, the right-hand side when the
        // overlaps are complete too
        if (c.tid < kGsInvert) {
          asm volatile("bar.arrive 4, 512;" ::: "memory");
          asm volatile("bar.sync 3, 512;" ::: "memory");
        } else {
          asm volatile("bar.arrive 3, 512;" ::: "memory");
          update_overlaps(c, j, jn, nk);
          asm volatile("bar.sync 4, 512;" ::: "memory");
        }
      }
    }
    __syncthreads();
    finish_vector(c, p, iv, true);
  }
  if (c.rank == 0 && c.tid == 0 && c.a.flags[1]) atomicOr(p.status, 1);
  // no CTA leaves while a peer may still store into its shared memory
  cl_wait();
}

// CTAs per cluster: 16 (the non-portable maximum) unless the block is
// smaller or the caller asks for `pref` (the measured choice of
// gs_tuned_cluster); MLCP_GB300_GS_CLUSTER fixes a size (measurements).
int gs_cluster_size(int nbloc, int pref) {
  int cl = pref > 0 ? std::max(2, std::min(16, pref)) : 16;
  if (const char* e = getenv("MLCP_GB300_GS_CLUSTER")) cl = std::max(2, std::min(16, atoi(e)));
  return nbloc > cl ? cl : (nbloc > 1 ? nbloc - 1 : 1);
}

namespace {

// Cluster sizes the search tries (each clamped to the block).
constexpr int kClusterCandidates[] = {16, 12, 8};

int gs_nkmax(int nbloc, int nc) { return std::max(1, (nbloc - 1 + nc - 1) / nc); }

// Bytes of the one-cluster form with clusters of cl CTAs.
size_t gs_bytes(const GsParams& p, int cl, int level) {
  GsArrays a;
  return gs_carve(GsDims{p.R, p.D, p.nD, p.npmax, gs_nkmax(p.nbloc, cl), cl, level}, &a, nullptr);
}

// How one cluster of cl CTAs can run the block: the smallest level that fits, or -1 (the grid
// form).  With P in global memory a step of 150 vectors, rank 16, takes 9.0 us and 10.8 in the
// grid form; with the leading products there too, 250 vectors take 12.4 and 11.0, so that stays out.
int gs_level(const GsParams& p, int cl, int smem_max) {
  if (p.R > kGsRank || p.D < 2) return -1;
  for (int level = 0; level < 2; ++level)
    if (gs_bytes(p, cl, level) <= (size_t)smem_max) return level;
  return -1;
}

// Shared memory that a shape may not exceed: what one CTA of the form before these two needed of a
// mode step (normal equations and two inverses, six right-hand sides, a coefficient per
// chunk of the overlaps of nkm vectors, its reductions).  Kept as the limit on purpose: what
// was refused stays refused, and both forms need less.
size_t gs_core_bytes(int R, int D, int npm, int nkm) {
  const size_t RR = (size_t)R * R, Rn = (size_t)R * npm;
  size_t o = 0;
  for (size_t bytes : {8 * (size_t)R, 8 * Rn, 8 * RR, 8 * RR, 8 * RR, 8 * nkm * ((RR + 31) / 32), 8 * (size_t)nkm, 16 * Rn,
                       8 * Rn, 8 * Rn, 8 * Rn, 8 * (size_t)R, 8 * (size_t)R, (size_t)128, (size_t)32, 8 * RR, (size_t)16,
                       (size_t)256, (size_t)2048, (size_t)4096, 4 * (size_t)(D + 1), 4 * (size_t)(D + 1),
                       (size_t)16, sizeof(FastDiv) * (D + 3)})
    o += (bytes + 15) / 16 * 16;
  return o;
}

}  // namespace

size_t gs_work_doubles(int nbloc, int R, int nD, int D, int npm) {
  // the overlaps of 16 CTAs' vectors (fewer CTAs: fewer vectors in all), or the grid form's
  return std::max(gs_grid_dw(nbloc, R, nD, D, npm), ((size_t)nbloc + 16) * D * R * R);
}

int gs_launch(const GsParams& prm, cudaStream_t st) {
  GsParams p = prm;
  const int cl = gs_cluster_size(p.nbloc, p.cl);
  int dev = 0, smem_max = 0, nsm = 0;
  MLCP_CUDA_TRY(cudaGetDevice(&dev));
  MLCP_CUDA_TRY(cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  MLCP_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  // shapes beyond what one CTA can hold of a mode step are refused
  if (gs_core_bytes(p.R, p.D, p.npmax, gs_nkmax(p.nbloc, std::min(nsm, 9 * cl))) > (size_t)smem_max) {
    set_error("intertwinecpp_: Gram-Schmidt needs more shared memory than %d bytes (rank %d)", smem_max, p.R);
    return kTooLarge;
  }
  p.level = gs_level(p, cl, smem_max);
  if (p.level < 0) return gs_grid_launch(p, st);
  const size_t smem = gs_bytes(p, cl, p.level);
  p.nkmax = gs_nkmax(p.nbloc, cl);
  void (*kern)(GsParams) = p.R == kGsRank ? gs_kernel<kGsRank> : gs_kernel<0>;
  MLCP_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  if (cl > 8) MLCP_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cl);
  cfg.blockDim = dim3(kGsThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cl;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  MLCP_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, p));
  return kOk;
}

// ---------------------------------------------------------------------------
// Cluster-size search
// ---------------------------------------------------------------------------
// A larger cluster spreads the earlier vectors over more CTAs but pays a
// longer gather and cluster barrier at every mode step; which wins depends on
// the block, and the grid form takes the blocks whose arrays 16 CTAs cannot hold
// (measured on the 40-vector rank-16 block, ten sweeps: 16 CTAs 13.7 ms,
// 12 CTAs 14.1, 8 CTAs 15.5).  The first cycle of a block shape runs
// one Gram-Schmidt sweep (nals = 1) twice with each candidate size on a
// scratch copy of the block, times it with CUDA events on the cycle's stream
// and caches the size of the fastest run for the process, per device and
// shape.  Off with
// mlcp_gb300_set_autotune(0) / MLCP_GB300_AUTOTUNE=0 or a fixed
// MLCP_GB300_GS_CLUSTER (then the 16-CTA rule applies).

namespace {

struct GsTuneKey {
  int device, nbloc, R, D, nD, npmax, ragged;
  bool operator<(const GsTuneKey& o) const {
    return std::tie(device, nbloc, R, D, nD, npmax, ragged) <
           std::tie(o.device, o.nbloc, o.R, o.D, o.nD, o.npmax, o.ragged);
  }
};

struct GsTuneEntry {
  int cl = 0;
  std::vector<std::pair<int, float>> trials;  // (cluster size, ms of one sweep)
};

std::mutex g_gs_tune_mu;
std::map<GsTuneKey, GsTuneEntry> g_gs_tune;

}  // namespace

int gs_tuned_cluster(const GsParams& p, int device, double* scratch_base, double* scratch_coef, cudaStream_t st,
                     int* cl_out) {
  *cl_out = 0;
  if (getenv("MLCP_GB300_GS_CLUSTER") || p.nals <= 0) return kOk;
  const GsTuneKey key{device, p.nbloc, p.R, p.D, p.nD, p.npmax, p.rank_v != nullptr};
  {
    std::lock_guard<std::mutex> lk(g_gs_tune_mu);
    auto it = g_gs_tune.find(key);
    if (it != g_gs_tune.end()) {
      *cl_out = it->second.cl;
      return kOk;
    }
  }
  int smem_max = 0;
  MLCP_CUDA_TRY(cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, device));
  std::vector<int> cand;  // sizes whose CTAs hold the block
  for (int c : kClusterCandidates) {
    const int cl = gs_cluster_size(p.nbloc, c);
    if (gs_level(p, cl, smem_max) >= 0 && std::find(cand.begin(), cand.end(), cl) == cand.end())
      cand.push_back(cl);
  }
  GsTuneEntry entry;
  if (cand.size() > 1) {
    const size_t nvals = (size_t)p.nbloc * p.R * p.nD, ncoef = (size_t)p.nbloc * p.R;
    cudaEvent_t e0, e1;
    MLCP_CUDA_TRY(cudaEventCreate(&e0));
    MLCP_CUDA_TRY(cudaEventCreate(&e1));
    float best = 0.f;
    for (int cl : cand) {
      GsParams t = p;
      t.base = scratch_base;
      t.coef = scratch_coef;
      t.nals = 1;
      t.cl = cl;
      float ms = -1.f;
      for (int rep = 0; rep < 2; ++rep) {  // the faster of two runs
        MLCP_CUDA_TRY(cudaMemcpyAsync(scratch_base, p.base, sizeof(double) * nvals, cudaMemcpyDeviceToDevice, st));
        MLCP_CUDA_TRY(cudaMemcpyAsync(scratch_coef, p.coef, sizeof(double) * ncoef, cudaMemcpyDeviceToDevice, st));
        MLCP_CUDA_TRY(cudaEventRecord(e0, st));
        if (gs_launch(t, st) != kOk) {  // a size this GPU cannot launch for the block: no candidate
          cudaGetLastError();
          ms = -1.f;
          break;
        }
        MLCP_CUDA_TRY(cudaEventRecord(e1, st));
        MLCP_CUDA_TRY(cudaEventSynchronize(e1));
        float m = 0.f;
        MLCP_CUDA_TRY(cudaEventElapsedTime(&m, e0, e1));
        ms = (ms < 0.f || m < ms) ? m : ms;
      }
      if (ms < 0.f) continue;
      entry.trials.push_back({cl, ms});
      if (entry.trials.size() == 1 || ms < best) {
        best = ms;
        entry.cl = cl;
      }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
  } else {
    entry.cl = cand.empty() ? 0 : cand[0];
  }
  {
    std::lock_guard<std::mutex> lk(g_gs_tune_mu);
    g_gs_tune[key] = entry;
  }
  *cl_out = entry.cl;
  return kOk;
}

void gs_tune_report(std::string& out) {
  std::lock_guard<std::mutex> lk(g_gs_tune_mu);
  char line[160];
  for (const auto& kv : g_gs_tune) {
    const GsTuneKey& k = kv.first;
    snprintf(line, sizeof(line), "gs nbloc=%d R=%d ndof=%d nD=%d%s: cluster %d;", k.nbloc, k.R, k.D, k.nD,
             k.ragged ? " ragged" : "", kv.second.cl);
    out += line;
    for (const auto& t : kv.second.trials) {
      snprintf(line, sizeof(line), " %d=%.3fms", t.first, t.second);
      out += line;
    }
    out += "\n";
  }
}

}  // namespace mlcp
