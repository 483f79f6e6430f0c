// ALS-guided Gram-Schmidt over the whole GPU: the algorithm of gs.cu (see
// there for the definition and the precision) as two launches per mode step,
// for blocks whose arrays do not fit the shared memory of one cluster.
//
// Vector iv, with the earlier vectors k < iv finished:
//   gsg_overlap_kernel  the overlaps P_k,d(r,i) = <Q_k,r^d, F_i^d> of every k
//                       and mode with the starting F, and F's Grams, as the
//                       overlaps of F with itself (k = iv); one CTA per (k, d);
// then for every mode step j (jp the mode solved before it):
//   gsg_accum_kernel    a CTA for every slab of at most 16 rows r of every
//                       k <= iv: P_k,jp with the new factor, the products over
//                       d != j, the slab's share of the coefficient <Q_k, F>
//                       and of the right-hand side, summed over the eight
//                       CTAs of a cluster; one more CTA: the normal equations
//                       and their FP32 inverse;
//   gsg_solve_kernel    one cluster of eight CTAs, each solving an eighth of the
//                       columns (they are independent but for the row norms);
// and gsg_finish_kernel for the norm.  The step launches overlap (programmatic
// dependent launch): what a kernel reads that is older than its predecessor
// it fetches while that one still runs.
//
// The weights of F enter every step linearly, so they are only rescaled by a
// power of two per step (exact) and divided by |F| once, when the vector is
// finished, instead of after every step.  A vector of a ragged block is fitted
// at its own rank; its padding terms get the first unit vector and no weight,
// as the padded solve of the one-cluster form leaves them.
//
// What bounds it: the chain of 2 nals D launches per vector, each a few
// thousand cycles of double-word work spread over iv CTAs.  A mode step takes 10 to 13 us
// for ranks up to 30 and small bases, 20 us for rank 30 and 48 basis functions and
// 28 us at rank 48 (12 modes of 8); the block spread over several clusters that
// exchanged through global memory and met at a grid barrier, which it replaces, took 15 to 25,
// 79 and 103 us.  Blocks of rank 16 that one cluster can hold are faster there (gs.cu): 5.7 and
// 13 us for 40 vectors with 10 basis functions in 6 modes; the 250 vectors that it
// cannot hold take 11.0 us (10.9 over several clusters).
#include <algorithm>

#include "common.cuh"
#include "dword.cuh"
#include "dwsolve.cuh"
#include "intertwine.cuh"

namespace mlcp {

namespace {

constexpr int kAccThreads = 512;
constexpr int kSolThreads = 256;
constexpr int kCl = 8;  // CTAs of a cluster (portable size)

__device__ __forceinline__ void gg_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void gg_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// Waits until the kernel launched before this one has finished; kernels before
// that one have then finished too.
__device__ __forceinline__ void gg_after_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// Lets the next kernel's CTAs start.  After gg_after_previous only, so that what
// they read before their own wait is at least two kernels old.
__device__ __forceinline__ void gg_release_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Asynchronous global -> shared copies of 8 and 4 bytes.
__device__ __forceinline__ void gg_cp8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void gg_cp4(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

// Stores v at the place of `p` in CTA `r` of the cluster (which has arrived at
// a cluster barrier, so it runs); visible there after the next cluster barrier.
__device__ __forceinline__ void gg_push(dw* p, int r, dw v) {
  const uint32_t local = (uint32_t)__cvta_generic_to_shared(p);
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(r));
  asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(remote), "f"(v.hi), "f"(v.lo) : "memory");
}

// Scratch.  Factors are stored per vector and mode: mode d of vector k at
// qf + k R nD + R off_d, [R][n_d].
struct GgScratch {
  dw *qf;    // [B][R nD] finished vectors' factors, and the one being fitted
  dw *qc;    // [B][R] their weights
  dw *P;     // [B][D][R R] overlaps of the vector being fitted with k <= iv
  dw *fc;    // [R] its weights
  dw *pg;    // [R R] products of F's Grams over d not in {mode being solved, next mode}
  dw *bb;    // [R R] normal equations (ld rv)
  dw *iv;    // [R R] their inverse (ld rv; ranks up to 16)
  dw *part;  // [clusters][R npmax] parts of the right-hand side (i + m R)
  dw *pen;   // [1]
  float *inv;  // [R R] FP32 inverse of bb (ld rv)
  int *flag;   // [0] inverse usable, [1] non-positive pivot seen
};

// Slabs of rows per vector (a divisor of kCl), their height, and the clusters
// of an accumulation over nk vectors.
__host__ __device__ inline int gg_slabs(int R) { return R <= 16 ? 1 : R <= 32 ? 2 : 4; }
__host__ __device__ inline int gg_slab_rows(int R) { return (R + gg_slabs(R) - 1) / gg_slabs(R); }
__host__ __device__ inline int gg_clusters(int nk, int R) { return (nk * gg_slabs(R) + kCl - 1) / kCl; }

__host__ __device__ inline size_t gg_carve(int B, int R, int D, int nD, int npm, dw* base, GgScratch* s) {
  size_t o = 0;
  auto take = [&](size_t n) -> dw* {
    dw* r = base ? base + o : nullptr;
    o += (n + 1) / 2 * 2;
    return r;
  };
  const size_t RR = (size_t)R * R;
  s->qf = take((size_t)B * R * nD);
  s->qc = take((size_t)B * R);
  s->P = take((size_t)B * D * RR);
  s->fc = take(R);
  s->pg = take(RR);
  s->bb = take(RR);
  s->iv = take(RR);
  s->part = take((size_t)gg_clusters(B, R) * R * npm);
  s->pen = take(1);
  s->inv = reinterpret_cast<float*>(take((RR + 1) / 2));
  s->flag = reinterpret_cast<int*>(take(1));
  return o;
}

__device__ __forceinline__ GgScratch gg_scratch(const GsParams& p) {
  GgScratch s;
  gg_carve(p.nbloc, p.R, p.D, p.nD, p.npmax, reinterpret_cast<dw*>(p.work), &s);
  return s;
}

// Whether the steps are solved a row per warp (gsg_solve_rows_kernel).
__host__ __device__ inline bool gg_by_rows(int R) { return R <= dwsolve::kRowRank; }

__device__ __forceinline__ int gg_rank(const GsParams& p, int v) { return p.rank_v ? p.rank_v[v] : p.R; }

// Sum over the block; every thread gets the result (fixed order; dw_add is
// commutative).  red: [warps].
template <int NT>
__device__ dw gg_block_sum(dw v, dw* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int o = 16; o > 0; o >>= 1) v = dw_add(v, dwsolve::dw_shfl_xor(v, o));
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  dw s = red[lane % (NT / 32)];
  for (int o = NT / 64; o > 0; o >>= 1) s = dw_add(s, dwsolve::dw_shfl_xor(s, o));
  return s;
}

// out(r, i) = sum_m X[r][m] Y[i][m], r < nr, i < ni (X, Y in shared memory, ld
// ldx): LX lanes along i, NT / LX rows at a time.  pre(r, i) runs before the
// products of an entry (loads to be in flight meanwhile) and its value goes
// to emit(r, i, value, pre's).  With `half`, entries i <= r only.
template <int NT, int LX, class Pre, class Emit>
__device__ __forceinline__ void gg_tile(const dw* X, const dw* Y, int ldx, int nr, int ni, int n, Pre&& pre,
                                        Emit&& emit) {
  constexpr int TY = NT / LX;
  const int tx = threadIdx.x % LX, ty = threadIdx.x / LX;
  for (int r = ty; r < nr; r += TY)
    for (int i = tx; i < ni; i += LX) {
      const auto held = pre(r, i);
      const dw *x = X + (size_t)r * ldx, *y = Y + (size_t)i * ldx;
      dw_acc acc = acc_zero();
#pragma unroll 4
      for (int m = 0; m < n; ++m) acc_fma(acc, x[m], y[m]);
      emit(r, i, acc_value(acc), held);
    }
}

template <int NT, class Pre, class Emit>
__device__ __forceinline__ void gg_products(const dw* X, const dw* Y, int ldx, int nr, int ni, int n,
                                            Pre&& pre, Emit&& emit) {
  if (ni > 16) gg_tile<NT, 32>(X, Y, ldx, nr, ni, n, pre, emit);
  else gg_tile<NT, 16>(X, Y, ldx, nr, ni, n, pre, emit);
}
struct GgNothing {};

// The entries v[d stride], d < D but ex1 and ex2 (global memory): the first
// eight are loaded together, later ones with the product.
struct GgChain {
  dw y[8];
};
__device__ __forceinline__ GgChain gg_fetch(const dw* v, size_t stride, int D, int ex1, int ex2, int d0 = 0) {
  GgChain c;
#pragma unroll
  for (int u = 0; u < 8; ++u)
    c.y[u] = d0 + u < D && d0 + u != ex1 && d0 + u != ex2 ? v[(size_t)(d0 + u) * stride] : dw_make(1.f);
  return c;
}
// x times their product.
__device__ __forceinline__ dw gg_chain(dw x, GgChain c, const dw* v, size_t stride, int D, int ex1, int ex2) {
  for (int d0 = 0; d0 < D; d0 += 8) {
    if (d0) c = gg_fetch(v, stride, D, ex1, ex2, d0);
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (d0 + u < D && d0 + u != ex1 && d0 + u != ex2) x = dw_mul(x, c.y[u]);
  }
  return x;
}

// The part of the right-hand side of rows r: out(i, m) = sum_r A[r][m] W[r][i]
// (A [nr][n], W ld ldw), LX lanes along i.
template <int NT, int LX, class Emit>
__device__ __forceinline__ void gg_part(const dw* A, const dw* W, int ldw, int nr, int n, int rv, Emit&& emit) {
  const int tx = threadIdx.x % LX, ty = threadIdx.x / LX;
  for (int i = tx; i < rv; i += LX)
    for (int m = ty; m < n; m += NT / LX) {
      dw_acc a = acc_zero();
#pragma unroll 4
      for (int r = 0; r < nr; ++r) acc_fma(a, A[r * n + m], W[r * ldw + i]);
      emit(i, m, acc_value(a));
    }
}

// Rows of a factor slice [rows][n] into shared memory with an odd leading
// dimension (16 lanes along the rows then read distinct banks).
__device__ __forceinline__ int gg_ld(int n) { return n | 1; }
__device__ __forceinline__ void gg_load(dw* dst, const dw* src, int rows, int n, int nt) {
  const int ld = gg_ld(n);
  for (int e = threadIdx.x; e < rows * n; e += nt) {
    const int r = e / n;
    dst[r * ld + (e - r * n)] = src[e];
  }
}
// The same from a vector's FP64 factors (row stride nD).
__device__ __forceinline__ void gg_load64(dw* dst, const double* src, int rows, int n, int nD, int nt) {
  const int ld = gg_ld(n);
  for (int e = threadIdx.x; e < rows * n; e += nt) {
    const int r = e / n;
    dst[r * ld + (e - r * n)] = dw_from_double(src[(size_t)r * nD + (e - r * n)]);
  }
}

// Vector v finished (one CTA): its last mode's Gram when it was fitted (the
// others are P's slot v), weights divided by |F|.
template <int NT>
__device__ void gg_finish(const GsParams& p, const GgScratch& s, int v, bool fitted, dw* sm, dw* red) {
  const int R = p.R, RR = R * R, rv = gg_rank(p, v);
  const dw* f = s.qf + (size_t)v * R * p.nD;
  dw* G = s.P + (size_t)v * p.D * RR;
  if (fitted) {
    const int d = p.D - 1, n = p.nbas[d];
    gg_load(sm, f + (size_t)R * p.off[d], rv, n, NT);
    __syncthreads();
    gg_products<NT>(sm, sm, gg_ld(n), rv, rv, n, [](int, int) { return GgNothing(); },
                    [&](int r, int i, dw x, GgNothing) { G[(size_t)d * RR + r * R + i] = x; });
    __syncthreads();
  }
  const dw* c = fitted ? s.fc : s.qc + (size_t)v * R;
  dw sum = dw_make(0.f);
  for (int e = threadIdx.x; e < rv * rv; e += NT) {
    const int a = e / rv, b = e - a * rv;
    const dw* g = G + a * R + b;
    const GgChain ch = gg_fetch(g, RR, p.D, -1, -1);
    sum = dw_add(sum, gg_chain(dw_mul(c[a], c[b]), ch, g, RR, p.D, -1, -1));
  }
  const dw q = dw_sqrt(dw_abs(gg_block_sum<NT>(sum, red)));
  for (int i = threadIdx.x; i < R; i += NT) {
    const dw x = i < rv ? dw_div(c[i], q) : dw_make(0.f);
    s.qc[(size_t)v * R + i] = x;
    p.coef[(size_t)v * R + i] = dw_to_double(x);
  }
}

// Vector 0 (its factors stay as they are), one CTA: double-word copy, Grams, norm.
__global__ void __launch_bounds__(kAccThreads) gsg_first_kernel(GsParams p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ dw red[kAccThreads / 32];
  dw* sm = reinterpret_cast<dw*>(smem_raw);
  const GgScratch s = gg_scratch(p);
  const int R = p.R, RR = R * R, rv = gg_rank(p, 0);
  if (threadIdx.x == 0) {
    s.flag[0] = 1;
    s.flag[1] = 0;
  }
  for (int d = 0; d < p.D; ++d) {
    const int n = p.nbas[d], ld = gg_ld(n);
    gg_load64(sm, p.base + p.off[d], R, n, p.nD, kAccThreads);
    __syncthreads();
    for (int e = threadIdx.x; e < R * n; e += kAccThreads) s.qf[(size_t)R * p.off[d] + e] = sm[e / n * ld + e % n];
    gg_products<kAccThreads>(sm, sm, ld, rv, rv, n, [](int, int) { return GgNothing(); },
                             [&](int r, int i, dw x, GgNothing) { s.P[(size_t)d * RR + r * R + i] = x; });
    __syncthreads();
  }
  for (int i = threadIdx.x; i < R; i += kAccThreads) s.qc[i] = dw_from_double(p.coef[i]);
  __syncthreads();
  gg_finish<kAccThreads>(p, s, 0, false, sm, red);
}

// Vector iv begins: CTA (k, d), k < iv: the overlaps of Q_k with F in mode d;
// k = iv: F's double-word copy and Gram of mode d, its weights and penalty.
template <int NT>
__global__ void __launch_bounds__(NT) gsg_overlap_kernel(GsParams p, int iv) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  dw* F = reinterpret_cast<dw*>(smem_raw);
  const GgScratch s = gg_scratch(p);
  const int k = blockIdx.x, d = blockIdx.y, R = p.R, RR = R * R, n = p.nbas[d], ld = gg_ld(n);
  const int rv = gg_rank(p, iv), rk = gg_rank(p, k);
  dw* Q = F;
  gg_load64(F, p.base + (size_t)iv * R * p.nD + p.off[d], R, n, p.nD, NT);
  if (k < iv) {
    Q = F + (size_t)R * ld;
    gg_load(Q, s.qf + (size_t)k * R * p.nD + (size_t)R * p.off[d], rk, n, NT);
  }
  __syncthreads();
  dw* P = s.P + ((size_t)k * p.D + d) * RR;
  gg_products<NT>(Q, F, ld, rk, rv, n, [](int, int) { return GgNothing(); },
                           [&](int r, int i, dw x, GgNothing) { P[r * R + i] = x; });
  if (k < iv) return;
  dw* f = s.qf + (size_t)iv * R * p.nD + (size_t)R * p.off[d];
  for (int e = threadIdx.x; e < R * n; e += NT) f[e] = F[e / n * ld + e % n];
  if (d == 0) {
    for (int i = threadIdx.x; i < R; i += NT)
      s.fc[i] = i < rv ? dw_from_double(p.coef[(size_t)iv * R + i]) : dw_make(0.f);
    if (threadIdx.x == 0) {
      double pen = p.coef[(size_t)iv * R];
      for (int i = 1; i < R; ++i) pen = fmax(pen, p.coef[(size_t)iv * R + i]);
      s.pen[0] = dw_from_double(pen * 1.0e-10);  // FP64-build rule of the reference for this stage
    }
  }
}

// A fitted vector's last Gram and norm (one CTA), before the next one begins.
__global__ void __launch_bounds__(kAccThreads) gsg_finish_kernel(GsParams p, int v) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ dw red[kAccThreads / 32];
  const GgScratch s = gg_scratch(p);
  gg_finish<kAccThreads>(p, s, v, true, reinterpret_cast<dw*>(smem_raw), red);
  if (v == p.nbloc - 1 && threadIdx.x == 0 && s.flag[1]) atomicOr(p.status, 1);
}

// Shared memory of the accumulation CTAs (dw): the slab's factors of modes jp
// and j, F's of mode jp, the slab's products, the parts received from the
// cluster and their coefficients; or (equations CTA) F's factor and the normal
// equations.
__host__ __device__ inline size_t acc_dw(int R, int npm) {
  const size_t row = npm | 1, sl = gg_slab_rows(R), RR = (size_t)R * R;
  const size_t slab = 2 * sl * row + R * row + sl * R + (size_t)R * npm + kCl * kCl + kCl, eq = R * row + RR;
  return slab > eq ? slab : eq;
}

// The equations CTA of mode step j: G_jp from the new factor (times the other
// modes' product, formed while mode jp was solved),
// BB = prod_{d != j} G_d + pen I and its FP32 inverse.
template <int NT>
__device__ void gg_equations(const GsParams& p, const GgScratch& s, int iv, int j, int jp, dw* sm, float* prow,
                             int* flag) {
  const int R = p.R, RR = R * R, D = p.D, rv = gg_rank(p, iv);
  const dw* G = s.P + (size_t)iv * D * RR;
  dw* bb = sm;  // [rv][rv]
  dw* F = sm + RR;
  if (threadIdx.x == 0) *flag = 1;
  gg_after_previous();
  gg_release_next();
  const dw pen = s.pen[0];
  const bool gram = jp >= 0 && jp != j;
  const int n = gram ? p.nbas[jp] : 0, ld = gg_ld(n);
  if (gram) gg_load(F, s.qf + (size_t)iv * R * p.nD + (size_t)R * p.off[jp], rv, n, NT);
  __syncthreads();
  // entries (a, b), b <= a, one after the other over the threads
  for (int e = threadIdx.x; e < rv * (rv + 1) / 2; e += NT) {
    int a = (int)((sqrtf(8.f * e + 1.f) - 1.f) * 0.5f);
    while ((a + 1) * (a + 2) / 2 <= e) ++a;
    while (a * (a + 1) / 2 > e) --a;
    const int b = e - a * (a + 1) / 2;
    dw x;
    if (gram) {
      const dw pg = s.pg[a * R + b];
      const dw *y = F + (size_t)a * ld, *z = F + (size_t)b * ld;
      dw_acc acc = acc_zero();
#pragma unroll 4
      for (int m = 0; m < n; ++m) acc_fma(acc, y[m], z[m]);
      x = dw_mul(acc_value(acc), pg);
    } else {
      const dw* g = G + a * R + b;
      x = gg_chain(dw_make(1.f), gg_fetch(g, RR, D, j, -1), g, RR, D, j, -1);
    }
    if (a == b) x = dw_add(x, pen);
    bb[a * rv + b] = bb[b * rv + a] = x;
    s.bb[a * rv + b] = s.bb[b * rv + a] = x;
  }
  __syncthreads();
  if (!gg_by_rows(R)) {
    if ((int)threadIdx.x < 32 * dwsolve::invert_warps(rv)) dwsolve::invert_any(bb, rv, s.inv, prow, flag);
    __syncthreads();
    if (threadIdx.x == 0) s.flag[0] = *flag;
    return;
  }
  constexpr int kRR = dwsolve::kRowRank * dwsolve::kRowRank;
  __shared__ dw Iv[kRR];
  __shared__ float gi[kRR], Ef[kRR], emax[dwsolve::kSolverWarps];
  if (threadIdx.x < dwsolve::kSolverThreads) {
    if (threadIdx.x < 32) dwsolve::invert_any(bb, rv, gi, prow, flag);
    dwsolve::solver_sync();
    const bool ok = *flag != 0 && dwsolve::correct_inverse<0>(bb, rv, gi, Iv, Ef, emax);
    dwsolve::solver_sync();
    for (int e = threadIdx.x; e < rv * rv; e += dwsolve::kSolverThreads) s.iv[e] = Iv[e];
    if (threadIdx.x == 0) s.flag[0] = ok;
  }
}

// Mode step j of vector iv, mode jp solved just before (jp < 0: none yet).
template <int NT>
__global__ void __launch_bounds__(NT, 1024 / NT) gsg_accum_kernel(GsParams p, int iv, int j, int jp) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ dw red[NT / 32];
  __shared__ float prow[2 * 72];
  __shared__ int flag;
  const GgScratch s = gg_scratch(p);
  const int R = p.R, RR = R * R, D = p.D, nj = p.nbas[j], rv = gg_rank(p, iv), npm = p.npmax;
  const int S = gg_slabs(R), H = gg_slab_rows(R), last = gridDim.x - kCl;  // the last cluster: the equations
  const int rank = blockIdx.x % kCl, k = blockIdx.x / S, r0 = blockIdx.x % S * H;
  dw* sm = reinterpret_cast<dw*>(smem_raw);
  if ((int)blockIdx.x >= last) {
    if ((int)blockIdx.x == last) gg_equations<NT>(p, s, iv, j, jp, sm, prow, &flag);
    return;
  }
  gg_arrive();  // this CTA runs: its peers may store into it once all have arrived
  const size_t row = npm | 1;
  dw* Qp = sm;                       // [H] rows of Q_k^jp
  dw* A = Qp + H * row;              // [H][nj] rows of c Q_k^j
  dw* F = A + H * row;               // [rv] rows of F^jp
  dw* W = F + R * row;               // [H][R] products over d != j
  dw* bs = W + (size_t)H * R;        // [8][an eighth of the entries] parts received
  dw* gs = bs + (size_t)R * npm + kCl * kCl;  // [8] shares of the coefficients received
  // entry o = i + m rv of the part is summed by CTA o / per of the cluster,
  // which receives it from CTA q at bs[q per + o mod per]
  const int per = (rv * nj + kCl - 1) / kCl;
  const int nr = k <= iv ? min(H, gg_rank(p, k) - r0) : 0;
  if (nr > 0) {
    const dw* q = s.qf + (size_t)k * R * p.nD;
    dw* P = s.P + (size_t)k * D * RR + (size_t)r0 * R;
    const bool self = k == iv;
    const int np = jp >= 0 ? p.nbas[jp] : 0, ld = gg_ld(np);
    const dw* qp = q + (jp >= 0 ? (size_t)R * p.off[jp] + (size_t)r0 * np : 0);
    const dw* qj = q + (size_t)R * p.off[j] + (size_t)r0 * nj;
    const dw* qc = s.qc + (size_t)k * R + r0;
    if (!self) {  // finished vectors: older than the previous kernel
      for (int e = threadIdx.x; e < nr * np; e += NT) {
        const int r = e / np;
        gg_cp8(Qp + r * ld + (e - r * np), qp + e);
      }
      for (int e = threadIdx.x; e < nr * nj; e += NT) A[e] = dw_mul(qc[e / nj], qj[e]);
    }
    gg_after_previous();
    gg_release_next();
    for (int e = threadIdx.x; e < rv * np; e += NT) {
      const int r = e / np;
      gg_cp8(F + r * ld + (e - r * np), s.qf + (size_t)iv * R * p.nD + (size_t)R * p.off[jp] + e);
    }
    if (self) {
      for (int e = threadIdx.x; e < nr * np; e += NT) {
        const int r = e / np;
        gg_cp8(Qp + r * ld + (e - r * np), qp + e);
      }
      for (int e = threadIdx.x; e < nr * nj; e += NT) A[e] = dw_mul(s.fc[r0 + e / nj], qj[e]);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    // products over d != j of entry (r, i) and its share of <Q_k, F>
    dw sum = dw_make(0.f);
    struct Held {
      GgChain c;
      dw pj, w;
    };
    auto pre = [&](int r, int i) {
      Held h;
      const dw* v = P + r * R + i;
      h.c = gg_fetch(v, RR, D, j, jp);
      h.pj = jp == j ? dw_make(1.f) : v[(size_t)j * RR];
      h.w = self ? dw_make(0.f) : dw_mul(qc[r], s.fc[i]);
      return h;
    };
    auto emit = [&](int r, int i, dw x, const Held& h) {
      const dw* v = P + r * R + i;
      const dw pj = jp == j ? x : h.pj;
      if (jp >= 0) P[(size_t)jp * RR + r * R + i] = x;
      x = gg_chain(jp >= 0 && jp != j ? x : dw_make(1.f), h.c, v, RR, D, j, jp);
      W[r * R + i] = x;
      if (!self) sum = dw_add(sum, dw_mul(dw_mul(x, pj), h.w));
    };
    if (jp >= 0) gg_products<NT>(Qp, F, ld, nr, rv, np, pre, emit);
    else
      for (int e = threadIdx.x; e < nr * rv; e += NT) emit(e / rv, e % rv, dw_make(1.f), pre(e / rv, e % rv));
    const dw g = gg_block_sum<NT>(sum, red);  // its barriers also order W
    gg_wait();
    if (threadIdx.x < kCl) gg_push(gs + rank, threadIdx.x, self ? dw_make(1.f) : dw_neg(g));
    auto push = [&](int i, int m, dw x) {
      const int o = i + m * rv, r = o / per;
      gg_push(bs + rank * per + (o - r * per), r, x);
    };
    if (rv > 16) gg_part<NT, 32>(A, W, R, nr, nj, rv, push);
    else gg_part<NT, 16>(A, W, R, nr, nj, rv, push);
  } else {
    gg_after_previous();
    gg_release_next();
    gg_wait();
    if (threadIdx.x < kCl) gg_push(gs + rank, threadIdx.x, dw_make(0.f));
  }
  gg_arrive();
  gg_wait();
  // coefficients of the cluster's slabs (their vector's shares added up); an
  // empty slab's part was not written
  __shared__ dw gt[kCl];
  __shared__ int used[kCl];
  if (threadIdx.x < kCl) {
    const int q = threadIdx.x, kk = (blockIdx.x - rank + q) / S, c0 = q - q % S;
    dw g = gs[c0];
    if (kk < iv)
      for (int u = 1; u < S; ++u) g = dw_add(g, gs[c0 + u]);
    gt[q] = g;
    used[q] = kk <= iv && q % S * H < gg_rank(p, kk);
  }
  __syncthreads();
  dw* part = s.part + (size_t)(blockIdx.x / kCl) * R * npm;
  for (int e = threadIdx.x; e < per && rank * per + e < rv * nj; e += NT) {
    const int o = rank * per + e, m = o / rv, i = o - m * rv;
    dw_acc acc = acc_zero();
#pragma unroll
    for (int q = 0; q < kCl; ++q)
      if (used[q]) acc_fma(acc, gt[q], bs[q * per + e]);
    part[i + m * R] = acc_value(acc);
  }
}

// Shared memory of the solve CTAs: BB, its inverse, and an eighth of the columns.
struct SolSmem {
  dw *BB, *X, *b0, *res, *dinv, *u, *norm;  // norm: [8][2][R] row maxima and scaled sums of squares of the cluster
  float *inv, *rred;
};
__host__ __device__ inline size_t sol_carve(int R, int npm, unsigned char* base, SolSmem* s) {
  size_t o = 0;
  auto take = [&](size_t bytes) -> unsigned char* {
    const size_t r = o;
    o += (bytes + 15) / 16 * 16;
    return base ? base + r : nullptr;
  };
  const size_t cols = (npm + kCl - 1) / kCl, Rn = (size_t)R * cols, RR = (size_t)R * R;
  s->BB = (dw*)take(sizeof(dw) * RR);
  s->X = (dw*)take(sizeof(dw) * Rn);
  s->b0 = (dw*)take(sizeof(dw) * Rn);
  s->res = (dw*)take(sizeof(dw) * Rn);
  s->dinv = (dw*)take(sizeof(dw) * R);
  s->u = (dw*)take(sizeof(dw) * R);
  s->norm = (dw*)take(sizeof(dw) * kCl * 2 * R);
  s->inv = (float*)take(sizeof(float) * RR);
  s->rred = (float*)take(sizeof(float) * 4);
  return o;
}

// Entry of the right-hand side: the clusters' parts in order.
__device__ __forceinline__ dw gg_sum_parts(const dw* q, int nparts, size_t stride) {
  dw_acc acc = acc_zero();
  for (int g0 = 0; g0 < nparts; g0 += 16) {
    dw v[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) v[u] = g0 + u < nparts ? q[(size_t)(g0 + u) * stride] : dw_make(0.f);
#pragma unroll
    for (int u = 0; u < 16; ++u) acc_add(acc, v[u]);
  }
  return acc_value(acc);
}

// The Grams' products over the modes other than j (solved now) and jn (the next one): the
// mode solved before j is up to date.  Entries e0, e0 + step, ...
__device__ __forceinline__ void gg_gram_products(const GsParams& p, const GgScratch& s, int iv, int j, int jn, int n, int e0,
                                                 int step) {
  const int R = p.R, RR = R * R;
  const dw* G = s.P + (size_t)iv * p.D * RR;
  for (int e = e0; e < R * n; e += step) {
    const dw* g = G + e;
    if (e % R < n) s.pg[e] = gg_chain(dw_make(1.f), gg_fetch(g, RR, p.D, j, jn), g, RR, p.D, j, jn);
  }
}

// The weights (one warp): the row norms, scaled by the power of two that brings the largest
// into [0.5, 1); padding terms none.
__device__ __forceinline__ void gg_put_weights(const GgScratch& s, const dw* nrm, int n, int R) {
  const int lane = threadIdx.x & 31;
  float big = 0.f;
  for (int i = lane; i < n; i += 32) big = fmaxf(big, fabsf(nrm[i].hi));
  for (int o = 16; o > 0; o >>= 1) big = fmaxf(big, __shfl_xor_sync(0xffffffffu, big, o));
  int ex = 0;
  if (big > 0.f && big <= 3.4028235e38f) frexpf(big, &ex);
  for (int i = lane; i < R; i += 32)
    s.fc[i] = i < n ? dw_make(ldexpf(nrm[i].hi, -ex), ldexpf(nrm[i].lo, -ex)) : dw_make(0.f);
}

// The solve of mode step j: CTA `rank` of the cluster has columns m0 .. m0 + nc.
// A second cluster forms the Grams' products over the modes other than j and
// the next one, jn (jn < 0: no next step), for the next step's equations.
__global__ void __launch_bounds__(kSolThreads) gsg_solve_kernel(GsParams p, int iv, int j, int jn, int nparts,
                                                                int write64) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  SolSmem m;
  sol_carve(p.R, p.npmax, smem_raw, &m);
  const GgScratch s = gg_scratch(p);
  const int R = p.R, nj = p.nbas[j], n = gg_rank(p, iv), npm = p.npmax, rank = blockIdx.x % kCl;
  if (blockIdx.x >= kCl) {
    gg_after_previous();
    gg_release_next();
    gg_gram_products(p, s, iv, j, jn, n, rank * kSolThreads + threadIdx.x, kCl * kSolThreads);
    return;
  }
  const int per = (nj + kCl - 1) / kCl, m0 = min(nj, rank * per), nc = min(nj, m0 + per) - m0;
  gg_arrive();  // this CTA runs: its peers may store into it once all have arrived
  gg_after_previous();
  gg_release_next();
  for (int e = threadIdx.x; e < n * n; e += kSolThreads) {
    gg_cp8(m.BB + e, s.bb + e);
    gg_cp4(m.inv + e, s.inv + e);
  }
  // the right-hand side: the clusters' parts in order
  for (int e = threadIdx.x; e < n * nc; e += kSolThreads) {
    const int c = e / n, i = e - c * n;
    m.b0[e] = gg_sum_parts(s.part + i + (size_t)(m0 + c) * R, nparts, (size_t)R * npm);
  }
  const bool gj_ok = s.flag[0] != 0;
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  if (nc > 0 && !(gj_ok && dwsolve::refine_any<kSolThreads>(m.BB, n, m.b0, m.X, nc, m.inv, m.res, m.rred))) {
    if (threadIdx.x < dwsolve::kSolverThreads) {
      for (int e = threadIdx.x; e < n * nc; e += dwsolve::kSolverThreads) m.X[e] = m.b0[e];
      const int bad = dwsolve::dw_ldlt(m.BB, n, m.dinv, m.u);
      dwsolve::dw_ldlt_solve(m.BB, n, m.dinv, m.X, nc);
      if (threadIdx.x == 0 && bad) s.flag[1] = 1;
    }
  }
  __syncthreads();
  gg_wait();
  // row norms: this CTA's largest |x| and sum of squares scaled by it, then
  // the cluster's
  for (int i = threadIdx.x; i < n; i += kSolThreads) {
    float big = 0.f;
    for (int c = 0; c < nc; ++c) big = fmaxf(big, fabsf(m.X[i + c * n].hi));
    dw_acc sq = acc_zero();
    if (big > 0.f) {
      const dw il = dw_rcp(dw_make(big));
      for (int c = 0; c < nc; ++c) {
        const dw y = dw_mul(m.X[i + c * n], il);
        acc_fma(sq, y, y);
      }
    }
    const dw sum = acc_value(sq);
#pragma unroll
    for (int r = 0; r < kCl; ++r) {
      gg_push(m.norm + 2 * rank * R + i, r, dw_make(big));
      gg_push(m.norm + (2 * rank + 1) * R + i, r, sum);
    }
  }
  gg_arrive();
  gg_wait();
  dw* nrm = m.dinv;  // norm and its reciprocal
  dw* rcp = m.u;
  for (int i = threadIdx.x; i < n; i += kSolThreads) {
    float big = 0.f;
#pragma unroll
    for (int r = 0; r < kCl; ++r) big = fmaxf(big, m.norm[2 * r * R + i].hi);
    if (!(big > 0.f)) {  // NaN, as the reference's zero-row norm
      nrm[i] = rcp[i] = dw_make(__int_as_float(0x7fffffff));
      continue;
    }
    const dw il = dw_rcp(dw_make(big));
    dw_acc sum = acc_zero();
#pragma unroll
    for (int r = 0; r < kCl; ++r) {
      const dw t = dw_mul(m.norm[2 * r * R + i], il);
      acc_fma(sum, m.norm[(2 * r + 1) * R + i], dw_mul(t, t));
    }
    const dw x = dw_mul(dw_make(big), dw_sqrt(acc_value(sum)));
    nrm[i] = x;
    rcp[i] = dw_rcp(x);
  }
  __syncthreads();
  // the new factor (padding terms: the first unit vector)
  dw* f = s.qf + (size_t)iv * R * p.nD + (size_t)R * p.off[j];
  double* fb = p.base + (size_t)iv * R * p.nD + p.off[j];
  for (int e = threadIdx.x; e < R * nc; e += kSolThreads) {
    const int i = e / nc, c = e - i * nc;
    const dw x = i < n ? dw_mul(m.X[i + c * n], rcp[i]) : dw_make(m0 + c == 0 ? 1.f : 0.f);
    f[i * nj + m0 + c] = x;
    if (write64) fb[(size_t)i * p.nD + m0 + c] = dw_to_double(x);
  }
  if (rank == 0 && threadIdx.x < 32) gg_put_weights(s, nrm, n, R);
}

// The solve of mode step j for ranks up to 16, by the inverse formed beside
// the accumulation: one CTA, a row of the solution per warp, its norm there too.  CTAs 1..8:
// the Grams' products, as the second cluster above.
constexpr int kRowThreads = 32 * dwsolve::kRowRank;
template <int NC>
__device__ __forceinline__ void gg_row(const GsParams& p, const GgScratch& s, int iv, int j, int n, const dw* Iv, const dw* b0,
                                       const dw* X, bool solved, int write64, dw* nrm) {
  const int R = p.R, nj = p.nbas[j], i = threadIdx.x >> 5, lane = threadIdx.x & 31;
  dw x[NC ? NC : 1], nr;
  if (i < n) {
    dwsolve::row_product<0, NC>(Iv + i, n, b0, nj, solved, X + i, x);
    dwsolve::row_normalise<NC>(x, &nr);
    if (lane == 0) nrm[i] = nr;
  }
  dw* f = s.qf + (size_t)iv * R * p.nD + (size_t)R * p.off[j] + (size_t)i * nj;
  double* fb = p.base + (size_t)iv * R * p.nD + p.off[j] + (size_t)i * p.nD;
#pragma unroll
  for (int q = 0; q < (NC ? NC : 1); ++q) {
    const int m = (NC ? lane : lane & 15) + 32 * q;
    if (m >= nj || (!NC && lane >= 16)) continue;
    const dw y = i < n ? x[q] : dw_make(m == 0 ? 1.f : 0.f);  // padding terms: the first unit vector
    f[m] = y;
    if (write64) fb[m] = dw_to_double(y);
  }
}
__global__ void __launch_bounds__(kRowThreads) gsg_solve_rows_kernel(GsParams p, int iv, int j, int jn, int nparts,
                                                                    int write64) {
  __shared__ dw Iv[dwsolve::kRowRank * dwsolve::kRowRank], b0[dwsolve::kRowRank * 64], nrm[dwsolve::kRowRank];
  const GgScratch s = gg_scratch(p);
  const int R = p.R, nj = p.nbas[j], n = gg_rank(p, iv), npm = p.npmax, t = threadIdx.x;
  gg_after_previous();
  gg_release_next();
  if (blockIdx.x > 0) {
    gg_gram_products(p, s, iv, j, jn, n, (blockIdx.x - 1) * kRowThreads + t, kCl * kRowThreads);
    return;
  }
  const bool solved = s.flag[0] != 0;
  if (t < n * n) Iv[t] = (solved ? s.iv : s.bb)[t];
  // the right-hand side: the clusters' parts in order
  for (int e = t; e < n * nj; e += kRowThreads) {
    const int m = e / n, i = e - m * n;
    b0[i * nj + m] = gg_sum_parts(s.part + i + (size_t)m * R, nparts, (size_t)R * npm);
  }
  __syncthreads();
  __shared__ dw X[dwsolve::kRowRank * 64], dinv[dwsolve::kRowRank], u[dwsolve::kRowRank];
  if (!solved) {
    if (t < dwsolve::kSolverThreads) {
      for (int e = t; e < n * nj; e += dwsolve::kSolverThreads) X[e] = b0[e % n * nj + e / n];
      const int bad = dwsolve::dw_ldlt(Iv, n, dinv, u);
      dwsolve::dw_ldlt_solve(Iv, n, dinv, X, nj);
      if (t == 0 && bad) s.flag[1] = 1;
    }
    __syncthreads();
  }
  if (t >> 5 < R) {
    if (nj <= 16) gg_row<0>(p, s, iv, j, n, Iv, b0, X, solved, write64, nrm);
    else if (nj <= 32) gg_row<1>(p, s, iv, j, n, Iv, b0, X, solved, write64, nrm);
    else gg_row<2>(p, s, iv, j, n, Iv, b0, X, solved, write64, nrm);
  }
  __syncthreads();
  if (t < 32) gg_put_weights(s, nrm, n, R);
}

// A launch (in clusters of eight, or of single CTAs) whose CTAs may start before the previous
// kernel has finished (they wait for it themselves).
template <class... Args>
int gg_step_launch(void (*kern)(Args...), int grid, int cluster, int threads, size_t smem, cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  MLCP_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, args...));
  return kOk;
}

}  // namespace

size_t gs_grid_dw(int nbloc, int R, int nD, int D, int npm) {
  GgScratch s;
  return gg_carve(nbloc, R, D, nD, npm, nullptr, &s);
}

int gs_grid_launch(const GsParams& p, cudaStream_t st) {
  const int R = p.R, npm = p.npmax;
  SolSmem m;
  const size_t s_acc = sizeof(dw) * acc_dw(R, npm), s_two = sizeof(dw) * 2 * (size_t)R * (npm | 1),
               s_sol = sol_carve(R, npm, nullptr, &m);
  MLCP_CUDA_TRY(cudaFuncSetAttribute(gsg_first_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s_two));
  MLCP_CUDA_TRY(cudaFuncSetAttribute(gsg_finish_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s_two));
  // ranks up to 16 have at most 256 entries per slab: CTAs of 256 threads, four to an SM
  const int acc_threads = R <= 16 ? kAccThreads / 2 : kAccThreads;
  void (*accum)(GsParams, int, int, int) = R <= 16 ? gsg_accum_kernel<kAccThreads / 2> : gsg_accum_kernel<kAccThreads>;
  void (*overlap)(GsParams, int) = R <= 16 ? gsg_overlap_kernel<kAccThreads / 2> : gsg_overlap_kernel<kAccThreads>;
  MLCP_CUDA_TRY(cudaFuncSetAttribute(overlap, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s_two));
  MLCP_CUDA_TRY(cudaFuncSetAttribute(accum, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s_acc));
  MLCP_CUDA_TRY(cudaFuncSetAttribute(gsg_solve_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s_sol));
  gsg_first_kernel<<<1, kAccThreads, s_two, st>>>(p);
  MLCP_CUDA_TRY(cudaGetLastError());
  for (int iv = 1; iv < p.nbloc; ++iv) {
    overlap<<<dim3(iv + 1, p.D), acc_threads, s_two, st>>>(p, iv);
    MLCP_CUDA_TRY(cudaGetLastError());
    const int ncl = gg_clusters(iv + 1, R);
    int jp = -1;
    for (int it = 0; it < p.nals; ++it)
      for (int j = 0; j < p.D; ++j) {
        if (int rc = gg_step_launch(accum, (ncl + 1) * kCl, kCl, acc_threads, s_acc, st, p, iv, j, jp))
          return rc;
        const bool more = it + 1 < p.nals || j + 1 < p.D;
        const int jn = j + 1 < p.D ? j + 1 : 0, last = it == p.nals - 1 ? 1 : 0;
        if (int rc = gg_by_rows(R)
                         ? gg_step_launch(gsg_solve_rows_kernel, more ? 1 + kCl : 1, 1, kRowThreads, (size_t)0, st, p, iv, j,
                                          jn, ncl, last)
                         : gg_step_launch(gsg_solve_kernel, more ? 2 * kCl : kCl, kCl, kSolThreads, s_sol, st, p, iv, j, jn,
                                          ncl, last))
          return rc;
        jp = j;
      }
    gsg_finish_kernel<<<1, kAccThreads, s_two, st>>>(p, iv);
    MLCP_CUDA_TRY(cudaGetLastError());
  }
  return kOk;
}

}  // namespace mlcp
