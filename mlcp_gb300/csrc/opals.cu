// ALS-fitted Hamiltonian applications, one persistent CTA per vector (small
// nodes; opals_grid.cu has the form for larger ones).
//
// Reference: POW_ALS (src/intertw_mvp.cu:452-497) and PRODHV_ALS (:501-549)
// with mvp_build_linear_system (:380-448).  For mode j the reference builds,
// for every term t, G = h_t Fo (all modes, mvp_kernel :39), then
// PS = prod_{d!=j} <G^d, F^d> (constpstot) and accumulates
// b(i,n) += sum_r c_r G_r^j(n) PS(r,i) (constbjk): 3T launches per mode step.
//
// Here the same b is assembled from per-mode operator Grams
//   M[d][u](r,i) = <h_u Fo_r^d, F_i^d>     (one R x R matrix per distinct operator u of mode d)
// which change only when mode d of F changes:
//   W_u = sum_{t: op(t,j) = u} alpha_t prod_{d!=j} M[d][op(t,d)]
//   b(i,n) = sum_u sum_r c_r W_u(r,i) (h_u Fo_r^j)(n)
// so a mode step costs O(T R^2 D) instead of O(T R (sum_d n_d^2 + R nD)).
// The energy shift enters as an identity term with weight -E; for ishift < 0
// b changes sign, as in the reference.
//
// Precision.  The penalty is the reference's FP64-build rule (1e-10 max c,
// src/als.cu:248-267).  With it the normal equations of a nearly converged
// vector (whose terms are close to linearly dependent) have condition
// numbers up to 1e10, so any noise in b along their near-null directions is
// amplified by up to 1e10: FP32 right-hand sides (24 bits) made the weights
// blow up over successive cycles.  Everything here therefore runs in
// double-word arithmetic (dword.cuh, about 48 bits): the factors of F and Fo,
// the operators, the operator Grams M, the term products W, h_u Fo_j, the
// right-hand sides, the normal equations (prod_{d!=j} F_d F_d^T + pen I),
// their solve (FP32 inverse as the preconditioner of a double-word
// refinement, or a double-word LDL^T), the F Grams and the weight
// normalisation; the factors are written out in FP64.  In POW the weights
// are rescaled by a power of two after every mode step
// (rescale_weights_warp), which keeps them in the FP32 exponent range of
// the double-word values without changing the sweep's result.
#include <algorithm>

#include "common.cuh"
#include "dword.cuh"
#include "dwsolve.cuh"
#include "fastdiv.cuh"
#include "intertwine.cuh"
#include "opstep.cuh"

namespace mlcp {

namespace {

constexpr int kThreads = kStepThreads;

struct OpSmem {
  StepSmem st;    // the step from the normal equations on
  dw* f;          // [R][ldf] current F
  dw* fo;         // [R][ldf] Fo; aliases f for POW
  dw* cfo;        // [R] weights of Fo
  int* moff;      // [T][D] offset of each term's operator Gram per mode
  int* ord;       // [D][T] terms grouped by their operator at each mode
  int* gst;       // [D][umax+1] group starts
  dw* alpha;      // [T] term coefficients
  dw *Ms, *Ws, *Zs;  // operator Grams, term products, h_u Fo_j
  dw* hs;         // [utot][npmax][ldh] the operators
  dw* G;          // [D][R][R] Grams of F (with zmodes; else in global memory)
  FastDiv* fd;    // [2 D] divisors n_d and R n_d (index splits by multiplication)
  FastDiv fdr, fdrr;  // R, R R
  int ldf, ldh;   // row strides: odd, so that lanes on different rows read different banks
  int zmodes;     // 1: h_u Fo_j of every mode is kept in Zs, else of the current one
};

// Terms x modes up to which the one-CTA form tabulates the Gram offsets.
constexpr int kMoffMax = 8192;
// Multiply-adds per mode step and vector up to which the one-CTA form is
// taken: a grid step costs four launches (22 us at least, whatever the block),
// a step of the one-CTA form what its one CTA takes.  Measured steps, one CTA
// against grid: 6 modes of 10, rank 16 (45 k) 13.3 against 23.7 us; 4 of 6,
// rank 8, 40 terms (31 k) 14.8 against 34; 8 of 10, rank 20 (90 k) 22 against
// 35; 8 of 20, rank 16 (106 k) 19.8 against 28; 3 of 30, rank 16 (132 k) 27.5
// against 37; 2 of 24, rank 24 (168 k) 52 against 64.  Shapes beyond that hardly
// fit one CTA's shared memory.
constexpr double kOneCtaWork = 1.8e5;
// What bounds a step of the one-CTA form is the latency of its phases (about 23 k cycles for
// 6 modes of 10 at rank 16: products of the longest term group 8 k, solve 7 k,
// right-hand side 3 k, operators and their Grams 5 k), hence 512 threads, row strides
// without bank conflicts, index splits by multiplication and h_u Fo_j kept from the step
// before where it fits: 18.5 us a step before, 13.3 now.


// Carves the shared memory (null base: sizes only); returns the bytes.  `keep`: h_u Fo_j of
// every mode is kept.
__host__ __device__ inline size_t carve(OpSmem& s, unsigned char* base, const OpTable& t, bool separate_fo, bool keep) {
  size_t o = (step_carve(s.st, base, t.R, t.npmax) + 15) / 16 * 16;
  auto take = [&](size_t bytes) -> unsigned char* {
    const size_t r = o;
    o += (bytes + 15) / 16 * 16;
    return base ? base + r : nullptr;
  };
  const size_t Rn = (size_t)t.R * t.npmax, RR = (size_t)t.R * t.R;
  s.ldf = t.nDp | 1;
  s.ldh = t.npmax | 1;
  s.f = (dw*)take(sizeof(dw) * t.R * s.ldf);
  s.fo = separate_fo ? (dw*)take(sizeof(dw) * t.R * s.ldf) : s.f;
  s.G = keep ? (dw*)take(sizeof(dw) * t.D * RR) : nullptr;
  s.cfo = (dw*)take(sizeof(dw) * t.R);
  s.moff = (int*)take(sizeof(int) * t.T * t.D);
  s.ord = (int*)take(sizeof(int) * t.T * t.D);
  s.gst = (int*)take(sizeof(int) * t.D * (t.umax + 1));
  s.alpha = (dw*)take(sizeof(dw) * t.T);
  s.fd = (FastDiv*)take(sizeof(FastDiv) * 2 * t.D);
  s.hs = (dw*)take(sizeof(dw) * t.utot * t.npmax * s.ldh);
  s.Ms = (dw*)take(sizeof(dw) * t.utot * RR);
  s.Ws = (dw*)take(sizeof(dw) * t.umax * RR);
  s.zmodes = keep ? 1 : 0;
  s.Zs = (dw*)take(sizeof(dw) * (keep ? t.utot : t.umax) * Rn);
  return o;
}

// Z_u(r, m) = sum_k h_u(m, k) x_r(k) for the operators u of mode j (identity operators copy),
// Z [nu][R][npmax]; threads t0, t0 + nt, ...
__device__ __forceinline__ void apply_operators(const OpTable& t, const OpSmem& s, const dw* x, int j, dw* Z, int t0, int nt) {
  const int R = t.R, n = t.nbas[j], op = t.offp[j], npm = t.npmax, nu = t.uoff[j + 1] - t.uoff[j];
  for (int item = t0; item < nu * R * n; item += nt) {
    int u, rem, r, m;
    s.fd[2 * j + 1].divmod((unsigned)item, &u, &rem);
    s.fd[2 * j].divmod((unsigned)rem, &r, &m);
    const int ug = t.uoff[j] + u;
    const dw* xr = x + r * s.ldf + op;
    dw val;
    if (t.ident[ug]) {
      val = xr[m];
    } else {
      const dw* h = s.hs + ((size_t)ug * npm + m) * s.ldh;
      dw_acc acc = acc_zero();
#pragma unroll 4
      for (int k = 0; k < n; ++k) acc_fma(acc, h[k], xr[k]);
      val = acc_value(acc);
    }
    Z[(size_t)u * R * npm + r * npm + m] = val;
  }
}

// M_u(r, i) = sum_m Z_u(r, m) F_i(m) for the operators u of mode j.
__device__ __forceinline__ void operator_grams(const OpTable& t, const OpSmem& s, const dw* Z, int j, dw* M) {
  const int R = t.R, RR = R * R, n = t.nbas[j], op = t.offp[j], npm = t.npmax, nu = t.uoff[j + 1] - t.uoff[j];
  for (int item = threadIdx.x; item < nu * RR; item += kThreads) {
    int u, e, r, i;
    s.fdrr.divmod((unsigned)item, &u, &e);
    s.fdr.divmod((unsigned)e, &r, &i);
    const dw *z = Z + (size_t)u * R * npm + r * npm, *fi = s.f + i * s.ldf + op;
    dw_acc acc = acc_zero();
#pragma unroll 4
    for (int m = 0; m < n; ++m) acc_fma(acc, z[m], fi[m]);
    M[(size_t)(t.uoff[j] + u) * RR + e] = acc_value(acc);
  }
}

// Double-word Gram of mode d of F from the FP64 factors (set-up only).
__device__ void f_gram_from64(const OpTable& t, int d, const double* fb, int nD, dw* G) {
  const int R = t.R, n = t.nbas[d], o = t.off[d];
  for (int e = threadIdx.x; e < R * R; e += blockDim.x) {
    const int i = e % R, i2 = e / R;
    double acc = 0.0;
    for (int q = 0; q < n; ++q) acc += fb[(size_t)i * nD + o + q] * fb[(size_t)i2 * nD + o + q];
    G[e] = dw_from_double(acc);
  }
}

}  // namespace

__global__ void __launch_bounds__(kThreads, 1) opals_kernel(OpAlsParams p) {
  const OpTable& t = p.ops;
  const int v = blockIdx.x;
  const int R = t.R, D = t.D, T = t.T, npm = t.npmax, nD = p.nD, RR = R * R;
  const bool pow_mode = (p.mode == 0);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  OpSmem s;
  carve(s, smem_raw, t, !pow_mode, p.keep != 0);

  const double* fob = p.fo_base + (size_t)v * R * nD;
  const double* foc = p.fo_coef + (size_t)v * R;
  double* fb = p.f_base + (size_t)v * R * nD;
  double* fc = p.f_coef + (size_t)v * R;
  s.fdr = FastDiv((unsigned)R);
  s.fdrr = FastDiv((unsigned)RR);
  for (int q = threadIdx.x; q < 2 * D; q += blockDim.x) s.fd[q] = FastDiv((unsigned)(t.nbas[q / 2] * (q % 2 ? R : 1)));
  dw* M = s.Ms;
  dw* W = s.Ws;
  dw* Z = s.Zs;
  const int* moff = s.moff;
  for (int e = threadIdx.x; e < T * D; e += blockDim.x) {
    s.moff[e] = t.slot[e] * RR;
    s.ord[e] = t.order[e];
  }
  for (int e = threadIdx.x; e < D * (t.umax + 1); e += blockDim.x) s.gst[e] = t.gstart[e];
  for (int e = threadIdx.x; e < T; e += blockDim.x) s.alpha[e] = t.alphadw[e];
  for (int e = threadIdx.x; e < t.utot * npm * npm; e += blockDim.x) s.hs[(size_t)(e / npm) * s.ldh + e % npm] = t.hdw[e];
  dw* G = s.zmodes ? s.G : reinterpret_cast<dw*>(p.g64) + (size_t)v * D * RR;  // F's Grams per mode

  // ---- set-up: F (= Fo for PRODHV), double-word copies, Grams, penalty ----
  if (!pow_mode) {
    for (int e = threadIdx.x; e < R * nD; e += blockDim.x) fb[e] = fob[e];
    for (int e = threadIdx.x; e < R; e += blockDim.x) fc[e] = foc[e];
  }
  __syncthreads();
  for (int e = threadIdx.x; e < R * t.nDp; e += blockDim.x) {
    const int r = e / t.nDp, q = e % t.nDp;
    int d = 0;
    while (d + 1 < D && t.offp[d + 1] <= q) ++d;
    const int k = q - t.offp[d];
    const dw x = dw_from_double((k < t.nbas[d]) ? fob[(size_t)r * nD + t.off[d] + k] : 0.0);
    s.f[r * s.ldf + q] = x;
    if (!pow_mode) s.fo[r * s.ldf + q] = x;
  }
  for (int e = threadIdx.x; e < R; e += blockDim.x) {
    s.st.cf[e] = dw_from_double(fc[e]);
    s.cfo[e] = dw_from_double(foc[e]);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double pen = foc[0];
    for (int i = 1; i < R; ++i) pen = foc[i] > pen ? foc[i] : pen;
    s.st.misc[0] = dw_from_double(pen * p.pen_factor);
    s.st.flags[1] = 0;
    s.st.flags[2] = 1;
  }
  for (int d = 0; d < D; ++d) f_gram_from64(t, d, fb, nD, G + (size_t)d * R * R);
  __syncthreads();
  const dw pen = s.st.misc[0];
  const int rv = p.rank_v ? p.rank_v[v] : R;  // ragged: this vector's rank
  const size_t Rn = (size_t)R * npm;
  for (int d = 0; d < D; ++d) {
    dw* z = Z + (s.zmodes ? t.uoff[d] * Rn : 0);
    apply_operators(t, s, s.fo, d, z, threadIdx.x, kThreads);
    __syncthreads();
    operator_grams(t, s, z, d, M);
    if (!s.zmodes) __syncthreads();
  }
  __syncthreads();
  const dw eshift = dw_from_double(-(p.eshift_v ? p.eshift_v[v] : p.eshift));

  for (int sw = 0; sw < p.nsweeps; ++sw) {
    for (int j = 0; j < D; ++j) {
      const int nj = t.nbas[j], opj = t.offp[j];
      const int nu = t.uoff[j + 1] - t.uoff[j];
      const int* ord = s.ord + (size_t)j * T;
      const int* gs = s.gst + (size_t)j * (t.umax + 1);
      // -- normal equations from the Grams of the previous step:
      //    prod_{d != j} G_d + pen I --
      for (int e = threadIdx.x; e < RR; e += blockDim.x) {
        int i2, i;
        s.fdr.divmod((unsigned)e, &i2, &i);
        s.st.BB[e] = normal_equation(G, D, j, i, i2, R, rv, pen);
      }
      __syncthreads();
      // -- their FP32 inverse (the first warps) while the others form the
      //    right-hand side --
      const int w0 = 32 * dwsolve::invert_warps(R);
      dw* Zj = Z + (s.zmodes ? t.uoff[j] * Rn : 0);  // h_u Fo_j
      if (threadIdx.x < w0) {
        dwsolve::invert_any(s.st.BB, R, s.st.gi, s.st.prow, s.st.flags + 2);
      } else {
        const int wt = threadIdx.x - w0, nw = kThreads - w0;
        const dw* cg = pow_mode ? s.st.cf : s.cfo;
        // grouped term products W_u(r,i) = sum_{t in group u} alpha_t prod_{d != j} M[d][op(t,d)](r,i),
        // four terms at a time
        for (int item = wt; item < nu * RR; item += nw) {
          int u, e;
          s.fdrr.divmod((unsigned)item, &u, &e);
          dw_acc acc = acc_zero();
          for (int q = gs[u]; q < gs[u + 1]; q += 4) {
            dw pr[4];
            int tb[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const bool live = q + k < gs[u + 1];
              const int term = ord[live ? q + k : q];
              pr[k] = live ? s.alpha[term] : dw_make(0.f);
              tb[k] = term * D;
            }
            for (int d = 0; d < D; ++d) {
              if (d == j) continue;
#pragma unroll
              for (int k = 0; k < 4; ++k)
                pr[k] = dw_mul(pr[k], M[moff[tb[k] + d] + e]);
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) acc_add(acc, pr[k]);
          }
          if (u == 0 && p.ishift != 0) {
            dw prod = eshift;
            for (int d = 0; d < D; ++d)
              if (d != j) prod = dw_mul(prod, M[(size_t)t.uoff[d] * RR + e]);
            acc_add(acc, prod);
          }
          W[(size_t)u * RR + e] = dw_mul(acc_value(acc), cg[s.fdr.div((unsigned)e)]);
        }
        if (!s.zmodes) apply_operators(t, s, s.fo, j, Zj, wt, nw);
        asm volatile("bar.sync 2, %0;" ::"r"(nw) : "memory");
        // right-hand side b(i,n) = sum_u sum_r W_u(r,i) c_r Z_u(r,n)
        for (int e = wt; e < R * nj; e += nw) {
          int m, i;
          s.fdr.divmod((unsigned)e, &m, &i);
          dw_acc acc = acc_zero();
          for (int u = 0; u < nu; ++u) {
            const dw *w = W + (size_t)u * RR + i, *z = Zj + (size_t)u * Rn + m;
#pragma unroll 4
            for (int r = 0; r < R; ++r) acc_fma(acc, w[r * R], z[r * npm]);
          }
          const dw b = acc_value(acc);
          s.st.b0[i + m * R] = i >= rv ? dw_make(m == 0 ? 1.f : 0.f) : (p.ishift < 0 ? dw_neg(b) : b);
        }
      }
      __syncthreads();
      step_solve(s.st, R, nj);
      // -- the new factor: FP64 output, double-word copy and Gram --
      step_weights(s.st, R, rv, pow_mode, fc);
      step_factor(s.st, R, nj, fb + t.off[j], nD, s.f + opj, s.ldf, G + (size_t)j * RR);
      __syncthreads();
      // -- operator Grams of mode j with the new factor: h_u F_j for every
      //    operator (POW; PRODHV keeps h_u Fo_j), then M_u = (h_u F_j) F_j^T --
      if (pow_mode) {
        apply_operators(t, s, s.f, j, Zj, threadIdx.x, kThreads);
        __syncthreads();
      }
      operator_grams(t, s, Zj, j, M);
      if (threadIdx.x == 0) s.st.flags[2] = 1;
      __syncthreads();
    }
    if (pow_mode) step_renormalise(s.st, R, D, G, fc);
  }
  if (threadIdx.x == 0 && s.st.flags[1]) atomicOr(&p.status[v], 1);
}

// F, Fo and one mode step: what both forms' callers check against the
// device's limit.  (The grid form alone would need less; shapes beyond stay refused.)
size_t opals_smem_bytes(const OpTable& t) {
  StepSmem m;
  return step_carve(m, nullptr, t.R, t.npmax) +
         sizeof(dw) * ((size_t)2 * t.R * t.nDp + (size_t)t.R * t.npmax + (size_t)t.R);
}

namespace {

// Scratch that the vectors of one launch may take together.  The operator Grams, term products
// and h Fo of a vector are 8 (utot (R^2 + R n) + umax R^2) bytes: 48 MB at rank 30 on six
// modes of 48 functions and 400 operators each, so 16 GB are 360 such vectors, more than fill
// the GPU.  (Held for a whole block, h Fo of every mode would halve the longest operator list
// that 160 of them can have.)
constexpr size_t kScratchBytes = (size_t)16 << 30;
constexpr int kMaxVectors = 65535;  // gridDim.y and z of the grid form

int launch_vectors(const OpAlsParams& p, cudaStream_t st) {
  int dev = 0, limit = 0;
  MLCP_CUDA_TRY(cudaGetDevice(&dev));
  MLCP_CUDA_TRY(cudaDeviceGetAttribute(&limit, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  OpSmem s;
  OpAlsParams q = p;
  q.keep = carve(s, nullptr, p.ops, p.mode != 0, true) <= (size_t)limit ? 1 : 0;
  const size_t res = carve(s, nullptr, p.ops, p.mode != 0, q.keep != 0);
  // multiply-adds of one mode step of one vector: term products, operators
  // applied, operator Grams and right-hand side (mean over the modes)
  const OpTable& t = p.ops;
  const double R = t.R, nu = (double)t.utot / t.D, n = (double)t.nDp / t.D;
  const double work = (double)t.T * R * R * (t.D - 1) + nu * R * n * (n + 2.0 * R);
  const bool one = t.T * t.D <= kMoffMax && res <= (size_t)limit && work <= kOneCtaWork;
  if (!one) return opals_grid_launch(p, st);
  MLCP_CUDA_TRY(cudaFuncSetAttribute(opals_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)res));
  opals_kernel<<<p.nvec, kThreads, res, st>>>(q);
  MLCP_CUDA_TRY(cudaGetLastError());
  return kOk;
}

}  // namespace

int opals_vectors(const OpTable& t, int nvec) {
  const size_t per = sizeof(dw) * ((size_t)(t.utot + t.umax) * t.R * t.R + (size_t)t.utot * t.R * t.npmax);
  return (int)std::max<size_t>(1, std::min<size_t>(std::min(nvec, kMaxVectors), kScratchBytes / per));
}

int opals_launch(const OpAlsParams& p, cudaStream_t st) {
  const int most = opals_vectors(p.ops, p.nvec);
  const size_t R = p.ops.R;
  for (int v = 0; v < p.nvec; v += most) {
    OpAlsParams q = p;
    q.nvec = std::min(most, p.nvec - v);
    q.fo_base += v * R * p.nD;
    q.fo_coef += v * R;
    q.f_base += v * R * p.nD;
    q.f_coef += v * R;
    q.status += v;
    if (p.eshift_v) q.eshift_v += v;
    if (p.rank_v) q.rank_v += v;
    if (int rc = launch_vectors(q, st)) return rc;
  }
  return kOk;
}

}  // namespace mlcp
