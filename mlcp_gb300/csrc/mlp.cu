// Learned ALS warm start: training and inference kernels of a small MLP
// (BF16 weights and activations, FP32 accumulation) that proposes the
// starting factors of an ALS rank reduction.  No counterpart in the
// reference, which starts its GPU ALS from a random CP vector
// (GPU_ALS_AA, src/GPUIterate.f90:191-210, GetRandomCPvec) or from a
// randomised interpolative decomposition on the CPU (reduc_RID,
// src/REDUCTIONML.f90:483-551).
//
// GEMM on the 5th-generation tensor cores: C[M x N] = A[M x K] B[N x K]^T
// with A and B BF16, K-major (row-major, K contiguous), one CTA of 4 warps
// per 128 x BN output tile.  Per 64-wide K slice the operands are copied with
// cp.async into shared memory in the canonical no-swizzle K-major layout
// (8-row x 16-byte core matrices: core (r/8, k/8) at ((r/8) 8 + k/8) 128
// bytes, so the core-matrix stride is 128 B along K and 1024 B along M/N),
// through a ring of up to eight stages; one elected thread issues four
// tcgen05.mma (kind::f16, M = 128, K = 16 each) into a TMEM accumulator and
// commits them to the stage's mbarrier, which the copies into that stage
// wait on (bounded waits: on expiry the kernel records status bit 1, stops
// issuing and still frees its tensor memory).  The epilogue reads the
// accumulator with tcgen05.ld (warp w: rows 32w..32w+31) and applies bias,
// ReLU or the ReLU derivative, writing FP32 and/or BF16 (16 bytes at a time)
// and a transposed BF16 copy (coalesced along the rows; the operand layouts
// of the backward GEMMs).
//
// What bounds it: the network's GEMMs (768 x 256 x 576 and smaller) are 0.1 us
// of tensor work; their time is the latency of the first operand slices, the
// epilogue and the launch.  So the tile width BN is the widest that still
// gives every SM a tile, the whole K range is in flight at once when it fits
// the ring, and no lane writes single elements across rows.  With 256-wide
// tiles (six CTAs), two stages and element-wise stores the five shapes of a
// training step took 51-77 us each.
#include <algorithm>

#include <cuda_bf16.h>

#include <cstdint>

#include "common.cuh"
#include "mlp.cuh"

namespace mlcp {

namespace {

constexpr int kGemmThreads = 128;
constexpr int kBM = 128;
constexpr int kBK = 64;
constexpr int kMaxBN = 256;
constexpr int kMinBN = 32;
constexpr int kStageA = kBM * kBK * 2;       // bytes
constexpr int kWaitLimit = 1 << 22;

__device__ __forceinline__ uint32_t saddr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(saddr(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(saddr(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait; false when the limit was reached.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
  for (int it = 0; it < kWaitLimit; ++it)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(saddr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// All but the latest N committed groups of this thread have landed.
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Shared-memory matrix descriptor, no swizzle, K-major canonical layout:
// start address, leading (K-direction) core-matrix offset 128 B, stride
// (M/N-direction) core-matrix offset 1024 B, descriptor version 1.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr >> 4) & 0x3FFFu);
  d |= (uint64_t)(128u >> 4) << 16;
  d |= (uint64_t)(1024u >> 4) << 32;
  d |= (uint64_t)1 << 46;
  return d;
}

// Instruction descriptor of kind::f16: BF16 A and B, FP32 D, both K-major,
// M = 128, N = n.
__device__ __forceinline__ uint32_t idesc_bf16(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kBM >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(saddr(bar))
               : "memory");
}

// 32 consecutive FP32 columns of this warp's 32 TMEM lanes (lane = row).
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int q = 0; q < 32; ++q) v[q] = __uint_as_float(r[q]);
}

// Copy rows [r0, r0 + rows) x K slice [k0, k0 + 64) of a K-major BF16 matrix
// into the core-matrix layout at dst (one 16-byte chunk per copy).
__device__ __forceinline__ void stage_tile(unsigned char* dst, const __nv_bfloat16* src, int ld, int r0, int rows,
                                           int k0) {
  for (int c = threadIdx.x; c < rows * 8; c += kGemmThreads) {
    const int r = c >> 3, kc = c & 7;
    unsigned char* d = dst + (((r >> 3) * 8 + kc) << 7) + ((r & 7) << 4);
    cp_async16(d, src + (size_t)(r0 + r) * ld + k0 + kc * 8);
  }
}

// Ring stages for tiles of BN columns.
__host__ __device__ constexpr int gemm_stages(int bn) { return bn <= 64 ? 8 : 4; }

// Eight consecutive BF16 values as 16 bytes.
__device__ __forceinline__ uint4 pack8(const __nv_bfloat16 (&x)[8]) {
  uint32_t w[4];
#pragma unroll
  for (int q = 0; q < 4; ++q)
    w[q] = (uint32_t)__bfloat16_as_ushort(x[2 * q]) | ((uint32_t)__bfloat16_as_ushort(x[2 * q + 1]) << 16);
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// Whether rows of `ld` elements of `size` bytes at `ptr` start on 16-byte
// boundaries (their 8-element groups then do too).
__device__ __forceinline__ bool rows_aligned(const void* ptr, int ld, int size) {
  return ((reinterpret_cast<uintptr_t>(ptr) | (uintptr_t)((size_t)ld * size)) & 15u) == 0;
}

}  // namespace

// BN: the tile width (32, 64, 128 or 256); S = gemm_stages(BN).
template <int BN>
__global__ void __launch_bounds__(kGemmThreads, 1) mlp_gemm_kernel(MlpGemm p) {
  constexpr int S = gemm_stages(BN), kStageB = BN * kBK * 2;
  extern __shared__ __align__(1024) unsigned char gsm[];
  unsigned char* sA = gsm;                 // [S][kStageA]
  unsigned char* sB = gsm + S * kStageA;   // [S][kStageB]
  __shared__ __align__(8) uint64_t bar[S];
  __shared__ uint32_t tmem_base;
  const int m0 = blockIdx.x * kBM, n0 = blockIdx.y * BN;
  const int bn = min(BN, p.N - n0);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int KT = p.K / kBK;
  auto load = [&](int kt) {
    const int st = kt % S;
    stage_tile(sA + st * kStageA, p.A, p.lda, m0, kBM, kt * kBK);
    stage_tile(sB + st * kStageB, p.B, p.ldb, n0, bn, kt * kBK);
  };
  // one group per slice, empty ones past the end, so that the wait below
  // always means "slice kt has landed"
#pragma unroll
  for (int kt = 0; kt < S - 1; ++kt) {
    if (kt < KT) load(kt);
    cp_async_commit();
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) mbar_init(&bar[s], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(saddr(&tmem_base)),
                 "r"(BN)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base;
  const uint32_t idesc = idesc_bf16(bn);
  bool failed = false, aborted = false;
  for (int kt = 0; kt < KT; ++kt) {
    cp_async_wait<S - 2>();
    fence_proxy_async();
    aborted = __syncthreads_or(failed);
    if (aborted) break;
    const int st = kt % S;
    if (threadIdx.x == 0) {
      tc_fence_after();
      const uint32_t a0 = saddr(sA + st * kStageA), b0 = saddr(sB + st * kStageB);
#pragma unroll
      for (int kk = 0; kk < kBK / 16; ++kk)
        mma_bf16(tmem, smem_desc(a0 + kk * 256), smem_desc(b0 + kk * 256), idesc, (kt > 0 || kk > 0) ? 1u : 0u);
      mma_commit(&bar[st]);
    }
    if (kt + S - 1 < KT) {  // into the stage whose MMAs were committed in the previous iteration
      if (kt > 0 && !mbar_wait(&bar[(kt - 1) % S], (uint32_t)((kt - 1) / S) & 1u)) failed = true;
      if (!failed) load(kt + S - 1);
    }
    cp_async_commit();
  }
  // the last commit covers every MMA issued before it
  if (!aborted && !failed && !mbar_wait(&bar[(KT - 1) % S], (uint32_t)((KT - 1) / S) & 1u)) failed = true;
  tc_fence_before();
  aborted = __syncthreads_or(failed) || aborted;
  tc_fence_after();
  if (!aborted) {
    const int row = m0 + warp * 32 + lane;
    const uint32_t trow = tmem + ((uint32_t)(warp * 32) << 16);
    const bool live = row < p.valid_m;
    const bool vc = p.C && rows_aligned(p.C, p.ldc, 4), vb = p.Cb && rows_aligned(p.Cb, p.ldcb, 2),
               vm = p.act == 2 && rows_aligned(p.mask, p.ldm, 2);
    for (int c0 = 0; c0 < bn; c0 += 32) {
      float v[32];
      tmem_ld32(trow + (uint32_t)c0, v);
#pragma unroll
      for (int g = 0; g < 4; ++g) {  // eight columns at a time (bn is a multiple of 16)
        if (c0 + 8 * g >= bn) break;
        const int col = n0 + c0 + 8 * g;
        float x[8];
        __nv_bfloat16 xb[8], mk[8];
        if (p.act == 2) {
          if (vm) {
            *reinterpret_cast<uint4*>(mk) = *reinterpret_cast<const uint4*>(p.mask + (size_t)row * p.ldm + col);
          } else {
#pragma unroll
            for (int q = 0; q < 8; ++q) mk[q] = p.mask[(size_t)row * p.ldm + col + q];
          }
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          x[q] = v[8 * g + q];
          if (p.bias) x[q] += p.bias[col + q];
          if (p.act == 1) x[q] = fmaxf(x[q], 0.f);
          if (p.act == 2) x[q] = (__bfloat162float(mk[q]) > 0.f) ? x[q] : 0.f;
          if (!live) x[q] = 0.f;
          xb[q] = __float2bfloat16_rn(x[q]);
        }
        if (p.C) {
          float* o = p.C + (size_t)row * p.ldc + col;
          if (vc) {
            reinterpret_cast<float4*>(o)[0] = make_float4(x[0], x[1], x[2], x[3]);
            reinterpret_cast<float4*>(o)[1] = make_float4(x[4], x[5], x[6], x[7]);
          } else {
#pragma unroll
            for (int q = 0; q < 8; ++q) o[q] = x[q];
          }
        }
        if (p.Cb) {
          __nv_bfloat16* o = p.Cb + (size_t)row * p.ldcb + col;
          if (vb) {
            *reinterpret_cast<uint4*>(o) = pack8(xb);
          } else {
#pragma unroll
            for (int q = 0; q < 8; ++q) o[q] = xb[q];
          }
        }
        if (p.Ct)
#pragma unroll
          for (int q = 0; q < 8; ++q) p.Ct[(size_t)(col + q) * p.ldct + row] = xb[q];
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(BN) : "memory");
  if (threadIdx.x == 0 && aborted && p.status) atomicOr(p.status, 2);
}

namespace {

template <int BN>
int gemm_launch_bn(const MlpGemm& g, cudaStream_t st) {
  constexpr size_t smem = (size_t)gemm_stages(BN) * (kStageA + BN * kBK * 2);
  MLCP_CUDA_TRY(cudaFuncSetAttribute(mlp_gemm_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  mlp_gemm_kernel<BN><<<dim3(g.M / kBM, (g.N + BN - 1) / BN), kGemmThreads, smem, st>>>(g);
  MLCP_CUDA_TRY(cudaGetLastError());
  return kOk;
}

}  // namespace

int mlp_gemm_launch(const MlpGemm& g, cudaStream_t st) {
  if (g.M % kBM || g.K % kBK || g.N % 16 || g.N <= 0 || g.K <= 0 || g.lda % 8 || g.ldb % 8) {
    set_error("mlp gemm: unsupported shape M=%d N=%d K=%d (M multiple of 128, N of 16, K of 64)", g.M, g.N, g.K);
    return kBadArgument;
  }
  // the widest tile that still makes a tile for every SM (wider tiles re-read
  // less of A), else the narrowest: one 768 x 256 x 576 GEMM takes 13.9 us
  // with 32-wide tiles (48 CTAs), and took 76.4 with 256-wide ones (6 CTAs,
  // two stages, element-wise stores; launch list, cold)
  int dev = 0, nsm = 0;
  MLCP_CUDA_TRY(cudaGetDevice(&dev));
  MLCP_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  int bn = kMaxBN;
  while (bn > kMinBN && (long long)(g.M / kBM) * ((g.N + bn - 1) / bn) < nsm) bn /= 2;
  switch (bn) {
    case 256: return gemm_launch_bn<256>(g, st);
    case 128: return gemm_launch_bn<128>(g, st);
    case 64: return gemm_launch_bn<64>(g, st);
    default: return gemm_launch_bn<32>(g, st);
  }
}

// ---------------------------------------------------------------------------
// Loss, bias gradients, optimiser
// ---------------------------------------------------------------------------

constexpr int kTileDim = 32;    // tiles of the kernels that also write a transposed copy
constexpr int kTileThreads = 256;

inline unsigned tile_count(int rows, int cols) {
  return (unsigned)((long long)((rows + kTileDim - 1) / kTileDim) * ((cols + kTileDim - 1) / kTileDim));
}

// Sum over the block (warp order; every thread of the block calls it); valid in thread 0.
__device__ float block_sum_f32(float v) {
  __shared__ float red[32];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  float s = 0.f;
  if (threadIdx.x == 0)
    for (int w = 0; w < (int)blockDim.x / 32; ++w) s += red[w];
  return s;
}

// Mean squared error over the valid block (rows < m, cols < n) of Y against
// T (both [rows_p][ld] FP32); dY = 2 (Y - T) / (m n) as BF16 [rows_p][ld] and
// transposed [ld][rows_p]; loss accumulated into *loss, one atomic per CTA.
// One 32 x 32 tile per CTA, transposed through shared memory so that both
// copies are written in rows (13 us -> 5.0 us for 768 x 256: element-wise
// transposed stores touched a sector per two bytes).
__global__ void __launch_bounds__(kTileThreads) mlp_loss_kernel(const float* Y, const float* T, int m, int n, int ld,
                                                                int rows_p, __nv_bfloat16* dY, __nv_bfloat16* dYt,
                                                                float* loss) {
  __shared__ __nv_bfloat16 tile[kTileDim][kTileDim + 2];
  const int tx = threadIdx.x % kTileDim, ty = threadIdx.x / kTileDim;
  const int across = (ld + kTileDim - 1) / kTileDim;
  const int r0 = blockIdx.x / across * kTileDim, c0 = blockIdx.x % across * kTileDim;
  const float scale = 2.f / ((float)m * (float)n);
  float part = 0.f;
#pragma unroll
  for (int u = 0; u < kTileDim; u += kTileThreads / kTileDim) {
    const int r = r0 + ty + u, c = c0 + tx;
    if (r >= rows_p || c >= ld) continue;
    const size_t e = (size_t)r * ld + c;
    float g = 0.f;
    if (r < m && c < n) {
      const float d = Y[e] - T[e];
      part += d * d;
      g = scale * d;
    }
    const __nv_bfloat16 gb = __float2bfloat16_rn(g);
    dY[e] = gb;
    tile[ty + u][tx] = gb;
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < kTileDim; u += kTileThreads / kTileDim) {
    const int c = c0 + ty + u, r = r0 + tx;
    if (r < rows_p && c < ld) dYt[(size_t)c * rows_p + r] = tile[tx][ty + u];
  }
  part = block_sum_f32(part);
  if (threadIdx.x == 0) atomicAdd(loss, part / ((float)m * (float)n));
}

// db[c] = sum over rows of G[r][c] (BF16 [rows][ld]) for up to three matrices
// (blockIdx.y): a CTA per 32 columns, each warp every 32nd row, the warps' sums added
// in order (one thread per column walked its rows alone: 45 us -> 5.1 us for 768 x 256).
__global__ void __launch_bounds__(1024) mlp_colsum_kernel(MlpColsums p) {
  __shared__ float red[32][33];
  const __nv_bfloat16* G = p.G[blockIdx.y];
  const int n = p.n[blockIdx.y], ld = p.ld[blockIdx.y];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = blockIdx.x * 32 + lane;
  float s = 0.f;
  if (c < n)
#pragma unroll 8
    for (int r = warp; r < p.rows; r += 32) s += __bfloat162float(G[(size_t)r * ld + c]);
  red[warp][lane] = s;
  __syncthreads();
  if (warp == 0 && c < n) {
    float t = 0.f;
    for (int w = 0; w < 32; ++w) t += red[w][lane];
    p.db[blockIdx.y][c] = t;
  }
}

// Adam step on FP32 master parameters [rows][cols] of up to six matrices, the tiles of
// one after those of the other; writes the BF16 copy and the transposed BF16 copy
// [cols][rows] where they are given (32 x 32 tiles, as in the loss kernel).
__global__ void __launch_bounds__(kTileThreads) mlp_adam_kernel(MlpAdam p) {
  __shared__ __nv_bfloat16 tile[kTileDim][kTileDim + 2];
  int b = blockIdx.x, k = 0;
  while (k + 1 < p.count && b >= p.tiles[k]) b -= p.tiles[k++];
  const MlpParam& s = p.param[k];
  const int rows = s.rows, cols = s.cols;
  const int tx = threadIdx.x % kTileDim, ty = threadIdx.x / kTileDim;
  const int across = (cols + kTileDim - 1) / kTileDim;
  const int r0 = b / across * kTileDim, x0 = b % across * kTileDim;
#pragma unroll
  for (int u = 0; u < kTileDim; u += kTileThreads / kTileDim) {
    const int r = r0 + ty + u, c = x0 + tx;
    if (r >= rows || c >= cols) continue;
    const size_t e = (size_t)r * cols + c;
    const float gv = s.g[e];
    const float a = p.b1 * s.m1[e] + (1.f - p.b1) * gv;
    const float v = p.b2 * s.m2[e] + (1.f - p.b2) * gv * gv;
    s.m1[e] = a;
    s.m2[e] = v;
    const float x = s.w[e] - p.lr * (a / p.c1) / (sqrtf(v / p.c2) + p.eps);
    s.w[e] = x;
    const __nv_bfloat16 xb = __float2bfloat16_rn(x);
    if (s.wb) s.wb[e] = xb;
    tile[ty + u][tx] = xb;
  }
  if (!s.wt) return;
  __syncthreads();
#pragma unroll
  for (int u = 0; u < kTileDim; u += kTileThreads / kTileDim) {
    const int c = x0 + ty + u, r = r0 + tx;
    if (r < rows && c < cols) s.wt[(size_t)c * rows + r] = tile[tx][ty + u];
  }
}

// out[c][r] = in[r][c], BF16, rows of `in` ld apart (32 x 32 tiles).
__global__ void __launch_bounds__(kTileThreads) mlp_transpose_kernel(const __nv_bfloat16* in, int ld, int rows, int cols,
                                                                     __nv_bfloat16* out) {
  __shared__ __nv_bfloat16 tile[kTileDim][kTileDim + 2];
  const int tx = threadIdx.x % kTileDim, ty = threadIdx.x / kTileDim;
  const int across = (cols + kTileDim - 1) / kTileDim;
  const int r0 = blockIdx.x / across * kTileDim, c0 = blockIdx.x % across * kTileDim;
#pragma unroll
  for (int u = 0; u < kTileDim; u += kTileThreads / kTileDim)
    if (r0 + ty + u < rows && c0 + tx < cols) tile[ty + u][tx] = in[(size_t)(r0 + ty + u) * ld + c0 + tx];
  __syncthreads();
#pragma unroll
  for (int u = 0; u < kTileDim; u += kTileThreads / kTileDim)
    if (c0 + ty + u < cols && r0 + tx < rows) out[(size_t)(c0 + ty + u) * rows + r0 + tx] = tile[tx][ty + u];
}

int mlp_loss_launch(const float* Y, const float* T, int m, int n, int ld, int rows_p, __nv_bfloat16* dY,
                    __nv_bfloat16* dYt, float* loss, cudaStream_t st) {
  mlp_loss_kernel<<<tile_count(rows_p, ld), kTileThreads, 0, st>>>(Y, T, m, n, ld, rows_p, dY, dYt, loss);
  MLCP_CUDA_TRY(cudaGetLastError());
  return kOk;
}

int mlp_colsums_launch(const MlpColsums& p, int count, cudaStream_t st) {
  int n = 0;
  for (int k = 0; k < count; ++k) n = std::max(n, p.n[k]);
  mlp_colsum_kernel<<<dim3((n + 31) / 32, count), 1024, 0, st>>>(p);
  MLCP_CUDA_TRY(cudaGetLastError());
  return kOk;
}

int mlp_colsum_launch(const __nv_bfloat16* G, int rows, int n, int ld, float* db, cudaStream_t st) {
  MlpColsums p{};
  p.rows = rows;
  p.G[0] = G; p.n[0] = n; p.ld[0] = ld; p.db[0] = db;
  return mlp_colsums_launch(p, 1, st);
}

int mlp_adam_launch(MlpAdam p, int step, cudaStream_t st) {
  p.c1 = 1.f - powf(p.b1, (float)step);
  p.c2 = 1.f - powf(p.b2, (float)step);
  int total = 0;
  for (int k = 0; k < p.count; ++k) total += p.tiles[k] = (int)tile_count(p.param[k].rows, p.param[k].cols);
  mlp_adam_kernel<<<total, kTileThreads, 0, st>>>(p);
  MLCP_CUDA_TRY(cudaGetLastError());
  return kOk;
}

namespace {
MlpGemm gemm_of(const __nv_bfloat16* A, int lda, const __nv_bfloat16* B, int ldb, int M, int N, int K, int valid_m,
                int* status) {
  MlpGemm g{};
  g.A = A; g.B = B; g.M = M; g.N = N; g.K = K; g.lda = lda; g.ldb = ldb;
  g.valid_m = valid_m; g.status = status;
  return g;
}
}  // namespace

int mlp_forward(const MlpStep& s, cudaStream_t st) {
  const int M = s.rows_p, h = s.h_p;
  MlpGemm g = gemm_of(s.X, s.ldx, s.w[0], s.in_p, M, h, s.in_p, s.rows, s.status);
  g.bias = s.b[0]; g.act = 1; g.Cb = s.H1; g.ldcb = h; g.Ct = s.H1t; g.ldct = M;
  if (int rc = mlp_gemm_launch(g, st)) return rc;
  g = gemm_of(s.H1, h, s.w[1], h, M, h, h, s.rows, s.status);
  g.bias = s.b[1]; g.act = 1; g.Cb = s.H2; g.ldcb = h; g.Ct = s.H2t; g.ldct = M;
  if (int rc = mlp_gemm_launch(g, st)) return rc;
  g = gemm_of(s.H2, h, s.w[2], h, M, s.out_p, h, s.rows, s.status);
  g.bias = s.b[2]; g.C = s.Y; g.ldc = s.out_p;
  return mlp_gemm_launch(g, st);
}

int mlp_backward(const MlpStep& s, cudaStream_t st) {
  const int M = s.rows_p, h = s.h_p, o = s.out_p;
  MLCP_CUDA_TRY(cudaMemsetAsync(s.loss, 0, sizeof(float), st));
  if (int rc = mlp_loss_launch(s.Y, s.T, s.rows, s.out_dim, o, M, s.dY, s.dYt, s.loss, st)) return rc;
  mlp_transpose_kernel<<<tile_count(M, s.in_p), kTileThreads, 0, st>>>(s.X, s.ldx, M, s.in_p, s.Xt);
  MLCP_CUDA_TRY(cudaGetLastError());
  // layer 3: dW3 = dY^T H2, dZ2 = (dY W3) * (H2 > 0)
  MlpGemm g = gemm_of(s.dYt, M, s.H2t, M, o, h, M, o, s.status);
  g.C = s.gw[2]; g.ldc = h;
  if (int rc = mlp_gemm_launch(g, st)) return rc;
  g = gemm_of(s.dY, o, s.wt[2], o, M, h, o, s.rows, s.status);
  g.act = 2; g.mask = s.H2; g.ldm = h; g.Cb = s.dZ2; g.ldcb = h; g.Ct = s.dZ2t; g.ldct = M;
  if (int rc = mlp_gemm_launch(g, st)) return rc;
  // layer 2
  g = gemm_of(s.dZ2t, M, s.H1t, M, h, h, M, h, s.status);
  g.C = s.gw[1]; g.ldc = h;
  if (int rc = mlp_gemm_launch(g, st)) return rc;
  g = gemm_of(s.dZ2, h, s.wt[1], h, M, h, h, s.rows, s.status);
  g.act = 2; g.mask = s.H1; g.ldm = h; g.Cb = s.dZ1; g.ldcb = h; g.Ct = s.dZ1t; g.ldct = M;
  if (int rc = mlp_gemm_launch(g, st)) return rc;
  // layer 1
  g = gemm_of(s.dZ1t, M, s.Xt, M, h, s.in_p, M, h, s.status);
  g.C = s.gw[0]; g.ldc = s.in_p;
  if (int rc = mlp_gemm_launch(g, st)) return rc;
  // the bias gradients: column sums of dY, dZ2, dZ1
  MlpColsums c{};
  c.rows = M;
  c.G[0] = s.dY; c.n[0] = c.ld[0] = o; c.db[0] = s.gb[2];
  c.G[1] = s.dZ2; c.n[1] = c.ld[1] = h; c.db[1] = s.gb[1];
  c.G[2] = s.dZ1; c.n[2] = c.ld[2] = h; c.db[2] = s.gb[0];
  return mlp_colsums_launch(c, 3, st);
}

}  // namespace mlcp
