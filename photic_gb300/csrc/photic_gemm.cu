// photic_gemm.cu -- BF16 "TN" GEMM on the tcgen05 tensor cores:
//   C[M x N] = A[M x K] * B[N x K]^T  (A, B row-major BF16, K contiguous)
// with the FP32 accumulator in tensor memory and a fused epilogue.  It is
// the building block of the surrogate MLP (photic_mlp.cu): forward layers
// (bias + SiLU), input gradients (times SiLU') and weight gradients.
//
// One CTA (8 warps) owns a 128 x BN output tile (or, split-K, one slice of
// K of it: the weight-gradient products have 128 x 128 outputs and K = the
// batch, so their K is spread over CTAs and photic_mlp.cu adds the partial
// sums in a fixed order).  K is consumed in chunks of 64 through two
// buffers: all threads stage the A and B chunks into shared memory in the
// canonical no-swizzle core-matrix layout (16-byte vector loads; an operand
// stored with K as its rows is transposed 8 x 8 in registers on the way), one
// thread issues four K=16 MMAs and commits them to the buffer's mbarrier while
// the others stage the next chunk, every wait is bounded, and the epilogue
// reads the accumulator back with tcgen05.ld, one TMEM lane (= output row) per
// thread, sixteen columns at a time in 16-byte accesses.
//
// At the MLP's sizes (8 192 x 128 x 128) the products are bound by the
// epilogue's and the staging's memory instructions, not by the tensor cores:
// with four warps and an element per access a forward layer took 49 us, now 15
// (from cold caches; half-width tiles on twice the SMs took as long).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "photic_kernels.h"
#include "photic_tc.cuh"

namespace photic {

namespace {

constexpr int kBM = 128, kBN = 128, kBK = 64;
constexpr int kThreads = 256;
constexpr uint32_t kTmemCols = 256;        // >= any N the descriptor can name here
constexpr uint32_t kWaitLimit = 1u << 26;  // bounded mbarrier spin

__device__ __forceinline__ float silu(float z) { return z / (1.0f + __expf(-z)); }
__device__ __forceinline__ float dsilu(float z) {
  const float s = 1.0f / (1.0f + __expf(-z));
  return s * (1.0f + z * (1.0f - s));
}

// Stage rows [r0, r0+rows) x cols [k0, k0+64) of a row-major BF16 matrix
// into the core-matrix layout: element (r, k) at byte
// ((r/8)*8 + k/8)*128 + (r%8)*16 + (k%8)*2.  Out-of-range parts are zero.
__device__ __forceinline__ void stage(const __nv_bfloat16 *src, int ld, int nrows_total,
                                      int r0, int rows, int k0, int K, unsigned char *dst) {
  const int vecs = rows * (kBK / 8);
  for (int v = threadIdx.x; v < vecs; v += blockDim.x) {
    const int r = v >> 3, c = v & 7;
    const int gr = r0 + r, gk = k0 + c * 8;
    uint4 val = make_uint4(0u, 0u, 0u, 0u);
    if (gr < nrows_total && gk < K)
      val = *reinterpret_cast<const uint4 *>(src + (size_t)gr * ld + gk);
    *reinterpret_cast<uint4 *>(dst + (((r >> 3) * 8 + c) * 128 + (r & 7) * 16)) = val;
  }
}

// The same from a matrix stored with K as its rows (element (r, k) at
// src[k * ld + r]): eight rows of eight values a thread, transposed in
// registers.  ld and r0 are multiples of 8 and the rows 16-byte aligned.
__device__ __forceinline__ void stage_k_rows(const __nv_bfloat16 *src, int ld, int nrows_total,
                                             int r0, int rows, int k0, int K, unsigned char *dst,
                                             int thread, int threads) {
  const int blocks = rows >> 3;
  for (int v = thread; v < blocks * (kBK / 8); v += threads) {
    const int rb = v % blocks, c = v / blocks;
    uint4 a[8];
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const int gk = k0 + c * 8 + k;
      a[k] = make_uint4(0u, 0u, 0u, 0u);
      if (gk < K && r0 + rb * 8 < nrows_total)
        a[k] = *reinterpret_cast<const uint4 *>(src + (size_t)gk * ld + r0 + rb * 8);
    }
#pragma unroll
    for (int m = 0; m < 8; m++) {
      uint32_t w[4];
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const uint4 &lo = a[2 * i], &hi = a[2 * i + 1];
        const uint32_t x = m < 2 ? lo.x : m < 4 ? lo.y : m < 6 ? lo.z : lo.w;
        const uint32_t y = m < 2 ? hi.x : m < 4 ? hi.y : m < 6 ? hi.z : hi.w;
        w[i] = __byte_perm(x, y, (m & 1) ? 0x7632 : 0x5410);
      }
      *reinterpret_cast<uint4 *>(dst + (rb * 8 + c) * 128 + m * 16) =
          make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
}

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  const __nv_bfloat162 h = __halves2bfloat162(__float2bfloat16(a), __float2bfloat16(b));
  return *reinterpret_cast<const uint32_t *>(&h);
}

// Columns [col, col + 16) of a row, 16-byte accesses.
__device__ __forceinline__ void store16(float *dst, const float (&v)[16]) {
#pragma unroll
  for (int j = 0; j < 4; j++)
    reinterpret_cast<float4 *>(dst)[j] =
        make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
}
__device__ __forceinline__ void store16(__nv_bfloat16 *dst, const float (&v)[16]) {
#pragma unroll
  for (int j = 0; j < 2; j++)
    reinterpret_cast<uint4 *>(dst)[j] =
        make_uint4(pack_bf16(v[8 * j], v[8 * j + 1]), pack_bf16(v[8 * j + 2], v[8 * j + 3]),
                   pack_bf16(v[8 * j + 4], v[8 * j + 5]), pack_bf16(v[8 * j + 6], v[8 * j + 7]));
}
__device__ __forceinline__ void epilogue16(const GemmArgs &g, __nv_bfloat16 *gO, int64_t row,
                                           int col, float (&v)[16]) {
  switch (g.epi) {
    case EPI_F32:
      store16(g.C + row * g.ldc + col, v);
      break;
    case EPI_BIAS_F32:
#pragma unroll
      for (int j = 0; j < 16; j++) v[j] = v[j] + g.bias[col + j];
      store16(g.C + row * g.ldc + col, v);
      break;
    case EPI_BIAS_SILU:
#pragma unroll
      for (int j = 0; j < 16; j++) v[j] = v[j] + g.bias[col + j];
      if (g.Z) store16(g.Z + row * g.ldz + col, v);
#pragma unroll
      for (int j = 0; j < 16; j++) v[j] = silu(v[j]);
      store16(gO + row * g.ldo + col, v);
      break;
    case EPI_DSILU: {
      float z[16];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const float4 t = reinterpret_cast<const float4 *>(g.Z + row * g.ldz + col)[j];
        z[4 * j] = t.x;
        z[4 * j + 1] = t.y;
        z[4 * j + 2] = t.z;
        z[4 * j + 3] = t.w;
      }
#pragma unroll
      for (int j = 0; j < 16; j++) v[j] = v[j] * dsilu(z[j]);
      store16(gO + row * g.ldo + col, v);
      break;
    }
    default:
      break;
  }
}
__device__ __forceinline__ void epilogue1(const GemmArgs &g, __nv_bfloat16 *gO, int64_t row,
                                          int col, float acc) {
  switch (g.epi) {
    case EPI_F32:
      g.C[row * g.ldc + col] = acc;
      break;
    case EPI_BIAS_F32:
      g.C[row * g.ldc + col] = acc + g.bias[col];
      break;
    case EPI_BIAS_SILU: {
      const float z = acc + g.bias[col];
      if (g.Z) g.Z[row * g.ldz + col] = z;
      gO[row * g.ldo + col] = __float2bfloat16(silu(z));
      break;
    }
    case EPI_DSILU:
      gO[row * g.ldo + col] = __float2bfloat16(acc * dsilu(g.Z[row * g.ldz + col]));
      break;
    default:
      break;
  }
}

// blockIdx.z: the product of the batch, and its slice of K.
__global__ void __launch_bounds__(kThreads) tn_gemm_kernel(const __grid_constant__ GemmBatch b) {
  const GemmArgs &g = b.g[blockIdx.z / b.slices];
  const int slice = blockIdx.z % b.slices;
  const __nv_bfloat16 *gA = reinterpret_cast<const __nv_bfloat16 *>(g.A);
  const __nv_bfloat16 *gB = reinterpret_cast<const __nv_bfloat16 *>(g.B);
  __nv_bfloat16 *gO = reinterpret_cast<__nv_bfloat16 *>(g.O);
  extern __shared__ __align__(1024) unsigned char smem[];
  constexpr int kBufBytes = (kBM + kBN) * kBK * 2;  // a chunk of A, then of B
  __shared__ __align__(8) uint64_t mbar[2];
  __shared__ uint32_t tmem_slot;

  const int m0 = blockIdx.x * kBM, n0 = blockIdx.y * kBN;
  const int ncols = min(kBN, g.N - n0);          // valid output columns of this tile
  const int mma_n = (ncols + 15) / 16 * 16;      // MMA N: multiple of 16, <= 128
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (warp == 0) tc::tmem_alloc(&tmem_slot, kTmemCols);
  if (tid == 0) {
    tc::mbar_init(&mbar[0], 1);
    tc::mbar_init(&mbar[1], 1);
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tmem_slot;
  const uint32_t idesc = tc::make_idesc_bf16(kBM, mma_n);

  bool ok = true;
  // split-K: CTA z takes chunks [c0, c1) of K and writes a partial sum
  const int nchunks = (g.K + kBK - 1) / kBK;
  const int per = (nchunks + b.slices - 1) / b.slices;  // (no slice is empty)
  const int c0 = slice * per;
  const int c1 = min(nchunks, c0 + per);
  // Wait for the MMAs of chunk kc (the n-th use of its buffer).  A wait that
  // runs out records the error and gives the tensor core a second bounded
  // chance to finish before the shared memory and TMEM go away.
  auto finished = [&](int kc) {
    const int u = kc - c0;
    const uint32_t parity = (uint32_t)(u >> 1) & 1u;
    if (tc::mbar_wait(&mbar[u & 1], parity, kWaitLimit)) return true;
    if (tid == 0) atomicOr(g.error, PHOTIC_DEVERR_MMA_TIMEOUT);
    tc::mbar_wait(&mbar[u & 1], parity, kWaitLimit);
    return false;
  };
  int issued = 0;  // chunks whose MMAs are committed
  for (int kc = c0; kc < c1; kc++) {
    const int k0 = kc * kBK;
    unsigned char *sA = smem + ((kc - c0) & 1) * kBufBytes, *sB = sA + kBM * kBK * 2;
    if (kc - c0 >= 2 && ok) ok = finished(kc - 2);
    if (!__syncthreads_and(ok)) {
      ok = false;
      break;
    }
    if (g.k_rows) {
      stage_k_rows(gA, g.lda, g.M, m0, kBM, k0, g.K, sA, tid, kThreads / 2);
      if (tid >= kThreads / 2)
        stage_k_rows(gB, g.ldb, g.N, n0, mma_n, k0, g.K, sB, tid - kThreads / 2, kThreads / 2);
    } else {
      stage(gA, g.lda, g.M, m0, kBM, k0, g.K, sA);
      stage(gB, g.ldb, g.N, n0, mma_n, k0, g.K, sB);
    }
    tc::fence_smem_async();
    __syncthreads();
    if (tid == 0) {
      tc::fence_after_sync();
      const uint32_t a0 = tc::smem_u32(sA), b0 = tc::smem_u32(sB);
#pragma unroll
      for (int kk = 0; kk < kBK / 16; kk++) {
        if (k0 + kk * 16 < g.K) {
          const uint64_t ad = tc::make_desc(a0 + kk * 256, g.lbo, g.sbo);
          const uint64_t bd = tc::make_desc(b0 + kk * 256, g.lbo, g.sbo);
          tc::mma_bf16(tmem, ad, bd, idesc, (kc > c0 || kk > 0) ? 1u : 0u);
        }
      }
      tc::mma_commit(&mbar[(kc - c0) & 1]);
    }
    issued++;
  }
  // no MMA stays in flight on any exit
  for (int u = issued > 2 ? issued - 2 : 0; u < issued; u++)
    if (!finished(c0 + u)) ok = false;
  ok = __syncthreads_and(ok) != 0;
  tc::fence_after_sync();

  const int64_t row = m0 + (warp & 3) * 32 + lane;
  if (ok) {
    // warps 0-3 and 4-7 share the TMEM lanes and take every other 16 columns
    for (int cc = (warp >> 2) * 16; cc < mma_n; cc += 32) {
      float v[16];
      tc::tmem_ld16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)cc, v);
      const int col = n0 + cc;
      if (row < g.M) {
        if (g.vec && cc + 16 <= ncols) {
          if (g.partial) store16(g.partial + ((size_t)slice * g.M + row) * g.N + col, v);
          else epilogue16(g, gO, row, col, v);
        } else {
#pragma unroll
          for (int j = 0; j < 16; j++) {
            if (cc + j >= ncols) break;
            if (g.partial) g.partial[((size_t)slice * g.M + row) * g.N + col + j] = v[j];
            else epilogue1(g, gO, row, col + j, v[j]);
          }
        }
      }
      __syncwarp();
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_free(tmem, kTmemCols);
}

}  // namespace

// Dynamic shared memory is sized to keep at most two CTAs per SM, so the
// TMEM of resident CTAs (2 x 256 of 512 columns) never over-subscribes.
size_t gemm_smem_bytes() { return 96 * 1024; }

namespace {

// 16-byte accesses of the epilogue: every row of every array that it touches
// on a 16-byte boundary.
int epilogue_vec(const GemmArgs &a) {
  auto rows16 = [](const void *p, int64_t row_bytes) {
    return p == nullptr || (((uintptr_t)p | (uintptr_t)row_bytes) & 15u) == 0;
  };
  return a.partial ? rows16(a.partial, (int64_t)a.N * 4)
                   : rows16(a.C, (int64_t)a.ldc * 4) && rows16(a.Z, (int64_t)a.ldz * 4) &&
                         rows16(a.O, (int64_t)a.ldo * 2);
}

cudaError_t launch_batch(const GemmBatch &b, int n, int M, int N, cudaStream_t s) {
  const size_t smem = gemm_smem_bytes();
  cudaError_t e = cudaFuncSetAttribute(tn_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem);
  if (e != cudaSuccess) return e;
  dim3 grid((unsigned)((M + kBM - 1) / kBM), (unsigned)((N + kBN - 1) / kBN),
            (unsigned)(b.slices * n));
  tn_gemm_kernel<<<grid, kThreads, smem, s>>>(b);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_gemm(const GemmArgs &g, cudaStream_t s) {
  if (g.M <= 0 || g.N <= 0) return cudaSuccess;
  GemmBatch b{};
  b.g[0] = g;
  b.g[0].partial = nullptr;
  b.g[0].vec = epilogue_vec(b.g[0]);
  b.slices = 1;
  return launch_batch(b, 1, g.M, g.N, s);
}

// Products of one M and K in one launch, each cut into up to `ksplit` slices
// of K and the partial sums left in their scratch: [slices][M][N] each.
// Returns the slices.
cudaError_t launch_gemm_partials(const GemmArgs *g, int n, int ksplit, int *slices,
                                 cudaStream_t s) {
  GemmBatch b{};
  const int nchunks = (g[0].K + kBK - 1) / kBK;
  const int per = (nchunks + ksplit - 1) / ksplit;
  b.slices = (nchunks + per - 1) / per;
  int N = 0;
  for (int i = 0; i < n; i++) {
    b.g[i] = g[i];
    b.g[i].vec = epilogue_vec(b.g[i]);
    N = g[i].N > N ? g[i].N : N;
  }
  *slices = b.slices;
  return launch_batch(b, n, g[0].M, N, s);
}

}  // namespace photic
