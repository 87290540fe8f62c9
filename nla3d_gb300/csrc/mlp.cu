// Kernels of the learned Newton start: a small multilayer perceptron whose
// weights are stored in BF16 and whose products accumulate in FP32.  No
// counterpart in the reference (which always starts Newton from the previous
// converged state).
//
//   gemm:        C[m,n] = act( sum_k A[m,k] B[k,n] + bias[n] )  (A, B FP32 or BF16,
//                arbitrary strides so that X W^T, dZ^T X and dZ W use one kernel),
//                on the tensor cores (tcgen05, BF16 operands, FP32 accumulation)
//   tanh_bwd:    dZ = dY * (1 - Y^2)
//   column_sum:  s[n] = sum_m X[m,n]            (bias gradient)
//   mse_grad:    dY = scale * (Y - T)
//   adam:        FP32 master weights, moments, BF16 copy refreshed in place
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/nla3d_gpu.h"

namespace {

// ---- C = act(A B + bias) on the tensor cores (tcgen05.mma kind::f16, BF16) ----
//
// One CTA (512 threads) per 128 x 32 tile of C, K in chunks of 128, two
// shared-memory stages.  Both operands are staged as BF16 in the canonical
// K-major layout without swizzle (8-row x 16-byte core matrices; K-adjacent
// cores 128 B apart, 8-row groups 2 KB apart): A as its 128 rows m, B as its
// 32 columns n (the MMA computes D[m][n] = sum_k A[m][k] B'[n][k]).  An FP32
// operand (activations, gradients) is split into a BF16 high part and the
// BF16 rounding of the remainder, x = hi + lo + O(2^-16 |x|); a BF16 operand
// (the weights) is exact as it is.  One thread issues, per 16-wide K step,
// hi.hi, then hi.lo and lo.hi where an operand has a low part (BF16 x BF16
// products are exact in FP32), accumulating in FP32 in 32 TMEM columns, and
// commits them to the stage's mbarrier; a stage is refilled once its MMAs
// have released it, and a chunk's loads are issued before that wait.  The
// epilogue reads TMEM (warp w: lanes 32 (w % 4) .. +31 = rows, columns
// 8 (w / 4) .. +7), adds the bias, applies the activation and stores FP32.
// Every wait is bounded: on a timeout the tile's outputs, its row sums among
// them, are set to NaN and g_mlp_timeouts is incremented.
//
// The network's products (batch x 256 x 256) are far below the chip: what
// bounds one is the latency of its serial chunks.  128 x 128 tiles with
// 32-wide chunks ran 4 CTAs x 8 serial load-convert-multiply rounds, 51 us a
// product at batch 256 (ncu, cold); 128 x 32 tiles with 128-wide chunks run
// 16 CTAs x 2 rounds, each with all of a chunk's loads in flight, 14 us.
constexpr int kTcM = 128, kTcN = 32, kTcK = 128;
constexpr int kThreads = 512;
constexpr uint32_t kATile = kTcM * kTcK, kBTile = kTcN * kTcK;      // elements per operand part
constexpr uint32_t kStageElems = 2 * (kATile + kBTile);             // A hi, A lo, B hi, B lo
constexpr size_t kTcSmem = 2 * kStageElems * sizeof(__nv_bfloat16) + 64;
// instruction descriptor: D F32 (bit 4), A and B BF16 (bits 7, 10), both
// K-major, N / 8 at bit 17, M / 16 at bit 24
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) |
                            ((uint32_t)(kTcN >> 3) << 17) | ((uint32_t)(kTcM >> 4) << 24);
constexpr long long kSpinLimit = 1ll << 26;

__device__ unsigned int g_mlp_timeouts;

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// shared-memory matrix descriptor: start, leading (K) and stride (8-row) byte
// offsets, descriptor version 1, no swizzle
__device__ __forceinline__ uint64_t mat_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t phase) {
  for (long long it = 0; it < kSpinLimit; it++) {
    uint32_t done;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(mbar), "r"(phase)
        : "memory");
    if (done) return true;
  }
  return false;
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem, uint64_t a, uint64_t b, uint32_t acc) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.u32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
      "l"(a), "l"(b), "r"(kIdesc), "r"(acc));
}

__device__ __forceinline__ float load_elem(const void* p, int bf16, long i) {
  if (bf16) return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p)[i]);
  return reinterpret_cast<const float*>(p)[i];
}

// An operand chunk of R rows x kTcK is R kTcK / 8 units of (one row, 8
// consecutive k), one 16-byte core-matrix row each.  Eight consecutive
// threads take the eight rows of a core matrix (conflict-free 16-byte
// stores); where k runs contiguously in memory the next 24 threads take the
// next three core matrices along k (128 contiguous bytes per row), where
// rows do, along the rows.
template <int R>
__device__ __forceinline__ void unit_of(int u, bool k_fast, int& row, int& k) {
  const int g = u >> 3;
  if (k_fast) {
    row = (g / (kTcK / 8)) * 8 + (u & 7);
    k = (g % (kTcK / 8)) * 8;
  } else {
    row = (g % (R / 8)) * 8 + (u & 7);
    k = (g / (R / 8)) * 8;
  }
}

// `vec`: k runs contiguously and every unit starts on a 16-byte boundary, so
// a whole unit is two (FP32) or one (BF16) 16-byte loads
__device__ __forceinline__ bool vector_units(const void* p, int bf16, long ld_r, long ld_k) {
  return ld_k == 1 && (reinterpret_cast<uintptr_t>(p) & 15u) == 0 && ld_r % (bf16 ? 8 : 4) == 0;
}

template <int R>
__device__ __forceinline__ void load_units(float v[][8], const void* p, int bf16, bool vec,
                                           long ld_r, long ld_k, int r0, int rows, int k0, int K) {
#pragma unroll
  for (int q = 0; q < R * kTcK / 8 / kThreads; q++) {
    int row, k;
    unit_of<R>(threadIdx.x + q * kThreads, ld_k == 1, row, k);
    const long base = (long)(r0 + row) * ld_r + (long)(k0 + k) * ld_k;
    if (vec && r0 + row < rows && k0 + k + 8 <= K) {
      if (bf16) {
        const uint4 w = *reinterpret_cast<const uint4*>(
            reinterpret_cast<const __nv_bfloat16*>(p) + base);
        const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int e = 0; e < 4; e++) {
          v[q][2 * e] = __uint_as_float(u[e] << 16);
          v[q][2 * e + 1] = __uint_as_float(u[e] & 0xFFFF0000u);
        }
      } else {
        const float4 x = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(p) + base);
        const float4 y =
            *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(p) + base + 4);
        v[q][0] = x.x, v[q][1] = x.y, v[q][2] = x.z, v[q][3] = x.w;
        v[q][4] = y.x, v[q][5] = y.y, v[q][6] = y.z, v[q][7] = y.w;
      }
    } else {
#pragma unroll
      for (int e = 0; e < 8; e++)
        v[q][e] = (r0 + row < rows && k0 + k + e < K) ? load_elem(p, bf16, base + e * ld_k) : 0.f;
    }
  }
}

template <int R>
__device__ __forceinline__ void stage_units(__nv_bfloat16* hi, __nv_bfloat16* lo, bool split,
                                            bool k_fast, const float v[][8]) {
#pragma unroll
  for (int q = 0; q < R * kTcK / 8 / kThreads; q++) {
    int row, k;
    unit_of<R>(threadIdx.x + q * kThreads, k_fast, row, k);
    const uint32_t off = (uint32_t)(((row >> 3) * (kTcK / 8) + (k >> 3)) * 64 + (row & 7) * 8);
    __align__(16) __nv_bfloat16 h[8], l[8];
#pragma unroll
    for (int e = 0; e < 8; e++) {
      h[e] = __float2bfloat16_rn(v[q][e]);
      l[e] = __float2bfloat16_rn(v[q][e] - __bfloat162float(h[e]));
    }
    *reinterpret_cast<uint4*>(hi + off) = *reinterpret_cast<const uint4*>(h);
    if (split) *reinterpret_cast<uint4*>(lo + off) = *reinterpret_cast<const uint4*>(l);
  }
}

__global__ void __launch_bounds__(kThreads)
    tc_gemm_kernel(int M, int N, int K, const void* __restrict__ A, int a_bf16, long lda_m,
                   long lda_k, const void* __restrict__ B, int b_bf16, long ldb_k, long ldb_n,
                   float* __restrict__ C, long ldc, const float* __restrict__ bias, int act,
                   const float* __restrict__ Y, float* __restrict__ a_sum) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __nv_bfloat16* stage = reinterpret_cast<__nv_bfloat16*>(smem);
  uint64_t* mbar = reinterpret_cast<uint64_t*>(stage + 2 * kStageElems);   // one per stage
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(mbar + 2);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = blockIdx.y * kTcM, n0 = blockIdx.x * kTcN;
  const bool a_split = !a_bf16, b_split = !b_bf16;
  const bool a_vec = vector_units(A, a_bf16, lda_m, lda_k);
  const bool b_vec = vector_units(B, b_bf16, ldb_n, ldb_k);
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_addr(tmem_slot)),
                 "r"(kTcN));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(mbar)), "r"(1));
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(mbar + 1)), "r"(1));
    asm volatile("fence.mbarrier_init.release.cluster;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  const uint32_t lbo = 128, sbo = (kTcK / 8) * 128;
  const int n_chunks = (K + kTcK - 1) / kTcK;
  bool ok = true;
  float row_sum = 0.f;
  for (int c = 0; c < n_chunks && ok; c++) {
    float av[kATile / 8 / kThreads][8], bv[kBTile / 8 / kThreads][8];
    load_units<kTcM>(av, A, a_bf16, a_vec, lda_m, lda_k, m0, M, c * kTcK, K);
    load_units<kTcN>(bv, B, b_bf16, b_vec, ldb_n, ldb_k, n0, N, c * kTcK, K);
    if (a_sum) {
      // lda_k != 1: every unit of a thread has the same row (threads t + 128 j
      // share one), so its values add up here
#pragma unroll
      for (int u = 0; u < kATile / 8 / kThreads; u++)
        row_sum += ((av[u][0] + av[u][1]) + (av[u][2] + av[u][3])) +
                   ((av[u][4] + av[u][5]) + (av[u][6] + av[u][7]));
    }
    const int q = c & 1;
    if (c > 1) ok = mbar_wait(smem_addr(mbar + q), (uint32_t)(c / 2 - 1) & 1u);   // stage released
    __nv_bfloat16* Ahi = stage + q * kStageElems;
    __nv_bfloat16* Alo = Ahi + kATile;
    __nv_bfloat16* Bhi = Alo + kATile;
    __nv_bfloat16* Blo = Bhi + kBTile;
    if (ok) {
      stage_units<kTcM>(Ahi, Alo, a_split, lda_k == 1, av);
      stage_units<kTcN>(Bhi, Blo, b_split, ldb_k == 1, bv);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    ok = __syncthreads_and(ok ? 1 : 0) != 0;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (ok && threadIdx.x == 0) {
      const uint32_t ahi = smem_addr(Ahi), alo = smem_addr(Alo);
      const uint32_t bhi = smem_addr(Bhi), blo = smem_addr(Blo);
      const int steps = (min(K - c * kTcK, kTcK) + 15) / 16;   // the rest of a chunk is zeros
      for (int st = 0; st < steps; st++) {
        const uint32_t koff = st * 256;   // 16 K values = two core matrices
        const uint64_t dah = mat_desc(ahi + koff, lbo, sbo), dbh = mat_desc(bhi + koff, lbo, sbo);
        mma_bf16(tmem, dah, dbh, (c > 0 || st > 0) ? 1u : 0u);
        if (b_split) mma_bf16(tmem, dah, mat_desc(blo + koff, lbo, sbo), 1u);
        if (a_split) mma_bf16(tmem, mat_desc(alo + koff, lbo, sbo), dbh, 1u);
      }
      asm volatile(
          "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
              smem_addr(mbar + q))
          : "memory");
    }
  }
  // the last chunk's commit covers every MMA issued (they complete in order)
  if (ok && n_chunks > 0)
    ok = mbar_wait(smem_addr(mbar + ((n_chunks - 1) & 1)), (uint32_t)((n_chunks - 1) / 2) & 1u);
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  ok = __syncthreads_and(ok ? 1 : 0) != 0;
  if (a_sum && blockIdx.x == 0) {
    // (the stages are free: every MMA has completed)
    float* part = reinterpret_cast<float*>(smem);
    int r, k;
    unit_of<kTcM>(threadIdx.x, false, r, k);
    part[(threadIdx.x / kTcM) * kTcM + r] = ok ? row_sum : __uint_as_float(0x7FC00000u);
    __syncthreads();
    if (threadIdx.x < kTcM && m0 + threadIdx.x < M)
      a_sum[m0 + threadIdx.x] = (part[threadIdx.x] + part[kTcM + threadIdx.x]) +
                                (part[2 * kTcM + threadIdx.x] + part[3 * kTcM + threadIdx.x]);
  }
  const int row = (warp & 3) * 32 + lane;
  const int m = m0 + row;
  const int c0 = (warp >> 2) * 8;
  uint32_t v[8];
  if (ok && n_chunks > 0) {
    const uint32_t taddr = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c0;
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
          "=r"(v[7])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
  } else {
#pragma unroll
    for (int q = 0; q < 8; q++) v[q] = ok ? 0u : 0x7FC00000u;   // K = 0: zero; timeout: NaN
  }
  if (m < M)
#pragma unroll
    for (int q = 0; q < 8; q++) {
      const int n = n0 + c0 + q;
      if (n < N) {
        float y = __uint_as_float(v[q]) + (bias ? bias[n] : 0.f);
        if (act == 1) y = tanhf(y);
        if (Y) {
          const float t = Y[(long)m * ldc + n];
          y *= 1.0f - t * t;
        }
        C[(long)m * ldc + n] = y;
      }
    }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    if (!ok) {
      // after a timeout the MMAs may still run: one more bounded wait on each
      // stage and phase
      if (lane == 0) atomicAdd(&g_mlp_timeouts, 1u);
      for (int q = 0; q < 2; q++) {
        mbar_wait(smem_addr(mbar + q), 0);
        mbar_wait(smem_addr(mbar + q), 1);
      }
    }
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTcN));
  }
}

__global__ void tanh_bwd_kernel(const float* Y, float* dY, long n) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dY[i] *= 1.0f - Y[i] * Y[i];
}

// one block per 32 columns; threads stride over the rows, fixed order
__global__ void column_sum_kernel(const float* X, long rows, long cols, float* out) {
  __shared__ float part[8][33];
  const int c = blockIdx.x * 32 + (threadIdx.x % 32);
  const int r0 = threadIdx.x / 32;  // 0..7
  float s = 0.f;
  if (c < cols)
    for (long r = r0; r < rows; r += 8) s += X[r * cols + c];
  part[r0][threadIdx.x % 32] = s;
  __syncthreads();
  if (r0 == 0 && c < cols) {
    float t = 0.f;
    for (int k = 0; k < 8; k++) t += part[k][threadIdx.x % 32];
    out[c] = t;
  }
}

// every tensor of the network in one launch: one launch of 4.3 us where ten of
// 3.3 us each were almost all launch latency
constexpr int kAdamTensors = 16;
struct AdamTensors {
  int count;
  unsigned first[kAdamTensors + 1];   // first block of each tensor
  long n[kAdamTensors];
  float* w[kAdamTensors];
  const float* g[kAdamTensors];
  float* m[kAdamTensors];
  float* v[kAdamTensors];
  __nv_bfloat16* wb[kAdamTensors];
};

__device__ __forceinline__ void adam_update(float* w, const float* g, float* m, float* v, long i,
                                            float lr, float b1, float b2, float eps, float c1,
                                            float c2, __nv_bfloat16* w_bf16) {
  const float gi = g[i];
  const float mi = b1 * m[i] + (1.f - b1) * gi;
  const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  const float wi = w[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  w[i] = wi;
  if (w_bf16) w_bf16[i] = __float2bfloat16_rn(wi);
}

__global__ void adam_multi_kernel(const __grid_constant__ AdamTensors a, float lr, float b1,
                                  float b2, float eps, float c1, float c2) {
  int t = 0;
  while (t + 1 < a.count && blockIdx.x >= a.first[t + 1]) t++;
  const long i = (long)(blockIdx.x - a.first[t]) * blockDim.x + threadIdx.x;
  if (i < a.n[t])
    adam_update(a.w[t], a.g[t], a.m[t], a.v[t], i, lr, b1, b2, eps, c1, c2, a.wb[t]);
}

__global__ void adam_kernel(float* w, const float* g, float* m, float* v, long n, float lr,
                            float b1, float b2, float eps, float c1, float c2,
                            __nv_bfloat16* w_bf16) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) adam_update(w, g, m, v, i, lr, b1, b2, eps, c1, c2, w_bf16);
}

__global__ void mse_grad_kernel(const float* Y, const float* T, float* dY, long n, float scale) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dY[i] = scale * (Y[i] - T[i]);
}

__global__ void to_bf16_kernel(const float* x, __nv_bfloat16* y, long n) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = __float2bfloat16_rn(x[i]);
}

int status(cudaError_t e) { return e == cudaSuccess ? NLA3D_OK : NLA3D_ERR_CUDA; }

int launch_gemm(int M, int N, int K, const void* A, int a_bf16, int64_t lda_m, int64_t lda_k,
                const void* B, int b_bf16, int64_t ldb_k, int64_t ldb_n, float* C, int64_t ldc,
                const float* bias, int act, const float* Y, float* a_sum, cudaStream_t stream) {
  if (M == 0 || N == 0) return NLA3D_OK;
  // 160 KB of shared memory: above the default limit (an attribute of the
  // function on the current device, not of a stream)
  const cudaError_t e = cudaFuncSetAttribute(
      tc_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTcSmem);
  if (e != cudaSuccess) return status(e);
  const dim3 grid((N + kTcN - 1) / kTcN, (M + kTcM - 1) / kTcM);
  tc_gemm_kernel<<<grid, kThreads, kTcSmem, stream>>>(M, N, K, A, a_bf16, lda_m, lda_k, B, b_bf16,
                                                      ldb_k, ldb_n, C, ldc, bias, act, Y, a_sum);
  return status(cudaGetLastError());
}

}  // namespace

extern "C" {

int nla3d_mlp_gemm(int M, int N, int K, const void* A, int a_bf16, int64_t lda_m, int64_t lda_k,
                   const void* B, int b_bf16, int64_t ldb_k, int64_t ldb_n, float* C, int64_t ldc,
                   const float* bias, int act, void* stream) {
  if (M < 0 || N < 0 || K < 0 || (K > 0 && (!A || !B)) || !C || (act != 0 && act != 1))
    return NLA3D_ERR_ARG;
  return launch_gemm(M, N, K, A, a_bf16, lda_m, lda_k, B, b_bf16, ldb_k, ldb_n, C, ldc, bias, act,
                     nullptr, nullptr, (cudaStream_t)stream);
}

int nla3d_mlp_layer_grads(int batch, int n_out, int n_in, const float* dY, const float* X,
                          float* dW, float* db, void* stream) {
  if (batch < 0 || n_out < 0 || n_in < 0 || !dW || !db || (batch > 0 && (!dY || !X)))
    return NLA3D_ERR_ARG;
  // dW[o,i] = sum_b dY[b,o] X[b,i], db[o] = sum_b dY[b,o]: A = dY^T (rows
  // contiguous), whose row sums the first column of tiles forms on the way.  One
  // output: dY^T runs contiguously along the batch too and its units are dealt
  // out that way, a thread's in different rows, so its sum takes a launch of its
  // own (dealing them out along the rows by a flag made the input gradients'
  // launches slower, 14.9 -> 16.3 us at batch 256)
  const bool apart = n_in == 0 || n_out == 1;
  if (n_in > 0) {
    const int rc = launch_gemm(n_out, n_in, batch, dY, 0, 1, n_out, X, 0, n_in, 1, dW, n_in,
                               nullptr, 0, nullptr, apart ? nullptr : db, (cudaStream_t)stream);
    if (rc != NLA3D_OK || !apart) return rc;
  }
  return nla3d_mlp_column_sum(dY ? dY : db, batch, n_out, db, stream);
}

int nla3d_mlp_input_grad(int batch, int n_out, int n_in, const float* dY, const uint16_t* W_bf16,
                         const float* Y, float* dX, void* stream) {
  if (batch < 0 || n_out < 0 || n_in < 0 || !dX || (batch > 0 && n_out > 0 && (!dY || !W_bf16)))
    return NLA3D_ERR_ARG;
  // dX[b,i] = (sum_o dY[b,o] W[o,i]) (1 - Y[b,i]^2), Y the layer's tanh input
  return launch_gemm(batch, n_in, n_out, dY, 0, n_out, 1, W_bf16, 1, n_in, 1, dX, n_in, nullptr, 0,
                     Y, nullptr, (cudaStream_t)stream);
}

int nla3d_mlp_status(uint32_t* timeouts) {
  if (!timeouts) return NLA3D_ERR_ARG;
  unsigned int v = 0, zero = 0;
  cudaError_t e = cudaMemcpyFromSymbol(&v, g_mlp_timeouts, sizeof(v));
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_mlp_timeouts, &zero, sizeof(zero));
  *timeouts = v;
  return status(e);
}

int nla3d_mlp_tanh_backward(const float* Y, float* dY, int64_t n, void* stream) {
  if (!Y || !dY || n < 0) return NLA3D_ERR_ARG;
  if (n == 0) return NLA3D_OK;
  tanh_bwd_kernel<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(Y, dY, n);
  return status(cudaGetLastError());
}

int nla3d_mlp_column_sum(const float* X, int64_t rows, int64_t cols, float* out, void* stream) {
  if (!X || !out || rows < 0 || cols < 0) return NLA3D_ERR_ARG;
  if (cols == 0) return NLA3D_OK;
  column_sum_kernel<<<(unsigned)((cols + 31) / 32), 256, 0, (cudaStream_t)stream>>>(X, rows, cols,
                                                                                     out);
  return status(cudaGetLastError());
}

int nla3d_mlp_adam(float* w, const float* g, float* m, float* v, int64_t n, float lr, float beta1,
                   float beta2, float eps, int step, uint16_t* w_bf16, void* stream) {
  if (!w || !g || !m || !v || n < 0 || step < 1) return NLA3D_ERR_ARG;
  if (n == 0) return NLA3D_OK;
  const float c1 = 1.f - powf(beta1, (float)step), c2 = 1.f - powf(beta2, (float)step);
  adam_kernel<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
      w, g, m, v, n, lr, beta1, beta2, eps, c1, c2, reinterpret_cast<__nv_bfloat16*>(w_bf16));
  return status(cudaGetLastError());
}

int nla3d_mlp_adam_multi(int count, float* const* w, const float* const* g, float* const* m,
                         float* const* v, const int64_t* n, uint16_t* const* w_bf16, float lr,
                         float beta1, float beta2, float eps, int step, void* stream) {
  if (count < 0 || step < 1 || (count > 0 && (!w || !g || !m || !v || !n || !w_bf16)))
    return NLA3D_ERR_ARG;
  for (int t = 0; t < count; t++)
    if (!w[t] || !g[t] || !m[t] || !v[t] || n[t] < 0 || (n[t] + 255) / 256 > 0x7FFFFFFF / kAdamTensors)
      return NLA3D_ERR_ARG;
  const float c1 = 1.f - powf(beta1, (float)step), c2 = 1.f - powf(beta2, (float)step);
  for (int t0 = 0; t0 < count; t0 += kAdamTensors) {
    AdamTensors a{};
    a.count = count - t0 < kAdamTensors ? count - t0 : kAdamTensors;
    for (int t = 0; t < a.count; t++) {
      a.n[t] = (long)n[t0 + t];
      a.w[t] = w[t0 + t];
      a.g[t] = g[t0 + t];
      a.m[t] = m[t0 + t];
      a.v[t] = v[t0 + t];
      a.wb[t] = reinterpret_cast<__nv_bfloat16*>(w_bf16[t0 + t]);
      a.first[t + 1] = a.first[t] + (unsigned)((n[t0 + t] + 255) / 256);
    }
    if (!a.first[a.count]) continue;
    adam_multi_kernel<<<a.first[a.count], 256, 0, (cudaStream_t)stream>>>(a, lr, beta1, beta2, eps,
                                                                          c1, c2);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return status(e);
  }
  return NLA3D_OK;
}

int nla3d_mlp_mse_grad(const float* Y, const float* T, float* dY, int64_t n, float scale,
                       void* stream) {
  if (!Y || !T || !dY || n < 0) return NLA3D_ERR_ARG;
  if (n == 0) return NLA3D_OK;
  mse_grad_kernel<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(Y, T, dY, n,
                                                                                  scale);
  return status(cudaGetLastError());
}

int nla3d_mlp_to_bf16(const float* x, uint16_t* y, int64_t n, void* stream) {
  if (!x || !y || n < 0) return NLA3D_ERR_ARG;
  if (n == 0) return NLA3D_OK;
  to_bf16_kernel<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
      x, reinterpret_cast<__nv_bfloat16*>(y), n);
  return status(cudaGetLastError());
}

}  // extern "C"
