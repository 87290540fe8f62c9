// Supernodal multifrontal LDL^T on the device for a symmetric K(2) held in
// the reference's upper CSR layout (SparseSymMatrix, SparseMatrix.h:206-221):
// the GPU counterpart of EquationSolver::factorizeEquations /
// substituteEquations (EquationSolver.h:19-34).  No counterpart exists in the
// reference's own sources for the device; its host PARDISO / dense Gauss
// solvers are what this replaces.
//
// Numeric factorisation, level by level of the supernodal tree (all fronts
// of a level are independent):
//   1. every front is zeroed and the matrix values are scattered into it
//      (one map entry per stored value, computed by the symbolic analysis);
//   2. extend-add: each child's update matrix is added into its parent's
//      front, a warp per parent column taking the children in order, so that
//      no two threads add into one entry and the sums keep a fixed order;
//   3. partial LDL^T of the front's k pivot columns, right-looking, without
//      pivoting (the u/p blocks are quasi-definite: K_uu > 0, K_pp < 0, and
//      constraint rows are ordered last by the caller); a pivot below
//      tau = pivot_rel * max|A| is replaced by +-tau and counted, and the
//      solve's iterative refinement recovers the accuracy.
//      Fronts of <= kSmallFront rows: one thread block per front, the front
//      in shared memory, all fronts of the level in one launch.  Larger
//      fronts: all of the level's together, blocked, 64 columns per panel
//      (diagonal block and its inverse, panel rows) in outer blocks of 256
//      columns: each panel's rank-64 update reaches only the rest of its
//      outer block; the columns after the block take one rank-256 update
//      per block, so each trailing tile is read and written once per 256
//      pivots instead of once per 64 (FMA tiles, or tcgen05 TF32 split MMAs
//      for FP32 fronts with precision 2).
// Solve (multifrontal, vectors): forward by levels with the same extend-add
// on the update vectors, D^-1, backward by levels top-down gathering the
// solved ancestor entries; FP64 refinement r = b - A x with A's
// both-triangle CSR in the input numbering (accelerated steps with FP32
// fronts, plain ones with FP64, then GMRES preconditioned by the factor).
// Factorisation and solve are captured once into CUDA graphs and replayed.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <string>
#include <vector>

#include "../../include/nla3d_gpu.h"
#include "ldlt.hpp"

namespace {

constexpr int kThreads = 256;
constexpr int kSmallFront = 128;   // fronts up to this many rows: one block each, in smem
constexpr int kPanel = 64;         // panel width of the blocked path
constexpr int kOuter = 256;        // outer block of the blocked path (4 panels)
constexpr int kInv = 512;          // pivots whose triangle is kept inverted for the solves
constexpr int kDoublings = kInv == 512 ? 3 : kInv == 256 ? 2 : kInv == 128 ? 1 : 0;
constexpr int kNarrow = kPanel;    // fronts with up to this many pivots: one CTA per solve pass
constexpr int kNarrowRows = 4096;  // ... and up to this many rows

struct LdltDev {
  const uint64_t* front_off;
  const uint64_t* vec_off;
  const int64_t* row_ptr;
  const int32_t* rows;
  const int32_t* sn_first;
  const int64_t* rel_ptr;
  const uint32_t* rel;
  const int32_t* inv_first;   // per supernode: its first kInv-pivot block (large fronts)
  float* inv_error;           // per block: the error of its joined inverse, see inv_probe_kernel
};

// ---- factorisation kernels ----

template <typename T>
__global__ void scatter_values_kernel(uint64_t nnz, const uint64_t* __restrict__ dest,
                                      const double* __restrict__ values, T* __restrict__ front) {
  for (uint64_t q = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; q < nnz;
       q += (uint64_t)gridDim.x * blockDim.x)
    front[dest[q]] = (T)values[q];
}

// max |A| over the stored values: per-block maxima, then one block over them
constexpr int kMaxBlocks = 1024;
__global__ void maxabs_kernel(uint64_t nnz, const double* __restrict__ values,
                              double* __restrict__ part) {
  __shared__ double red[kThreads];
  double m = 0.0;
  for (uint64_t q = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; q < nnz;
       q += (uint64_t)gridDim.x * blockDim.x)
    m = fmax(m, fabs(values[q]));
  red[threadIdx.x] = m;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) red[threadIdx.x] = fmax(red[threadIdx.x], red[threadIdx.x + s]);
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = red[0];
}

__global__ void maxabs_final_kernel(int n, const double* __restrict__ part, double* out) {
  __shared__ double red[kThreads];
  double m = 0.0;
  for (int q = threadIdx.x; q < n; q += blockDim.x) m = fmax(m, part[q]);
  red[threadIdx.x] = m;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) red[threadIdx.x] = fmax(red[threadIdx.x], red[threadIdx.x + s]);
    __syncthreads();
  }
  if (threadIdx.x == 0) out[0] = red[0];
}

// Extend-add of one level in one launch: the front rows of the level are
// contiguous in the solve vectors' order, and the lists that the forward pass
// gathers with (per row: the children's update rows, in child order) are the
// columns that meet in that row's column.  A warp owns a parent column and adds
// the children's columns one after the other, four loads a lane in flight, so
// every entry sums in child order and no two warps share one.
// Memory bounds the wide levels (a child's triangle read, the parent's read
// and written), dependent index loads the others.  A launch per child ordinal
// with at most u / 32 blocks a child had too few loads in flight: 3.0 ms in
// 100 launches of the 139k-equation bar's factor, now 1.2 in 16; 8.2 ms of the
// 457k-equation bar's, now 4.4.  A block per column of the narrow levels, and
// two, three or eight loads a lane, measured the same or slower.
template <typename T>
__global__ void __launch_bounds__(kThreads)
    extend_add_kernel(uint64_t r0, uint64_t r1, const uint32_t* __restrict__ ptr,
                      const uint32_t* __restrict__ src, const int32_t* __restrict__ row_sn,
                      LdltDev d, T* __restrict__ front) {
  const int lane = threadIdx.x & 31;
  const uint64_t r = r0 + blockIdx.x * (uint64_t)(kThreads / 32) + (threadIdx.x >> 5);
  if (r >= r1) return;
  const uint32_t b = ptr[r], e = ptr[r + 1];
  if (b == e) return;
  const int p = row_sn[r];
  const int64_t mp = d.row_ptr[p + 1] - d.row_ptr[p];
  T* dst = front + d.front_off[p] + (int64_t)(r - d.vec_off[p]) * mp;
  for (uint32_t q = b; q < e; q++) {
    const uint32_t sr = src[q];
    const int c = row_sn[sr];
    const int64_t mc = d.row_ptr[c + 1] - d.row_ptr[c];
    const int64_t kc = d.sn_first[c + 1] - d.sn_first[c];
    const int64_t pj = (int64_t)(sr - d.vec_off[c]);   // the child's column, in its front
    const T* col = front + d.front_off[c] + pj * mc;
    const uint32_t* rel = d.rel + d.rel_ptr[c];
    constexpr int kU = 4;
    for (int64_t i0 = pj + lane; i0 < mc; i0 += kU * 32) {
      T v[kU], w[kU];
      uint32_t t[kU];
#pragma unroll
      for (int x = 0; x < kU; x++) {
        const int64_t i = i0 + x * 32;
        t[x] = i < mc ? rel[i - kc] : 0u;
        v[x] = i < mc ? col[i] : T(0);
      }
#pragma unroll
      for (int x = 0; x < kU; x++)
        if (i0 + x * 32 < mc) w[x] = dst[t[x]];
#pragma unroll
      for (int x = 0; x < kU; x++)
        if (i0 + x * 32 < mc) dst[t[x]] = w[x] + v[x];
    }
    __syncwarp();
  }
}

// the guarded pivot without counting it
template <typename T>
__device__ __forceinline__ T guard_value(T dv, T tau) {
  if (!(fabs(dv) >= tau) && dv == dv) return dv < T(0) ? -tau : tau;
  return dv;
}

template <typename T>
__device__ __forceinline__ T guard_pivot(T dv, T tau, int* perturbed) {
  if (!(fabs(dv) >= tau)) {   // also catches NaN
    if (dv != dv) {
      atomicAdd(perturbed + 1, 1);
      return dv;
    }
    atomicAdd(perturbed, 1);
    return dv < T(0) ? -tau : tau;
  }
  return dv;
}

// one block per front (m <= kSmallFront), the front held in shared memory
// (column-major, leading dimension m+1): right-looking LDL^T of the k pivot
// columns, the trailing (m-k)^2 block left as the update matrix.  A warp per
// column, lane = row.  FP64: warp 0, which updates the next pivot's column
// first, inverts that pivot for everyone (a division per column and pivot kept
// the FP64 pipe busy longer than the update: 311 -> 89 us for a level of the
// 12^3 block's 46 fronts); FP32 divides (111 -> 65 us for 93 of the 139k-equation
// bar's, the columns loaded side by side).
template <typename T>
__global__ void __launch_bounds__(kThreads)
    factor_small_kernel(const int32_t* __restrict__ list, LdltDev d, T* __restrict__ front,
                        const double* __restrict__ tau_p, double pivot_rel, int* perturbed) {
  constexpr bool kShare = std::is_same<T, double>::value;
  extern __shared__ unsigned char smem_raw[];
  T* S = reinterpret_cast<T*>(smem_raw);
  __shared__ T winv[2];
  const int s = list[blockIdx.x];
  const int m = (int)(d.row_ptr[s + 1] - d.row_ptr[s]);
  const int k = d.sn_first[s + 1] - d.sn_first[s];
  const int ld = m + 1;
  T* F = front + d.front_off[s];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  // the lower triangle, four columns a warp in flight
  for (int c0 = ty; c0 < m; c0 += 32)
    for (int r0 = c0 & ~31; r0 < m; r0 += 32) {
      T v[4];
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const int c = c0 + 8 * u, r = r0 + tx;
        v[u] = c < m && r >= c && r < m ? F[r + (int64_t)c * m] : T(0);
      }
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const int c = c0 + 8 * u, r = r0 + tx;
        if (c < m && r >= c && r < m) S[r + c * ld] = v[u];
      }
    }
  __syncthreads();
  // the pivot bound in the front's precision (the guards compare in it)
  const T tau = (T)(pivot_rel * tau_p[0]);
  if (kShare) {
    if (threadIdx.x == 0) winv[0] = T(1) / guard_value(S[0], tau);
    __syncthreads();
  }
  // one barrier per pivot: the columns right of p are updated with the
  // unscaled column p (A_ij -= w_i w_j / d), which no later step writes; the
  // pivot columns are scaled after the loop
  for (int p = 0; p < k; p++) {
    // every thread guards the pivot itself (thread 0 counts)
    const T raw = S[p + p * ld];
    const T dv = threadIdx.x == 0 ? guard_pivot(raw, tau, perturbed) : guard_value(raw, tau);
    const T inv = kShare ? winv[p & 1] : T(0);
    const T* colp = S + p * ld;
    for (int j = p + 1 + ty; j < m; j += 8) {
      const T lj = kShare ? colp[j] * inv : colp[j] / dv;
      T* col = S + j * ld;
      for (int i = j + tx; i < m; i += 32) col[i] -= colp[i] * lj;
      if (kShare && j == p + 1 && tx == 0) winv[j & 1] = T(1) / guard_value(col[j], tau);
    }
    __syncthreads();
  }
  // scale column p by its guarded pivot (its diagonal is unchanged since
  // step p), one warp per column
  for (int p = ty; p < k; p += 8) {
    T* colp = S + p * ld;
    const T dv = guard_value(colp[p], tau);
    for (int i = p + 1 + tx; i < m; i += 32) colp[i] = colp[i] / dv;
    __syncwarp();
    if (tx == 0) colp[p] = dv;
  }
  __syncthreads();
  for (int c = ty; c < m; c += 8)
    for (int r = (c & ~31) + tx; r < m; r += 32)
      if (r >= c) F[r + (int64_t)c * m] = S[r + c * ld];
}

// Small fronts of up to kTinyPivots pivots and kTinyRows rows, a warp each:
// lane = row (kU rows a lane), the pivot columns in registers, the trailing
// columns updated where they lie, kC in flight; the same operations in the
// same order as a block's.  Most are leaves of one pivot and some 25 rows, for
// which a block waited for its columns one after the other, with shared memory
// for the level's widest front: 1104 -> 80 us for the 42,511 of the
// 457k-equation bar, 211 -> 28 for the 17,280 of the batch.  At 128 rows a warp
// takes longer than a block (FP64: 122 us against 89).
constexpr int kTinyPivots = 8;
constexpr int kTinyRows = 64;   // the factorisation's limit: past it a block is faster

template <typename T, int kU, int kC>
__device__ __forceinline__ void factor_tiny(T* __restrict__ F, int m, int k, T tau,
                                            int* perturbed) {
  const int lane = threadIdx.x & 31;
  T w[kTinyPivots][kU], l[kTinyPivots][kU];   // unscaled and scaled pivot columns
#pragma unroll
  for (int p = 0; p < kTinyPivots; p++)
#pragma unroll
    for (int u = 0; u < kU; u++) {
      const int r = lane + 32 * u;
      w[p][u] = p < k && r >= p && r < m ? F[r + (int64_t)p * m] : T(0);
    }
#pragma unroll
  for (int p = 0; p < kTinyPivots; p++) {
    if (p >= k) break;
    const T raw = __shfl_sync(0xffffffffu, w[p][0], p);
    const T dv = lane == 0 ? guard_pivot(raw, tau, perturbed) : guard_value(raw, tau);
#pragma unroll
    for (int u = 0; u < kU; u++) l[p][u] = w[p][u] / dv;
#pragma unroll
    for (int q = p + 1; q < kTinyPivots; q++) {
      if (q >= k) break;
      const T lq = __shfl_sync(0xffffffffu, l[p][0], q);
#pragma unroll
      for (int u = 0; u < kU; u++) w[q][u] -= w[p][u] * lq;
    }
#pragma unroll
    for (int u = 0; u < kU; u++) {
      const int r = lane + 32 * u;
      if (r >= p && r < m) F[r + (int64_t)p * m] = r == p ? dv : l[p][u];
    }
  }
#pragma unroll
  for (int ub = 0; ub < kU; ub++)
    for (int jj = ub == 0 ? k / kC * kC : 0; jj < 32 && 32 * ub + jj < m; jj += kC) {
      T c[kC][kU];
#pragma unroll
      for (int v = 0; v < kC; v++)
#pragma unroll
        for (int u = ub; u < kU; u++) {
          const int j = 32 * ub + jj + v, r = lane + 32 * u;
          c[v][u] = j >= k && r >= j && r < m ? F[r + (int64_t)j * m] : T(0);
        }
#pragma unroll
      for (int p = 0; p < kTinyPivots; p++) {
        if (p >= k) break;
#pragma unroll
        for (int v = 0; v < kC; v++) {
          const T lj = __shfl_sync(0xffffffffu, l[p][ub], jj + v);
#pragma unroll
          for (int u = ub; u < kU; u++) c[v][u] -= w[p][u] * lj;
        }
      }
#pragma unroll
      for (int v = 0; v < kC; v++)
#pragma unroll
        for (int u = ub; u < kU; u++) {
          const int j = 32 * ub + jj + v, r = lane + 32 * u;
          if (j >= k && r >= j && r < m) F[r + (int64_t)j * m] = c[v][u];
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(kThreads)
    factor_tiny_kernel(const int32_t* __restrict__ list, int n, LdltDev d, T* __restrict__ front,
                       const double* __restrict__ tau_p, double pivot_rel, int* perturbed) {
  const int q = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
  if (q >= n) return;   // warp-uniform; no block barrier follows
  const int s = list[q];
  const int m = (int)(d.row_ptr[s + 1] - d.row_ptr[s]);
  const int k = d.sn_first[s + 1] - d.sn_first[s];
  T* F = front + d.front_off[s];
  const T tau = (T)(pivot_rel * tau_p[0]);
  if (m <= 32)
    factor_tiny<T, 1, 8>(F, m, k, tau, perturbed);
  else
    factor_tiny<T, kTinyRows / 32, 4>(F, m, k, tau, perturbed);
}

// Blocked path for the fronts above kSmallFront rows, batched: every launch
// works on panel p0 of all large fronts of one level (blockIdx.z / .x picks
// the front; fronts with k <= p0 return).  W: per front an m x min(kOuter,
// k rounded up to kPanel) block, W[i + c m] = (L D)[i][o0 + c] for the rows
// i past the panel of column o0 + c (o0: the current outer block).
struct BigBatch {
  const int32_t* list;
  const uint64_t* w_off;
  const uint64_t* li_off;   // the front's inverted diagonal blocks, 64 x 64 per panel
  const uint64_t* pk_off;   // tensor-core fronts: the front's packed outer-block operands
};

// step 1: LDL^T of the pb x pb diagonal block, and the inverse of its unit
// lower factor (64 x 64 column-major, kept per panel for step 2 and the solves).
//
// One CTA per front: a chain of 64 pivots, bound by the latency of one step.
// Thread (r, cg) keeps row r, columns 16 cg .. +15 in registers (the front's
// columns are read and written coalesced along r); the group that owns column p
// publishes it (unscaled) in shared memory, and one barrier later every thread
// scales its own row's entry by the pivot and updates its columns.  FP64: the
// pivot's thread inverts it for everyone, since 256 FP64 divisions a step keep
// the pipe busy longer than the update; FP32: every thread divides, off the
// chain of the pivot's thread.
//
// The inverse is formed by substitution, which stays accurate where pivots are
// small (joined from inverses of 16 and 32 rows it left 0.4 instead of 1e-3 of
// the right-hand side after one FP32 application, on a block with three pivots
// of 1e-4).  FP64: along the way, the same row operations on the identity by
// the column groups whose own columns are final, which costs nothing where the
// pipe is the bound.  FP32: afterwards, four threads a column with 16 rows each
// in registers, x_p passed on by shuffle; along the way its loads and stores
// lengthened every step (26 us a launch).
//
// Against the block in shared memory, where each step's update ran as a chain
// of dependent accesses and the inverse row by row as another: 54 -> 21 us
// (FP32; 25 with its own part of an update) and 136 -> 64 us (FP64) a launch.
template <typename T>
constexpr int kDiagLdOf = std::is_same<T, double>::value ? kPanel + 1 : kPanel + 4;

template <typename T>
__global__ void __launch_bounds__(kThreads)
    batched_diag_kernel(BigBatch b, LdltDev d, T* __restrict__ front, int64_t p0,
                        T* __restrict__ Linv, const double* __restrict__ tau_p, double pivot_rel,
                        int* perturbed, int update) {
  static_assert(kThreads == 4 * kPanel, "four column groups of 16");
  constexpr bool kShare = std::is_same<T, double>::value;
  constexpr int kDiagLd = kDiagLdOf<T>;
  // FP64: X[r * kDiagLd + c], to be written transposed; FP32: L, column p at p * kDiagLd
  __shared__ __align__(16) T X[kPanel * kDiagLd];
  __shared__ __align__(16) T wcol[2][kPanel];    // column p, unscaled
  __shared__ __align__(16) T xrow[2][kPanel];    // row p of the inverse
  __shared__ T winv[2];
  const int s = b.list[blockIdx.x];
  const int64_t m = d.row_ptr[s + 1] - d.row_ptr[s];
  const int64_t k = d.sn_first[s + 1] - d.sn_first[s];
  if (p0 >= k) return;
  const int pb = (int)(k - p0 < kPanel ? k - p0 : kPanel);
  T* F = front + d.front_off[s] + p0 + p0 * m;
  const int r = threadIdx.x & (kPanel - 1), cg = threadIdx.x / kPanel;
  T a[16], x[16];
#pragma unroll
  for (int j = 0; j < 16; j++) {
    const int c = 16 * cg + j;
    a[j] = r < pb && c <= r ? F[r + c * m] : (r == c ? T(1) : T(0));
    x[j] = kShare && r == c ? T(1) : T(0);
  }
  if (!kShare && update) {
    // the block's own part of the update that runs meanwhile: A -= L D L^T over
    // the panel before (update 1) or the outer block before (2), 64 columns at
    // a time through X, the next 64 on their way into registers
    const int64_t kw = update == 1 ? kPanel : kOuter;
    const T* Lp = front + d.front_off[s] + (p0 + r) + (p0 - kw) * m;
    const T* Dp = front + d.front_off[s] + (p0 - kw) * (m + 1);
#pragma unroll
    for (int j = 0; j < 16; j++) x[j] = r < pb ? Lp[(int64_t)(16 * cg + j) * m] : T(0);
    T dv = cg == 0 ? Dp[(int64_t)r * (m + 1)] : T(0);
    for (int64_t c0 = 0; c0 < kw; c0 += kPanel) {
      __syncthreads();
#pragma unroll
      for (int j = 0; j < 16; j++) X[(16 * cg + j) * kDiagLd + r] = x[j];
      if (cg == 0) wcol[0][r] = dv;
      __syncthreads();
      if (c0 + kPanel < kw) {
#pragma unroll
        for (int j = 0; j < 16; j++)
          x[j] = r < pb ? Lp[(c0 + kPanel + 16 * cg + j) * m] : T(0);
        if (cg == 0) dv = Dp[(c0 + kPanel + r) * (m + 1)];
      }
      if ((r | 31) < 16 * cg) continue;   // above the diagonal
#pragma unroll 8
      for (int c = 0; c < kPanel; c++) {
        const T l = X[c * kDiagLd + r] * wcol[0][c];
        const float4* w = reinterpret_cast<const float4*>(X + c * kDiagLd + 16 * cg);
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const float4 v = w[u];
          a[4 * u] -= l * v.x;
          a[4 * u + 1] -= l * v.y;
          a[4 * u + 2] -= l * v.z;
          a[4 * u + 3] -= l * v.w;
        }
      }
    }
    __syncthreads();
  }
  // the pivot bound in the front's precision (the guards compare in it)
  const T tau = (T)(pivot_rel * tau_p[0]);
  for (int blk = 0; blk < 4; blk++) {
#pragma unroll
    for (int j = 0; j < 16; j++) {
      const int p = 16 * blk + j;
      if (p >= pb) break;
      T* w = wcol[p & 1];
      T* xr = xrow[p & 1];
      const bool own = cg == blk && r == p;
      if (cg == blk) w[r] = a[j];
      if (kShare && r == p && cg <= blk) {
#pragma unroll
        for (int c = 0; c < 16; c++) xr[16 * cg + c] = x[c];
      }
      if (kShare && own) {
        a[j] = guard_pivot(a[j], tau, perturbed);
        winv[p & 1] = T(1) / a[j];
      }
      __syncthreads();
      // (rows up to p are final, rows above a group's columns not wanted; a warp
      // holds 32 rows of one column group)
      if ((r | 31) < p || (r | 31) < 16 * cg || (!kShare && cg < blk)) continue;
      T l;
      if (kShare) {
        l = w[r] * winv[p & 1];
      } else {
        // every thread guards the pivot itself; its owner counts and keeps it
        const T dv = own ? guard_pivot(w[p], tau, perturbed) : guard_value(w[p], tau);
        if (own) a[j] = dv;
        l = w[r] / dv;
      }
      if (cg > blk) {
#pragma unroll
        for (int c = 0; c < 16; c++) a[c] -= l * w[16 * cg + c];
      } else if (cg == blk) {
#pragma unroll
        for (int c = j + 1; c < 16; c++) a[c] -= l * w[16 * blk + c];
        if (r > p) {
          a[j] = l;
          if (kShare) {
#pragma unroll
            for (int c = 0; c <= j; c++) x[c] -= l * xr[16 * blk + c];
          }
        }
      } else if (r > p) {
#pragma unroll
        for (int c = 0; c < 16; c++) x[c] -= l * xr[16 * cg + c];
      }
    }
  }
  T* Li = Linv + b.li_off[blockIdx.x] + (uint64_t)(p0 / kPanel) * kPanel * kPanel;
#pragma unroll
  for (int j = 0; j < 16; j++) {
    const int c = 16 * cg + j;
    if (r < pb && c <= r) F[r + c * m] = a[j];
    if (kShare) {
      if (r < pb && c < pb) Li[r + c * kPanel] = x[j];
      X[r * kDiagLd + c] = x[j];
    } else {
      X[c * kDiagLd + r] = r > c && r < pb ? a[j] : T(0);
    }
  }
  __syncthreads();
  if constexpr (kShare) {
    // the inverse for the solves too, in the front's unused upper triangle: row
    // c of it down column c (here r runs over the row's entries)
#pragma unroll
    for (int j = 0; j < 16; j++) {
      const int c = 16 * cg + j;
      if (r < c && c < pb) F[r + c * m] = X[c * kDiagLd + r];
    }
  } else {
    // column c of the inverse, rows 16 h .. +15 in this thread: x -= L[:,p] x_p
    const int c = threadIdx.x >> 2, h = threadIdx.x & 3, lane = threadIdx.x & 31;
#pragma unroll
    for (int i = 0; i < 16; i++) x[i] = 16 * h + i == c ? T(1) : T(0);
    const int first = (threadIdx.x >> 5) * 8;   // the warp's first column: zeros above it
    for (int blk = first / 16; blk < 4; blk++) {
#pragma unroll
      for (int j = 0; j < 16; j++) {
        const T xp = __shfl_sync(0xffffffffu, x[j], (lane & ~3) | blk);
        const float4* Lp = reinterpret_cast<const float4*>(X + (16 * blk + j) * kDiagLd + 16 * h);
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const float4 l = Lp[u];   // zero up to row p
          x[4 * u] -= l.x * xp;
          x[4 * u + 1] -= l.y * xp;
          x[4 * u + 2] -= l.z * xp;
          x[4 * u + 3] -= l.w * xp;
        }
      }
    }
    // (Li's 64 x 64 entries are all there; past pb the unit columns)
    float4* Lc = reinterpret_cast<float4*>(Li + c * kPanel + 16 * h);
#pragma unroll
    for (int u = 0; u < 4; u++)
      Lc[u] = make_float4(x[4 * u], x[4 * u + 1], x[4 * u + 2], x[4 * u + 3]);
    // and for the solves in the front's unused upper triangle
#pragma unroll
    for (int i = 0; i < 16; i++)
      if (c < 16 * h + i && 16 * h + i < pb) F[c + (16 * h + i) * m] = x[i];
  }
}

// ---- inverses of the kInv x kInv diagonal blocks, for the solves ----
//
// A substitution through 64-pivot blocks is a chain of dependent launches as
// long as the front's pivots; through the inverses X of larger blocks it is
// two products per block.  Once a level is factored, its fronts' inverses are
// joined in pairs on a second stream while the next levels are factored:
// blocks of s = 64, 128, 256 pivots, X_CA = -X_C (L_CA X_A), two launches per
// doubling over all pairs of the level.  X (unit lower triangular, diagonal
// not stored) lies transposed in the front's upper triangle, X[i][j] at
// row j of column i: it needs no memory, no kernel of the factorisation reads
// there, and a row of X is contiguous.  kInv = 512: the joins of the
// 139k-equation bar take 0.9 ms of kernels beside an 11 ms factorisation; a
// doubling more costs four times the work of all before it.
struct InvTask {
  uint32_t z, j0;     // large front (index in the level's list), first pivot of the pair
  uint32_t tile;      // row tile of C << 16 | column tile of A
};

template <typename T>
struct InvTile {
  static constexpr int BT = 64, RT = 4;
};
template <>
struct InvTile<double> {
  static constexpr int BT = 32, RT = 2;   // as the trailing updates
};

// pass 0: T = L_CA X_A;  pass 1: X_CA = -X_C T.  T: row c, kInv / 2 columns
template <typename T>
__global__ void __launch_bounds__(kThreads)
    inv_join_kernel(const InvTask* __restrict__ tasks, BigBatch b, LdltDev d,
                    T* __restrict__ front, const uint64_t* __restrict__ t_off,
                    T* __restrict__ work, int s, int pass) {
  constexpr int BT = InvTile<T>::BT, RT = InvTile<T>::RT, KS = 16;
  constexpr int LPT = KS * BT / kThreads;
  constexpr int kLdT = kInv / 2;
  __shared__ T As[KS][BT + 1];
  __shared__ T Bs[KS][BT + 1];
  const InvTask t = tasks[blockIdx.x];
  const int sn = b.list[t.z];
  const int64_t m = d.row_ptr[sn + 1] - d.row_ptr[sn];
  const int k = d.sn_first[sn + 1] - d.sn_first[sn];
  T* F = front + d.front_off[sn];
  T* W = work + t_off[t.z];
  const int j0 = (int)t.j0, c0 = j0 + s + (int)(t.tile >> 16) * BT;
  const int a0 = j0 + (int)(t.tile & 0xFFFFu) * BT;
  const int cend = min(j0 + 2 * s, k);
  const int qbeg = pass == 0 ? a0 : j0 + s;
  const int qend = pass == 0 ? j0 + s : min(c0 + BT, cend);
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  T acc[RT][RT] = {};
  T ra[LPT], rb[LPT];
  auto load = [&](int q0) {
#pragma unroll
    for (int e = 0; e < LPT; e++) {
      const int i = threadIdx.x + e * kThreads;
      const int rr = i % BT, q = q0 + i / BT;
      if (pass == 0) {
        const int c = c0 + rr, a = a0 + rr;
        ra[e] = c < cend && q < qend ? F[c + (int64_t)q * m] : T(0);
        rb[e] = q >= qend ? T(0) : q > a ? F[a + (int64_t)q * m] : q == a ? T(1) : T(0);
      } else {
        // X_C's rows run along q
        const int q2 = q0 + i % KS, c = c0 + i / KS;
        ra[e] = c >= cend || q2 >= qend ? T(0)
                : c > q2                ? F[q2 + (int64_t)c * m]
                : c == q2               ? T(1)
                                        : T(0);
        rb[e] = q < qend ? W[(uint64_t)q * kLdT + (a0 - j0) + rr] : T(0);
      }
    }
  };
  load(qbeg);
  for (int q0 = qbeg; q0 < qend; q0 += KS) {
#pragma unroll
    for (int e = 0; e < LPT; e++) {
      const int i = threadIdx.x + e * kThreads;
      if (pass == 0) As[i / BT][i % BT] = ra[e];
      else As[i % KS][i / KS] = ra[e];
      Bs[i / BT][i % BT] = rb[e];
    }
    __syncthreads();
    if (q0 + KS < qend) load(q0 + KS);
#pragma unroll
    for (int q = 0; q < KS; q++) {
      T av[RT], bv[RT];
#pragma unroll
      for (int u = 0; u < RT; u++) av[u] = As[q][ty + 16 * u];
#pragma unroll
      for (int v = 0; v < RT; v++) bv[v] = Bs[q][tx + 16 * v];
#pragma unroll
      for (int u = 0; u < RT; u++)
#pragma unroll
        for (int v = 0; v < RT; v++) acc[u][v] += av[u] * bv[v];
    }
    __syncthreads();
  }
#pragma unroll
  for (int u = 0; u < RT; u++) {
    const int c = c0 + ty + 16 * u;
    if (c >= cend) continue;
#pragma unroll
    for (int v = 0; v < RT; v++) {
      const int a = a0 + tx + 16 * v;
      if (pass == 0) W[(uint64_t)c * kLdT + a - j0] = acc[u][v];
      else F[a + (int64_t)c * m] = -acc[u][v];
    }
  }
}

// step 3: update of the lower triangle, F[i][j] -= sum_c L[i][lc0 + c] W[j][wc0 + c]
// for jb <= j < je, i >= j:
//   inner (outer == 0, after panel p0): the panel's kw = pb columns into the
//     rest of its outer block, jb = p0 + pb, je = min(o0 + kOuter, k);
//   outer (outer == 1, p0 = o0): the whole outer block, kw = min(k, o0 +
//     kOuter) - o0 columns, into everything after it, jb = o0 + kw, je = m.
// Every front's (lc0, wc0, kw, jb, je) follow from its own k and m.
struct UpdateRange {
  int64_t lc0, wc0, kw, jb, je;
};

__device__ __forceinline__ bool update_range(int64_t p0, int outer, int64_t k, int64_t m,
                                             UpdateRange& u) {
  if (p0 >= k) return false;
  if (!outer) {
    const int64_t pb = k - p0 < kPanel ? k - p0 : kPanel;
    const int64_t o0 = p0 - p0 % kOuter;
    u.lc0 = p0;
    u.wc0 = p0 % kOuter;
    u.kw = pb;
    u.jb = p0 + pb;
    u.je = o0 + kOuter < k ? o0 + kOuter : k;
  } else {
    const int64_t oe = p0 + kOuter < k ? p0 + kOuter : k;
    u.lc0 = p0;
    u.wc0 = 0;
    u.kw = oe - p0;
    u.jb = oe;
    u.je = m;
  }
  return u.jb < u.je;
}

// the first row past the front's next diagonal block (0: no such block)
__device__ __forceinline__ int64_t next_block_end(const UpdateRange& u, int64_t k) {
  return u.jb < k ? u.jb + (k - u.jb < kPanel ? k - u.jb : kPanel) : 0;
}

// BT x BT tiles (blockIdx.x rows from row_tile0, .y columns, both from jb), front
// blockIdx.z, RT x RT outputs per thread (32 / 2 for FP64: its pipe bounds the
// kernel, one SM takes 64 us for a 64 x 64 tile of a rank-64 update, and
// smaller tiles reach more SMs; 128 / 8 for FP32).  A thread owns rows tx + 16u and
// columns ty + 16v: shared-memory reads are conflict-free or broadcast and
// the stores run down the columns.  The next 16-wide slice of the operands
// is loaded into registers while the current one is multiplied.  ahead: the
// next diagonal block is left out (its own kernel updates it meanwhile).
template <typename T, int BT, int RT>
__global__ void __launch_bounds__(kThreads)
    batched_trailing_kernel(BigBatch b, LdltDev d, T* __restrict__ front, int64_t p0, int outer,
                            const T* __restrict__ Wbuf, int row_tile0, int ahead) {
  static_assert((BT / RT) * (BT / RT) == kThreads, "one output block per thread");
  static_assert(BT / RT == 16, "16 x 16 threads");
  constexpr int LPT = 16 * BT / kThreads;   // slice elements each thread loads per operand
  const int ti = blockIdx.x + row_tile0, tj = blockIdx.y;
  if (tj > ti) return;
  const int s = b.list[blockIdx.z];
  const int64_t m = d.row_ptr[s + 1] - d.row_ptr[s];
  const int64_t k = d.sn_first[s + 1] - d.sn_first[s];
  UpdateRange ur;
  if (!update_range(p0, outer, k, m, ur)) return;
  const int64_t i0 = ur.jb + (int64_t)ti * BT, j0 = ur.jb + (int64_t)tj * BT;
  if (i0 >= m || j0 >= ur.je) return;
  T* F = front + d.front_off[s];
  const T* W = Wbuf + b.w_off[blockIdx.z];
  const int kw = (int)ur.kw;
  __shared__ T As[16][BT];
  __shared__ T Bs[16][BT];
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  T acc[RT][RT] = {};
  T ra[LPT], rb[LPT];
  auto load = [&](int c0) {
#pragma unroll
    for (int q = 0; q < LPT; q++) {
      const int t = threadIdx.x + q * kThreads;
      const int cc = t / BT, rr = t % BT;
      const int c = c0 + cc;
      const int64_t i = i0 + rr, j = j0 + rr;
      ra[q] = (c < kw && i < m) ? F[i + (ur.lc0 + c) * m] : T(0);
      rb[q] = (c < kw && j < ur.je) ? W[j + (ur.wc0 + c) * m] : T(0);
    }
  };
  load(0);
  for (int c0 = 0; c0 < kw; c0 += 16) {
#pragma unroll
    for (int q = 0; q < LPT; q++) {
      const int t = threadIdx.x + q * kThreads;
      As[t / BT][t % BT] = ra[q];
      Bs[t / BT][t % BT] = rb[q];
    }
    __syncthreads();
    if (c0 + 16 < kw) load(c0 + 16);
#pragma unroll
    for (int cc = 0; cc < 16; cc++) {
      T a[RT], bb[RT];
#pragma unroll
      for (int u = 0; u < RT; u++) a[u] = As[cc][tx + 16 * u];
#pragma unroll
      for (int v = 0; v < RT; v++) bb[v] = Bs[cc][ty + 16 * v];
#pragma unroll
      for (int u = 0; u < RT; u++)
#pragma unroll
        for (int v = 0; v < RT; v++) acc[u][v] += a[u] * bb[v];
    }
    __syncthreads();
  }
  const int64_t i_min = ahead ? next_block_end(ur, k) : 0;
#pragma unroll
  for (int v = 0; v < RT; v++) {
    const int64_t j = j0 + ty + 16 * v;
    if (j >= ur.je) continue;
#pragma unroll
    for (int u = 0; u < RT; u++) {
      const int64_t i = i0 + tx + 16 * u;
      if (i < m && j <= i && i >= i_min) F[i + j * m] -= acc[u][v];
    }
  }
}

template <typename T>
struct TrailingShape {
  static constexpr int BT = 32, RT = 2;
};
template <>
struct TrailingShape<float> {
  static constexpr int BT = 128, RT = 8;
};

// ---- tensor-core helpers (tcgen05, kind::tf32) ----
//
// Operands are split into TF32 high and low parts (x = hi + lo, hi = x
// rounded to TF32) and staged in shared memory in the canonical K-major
// layout without swizzle (8-row x 16-byte core matrices; K-adjacent cores
// 128 B apart, 8-row groups 1 KB apart); an update tile is 128 x 128, its
// operands taken in chunks of 32 columns, each chunk 4 k-steps x 3 MMAs
// (hi.hi + hi.lo + lo.hi, FP32 accumulation in TMEM).
constexpr int kTcM = 128, kTcN = 128, kTcKH = 32;   // tile rows, columns, K per chunk
constexpr uint32_t kTcTileFloats = kTcM * kTcKH;     // one 128 x 32 operand chunk
// instruction descriptor: D F32 (bit 4), A and B TF32 (bits 7, 10), both
// K-major, N / 8 at bit 17, M / 16 at bit 24
constexpr uint32_t kTcIdesc =
    (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(kTcN >> 3) << 17) | ((uint32_t)(kTcM >> 4) << 24);
constexpr long long kTcSpinLimit = 1ll << 26;

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// shared-memory matrix descriptor: start, leading (K) and stride (8-row) byte
// offsets, descriptor version 1, no swizzle
__device__ __forceinline__ uint64_t tc_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

__device__ __forceinline__ float tf32_hi(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return __uint_as_float(r);
}

// offset (floats) of element (row r, k) of a 128 x 32 K-major operand chunk
__device__ __forceinline__ uint32_t tc_off(int r, int k) {
  return (uint32_t)(((r >> 3) * (kTcKH / 4) + (k >> 2)) * 32 + (r & 7) * 4 + (k & 3));
}

__device__ __forceinline__ bool tc_wait(uint32_t mbar, uint32_t phase) {
  for (long long it = 0; it < kTcSpinLimit; it++) {
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

__device__ __forceinline__ void tc_mma(uint32_t tmem, uint64_t a, uint64_t b, uint32_t acc) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.u32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
      "l"(a), "l"(b), "r"(kTcIdesc), "r"(acc));
}

// ---- the updates from packed operands (tensor-core fronts) ----
//
// An update (update_range: the rank-256 one after an outer block, or a
// panel's rank-64 one inside its block) reads the same operands from every
// tile of a row or column: L and W = L D of its columns.  batched_panel_kernel
// writes them once, split into TF32 high and low parts: per 128-row block
// (counted from the outer block's first row o0) and 32-column chunk, four 16
// KB tiles (A = L hi, lo, B = W hi, lo) in the MMA's shared-memory layout
// (tc_off), so a panel's chunks serve its own update and the outer block's.
// Tiles are aligned to o0; rows and columns of a tile outside the update's
// range are computed from whatever their slots hold and not stored.
// tc_packed_kernel is persistent
// (one CTA per SM walking a host-built list of the level's tiles) and
// warp-specialised:
//   warp 0 (one lane): copies each chunk's four tiles into a ring of
//     kPkStages shared-memory stages with asynchronous bulk copies
//     (cp.async.bulk, completion counted on the stage's `full` mbarrier);
//   warp 1 (one lane): waits for a stage, issues its 12 MMAs (hi.hi, hi.lo,
//     lo.hi per 8-wide k step) into one of two 128-column TMEM
//     accumulators and commits them to the stage's `empty` mbarrier (the
//     stage is refilled once they have read it) and, after a tile's last
//     chunk, to the accumulator's `acc_full` mbarrier;
//   warps 2-9: load their 32 rows x 64 columns of the front tile into
//     registers while the tile's MMAs run, then read the same part of the
//     finished accumulator from TMEM, release it (`acc_empty`, one arrival
//     per warp) and store the difference, while the MMAs of the next tile
//     run into the other accumulator.
// Every wait is bounded: on a timeout the role stops, err[0] is set and the
// copies and MMAs still in flight get one more bounded wait each before the
// CTA releases its shared memory and TMEM.
constexpr int kPkChunks = kOuter / kTcKH;                  // 8 chunks of 32 columns
constexpr uint32_t kPkTile = kTcTileFloats;                // floats per 128 x 32 tile
constexpr uint32_t kPkBlock = 4 * kPkTile * kPkChunks;    // floats per 128-row block
constexpr int kPkStages = 3;
constexpr size_t kPkSmem = (size_t)kPkStages * 4 * kPkTile * sizeof(float) + 256;
constexpr int kOuterThreads = 320;   // tc_packed_kernel: producer, MMA, 8 epilogue warps

// step 2: the panel rows i >= q0 = p0+pb: W = F21 Linv^T (W = L21 D), F21 <- W
// D^-1; PanelRows<T> rows per CTA, all 64 columns of both operands loaded at
// once.  Thread (tx, ty) owns columns 4 tx .. +3 of rows ty + 16 u; a warp
// holds two neighbouring tx, so it stops its sum where its columns of Linv^T
// (upper triangular) end.  FP64: 16 rows per CTA, since one SM's FP64 pipe
// would take 64 us for 64 rows and most launches have fewer tiles than SMs.
// Tensor-core fronts (kPack): instead of W, both operands of the updates that
// follow are written here, split and in the MMA's layout (see tc_packed_kernel).
template <typename T>
struct PanelRows {
  static constexpr int value = 64;
};
template <>
struct PanelRows<double> {
  static constexpr int value = 16;
};

template <typename T, bool kPack>
__global__ void __launch_bounds__(kThreads)
    batched_panel_kernel(BigBatch b, LdltDev d, T* __restrict__ front, int64_t p0,
                         const T* __restrict__ Linv, T* __restrict__ Wbuf,
                         float* __restrict__ packed) {
  constexpr int R = PanelRows<T>::value, RU = R / 16;
  __shared__ T As[kPanel][R];
  __shared__ __align__(16) T Bs[kPanel][kPanel];
  __shared__ T Dv[kPanel];
  const int s = b.list[blockIdx.y];
  const int64_t m = d.row_ptr[s + 1] - d.row_ptr[s];
  const int64_t k = d.sn_first[s + 1] - d.sn_first[s];
  if (p0 >= k) return;
  const int pb = (int)(k - p0 < kPanel ? k - p0 : kPanel);
  const int64_t q0 = p0 + pb;
  const int64_t i0 = q0 + (int64_t)blockIdx.x * R;
  if (i0 >= m) return;
  T* F = front + d.front_off[s];
  const T* Li = Linv + b.li_off[blockIdx.y] + (uint64_t)(p0 / kPanel) * kPanel * kPanel;
  if (threadIdx.x < kPanel)
    Dv[threadIdx.x] = threadIdx.x < pb ? F[(p0 + threadIdx.x) * (m + 1)] : T(1);
#pragma unroll
  for (int q = 0; q < kPanel * R / kThreads; q++) {
    const int t = threadIdx.x + q * kThreads;
    const int rr = t % R, c2 = t / R;
    As[c2][rr] = (c2 < pb && i0 + rr < m) ? F[i0 + rr + (p0 + c2) * m] : T(0);
  }
#pragma unroll
  for (int q = 0; q < kPanel * kPanel / kThreads; q++) {
    const int t = threadIdx.x + q * kThreads;
    const int c = t % kPanel, c2 = t / kPanel;
    Bs[c2][c] = (c2 < pb && c < pb) ? Li[c + c2 * kPanel] : T(0);   // Linv[c][c2]
  }
  __syncthreads();
  const int tx = threadIdx.x / 16, ty = threadIdx.x % 16;
  const int end = min(pb, 8 * (int)(threadIdx.x / 32) + 8);
  T acc[RU][4] = {};
#pragma unroll 4
  for (int c2 = 0; c2 < end; c2++) {
    T bb[4];
#pragma unroll
    for (int v = 0; v < 4; v++) bb[v] = Bs[c2][tx * 4 + v];
#pragma unroll
    for (int u = 0; u < RU; u++) {
      const T av = As[c2][ty + 16 * u];
#pragma unroll
      for (int v = 0; v < 4; v++) acc[u][v] += av * bb[v];
    }
  }
#pragma unroll
  for (int u = 0; u < RU; u++) {
    const int64_t i = i0 + ty + 16 * u;
    if (i >= m) continue;
    T l[4];
#pragma unroll
    for (int v = 0; v < 4; v++) {
      const int c = tx * 4 + v;
      l[v] = acc[u][v] / Dv[c];
      if (c >= pb) continue;
      F[i + (p0 + c) * m] = l[v];
      if constexpr (!kPack)
        Wbuf[b.w_off[blockIdx.y] + i + (int64_t)(p0 % kOuter + c) * m] = acc[u][v];
    }
    if constexpr (kPack) {
      // columns past pb are zeros: they end the update's last chunk
      const int64_t rel = i - (p0 - p0 % kOuter);
      const int c = (int)(p0 % kOuter) + tx * 4;
      float* P = packed + b.pk_off[blockIdx.y] +
                 ((uint64_t)(rel / kTcM) * kPkChunks + c / kTcKH) * 4 * kPkTile +
                 tc_off((int)(rel % kTcM), c % kTcKH);
      float h[4], e[4];
#pragma unroll
      for (int v = 0; v < 4; v++) {
        h[v] = tf32_hi(l[v]);
        e[v] = l[v] - h[v];
      }
      *reinterpret_cast<float4*>(P) = make_float4(h[0], h[1], h[2], h[3]);
      *reinterpret_cast<float4*>(P + kPkTile) = make_float4(e[0], e[1], e[2], e[3]);
#pragma unroll
      for (int v = 0; v < 4; v++) {
        h[v] = tf32_hi(acc[u][v]);
        e[v] = acc[u][v] - h[v];
      }
      *reinterpret_cast<float4*>(P + 2 * kPkTile) = make_float4(h[0], h[1], h[2], h[3]);
      *reinterpret_cast<float4*>(P + 3 * kPkTile) = make_float4(e[0], e[1], e[2], e[3]);
    }
  }
}

__device__ __forceinline__ void bulk_copy(uint32_t dst, const void* src, uint32_t bytes,
                                          uint32_t mbar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
          "r"(dst), "l"(src), "r"(bytes), "r"(mbar)
      : "memory");
}

__device__ __forceinline__ void expect_tx(uint32_t mbar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar), "r"(bytes)
               : "memory");
}

// one update tile of a level's list: large front z (index in the level's
// list), 128-row block ti and 128-column block tj <= ti from the outer block's
// first row
struct OuterTile {
  uint32_t z, tij;   // tij = ti << 16 | tj
};

__global__ void __launch_bounds__(kOuterThreads, 1)
    tc_packed_kernel(BigBatch b, LdltDev d, float* __restrict__ front, int64_t p0, int outer,
                     const float* __restrict__ packed, const OuterTile* __restrict__ tiles,
                     int n_tiles, int* __restrict__ err, int ahead) {
  extern __shared__ __align__(1024) unsigned char pk_smem[];
  float* stage0 = reinterpret_cast<float*>(pk_smem);
  uint64_t* full = reinterpret_cast<uint64_t*>(stage0 + (size_t)kPkStages * 4 * kPkTile);
  uint64_t* empty = full + kPkStages;
  uint64_t* acc_full = empty + kPkStages;
  uint64_t* acc_empty = acc_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_addr(tmem_slot)),
                 "r"(2 * kTcN));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (threadIdx.x == 32) {
    for (int q = 0; q < kPkStages; q++) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(full + q)), "r"(1));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(empty + q)), "r"(1));
    }
    for (int q = 0; q < 2; q++) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(acc_full + q)),
                   "r"(1));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(acc_empty + q)),
                   "r"(8));
    }
    asm volatile("fence.mbarrier_init.release.cluster;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  constexpr uint32_t kTileBytes = kPkTile * sizeof(float);
  auto stage_addr = [&](int q, int t) {   // t: 0 A hi, 1 A lo, 2 B hi, 3 B lo
    return smem_addr(stage0 + (size_t)(q * 4 + t) * kPkTile);
  };
  // the front of a tile: rows m, update range, chunks
  struct TileInfo {
    int64_t m, jb, je, i0, j0, i_min;
    int nch;
    const float* pa;
    const float* pb;
    float* F;
  };
  auto info = [&](int t, TileInfo& ti) {
    const OuterTile ot = tiles[t];
    const int s = b.list[ot.z];
    const int64_t m = d.row_ptr[s + 1] - d.row_ptr[s];
    const int64_t k = d.sn_first[s + 1] - d.sn_first[s];
    UpdateRange ur;
    update_range(p0, outer, k, m, ur);   // the host listed only fronts whose range is not empty
    const uint32_t rI = ot.tij >> 16, rJ = ot.tij & 0xFFFFu;
    const int64_t o0 = p0 - p0 % kOuter;
    ti.m = m;
    ti.jb = ur.jb;
    ti.je = ur.je;
    ti.i_min = ahead ? next_block_end(ur, k) : 0;
    ti.i0 = o0 + (int64_t)rI * kTcM;
    ti.j0 = o0 + (int64_t)rJ * kTcN;
    ti.nch = (int)((ur.kw + kTcKH - 1) / kTcKH);
    const uint64_t chunk = (uint64_t)(ur.wc0 / kTcKH) * 4 * kPkTile;
    ti.pa = packed + b.pk_off[ot.z] + (uint64_t)rI * kPkBlock + chunk;
    ti.pb = packed + b.pk_off[ot.z] + (uint64_t)rJ * kPkBlock + chunk;
    ti.F = front + d.front_off[s];
  };
  bool ok = true;
  if (warp == 0) {
    if (lane == 0) {
      // producer: the ring of stages, in the MMA warp's order
      uint32_t g = 0, issued = 0;
      for (int t = blockIdx.x; t < n_tiles && ok; t += gridDim.x) {
        TileInfo ti;
        info(t, ti);
        for (int c = 0; c < ti.nch && ok; c++, g++) {
          const int q = g % kPkStages;
          if (g >= kPkStages) ok = tc_wait(smem_addr(empty + q), (g / kPkStages - 1) & 1u);
          if (!ok) break;
          const uint32_t fb = smem_addr(full + q);
          expect_tx(fb, 4 * kTileBytes);
          const float* a = ti.pa + (size_t)c * 4 * kPkTile;
          const float* bb = ti.pb + (size_t)c * 4 * kPkTile;
          bulk_copy(stage_addr(q, 0), a, kTileBytes, fb);
          bulk_copy(stage_addr(q, 1), a + kPkTile, kTileBytes, fb);
          bulk_copy(stage_addr(q, 2), bb + 2 * kPkTile, kTileBytes, fb);
          bulk_copy(stage_addr(q, 3), bb + 3 * kPkTile, kTileBytes, fb);
          issued = g + 1;
        }
      }
      if (!ok) {
        atomicExch(err, 1);
        // the copies of the last kPkStages chunks may still be in flight
        for (uint32_t h = issued > kPkStages ? issued - kPkStages : 0; h < issued; h++)
          tc_wait(smem_addr(full + h % kPkStages), (h / kPkStages) & 1u);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // MMA issuer
      const uint32_t lbo = 128, sbo = (kTcKH / 4) * 128;
      uint32_t g = 0, it = 0, committed_acc = 0;
      for (int t = blockIdx.x; t < n_tiles && ok; t += gridDim.x, it++) {
        TileInfo ti;
        info(t, ti);
        const uint32_t a = it & 1u;
        if (it >= 2) ok = tc_wait(smem_addr(acc_empty + a), (it / 2 - 1) & 1u);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t acc = tmem + a * kTcN;
        for (int c = 0; c < ti.nch && ok; c++, g++) {
          const int q = g % kPkStages;
          ok = tc_wait(smem_addr(full + q), (g / kPkStages) & 1u);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          for (int st = 0; st < kTcKH / 8; st++) {
            const uint32_t koff = st * 256;   // 8 K values = two core matrices
            const uint64_t dah = tc_desc(stage_addr(q, 0) + koff, lbo, sbo);
            const uint64_t dal = tc_desc(stage_addr(q, 1) + koff, lbo, sbo);
            const uint64_t dbh = tc_desc(stage_addr(q, 2) + koff, lbo, sbo);
            const uint64_t dbl = tc_desc(stage_addr(q, 3) + koff, lbo, sbo);
            tc_mma(acc, dah, dbh, (c > 0 || st > 0) ? 1u : 0u);
            tc_mma(acc, dah, dbl, 1u);
            tc_mma(acc, dal, dbh, 1u);
          }
          asm volatile(
              "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                  smem_addr(empty + q))
              : "memory");
        }
        if (!ok) break;
        asm volatile(
            "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                smem_addr(acc_full + a))
            : "memory");
        committed_acc = it + 1;
      }
      if (!ok) {
        atomicExch(err, 1);
        // MMAs complete in order: the last chunk commit covers every MMA issued
        if (g > 0) tc_wait(smem_addr(empty + (g - 1) % kPkStages), ((g - 1) / kPkStages) & 1u);
      } else if (committed_acc > 0) {
        tc_wait(smem_addr(acc_full + ((committed_acc - 1) & 1u)), ((committed_acc - 1) / 2) & 1u);
      }
    }
  } else {
    // epilogue warp (warps 2-9): TMEM lanes 32 (warp % 4) .. +31 = tile rows
    // (a warp reaches only its own lane quarter), columns 64 ((warp - 2) / 4)
    // .. +63
    const int lq = warp & 3, cb = ((warp - 2) >> 2) * 64;
    const int row = lq * 32 + lane;
    uint32_t it = 0;
    for (int t = blockIdx.x; t < n_tiles && ok; t += gridDim.x, it++) {
      TileInfo ti;
      info(t, ti);
      const uint32_t a = it & 1u;
      const int64_t i = ti.i0 + row;
      const bool row_in = i < ti.m && i >= ti.i_min;
      // the front's values of the first 32 columns first: their loads overlap
      // the tile's MMAs; the second 32 load while the first are stored
      float* fp = ti.F + i + (ti.j0 + cb) * ti.m;   // (i, j0 + cb); column stride m
      const int jlim = (int)((row_in ? (i < ti.je - 1 ? i : ti.je - 1) : -1) - (ti.j0 + cb));
      const int jlo = (int)(ti.jb - (ti.j0 + cb));
      float cv[32];
#pragma unroll
      for (int q = 0; q < 32; q++) cv[q] = q <= jlim ? fp[q * ti.m] : 0.0f;
      ok = tc_wait(smem_addr(acc_full + a), (it / 2) & 1u);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int h = 0; h < 2; h++) {
        uint32_t v[32];
#pragma unroll
        for (int c2 = 0; c2 < 2; c2++) {
          const uint32_t taddr = tmem + ((uint32_t)(lq * 32) << 16) + a * kTcN +
                                 (uint32_t)(cb + h * 32 + c2 * 16);
          asm volatile(
              "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, "
              "%10, %11, %12, %13, %14, %15}, [%16];"
              : "=r"(v[c2 * 16 + 0]), "=r"(v[c2 * 16 + 1]), "=r"(v[c2 * 16 + 2]),
                "=r"(v[c2 * 16 + 3]), "=r"(v[c2 * 16 + 4]), "=r"(v[c2 * 16 + 5]),
                "=r"(v[c2 * 16 + 6]), "=r"(v[c2 * 16 + 7]), "=r"(v[c2 * 16 + 8]),
                "=r"(v[c2 * 16 + 9]), "=r"(v[c2 * 16 + 10]), "=r"(v[c2 * 16 + 11]),
                "=r"(v[c2 * 16 + 12]), "=r"(v[c2 * 16 + 13]), "=r"(v[c2 * 16 + 14]),
                "=r"(v[c2 * 16 + 15])
              : "r"(taddr));
        }
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (h == 1) {
          // the accumulator is in registers: the MMAs of the tile after next may reuse it
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0)
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(acc_empty + a))
                         : "memory");
        }
        float nv[32];
        if (h == 0) {
#pragma unroll
          for (int q = 0; q < 32; q++)
            nv[q] = 32 + q <= jlim ? fp[(32 + q) * ti.m] : 0.0f;
        }
#pragma unroll
        for (int q = 0; q < 32; q++)
          if (h * 32 + q >= jlo && h * 32 + q <= jlim)
            fp[(h * 32 + q) * ti.m] = cv[q] - __uint_as_float(v[q]);
        if (h == 0) {
#pragma unroll
          for (int q = 0; q < 32; q++) cv[q] = nv[q];
        }
      }
    }
    if (!ok && lane == 0) atomicExch(err, 1);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(2 * kTcN));
}

// ---- solve kernels ----

// The vectors of one level's fronts before its forward pass, one thread per
// row: the right-hand side for a pivot row, plus the children's update rows in
// child order (a list per row, built with the schedule).  The rows of a level
// are contiguous, so this is one launch; adding one child ordinal per launch
// took 100 launches a pass on the 139k-equation bar (0.6 of 4.4 ms).
__global__ void gather_level_kernel(uint64_t p0, uint64_t p1, const int32_t* __restrict__ b_idx,
                                    const uint32_t* __restrict__ ptr,
                                    const uint32_t* __restrict__ src,
                                    const double* __restrict__ b, double* __restrict__ vec) {
  const uint64_t p = p0 + blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (p >= p1) return;
  const int32_t bi = b_idx[p];
  double v = bi >= 0 ? b[bi] : 0.0;
  const uint32_t e = ptr[p + 1];
  for (uint32_t q = ptr[p]; q < e; q++) v += vec[src[q]];
  vec[p] = v;
}

// Products of the large supernodes' solves.  With FP64 fronts they are FP64
// FMAs.  With FP32 fronts the FP64 pipe (1/64 of the FP32 rate on this part,
// and the float -> double conversion runs on it too) would bound every pass,
// so a product f x of a front entry f and a vector entry x = xh + xl (two
// floats, |xl| <= ulp(xh)/2) is formed exactly in FP32 (p = f xh, e = fma(f,
// xh, -p)) and summed into a double-word accumulator (h, l) by TwoSum, l
// collecting the rounding errors and f xl: the compensated dot product Dot2
// of Ogita, Rump and Oishi (2005), error <= u |sum| + gamma_n^2 sum |f x|
// with u = 2^-24, far below the FP32 factor's own error.  Each accumulator
// adds in a fixed order, so a pass is run-to-run identical.
template <typename T>
struct Dot;

template <>
struct Dot<double> {
  using X = double;
  double s = 0.0;
  __device__ static X split(double x) { return x; }
  __device__ void add(double f, X x) { s = fma(f, x, s); }
  __device__ void merge(const Dot& o) { s += o.s; }
  __device__ void shfl_xor(int lanemask) { s += __shfl_xor_sync(0xffffffffu, s, lanemask); }
  __device__ void shfl_down(int delta) { s += __shfl_down_sync(0xffffffffu, s, delta); }
  __device__ double value() const { return s; }
};

template <>
struct Dot<float> {
  using X = float2;
  float h = 0.0f, l = 0.0f;
  __device__ static X split(double x) {
    const float xh = __double2float_rn(x);
    return make_float2(xh, __double2float_rn(x - (double)xh));
  }
  // h + l += b (TwoSum of h and b; the error joins l)
  __device__ void two_sum(float b, float bl) {
    const float sum = __fadd_rn(h, b);
    const float bv = __fsub_rn(sum, h);
    const float err = __fadd_rn(__fsub_rn(h, __fsub_rn(sum, bv)), __fsub_rn(b, bv));
    h = sum;
    l = __fadd_rn(l, __fadd_rn(err, bl));
  }
  __device__ void add(float f, X x) {
    const float p = __fmul_rn(f, x.x);
    two_sum(p, __fmaf_rn(f, x.y, __fmaf_rn(f, x.x, -p)));
  }
  __device__ void merge(const Dot& o) { two_sum(o.h, o.l); }
  __device__ void shfl_xor(int lanemask) {
    Dot o;
    o.h = __shfl_xor_sync(0xffffffffu, h, lanemask);
    o.l = __shfl_xor_sync(0xffffffffu, l, lanemask);
    merge(o);
  }
  __device__ void shfl_down(int delta) {
    Dot o;
    o.h = __shfl_down_sync(0xffffffffu, h, delta);
    o.l = __shfl_down_sync(0xffffffffu, l, delta);
    merge(o);
  }
  __device__ double value() const { return (double)h + (double)l; }
};

// FP32 fronts, FP64 products (the accurate mode of the refinement): the
// entry widened exactly by integer operations (re-biased exponent, shifted
// mantissa; zero by a select, subnormals and non-finite values by the
// conversion instruction), so that each product takes one FP64 FMA
__device__ __forceinline__ double widen(float f) {
  const uint32_t bits = __float_as_uint(f);
  const uint32_t mag = bits & 0x7FFFFFFFu;
  const uint32_t ex = bits & 0x7F800000u;
  if (mag != 0u && (ex == 0u || ex == 0x7F800000u)) return (double)f;
  const uint32_t sign = bits & 0x80000000u;
  const uint32_t hi = mag ? (sign | ((mag >> 3) + (896u << 20))) : sign;
  const uint32_t lo = mag ? (bits << 29) : 0u;
  return __hiloint2double((int)hi, (int)lo);
}

__device__ __forceinline__ double widen(double f) { return f; }

struct DotWide {
  using X = double;
  double s = 0.0;
  __device__ static X split(double x) { return x; }
  __device__ void add(float f, X x) { s = fma(widen(f), x, s); }
  __device__ void merge(const DotWide& o) { s += o.s; }
  __device__ void shfl_xor(int lanemask) { s += __shfl_xor_sync(0xffffffffu, s, lanemask); }
  __device__ void shfl_down(int delta) { s += __shfl_down_sync(0xffffffffu, s, delta); }
  __device__ double value() const { return s; }
};

// Solves of the small fronts: one CTA per front, FP64 products whatever the
// fronts' type.  FP32 entries take the conversion instruction: these chains wait
// for latency, and widening by integer operations only lengthens them (a pass:
// 100,000 tridiagonal equations in one chain 121.6 instead of 104.1 ms, a band of
// 40 39.8 instead of 33.1, the 139k-equation bar 1.74 instead of 1.69, the batch
// 1.25 instead of 1.21).
// forward: v[0:k] <- D^-1 L11^-1 v[0:k], v[k:m] <- v[k:m] - L21 (L11^-1 v[0:k]);
// blocks of 64 pivots: the block's unit triangle in shared memory, then one
// pass over the rows below it
template <typename T>
__global__ void __launch_bounds__(kThreads)
    forward_kernel(const int32_t* __restrict__ list, LdltDev d, const T* __restrict__ front,
                   double* __restrict__ vec) {
  __shared__ double yb[kPanel];
  const int s = list[blockIdx.x];
  const int64_t m = d.row_ptr[s + 1] - d.row_ptr[s];
  const int64_t k = d.sn_first[s + 1] - d.sn_first[s];
  const T* F = front + d.front_off[s];
  double* v = vec + d.vec_off[s];
  for (int64_t c0 = 0; c0 < k; c0 += kPanel) {
    const int cb = (int)(k - c0 < kPanel ? k - c0 : kPanel);
    if (threadIdx.x < cb) yb[threadIdx.x] = v[c0 + threadIdx.x];
    __syncthreads();
    for (int c = 0; c < cb; c++) {
      const int t = threadIdx.x;
      if (t > c && t < cb) yb[t] -= (double)F[(c0 + t) + (c0 + c) * m] * yb[c];
      __syncthreads();
    }
    if (threadIdx.x < cb) v[c0 + threadIdx.x] = yb[threadIdx.x];
    for (int64_t i = c0 + cb + threadIdx.x; i < m; i += blockDim.x) {
      double acc = 0.0;
      for (int c = 0; c < cb; c++) acc += (double)F[i + (c0 + c) * m] * yb[c];
      v[i] -= acc;
    }
    __syncthreads();
  }
  for (int64_t c = threadIdx.x; c < k; c += blockDim.x) v[c] /= (double)F[c + c * m];
}

// backward: x[0:k] = L11^-T (v[0:k] - L21^T x_rest), x_rest gathered from the
// solved ancestors (factor order), written to xf; blocks of 64 pivots from the
// last: the contributions of the solved pivots below the block (a warp per
// column), then the block's triangle in shared memory
template <typename T>
__global__ void __launch_bounds__(kThreads)
    backward_kernel(const int32_t* __restrict__ list, LdltDev d, const T* __restrict__ front,
                    double* __restrict__ vec, double* __restrict__ xf) {
  __shared__ double xb[kPanel];
  const int s = list[blockIdx.x];
  const int64_t m = d.row_ptr[s + 1] - d.row_ptr[s];
  const int64_t k = d.sn_first[s + 1] - d.sn_first[s];
  const int32_t* rows = d.rows + d.row_ptr[s];
  const T* F = front + d.front_off[s];
  double* v = vec + d.vec_off[s];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nwarps = blockDim.x / 32;
  for (int64_t c = warp; c < k; c += nwarps) {
    double acc = 0.0, acc2 = 0.0;
    int64_t i = k + lane;
    for (; i + 32 < m; i += 64) {
      acc += (double)F[i + c * m] * xf[rows[i]];
      acc2 += (double)F[i + 32 + c * m] * xf[rows[i + 32]];
    }
    if (i < m) acc += (double)F[i + c * m] * xf[rows[i]];
    acc += acc2;
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if (lane == 0) v[c] -= acc;
  }
  __syncthreads();
  for (int64_t c0 = ((k - 1) / kPanel) * kPanel; c0 >= 0; c0 -= kPanel) {
    const int cb = (int)(k - c0 < kPanel ? k - c0 : kPanel);
    for (int c = warp; c < cb; c += nwarps) {
      double acc = 0.0;
      for (int64_t i = c0 + cb + lane; i < k; i += 32) acc += (double)F[i + (c0 + c) * m] * v[i];
      for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
      if (lane == 0) xb[c] = v[c0 + c] - acc;
    }
    __syncthreads();
    for (int c = cb - 1; c >= 0; c--) {
      const int t = threadIdx.x;
      if (t < c) xb[t] -= (double)F[(c0 + c) + (c0 + t) * m] * xb[c];
      __syncthreads();
    }
    if (threadIdx.x < cb) v[c0 + threadIdx.x] = xb[threadIdx.x];
    __syncthreads();
  }
  const int32_t f = d.sn_first[s];
  for (int64_t c = threadIdx.x; c < k; c += blockDim.x) xf[f + c] = v[c];
}

// Small fronts of up to kTinyPivots pivots: a warp per front, lane = row
// (kSmallFront / 32 rows each), the same FP64 products.  Forward: a column at
// a time, v_i -= L[i][c] y_c; then D^-1.  Backward: from the last pivot, x_c =
// v_c - sum_{i > c} L[i][c] x_i, the ancestors' entries gathered first.  Most
// small fronts are leaves of one pivot and some 25 rows (10,293 in the
// 139k-equation bar), for which a CTA each spent its time being launched;
// with more pivots the warp's chain of columns is longer than the CTA's.
constexpr int kSmallRows = kSmallFront / 32;

template <typename T>
__global__ void __launch_bounds__(kThreads)
    fwd_tiny_kernel(const int32_t* __restrict__ list, int n, LdltDev d, const T* __restrict__ front,
                   double* __restrict__ vec) {
  const int q = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
  if (q >= n) return;   // warp-uniform; no block barrier follows
  const int s = list[q], lane = threadIdx.x & 31;
  const int m = (int)(d.row_ptr[s + 1] - d.row_ptr[s]);
  const int k = d.sn_first[s + 1] - d.sn_first[s];
  const T* F = front + d.front_off[s];
  double* v = vec + d.vec_off[s];
  double x[kSmallRows];
#pragma unroll
  for (int u = 0; u < kSmallRows; u++) x[u] = lane + 32 * u < m ? v[lane + 32 * u] : 0.0;
  const double piv = lane < k ? widen(F[lane + lane * m]) : 1.0;
#pragma unroll 4
  for (int c = 0; c < k; c++) {
    const double yc = __shfl_sync(0xffffffffu, x[0], c);
#pragma unroll
    for (int u = 0; u < kSmallRows; u++) {
      const int r = lane + 32 * u;
      if (r > c && r < m) x[u] = fma(-widen(F[r + c * m]), yc, x[u]);
    }
  }
  if (lane < k) x[0] = x[0] / piv;
#pragma unroll
  for (int u = 0; u < kSmallRows; u++)
    if (lane + 32 * u < m) v[lane + 32 * u] = x[u];
}

template <typename T>
__global__ void __launch_bounds__(kThreads)
    bwd_tiny_kernel(const int32_t* __restrict__ list, int n, LdltDev d, const T* __restrict__ front,
                    const double* __restrict__ vec, double* __restrict__ xf) {
  const int q = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
  if (q >= n) return;   // warp-uniform; no block barrier follows
  const int s = list[q], lane = threadIdx.x & 31;
  const int m = (int)(d.row_ptr[s + 1] - d.row_ptr[s]);
  const int k = d.sn_first[s + 1] - d.sn_first[s];
  const int32_t* rows = d.rows + d.row_ptr[s];
  const T* F = front + d.front_off[s];
  const double* v = vec + d.vec_off[s];
  double x[kSmallRows];
#pragma unroll
  for (int u = 0; u < kSmallRows; u++) {
    const int r = lane + 32 * u;
    x[u] = r < k ? v[r] : r < m ? xf[rows[r]] : 0.0;
  }
#pragma unroll 2
  for (int c = k - 1; c >= 0; c--) {
    double acc = 0.0;
#pragma unroll
    for (int u = 0; u < kSmallRows; u++) {
      const int r = lane + 32 * u;
      if (r > c && r < m) acc = fma(widen(F[r + c * m]), x[u], acc);
    }
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == c) x[0] -= acc;
  }
  if (lane < k) xf[d.sn_first[s] + lane] = x[0];
}

// Solves of the large fronts, batched per level.  Fronts with up to kNarrow
// pivots (and kNarrowRows rows) take one CTA each and pass; wider ones go by
// blocks of kInv pivots, two launches per block and direction: the block
// through its inverse X, then the rows below it (forward) or the pivots before
// it (backward).  Every product chain is split so that its loads are issued
// together, and partial sums are merged in a fixed order (run-to-run
// identical).  The passes are bound by the latency of that chain of launches
// near the root and by the fronts' bytes below it.  Blocks of 256 pivots with
// 64 x 64 inverses took 59 block steps of 35 us a direction on the
// 139k-equation bar, 4.4 ms a pass; these take 34 steps, 1.7 ms a pass.

// forward, narrow fronts: y = X v, v[0:k] <- D^-1 y, v[k:m] -= L21 y
template <typename T, typename D>
__global__ void __launch_bounds__(kThreads)
    fwd_narrow_kernel(const int32_t* __restrict__ list, LdltDev d, const T* __restrict__ front,
                      double* __restrict__ vec) {
  using X = typename D::X;
  static_assert(kThreads == 4 * kNarrow, "four threads per pivot row");
  __shared__ X xs[kNarrow];
  __shared__ X ys[kNarrow];
  const int s = list[blockIdx.x];
  const int64_t m = d.row_ptr[s + 1] - d.row_ptr[s];
  const int k = d.sn_first[s + 1] - d.sn_first[s];
  const T* F = front + d.front_off[s];
  double* v = vec + d.vec_off[s];
  const int t = threadIdx.x;
  {
    const int r = t >> 2, q = t & 3;
    T f[kNarrow / 4];
#pragma unroll
    for (int u = 0; u < kNarrow / 4; u++) {
      const int j = q + 4 * u;
      f[u] = r < k && j < r ? F[j + r * m] : T(0);
    }
    if (t < k) xs[t] = D::split(v[t]);
    __syncthreads();
    D y;
#pragma unroll
    for (int u = 0; u < kNarrow / 4; u++)
      if (r < k && q + 4 * u < r) y.add(f[u], xs[q + 4 * u]);
    y.shfl_xor(1);
    y.shfl_xor(2);
    if (r < k && q == 0) {
      const double yv = v[r] + y.value();
      ys[r] = D::split(yv);
      v[r] = yv / (double)F[r + r * m];
    }
  }
  __syncthreads();
  for (int64_t i = k + t; i < m; i += kThreads) {
    const T* Fi = F + i;
    D a0, a1;
    int c = 0;
    // (FP64: 32 loads in flight where the columns are there, 0.51 -> 0.46 ms a
    // pass on the 12^3 block; FP32 loses warps by the registers)
    if constexpr (sizeof(T) == sizeof(double)) {
      for (; c + 32 <= k; c += 32) {
        T f[32];
#pragma unroll
        for (int u = 0; u < 32; u++) f[u] = Fi[(c + u) * m];
#pragma unroll
        for (int u = 0; u < 32; u += 2) {
          a0.add(f[u], ys[c + u]);
          a1.add(f[u + 1], ys[c + u + 1]);
        }
      }
    }
    for (; c < k; c += 16) {
      T f[16];
#pragma unroll
      for (int u = 0; u < 16; u++) f[u] = c + u < k ? Fi[(c + u) * m] : T(0);
#pragma unroll
      for (int u = 0; u < 16; u += 2) {
        if (c + u < k) a0.add(f[u], ys[c + u]);
        if (c + u + 1 < k) a1.add(f[u + 1], ys[c + u + 1]);
      }
    }
    a0.merge(a1);
    v[i] -= a0.value();
  }
}

// backward, narrow fronts: t = v[0:k] - L21^T x_rest, x = X^T t; a warp takes
// four columns of L21 at a time, 128 rows of each in flight
template <typename T, typename D>
__global__ void __launch_bounds__(kThreads)
    bwd_narrow_kernel(const int32_t* __restrict__ list, LdltDev d, const T* __restrict__ front,
                      const double* __restrict__ vec, double* __restrict__ xf) {
  using X = typename D::X;
  extern __shared__ __align__(16) unsigned char narrow_raw[];
  X* xr = reinterpret_cast<X*>(narrow_raw);   // m - k
  __shared__ X ts[kNarrow];
  __shared__ double td[kNarrow];
  const int s = list[blockIdx.x];
  const int64_t m = d.row_ptr[s + 1] - d.row_ptr[s];
  const int k = d.sn_first[s + 1] - d.sn_first[s];
  const int u = (int)(m - k);
  const int32_t* rows = d.rows + d.row_ptr[s] + k;
  const T* F = front + d.front_off[s];
  const double* v = vec + d.vec_off[s];
  for (int i = threadIdx.x; i < u; i += kThreads) xr[i] = D::split(xf[rows[i]]);
  const int j = threadIdx.x >> 2, q = threadIdx.x & 3;   // four threads per pivot
  T fx[kNarrow / 4];
#pragma unroll
  for (int w = 0; w < kNarrow / 4; w++) {
    const int i = q + 4 * w;
    fx[w] = j < i && i < k ? F[j + i * m] : T(0);
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int kCols = 4;
  for (int c = warp * kCols; c < k; c += kThreads / 32 * kCols) {
    const T* Fc = F + k + c * m;
    D a[kCols];
    const int nc = min(k - c, kCols);
    for (int i = lane; i < u; i += 128) {
      T f[4][kCols];
#pragma unroll
      for (int h = 0; h < 4; h++)
#pragma unroll
        for (int w = 0; w < kCols; w++)
          f[h][w] = w < nc && i + 32 * h < u ? Fc[i + 32 * h + w * m] : T(0);
#pragma unroll
      for (int h = 0; h < 4; h++) {
        if (i + 32 * h >= u) break;
        const X x = xr[i + 32 * h];
#pragma unroll
        for (int w = 0; w < kCols; w++) a[w].add(f[h][w], x);
      }
    }
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int w = 0; w < kCols; w++) a[w].shfl_xor(o);
#pragma unroll
    for (int w = 0; w < kCols; w++)
      if (lane == w && w < nc) {
        const double tv = v[c + w] - a[w].value();
        td[c + w] = tv;
        ts[c + w] = D::split(tv);
      }
  }
  __syncthreads();
  D x;
#pragma unroll
  for (int w = 0; w < kNarrow / 4; w++)
    if (j < q + 4 * w && q + 4 * w < k) x.add(fx[w], ts[q + 4 * w]);
  x.shfl_xor(1);
  x.shfl_xor(2);
  if (j < k && q == 0) xf[d.sn_first[s] + j] = td[j] + x.value();
}

// ---- which joined inverses the solves may use ----
//
// y = X v is not a substitution: where elimination has grown (a pressure's
// small pivot ahead of its displacements), the rounding of X, up to
// 2^-24 |X_C| |L_CA| |X_A|, shows in v - L y although every y_i follows from
// the ones before it within a rounding.  On the 7 x 8 x 14 block one
// application then left up to 170 times the residual of 64-pivot substitution.
// So each block is tried once it is joined: v = L e for signs e, y = X v, and
// the largest |v - L y|_i / (|L| |y|)_i, the componentwise backward error
// (Oettli and Prager, Numer. Math. 6, 1964), kept; and the same for L^T and
// X^T.  The solves take a block whose error is above kInvError units of the
// front type's rounding by 64-pivot substitution in one CTA (50 us for 331
// pivots, against 6 through X).  128: sound blocks measure 0.25 to 8 units, the
// few with small pivots 2^5 to 2^17, of which those up to 2^7 changed the
// residual by less than a tenth and those at 2^8 by half; two of some 1,000
// blocks of the 457k-equation bar are above, one or two of 550 of the batch of
// 24 blocks.  The probe takes 0.1 ms of the 139k-equation bar's 11.6 ms factor.
constexpr float kInvError = 128.0f;
struct ProbeTask {
  uint32_t z, j0;   // large front (index in the level's list), first pivot of the block
};

__device__ __forceinline__ float probe_abs(double x) { return (float)fabs(x); }
__device__ __forceinline__ float probe_abs(float2 x) { return fabsf(x.x); }
__device__ __forceinline__ double probe_sign(int j) {
  return (__popc((uint32_t)j * 2654435761u) & 1) ? -1.0 : 1.0;
}

// One tile of 32 outputs, forward (blockIdx.z = 0) or backward (1).  phase 0:
// v = L e, t = L^T e;  1: y = X v, x = X^T t;  2: the errors.  L[i][j] lies at
// (i, j), X[i][j] at (j, i) of the front: L and X^T products have the outputs
// along the contiguous index (lane = output, warps over the terms), the other
// two the terms (a warp per output).
template <typename T, typename D>
__global__ void __launch_bounds__(512)
    inv_probe_kernel(const ProbeTask* __restrict__ tasks, BigBatch b, LdltDev d,
                     const T* __restrict__ front, double* __restrict__ work, int phase) {
  using X = typename D::X;
  constexpr int kW = 16;
  __shared__ X xs[kInv];
  __shared__ D part[kW][32];
  __shared__ float apart[kW][32];
  const ProbeTask t = tasks[blockIdx.x];
  const int s = b.list[t.z];
  const int64_t m = d.row_ptr[s + 1] - d.row_ptr[s];
  const int k = d.sn_first[s + 1] - d.sn_first[s];
  const int n = min(k - (int)t.j0, kInv), p0 = blockIdx.y * 32;
  if (p0 >= n) return;
  const bool back = blockIdx.z != 0;
  const T* F = front + d.front_off[s] + (int64_t)t.j0 * (m + 1);
  double* vt = work + ((int64_t)blockIdx.x * 2 + blockIdx.z) * 2 * kInv;   // v or t
  double* yx = vt + kInv;                                                  // y or x
  for (int j = threadIdx.x; j < n; j += 512)
    xs[j] = D::split(phase == 0 ? probe_sign(j) : phase == 1 ? vt[j] : yx[j]);
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool after = back;                                 // terms q > p (else q < p)
  const bool along = (phase == 1) == back;                 // outputs along the contiguous index
  // outputs of this thread: along, p0 + lane, terms warp, warp + 16, ...; else
  // p0 + warp and p0 + warp + 16, terms lane, lane + 32, ...
  for (int h = 0; h < (along ? 1 : 2); h++) {
    const int p = along ? p0 + lane : p0 + warp + kW * h;
    D a[4];
    float absum = 0.0f;
    if (p < n) {
      const int q0 = along ? warp : lane, dq = along ? kW : 32;
      const T* Fp = along ? F + p : F + (int64_t)p * m;
      const int64_t step = along ? m : 1;
      const int lo = after ? p + 1 : 0, hi = after ? n : p;
      for (int q = q0; q < hi; q += 4 * dq) {
        T f[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const int t4 = q + u * dq;
          f[u] = t4 >= lo && t4 < hi ? Fp[t4 * step] : T(0);
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const int t4 = q + u * dq;
          if (t4 < lo || t4 >= hi) continue;
          a[u].add(f[u], xs[t4]);
          if (phase == 2) absum += fabsf((float)f[u] * probe_abs(xs[t4]));
        }
      }
    }
    a[0].merge(a[1]);
    a[2].merge(a[3]);
    a[0].merge(a[2]);
    if (along) {
      part[warp][lane] = a[0];
      apart[warp][lane] = absum;
      __syncthreads();
      if (warp == 0)
        for (int w = 1; w < kW; w++) {
          a[0].merge(part[w][lane]);
          absum += apart[w][lane];
        }
    } else {
      for (int o = 16; o > 0; o >>= 1) {
        a[0].shfl_xor(o);
        absum += __shfl_xor_sync(0xffffffffu, absum, o);
      }
    }
    if (p < n && (along ? warp : lane) == 0) {
      const double self = phase == 0 ? probe_sign(p) : phase == 1 ? vt[p] : yx[p];
      const double sum = self + a[0].value();   // the diagonal is one
      if (phase < 2) {
        (phase == 0 ? vt : yx)[p] = sum;
      } else {
        const float unit = std::is_same<T, double>::value ? 0x1p-53f : 0x1p-24f;
        const float err = (float)fabs(vt[p] - sum) / (unit * (absum + (float)fabs(self)));
        // non-negative floats order as their bits do, and a NaN above them
        atomicMax(reinterpret_cast<int*>(d.inv_error + d.inv_first[s] + t.j0 / kInv),
                  __float_as_int(err));
      }
    }
  }
}

// the n x n block at F on its way into L2 (a substitution's steps would wait
// for DRAM one after the other)
template <typename T>
__device__ __forceinline__ void prefetch_block(const T* F, int64_t m, int n) {
  constexpr int kLine = 128 / sizeof(T);
  const int lines = (n + kLine - 1) / kLine;
  for (int x = threadIdx.x; x < n * lines; x += blockDim.x) {
    const int c = x / lines, i = min((x - c * lines) * kLine, n - 1);
    asm volatile("prefetch.global.L2 [%0];" ::"l"(F + i + (int64_t)c * m));
  }
}

// y from v by 64-pivot blocks of the block at F (n <= kInv pivots): the
// blocks' own inverses, then the rows after them; one CTA of kThreads
template <typename T, typename D>
__device__ void fwd_substitute(const T* __restrict__ F, int64_t m, int n,
                               const double* __restrict__ v, double* __restrict__ y) {
  using X = typename D::X;
  __shared__ double vs[kInv];
  __shared__ X xs[kPanel], ys[kPanel];
  const int t = threadIdx.x, r = t >> 2, q = t & 3;
  prefetch_block(F, m, n);
  for (int i = t; i < n; i += kThreads) vs[i] = v[i];
  __syncthreads();
  for (int b0 = 0; b0 < n; b0 += kPanel) {
    const int nb = min(kPanel, n - b0);
    if (t < nb) xs[t] = D::split(vs[b0 + t]);
    __syncthreads();
    D a;
    const T* Xr = F + b0 + (int64_t)(b0 + r) * m;
    if (r < nb) {
      T f[kPanel / 4];
#pragma unroll
      for (int u = 0; u < kPanel / 4; u++) f[u] = q + 4 * u < r ? Xr[q + 4 * u] : T(0);
#pragma unroll
      for (int u = 0; u < kPanel / 4; u++)
        if (q + 4 * u < r) a.add(f[u], xs[q + 4 * u]);
    }
    a.shfl_xor(1);
    a.shfl_xor(2);
    if (r < nb && q == 0) {
      const double yr = vs[b0 + r] + a.value();
      y[b0 + r] = yr;
      ys[r] = D::split(yr);
    }
    __syncthreads();
    for (int i = b0 + nb + t; i < n; i += kThreads) {
      const T* Fi = F + i + (int64_t)b0 * m;
      D s[4];
      for (int c = 0; c < nb; c += 16) {
        T f[16];
#pragma unroll
        for (int u = 0; u < 16; u++) f[u] = c + u < nb ? Fi[(int64_t)(c + u) * m] : T(0);
#pragma unroll
        for (int u = 0; u < 16; u++)
          if (c + u < nb) s[u & 3].add(f[u], ys[c + u]);
      }
      s[0].merge(s[1]);
      s[2].merge(s[3]);
      s[0].merge(s[2]);
      vs[i] -= s[0].value();
    }
    __syncthreads();
  }
}

// x from t by 64-pivot blocks, last to first; one CTA of 1024 threads
template <typename T, typename D>
__device__ void bwd_substitute(const T* __restrict__ F, int64_t m, int n,
                               const double* __restrict__ t_in, double* __restrict__ x) {
  using X = typename D::X;
  __shared__ double ts[kInv];
  __shared__ X us[kPanel], xs[kPanel];
  const int t = threadIdx.x;
  prefetch_block(F, m, n);
  for (int i = t; i < n; i += 1024) ts[i] = t_in[i];
  __syncthreads();
  for (int b0 = (n - 1) / kPanel * kPanel; b0 >= 0; b0 -= kPanel) {
    const int nb = min(kPanel, n - b0);
    if (t < nb) us[t] = D::split(ts[b0 + t]);
    __syncthreads();
    const int j = t >> 4, q = t & 15;   // 16 threads a pivot
    D a;
    if (j < nb) {
      T f[kPanel / 16];
#pragma unroll
      for (int u = 0; u < kPanel / 16; u++) {
        const int i = q + 16 * u;
        f[u] = i > j && i < nb ? F[b0 + j + (int64_t)(b0 + i) * m] : T(0);
      }
#pragma unroll
      for (int u = 0; u < kPanel / 16; u++) {
        const int i = q + 16 * u;
        if (i > j && i < nb) a.add(f[u], us[i]);
      }
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) a.shfl_xor(o);
    if (j < nb && q == 0) {
      const double xj = ts[b0 + j] + a.value();
      x[b0 + j] = xj;
      xs[j] = D::split(xj);
    }
    __syncthreads();
    for (int c0 = 0; c0 < b0; c0 += 128) {   // eight lanes a column (b0: a multiple of 64)
      const int c = c0 + (t >> 3), h = t & 7;
      D s;
      if (c < b0) {
        T f[kPanel / 8];
#pragma unroll
        for (int u = 0; u < kPanel / 8; u++)
          f[u] = h + 8 * u < nb ? F[b0 + h + 8 * u + (int64_t)c * m] : T(0);
#pragma unroll
        for (int u = 0; u < kPanel / 8; u++)
          if (h + 8 * u < nb) s.add(f[u], xs[h + 8 * u]);
      }
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) s.shfl_xor(o);
      if (c < b0 && h == 0) ts[c] -= s.value();
    }
    __syncthreads();
  }
}

// forward, wide fronts, block o0: y = X v, a warp per row (a row of X is
// contiguous; all its loads in flight)
constexpr int kInvRows = kThreads / 32;
template <typename T, typename D>
__global__ void __launch_bounds__(kThreads, 4)
    fwd_inv_kernel(const int32_t* __restrict__ list, LdltDev d, const T* __restrict__ front,
                   int64_t o0, const double* __restrict__ vec, double* __restrict__ yv) {
  using X = typename D::X;
  __shared__ X xs[kInv];
  const int s = list[blockIdx.y];
  const int64_t m = d.row_ptr[s + 1] - d.row_ptr[s];
  const int64_t k = d.sn_first[s + 1] - d.sn_first[s];
  if (o0 >= k) return;
  const int ob = (int)(k - o0 < kInv ? k - o0 : kInv);
  const int r0 = blockIdx.x * kInvRows;
  if (r0 >= ob) return;
  const double* v = vec + d.vec_off[s] + o0;
  const float error = d.inv_error[d.inv_first[s] + o0 / kInv];   // looked at once X is on its way
  const int lane = threadIdx.x & 31, i = r0 + (threadIdx.x >> 5);
  T f[kInv / 32];
  if (i < ob) {
    const T* Fi = front + d.front_off[s] + o0 + (o0 + i) * m;
#pragma unroll
    for (int u = 0; u < kInv / 32; u++) f[u] = lane + 32 * u < i ? Fi[lane + 32 * u] : T(0);
  }
  const double vi = lane == 0 && i < ob ? v[i] : 0.0;
  for (int j = threadIdx.x; j < min(ob, r0 + kInvRows); j += kThreads) xs[j] = D::split(v[j]);
  __syncthreads();
  if (!(error <= kInvError)) {
    if (r0 == 0)
      fwd_substitute<T, D>(front + d.front_off[s] + o0 * (m + 1), m, ob, v, yv + d.vec_off[s] + o0);
    return;
  }
  if (i >= ob) return;
  D a[4];
#pragma unroll
  for (int u = 0; u < kInv / 32; u++)
    if (lane + 32 * u < i) a[u & 3].add(f[u], xs[lane + 32 * u]);
  a[0].merge(a[1]);
  a[2].merge(a[3]);
  a[0].merge(a[2]);
  for (int o = 16; o > 0; o >>= 1) a[0].shfl_down(o);
  if (lane == 0) yv[d.vec_off[s] + o0 + i] = vi + a[0].value();
}

// the warps' partial sums per lane, merged in a fixed order by warp 0
template <int kWarps, typename D>
__device__ __forceinline__ bool merge_warps(D& a, D (*part)[32]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  part[warp][lane] = a;
  __syncthreads();
  if (warp != 0) return false;
#pragma unroll
  for (int w = 1; w < kWarps; w++) a.merge(part[w][lane]);
  return true;
}

// forward, wide fronts, block o0: v[i] -= sum_c L[i][o0+c] y_c for the rows
// below the block: lane = row (each load one coalesced 32-row segment of a
// column), a warp per 32 columns and 32 rows.  The block's column groups take
// that many warps of the CTA; a block of few columns leaves warps for further
// row groups (16 warps where a level has blocks above 256 pivots, else 8).
template <typename T, typename D, int kWarps>
__global__ void __launch_bounds__(32 * kWarps)
    fwd_rows_kernel(const int32_t* __restrict__ list, LdltDev d, const T* __restrict__ front,
                    int64_t o0, const double* __restrict__ yv, double* __restrict__ vec) {
  using X = typename D::X;
  struct __align__(16) Pair {
    X a, b;
  };
  __shared__ __align__(16) X yb[kInv];
  __shared__ D part[kWarps][32];
  const int s = list[blockIdx.y];
  const int64_t m = d.row_ptr[s + 1] - d.row_ptr[s];
  const int64_t k = d.sn_first[s + 1] - d.sn_first[s];
  if (o0 >= k) return;
  const int ob = (int)(k - o0 < kInv ? k - o0 : kInv);
  const int groups = (ob + 31) / 32;   // <= kWarps: see the launch
  const int row_groups = kWarps / groups;
  const int64_t r0 = o0 + ob + (int64_t)blockIdx.x * 32 * row_groups;
  if (r0 >= m) return;
  double* v = vec + d.vec_off[s];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int rg = warp / groups, cb = (warp - rg * groups) * 32;
  const int64_t i = r0 + 32 * rg + lane;
  const int nc = rg < row_groups && i < m ? min(ob - cb, 32) : 0;   // this warp's columns
  const bool full = rg < row_groups && ob - cb >= 32;   // the warp's columns are all there
  T f[32];
  const T* Fi = front + d.front_off[s] + (i < m ? i : m - 1) + (o0 + cb) * m;
  if (full) {
#pragma unroll
    for (int u = 0; u < 32; u++) f[u] = Fi[(int64_t)u * m];
  } else {
#pragma unroll
    for (int u = 0; u < 32; u++) f[u] = u < nc ? Fi[(int64_t)u * m] : T(0);
  }
  for (int j = threadIdx.x; j < ob; j += 32 * kWarps)
    yb[j] = D::split(yv[d.vec_off[s] + o0 + j]);
  const double vi = cb == 0 && nc > 0 ? v[i] : 0.0;
  __syncthreads();
  D a[4];
  if (full) {
    const Pair* yp = reinterpret_cast<const Pair*>(yb + cb);
#pragma unroll
    for (int u = 0; u < 32; u += 2) {
      const Pair y = yp[u / 2];
      a[u & 3].add(f[u], y.a);
      a[(u + 1) & 3].add(f[u + 1], y.b);
    }
  } else {
#pragma unroll
    for (int u = 0; u < 32; u++)
      if (u < nc) a[u & 3].add(f[u], yb[cb + u]);
  }
  a[0].merge(a[1]);
  a[2].merge(a[3]);
  a[0].merge(a[2]);
  part[warp][lane] = a[0];
  __syncthreads();
  if (cb == 0 && nc > 0) {
    for (int w = 1; w < groups; w++) a[0].merge(part[warp + w][lane]);
    v[i] = vi - a[0].value();
  }
}

// backward, wide fronts: the solved ancestor entries x[rows[i]], i >= k,
// gathered into v[k:m] (the update rows' slots, free once the forward pass has
// added them into the parent), in the products' operand form (a double, or its
// two-float split in its 8 bytes)
template <typename T, typename D>
__global__ void gather_rest_kernel(const int32_t* __restrict__ list, LdltDev d,
                                   double* __restrict__ vec, const double* __restrict__ xf) {
  using X = typename D::X;
  static_assert(sizeof(X) == sizeof(double), "operand form fills a vector slot");
  const int s = list[blockIdx.y];
  const int64_t m = d.row_ptr[s + 1] - d.row_ptr[s];
  const int64_t k = d.sn_first[s + 1] - d.sn_first[s];
  const int64_t i = k + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  reinterpret_cast<X*>(vec + d.vec_off[s])[i] = D::split(xf[d.rows[d.row_ptr[s] + i]]);
}

// backward, wide fronts: t_c = y_c / d_c - sum_{i >= k} L[i][c] xr_i (xr
// gathered into v[k:m]), a warp per column: the column's contiguous segment
// and xr read by the lanes, eight loads of each in flight, eight partial sums
// merged in a fixed order
template <typename T, typename D>
__global__ void __launch_bounds__(kThreads)
    bwd_rest_kernel(const int32_t* __restrict__ list, LdltDev d, const T* __restrict__ front,
                    const double* __restrict__ yv, double* __restrict__ vec) {
  using X = typename D::X;
  const int s = list[blockIdx.y];
  const int64_t m = d.row_ptr[s + 1] - d.row_ptr[s];
  const int64_t k = d.sn_first[s + 1] - d.sn_first[s];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t c = (int64_t)blockIdx.x * (kThreads / 32) + warp;
  if (c >= k) return;   // warp-uniform; no block barrier follows
  const T* Fc = front + d.front_off[s] + c * m;
  double* v = vec + d.vec_off[s];
  const X* xr = reinterpret_cast<const X*>(v);
  const double yc = lane == 0 ? yv[d.vec_off[s] + c] : 0.0;
  const double dc = lane == 0 ? (double)Fc[c] : 1.0;
  D acc[8];
  int64_t i = k + lane;
  for (; i + 7 * 32 < m; i += 8 * 32) {
    T f[8];
    X x[8];
#pragma unroll
    for (int u = 0; u < 8; u++) {
      f[u] = Fc[i + 32 * u];
      x[u] = xr[i + 32 * u];
    }
#pragma unroll
    for (int u = 0; u < 8; u++) acc[u].add(f[u], x[u]);
  }
  for (; i < m; i += 32) acc[0].add(Fc[i], xr[i]);
#pragma unroll
  for (int u = 1; u < 8; u++) acc[0].merge(acc[u]);
  for (int o = 16; o > 0; o >>= 1) acc[0].shfl_down(o);
  if (lane == 0) v[c] = yc / dc - acc[0].value();
}

// backward, wide fronts, block o0: x = X^T t, lane = pivot j (row i of X gives
// each lane its entry, coalesced), warp w takes the rows w, w + 32, ... from
// the lanes' diagonal piece on; the solved pivots go to xf (factor order)
constexpr int kColThreads = 1024;
template <typename T, typename D>
__global__ void __launch_bounds__(kColThreads)
    bwd_inv_kernel(const int32_t* __restrict__ list, LdltDev d, const T* __restrict__ front,
                   int64_t o0, const double* __restrict__ vec, double* __restrict__ xf) {
  using X = typename D::X;
  __shared__ X ts[kInv];
  __shared__ D part[kColThreads / 32][32];
  const int s = list[blockIdx.y];
  const int64_t m = d.row_ptr[s + 1] - d.row_ptr[s];
  const int64_t k = d.sn_first[s + 1] - d.sn_first[s];
  if (o0 >= k) return;
  const int ob = (int)(k - o0 < kInv ? k - o0 : kInv);
  const int j0 = blockIdx.x * 32;
  if (j0 >= ob) return;
  const double* v = vec + d.vec_off[s] + o0;
  const float error = d.inv_error[d.inv_first[s] + o0 / kInv];   // looked at once X is on its way
  const int j = j0 + (threadIdx.x & 31), i0 = j0 + (threadIdx.x >> 5);
  const T* Fj = front + d.front_off[s] + o0 + j + (o0 + i0) * m;   // X[i][j], i = i0 + 32 u
  T f[kInv / 32];
#pragma unroll
  for (int u = 0; u < kInv / 32; u++)
    f[u] = i0 + 32 * u < ob && i0 + 32 * u > j ? Fj[(int64_t)(32 * u) * m] : T(0);
  for (int i = j0 + threadIdx.x; i < ob; i += kColThreads) ts[i] = D::split(v[i]);
  const double vj = threadIdx.x < 32 && j < ob ? v[j] : 0.0;
  __syncthreads();
  if (!(error <= kInvError)) {
    if (j0 == 0)
      bwd_substitute<T, D>(front + d.front_off[s] + o0 * (m + 1), m, ob, v, xf + d.sn_first[s] + o0);
    return;
  }
  D a[2];
#pragma unroll
  for (int u = 0; u < kInv / 32; u++)
    if (i0 + 32 * u < ob && i0 + 32 * u > j) a[u & 1].add(f[u], ts[i0 + 32 * u]);
  a[0].merge(a[1]);
  if (merge_warps<kColThreads / 32>(a[0], part) && j < ob)
    xf[d.sn_first[s] + o0 + j] = vj + a[0].value();
}

// backward, wide fronts, block o0: t[j] -= sum_c L[o0+c][j] x_c for the pivots
// j < o0 (a warp per column j, lanes over the block's rows)
template <typename T, typename D>
__global__ void __launch_bounds__(kThreads)
    bwd_cols_kernel(const int32_t* __restrict__ list, LdltDev d, const T* __restrict__ front,
                    int64_t o0, const double* __restrict__ xf, double* __restrict__ vec) {
  using X = typename D::X;
  __shared__ X xb[kInv];
  const int s = list[blockIdx.y];
  const int64_t m = d.row_ptr[s + 1] - d.row_ptr[s];
  const int64_t k = d.sn_first[s + 1] - d.sn_first[s];
  if (o0 >= k) return;
  const int64_t j = (int64_t)blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
  if ((int64_t)blockIdx.x * (kThreads / 32) >= o0) return;
  const int ob = (int)(k - o0 < kInv ? k - o0 : kInv);
  for (int c = threadIdx.x; c < ob; c += kThreads) xb[c] = D::split(xf[d.sn_first[s] + o0 + c]);
  __syncthreads();
  if (j >= o0) return;
  const int lane = threadIdx.x & 31;
  const T* Fj = front + d.front_off[s] + o0 + j * m;
  double* vj = vec + d.vec_off[s] + j;
  const double v0 = lane == 0 ? *vj : 0.0;
  D a[4];
  int c = lane;
  for (; c + 7 * 32 < ob; c += 8 * 32) {
    T f[8];
#pragma unroll
    for (int u = 0; u < 8; u++) f[u] = Fj[c + 32 * u];
#pragma unroll
    for (int u = 0; u < 8; u++) a[u & 3].add(f[u], xb[c + 32 * u]);
  }
  for (; c < ob; c += 32) a[0].add(Fj[c], xb[c]);
  a[0].merge(a[1]);
  a[2].merge(a[3]);
  a[0].merge(a[2]);
  for (int o = 16; o > 0; o >>= 1) a[0].shfl_down(o);
  if (lane == 0) *vj = v0 - a[0].value();
}

// x = xf in the input numbering, or x += xf; z: also the step itself
__global__ void solve_finish_kernel(int64_t n, const int32_t* __restrict__ perm,
                                    const double* __restrict__ xf, double* __restrict__ x,
                                    int accumulate, double* __restrict__ z) {
  const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (j >= n) return;
  const int32_t i = perm[j];
  const double v = xf[j];
  if (accumulate)
    x[i] += v;
  else
    x[i] = v;
  if (z) z[i] = v;
}

// (A x)_row, A by both-triangle rows: eight lanes a row with four sums each,
// entry q of the row in sum q % 32, and the 32 sums added pairwise as a warp a
// row would add them, so the rounding is that of chains a 32nd of the row long.
// The FP64 pipe bounds it (2 FMA a clock and SM): with a warp a row, the five
// adds of the reduction cost more than the three products of a typical row of
// 80 entries; with eight lanes a row, four rows share six adds.
constexpr int kRowLanes = 8;
constexpr int kRowsPerBlock = kThreads / kRowLanes;

__device__ __forceinline__ double row_product(int64_t row, const int64_t* __restrict__ ptr,
                                              const int32_t* __restrict__ col,
                                              const uint32_t* __restrict__ slot,
                                              const double* __restrict__ A,
                                              const double* __restrict__ x) {
  constexpr int kU = 32 / kRowLanes;
  double acc[kU] = {};
  const int64_t e = ptr[row + 1];
  for (int64_t q = ptr[row] + threadIdx.x % kRowLanes; q < e; q += 32) {
    double a[kU], v[kU];
#pragma unroll
    for (int u = 0; u < kU; u++) {
      const int64_t t = q + u * kRowLanes;
      a[u] = t < e ? A[slot[t]] : 0.0;
      v[u] = t < e ? x[col[t]] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < kU; u++)
      if (q + u * kRowLanes < e) acc[u] = fma(a[u], v[u], acc[u]);
  }
  return (acc[0] + acc[2]) + (acc[1] + acc[3]);
}

__device__ __forceinline__ double row_sum(double acc) {   // all lanes of the warp
#pragma unroll
  for (int o = kRowLanes / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  return acc;
}

// r = b - A x (dr: what r fell by) and the sums of r^2 and b^2 in `norms`: partial
// sums per block, added up in a fixed order by the block that finishes last (a
// launch of its own for them was 3 us of a small system's pass; copying the pairs
// to the host took as long as the residual on large ones).  `done` counts the
// blocks and returns to zero.  110 -> 45 us on the 139k-equation bar against a warp
// per row.
__global__ void __launch_bounds__(kThreads)
    residual_kernel(int64_t n, const int64_t* __restrict__ ptr, const int32_t* __restrict__ col,
                    const uint32_t* __restrict__ slot, const double* __restrict__ A,
                    const double* __restrict__ x, const double* __restrict__ b,
                    double* __restrict__ r, double* __restrict__ part, double* __restrict__ dr,
                    unsigned* __restrict__ done, double* __restrict__ norms) {
  __shared__ double red[2][kRowsPerBlock];
  __shared__ double sum[kThreads];
  __shared__ bool last;
  const int local = threadIdx.x / kRowLanes;
  const int64_t row = blockIdx.x * (int64_t)kRowsPerBlock + local;
  const double ax = row_sum(row < n ? row_product(row, ptr, col, slot, A, x) : 0.0);
  if (threadIdx.x % kRowLanes == 0) {
    double ri = 0.0, bi = 0.0;
    if (row < n) {
      bi = b[row];
      ri = bi - ax;
      if (dr) dr[row] = r[row] - ri;
      r[row] = ri;
    }
    red[0][local] = ri;
    red[1][local] = bi;
  }
  __syncthreads();
  static_assert(kRowsPerBlock == 32, "a warp holds the block's rows");
  if (threadIdx.x < 32) {
    double rr = red[0][threadIdx.x] * red[0][threadIdx.x];
    double bb = red[1][threadIdx.x] * red[1][threadIdx.x];
    for (int o = 16; o > 0; o >>= 1) {
      rr += __shfl_down_sync(0xffffffffu, rr, o);
      bb += __shfl_down_sync(0xffffffffu, bb, o);
    }
    if (threadIdx.x == 0) {
      part[2 * blockIdx.x] = rr;
      part[2 * blockIdx.x + 1] = bb;
      __threadfence();
      last = atomicInc(done, gridDim.x - 1) == gridDim.x - 1;
    }
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  const int which = threadIdx.x & 1;   // r^2 or b^2
  double acc = 0.0;
#pragma unroll 8
  for (int64_t q = threadIdx.x; q < 2 * (int64_t)gridDim.x; q += kThreads) acc += __ldcg(part + q);
  sum[threadIdx.x] = acc;
  __syncthreads();
  for (int s = kThreads / 2; s > 1; s >>= 1) {
    if (threadIdx.x < s) sum[threadIdx.x] += sum[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x < 2) norms[which] = sum[which];
}

// ---- vector kernels of the accelerated refinement steps ----
//
// A refinement step z = M^-1 r leaves r - A z, and after the first steps it
// falls by the same factor every time (0.03 a step on the 139k-equation bar,
// 0.08 on the 457k-equation one): a few modes of I - A M^-1 dominate it.  So
// the steps z_i and q_i = A z_i, which the next residual gives for nothing (r
// before it less r after it), are kept, q orthonormalised, and r's components
// along them taken out: r -= q_i <q_i, r>, x += z_i <q_i, r>, the least
// residual in the span (GCR; Eisenstat, Elman and Schultz, SIAM J. Numer.
// Anal. 20, 1983).  Two launches of short vectors save one or two of the six to
// nine applications of the factor.
constexpr int kDirs = 30;                // steps kept (GMRES's restart); then GMRES takes over
// Steps without a better x before that: the residual can stay level until the
// space holds the factor's bad modes, and a new basis with GMRES gives the steps
// away.  Twelve against six on 288 made systems (200 to 500 rows, every fourth to
// seventh pivot 1e-2 to 1e-5): 1,173 ms against 1,418, one solve of 54 instead of
// 70 steps among them; a Newton solve of the 457k-equation bar 89 steps where six
// did not reach 1e-10 in 100.  A factor of no help at all costs as much either way
// (2,095 and 2,207 ms a solve of the 1.07M-equation bar, 100 steps).
constexpr int kStalled = 12;
constexpr int kDirSums = 2 * kDirs + 2;
constexpr int kDirChunk = 8;             // directions per block of the sums
constexpr int kDirBlocks = 152;

// partial sums of <q, Q_i>, <r, Q_i> (i < k, kDirChunk a blockIdx.y), <q, q>
// and <q, r>, q = Q_k
__global__ void __launch_bounds__(kThreads)
    direction_sums_kernel(int64_t n, int k, const double* __restrict__ Q,
                          const double* __restrict__ r, double* __restrict__ part) {
  constexpr int kSums = 2 * kDirChunk + 2;
  __shared__ double red[kSums][kThreads];
  const int i0 = blockIdx.y * kDirChunk, ni = min(k - i0, kDirChunk);
  double acc[kSums] = {};
  const double* q = Q + (int64_t)k * n;
  for (int64_t j = blockIdx.x * (int64_t)kThreads + threadIdx.x; j < n;
       j += (int64_t)gridDim.x * kThreads) {
    const double qj = q[j], rj = r[j];
#pragma unroll
    for (int i = 0; i < kDirChunk; i++) {
      if (i >= ni) break;
      const double v = Q[(int64_t)(i0 + i) * n + j];
      acc[2 * i] = fma(qj, v, acc[2 * i]);
      acc[2 * i + 1] = fma(rj, v, acc[2 * i + 1]);
    }
    if (i0 == 0) {
      acc[2 * kDirChunk] = fma(qj, qj, acc[2 * kDirChunk]);
      acc[2 * kDirChunk + 1] = fma(qj, rj, acc[2 * kDirChunk + 1]);
    }
  }
  // (eight threads a sum, 32 entries each: fewer FP64 adds than shuffles)
#pragma unroll
  for (int t = 0; t < kSums; t++) red[t][threadIdx.x] = acc[t];
  __syncthreads();
  const int t = threadIdx.x >> 3, h = threadIdx.x & 7;
  const bool dir = t < 2 * ni, own = i0 == 0 && t >= 2 * kDirChunk && t < kSums;
  if (!dir && !own) return;   // whole groups of eight lanes
  double v = 0.0;
#pragma unroll 8
  for (int w = 0; w < kThreads / 8; w++) v += red[t][h + 8 * w];
  for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(__activemask(), v, o);
  if (h == 0)
    part[blockIdx.x * kDirSums + (dir ? 2 * i0 + t : 2 * kDirs + t - 2 * kDirChunk)] = v;
}

// Q_k and Z_k orthonormalised from those sums, r's components along Q_0 .. Q_k
// taken out of r and into x; partial sums of the new r^2
__global__ void __launch_bounds__(kThreads)
    direction_step_kernel(int64_t n, int k, double* __restrict__ Q, double* __restrict__ Z,
                          double* __restrict__ r, double* __restrict__ x,
                          const double* __restrict__ part, double* __restrict__ rpart) {
  __shared__ double sum[kDirSums];
  __shared__ double red[kThreads / 32];
  static_assert(kDirSums * 4 <= kThreads && kDirBlocks % 4 == 0, "four threads a sum");
  if (threadIdx.x < kDirSums * 4) {
    const int t = threadIdx.x >> 2, h = threadIdx.x & 3;
    const unsigned lanes = __activemask();   // whole groups of four
    double v = 0.0;
    if (t < 2 * k || t >= 2 * kDirs)
#pragma unroll
      for (int b = 0; b < kDirBlocks / 4; b++) v += part[(4 * b + h) * kDirSums + t];
    for (int o = 2; o > 0; o >>= 1) v += __shfl_xor_sync(lanes, v, o);
    if (h == 0) sum[t] = v;
  }
  __syncthreads();
  const double qq = sum[2 * kDirs];
  double n2 = qq, qr = sum[2 * kDirs + 1];
  for (int i = 0; i < k; i++) {
    n2 = fma(-sum[2 * i], sum[2 * i], n2);
    qr = fma(-sum[2 * i], sum[2 * i + 1], qr);
  }
  // a step with nothing new in it is left as a null direction
  const double inv = n2 > 1e-12 * qq ? rsqrt(n2) : 0.0;
  const double beta = inv > 0.0 ? qr * inv : 0.0;
  double rr = 0.0;
  for (int64_t j = blockIdx.x * (int64_t)kThreads + threadIdx.x; j < n;
       j += (int64_t)gridDim.x * kThreads) {
    double q = Q[(int64_t)k * n + j], z = Z[(int64_t)k * n + j], dr = 0.0, dx = 0.0;
#pragma unroll 4
    for (int i = 0; i < k; i++) {
      const double qi = Q[(int64_t)i * n + j], zi = Z[(int64_t)i * n + j];
      q = fma(-sum[2 * i], qi, q);
      z = fma(-sum[2 * i], zi, z);
      dr = fma(sum[2 * i + 1], qi, dr);
      dx = fma(sum[2 * i + 1], zi, dx);
    }
    q *= inv;
    z *= inv;
    Q[(int64_t)k * n + j] = q;
    Z[(int64_t)k * n + j] = z;
    const double rj = r[j] - fma(beta, q, dr);
    r[j] = rj;
    x[j] += fma(beta, z, dx);
    rr = fma(rj, rj, rr);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int o = 16; o > 0; o >>= 1) rr += __shfl_down_sync(0xffffffffu, rr, o);
  if (lane == 0) red[warp] = rr;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kThreads / 32; w++) rr += red[w];
    rpart[blockIdx.x] = rr;
  }
}

// ---- vector kernels of the GMRES refinement (fixed-order reductions) ----
constexpr int kDotBlocks = 1024;

__global__ void dot_kernel(int64_t n, const double* __restrict__ a, const double* __restrict__ b,
                           double* __restrict__ part) {
  __shared__ double red[kThreads];
  double acc = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    acc += a[i] * b[i];
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = red[0];
}

// y += alpha x
__global__ void axpy_kernel(int64_t n, double alpha, const double* __restrict__ x,
                            double* __restrict__ y) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    y[i] += alpha * x[i];
}

// y = alpha x
__global__ void scale_kernel(int64_t n, double alpha, const double* __restrict__ x,
                             double* __restrict__ y) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    y[i] = alpha * x[i];
}

// y = A x
__global__ void __launch_bounds__(kThreads)
    spmv_kernel(int64_t n, const int64_t* __restrict__ ptr, const int32_t* __restrict__ col,
                const uint32_t* __restrict__ slot, const double* __restrict__ A,
                const double* __restrict__ x, double* __restrict__ y) {
  const int64_t row = blockIdx.x * (int64_t)kRowsPerBlock + threadIdx.x / kRowLanes;
  const double ax = row_sum(row < n ? row_product(row, ptr, col, slot, A, x) : 0.0);
  if (row < n && threadIdx.x % kRowLanes == 0) y[row] = ax;
}

}  // namespace

struct nla3d_ldlt {
  LdltSymbolic S;
  int prec = 0;   // 0: FP64 fronts, 1: FP32 fronts (FP64 refinement)
  bool tc = false;   // FP32 fronts with the trailing updates on the tensor cores
  int* d_err = nullptr;
  double pivot_rel = 1e-13;
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  std::string err;
  std::vector<void*> allocs;
  void* d_front = nullptr;
  double* d_vec = nullptr;
  double* d_y = nullptr;        // wide fronts: L^-1 of their pivots' entries
  double* d_xf = nullptr;
  double* d_r = nullptr;
  double* d_dx = nullptr;
  double* d_part = nullptr;     // the residual's partial sums,
  double* d_norm = nullptr;     // their totals: r^2, b^2,
  unsigned* d_done = nullptr;   // and the blocks that have written theirs
  double* d_V = nullptr;        // GMRES basis, (kRestart + 1) x n, allocated on first use
  double* d_dot = nullptr;
  double* d_dirs = nullptr;     // FP32 fronts: the refinement's Q and Z, kDirs x n each, and its best x, or null
  double* d_dirsum = nullptr;   // and their partial sums
  double* d_maxabs = nullptr;
  double* d_maxpart = nullptr;
  int* d_perturbed = nullptr;
  void* d_W = nullptr;
  void* d_Linv = nullptr;
  double* d_rhs = nullptr;      // the solve graph's right-hand side
  double* d_hb = nullptr;       // nla3d_ldlt_solve_host: b and x on the device
  double* d_hx = nullptr;
  cudaGraphExec_t factor_exec = nullptr, solve_exec = nullptr;
  // FP32 fronts: the solve with FP64 products (the refinement's accurate
  // mode, after the compensated-FP32 one stalls), and the mode in use
  cudaGraphExec_t solve_exec_acc = nullptr;
  int solve_accurate = 0;
  const double* factor_graph_values = nullptr;
  uint64_t* d_wo = nullptr;
  uint64_t* d_lio = nullptr;
  uint64_t* d_pko = nullptr;    // tensor-core fronts: packed outer-block operand offsets
  float* d_pk = nullptr;
  OuterTile* d_tiles = nullptr; // tensor-core fronts: every level's outer-block tile lists
  int n_sm = 0;
  InvTask* d_inv = nullptr;     // the inverses' joins: every level's tasks
  uint64_t* d_toff = nullptr;   // per large front: its part of the joins' workspace
  ProbeTask* d_probe = nullptr; // the joined blocks, per level, and their vectors
  double* d_probe_work = nullptr;
  size_t n_inv = 0;             // kInv-pivot blocks of large fronts
  void* d_work = nullptr;
  cudaStream_t side = nullptr;  // the joins run beside the next levels
  cudaEvent_t fork = nullptr, join = nullptr;
  cudaStream_t ahead = nullptr; // the next diagonal blocks run beside the updates
  cudaEvent_t join_ahead = nullptr;
  int32_t* d_bidx = nullptr;    // per front row (level order): its right-hand side entry or -1,
  uint32_t* d_gptr = nullptr;   // and its children's update rows
  uint32_t* d_gsrc = nullptr;
  int32_t* d_rsn = nullptr;     // per front row: its supernode
  uint64_t* d_adest = nullptr;
  int32_t* d_perm = nullptr;
  int32_t* d_lists = nullptr;   // per level: small, large, narrow and wide fronts
  int64_t* d_fptr = nullptr;
  int32_t* d_fcol = nullptr;
  uint32_t* d_fslot = nullptr;
  LdltDev dev{};
  // host schedule per level
  struct Level {
    int64_t small_off = 0, small_cnt = 0, tiny_cnt = 0, warp_cnt = 0;   // see the lists
    int32_t small_max_m = 0;
    int64_t large_off = 0, large_cnt = 0; // fronts above kSmallFront rows
    int64_t wo_off = 0;                   // their W offsets in d_wo
    int64_t large_max_m = 0, large_max_k = 0;
    std::vector<int64_t> tile_off, tile_cnt;  // tensor-core fronts: per outer block, its tiles
    std::vector<int64_t> itile_off, itile_cnt;  // and per panel, its in-block update's tiles
    int64_t inv_off[3] = {}, inv_cnt[3] = {};   // joins of 64-, 128-, 256-pivot blocks
    int64_t probe_off = 0, probe_cnt = 0;       // the joined blocks
    uint64_t vec0 = 0, vec1 = 0;                // its fronts' rows in the solve vectors
    int64_t narrow_off = 0, narrow_cnt = 0, narrow_max_u = 0;   // solves: large fronts by width
    int64_t wide_off = 0, wide_cnt = 0, wide_max_m = 0, wide_max_k = 0;
    bool has_children = false;
  };
  std::vector<Level> levels;
  bool factored = false;
  int perturbed[2] = {0, 0};
  uint64_t front_entries = 0;
};

namespace {

int fail(nla3d_ldlt* h, int code, const std::string& msg) {
  if (h) h->err = msg;
  return code;
}

int cuda_fail(nla3d_ldlt* h, cudaError_t e, const char* where) {
  return fail(h, NLA3D_ERR_CUDA, std::string(where) + ": " + cudaGetErrorString(e));
}

template <typename X>
cudaError_t dalloc(nla3d_ldlt* h, X** p, size_t count) {
  void* q = nullptr;
  cudaError_t e = cudaMalloc(&q, sizeof(X) * (count ? count : 1));
  if (e == cudaSuccess) {
    h->allocs.push_back(q);
    *p = static_cast<X*>(q);
  }
  return e;
}

template <typename X>
cudaError_t upload(nla3d_ldlt* h, X** p, const std::vector<X>& v) {
  cudaError_t e = dalloc(h, p, v.size());
  if (e == cudaSuccess && !v.empty())
    e = cudaMemcpyAsync(*p, v.data(), sizeof(X) * v.size(), cudaMemcpyHostToDevice, h->stream);
  return e;
}

template <typename T>
cudaError_t enqueue_factor(nla3d_ldlt* h, const double* values) {
  const LdltSymbolic& S = h->S;
  T* front = static_cast<T*>(h->d_front);
  cudaStream_t st = h->stream;
  cudaError_t e = cudaMemsetAsync(front, 0, sizeof(T) * h->front_entries, st);
  if (e != cudaSuccess) return e;
  e = cudaMemsetAsync(h->d_perturbed, 0, 2 * sizeof(int), st);
  if (e != cudaSuccess) return e;
  e = cudaMemsetAsync(h->dev.inv_error, 0, sizeof(float) * h->n_inv, st);
  if (e != cudaSuccess) return e;
  bool forked = false;
  {
    const int blocks = (int)std::max<uint64_t>(1, std::min<uint64_t>(
        kMaxBlocks, (S.nnz + kThreads - 1) / kThreads));
    maxabs_kernel<<<blocks, kThreads, 0, st>>>(S.nnz, values, h->d_maxpart);
    maxabs_final_kernel<<<1, kThreads, 0, st>>>(blocks, h->d_maxpart, h->d_maxabs);
  }
  if (S.nnz) {
    const unsigned blocks = (unsigned)std::min<uint64_t>((S.nnz + kThreads - 1) / kThreads, 152 * 16);
    scatter_values_kernel<T><<<blocks, kThreads, 0, st>>>(S.nnz, h->d_adest, values, front);
  }
  for (const auto& L : h->levels) {
    if (L.has_children) {
      constexpr uint64_t kCols = kThreads / 32;
      extend_add_kernel<T><<<(unsigned)((L.vec1 - L.vec0 + kCols - 1) / kCols), kThreads, 0, st>>>(
          L.vec0, L.vec1, h->d_gptr, h->d_gsrc, h->d_rsn, h->dev, front);
    }
    if (L.warp_cnt)
      factor_tiny_kernel<T>
          <<<(unsigned)((L.warp_cnt + kThreads / 32 - 1) / (kThreads / 32)), kThreads, 0, st>>>(
              h->d_lists + L.small_off, (int)L.warp_cnt, h->dev, front, h->d_maxabs, h->pivot_rel,
              h->d_perturbed);
    if (L.small_cnt > L.warp_cnt) {
      const size_t smem = sizeof(T) * (size_t)L.small_max_m * (L.small_max_m + 1);
      factor_small_kernel<T><<<(unsigned)(L.small_cnt - L.warp_cnt), kThreads, smem, st>>>(
          h->d_lists + L.small_off + L.warp_cnt, h->dev, front, h->d_maxabs, h->pivot_rel,
          h->d_perturbed);
    }
    if (L.large_cnt) {
      const BigBatch bb{h->d_lists + L.large_off, h->d_wo + L.wo_off, h->d_lio + L.wo_off,
                        h->d_pko ? h->d_pko + L.wo_off : nullptr};
      T* W = static_cast<T*>(h->d_W);
      T* Li = static_cast<T*>(h->d_Linv);
      const unsigned nf = (unsigned)L.large_cnt;
      constexpr int BT = TrailingShape<T>::BT, RT = TrailingShape<T>::RT;
      const bool tc = std::is_same<T, float>::value && h->tc;
      // one FMA update launch: rows from its range's first column (and row_tile0
      // tiles) to the largest front's last row, `col_tiles` tiles of columns
      auto update = [&](int64_t p, int outer, int64_t rows, unsigned col_tiles, int row_tile0,
                        int ahead) {
        const unsigned rt = (unsigned)((rows + BT - 1) / BT);
        if (rt <= (unsigned)row_tile0) return;
        const dim3 grid(rt - row_tile0, std::min(rt, col_tiles), nf);
        batched_trailing_kernel<T, BT, RT><<<grid, kThreads, 0, st>>>(
            bb, h->dev, front, p, outer, W, row_tile0, ahead);
      };
      auto diag = [&](int64_t p, int upd, cudaStream_t q) {
        batched_diag_kernel<T><<<nf, kThreads, 0, q>>>(bb, h->dev, front, p, Li, h->d_maxabs,
                                                       h->pivot_rel, h->d_perturbed, upd);
      };
      // Look-ahead: the next diagonal block, a chain on one SM, is updated and
      // factored beside the rest of the update that it would wait for.  FP32
      // blocks take their part of the update themselves; FP64 ones have its 64
      // rows updated first, in 16 x 16 tiles (4 us, where one SM would take 34).
      auto look_ahead = [&](int64_t p, int outer, int64_t next) {
        cudaError_t er = cudaEventRecord(h->fork, st);
        if (er == cudaSuccess) er = cudaStreamWaitEvent(h->ahead, h->fork, 0);
        if (er != cudaSuccess) return er;
        if constexpr (std::is_same<T, double>::value)
          batched_trailing_kernel<T, 16, 1><<<dim3(4, 4, nf), kThreads, 0, h->ahead>>>(
              bb, h->dev, front, p, outer, W, 0, 0);
        diag(next, std::is_same<T, double>::value ? 0 : outer + 1, h->ahead);
        return cudaEventRecord(h->join_ahead, h->ahead);
      };
      constexpr int kHeadTiles = std::is_same<T, double>::value ? kPanel / BT : 0;
      diag(0, 0, st);
      for (int64_t o0 = 0; o0 < L.large_max_k; o0 += kOuter) {
        const int64_t o_end = std::min<int64_t>(o0 + kOuter, L.large_max_k);
        for (int64_t p0 = o0; p0 < o_end; p0 += kPanel) {
          const int64_t rest = L.large_max_m - p0 - 1;   // rows past the smallest panel
          if (rest <= 0) continue;
          constexpr int R = PanelRows<T>::value;
          const dim3 panel_grid((unsigned)((rest + R - 1) / R), nf);
          const bool next = p0 + kPanel < o_end;
          if constexpr (std::is_same<T, float>::value) {
            if (tc)
              batched_panel_kernel<float, true><<<panel_grid, kThreads, 0, st>>>(
                  bb, h->dev, front, p0, Li, nullptr, h->d_pk);
          }
          if (!tc)
            batched_panel_kernel<T, false><<<panel_grid, kThreads, 0, st>>>(bb, h->dev, front, p0,
                                                                           Li, W, nullptr);
          if (next && (e = look_ahead(p0, 0, p0 + kPanel)) != cudaSuccess) return e;
          // the panel's columns into the rest of its outer block (at most
          // kOuter - kPanel columns)
          if constexpr (std::is_same<T, float>::value) {
            const int64_t pi = p0 / kPanel;
            const int nt = tc ? (int)L.itile_cnt[pi] : 0;
            if (nt > 0)
              tc_packed_kernel<<<(unsigned)std::min(nt, h->n_sm), kOuterThreads, kPkSmem, st>>>(
                  bb, h->dev, front, p0, 0, h->d_pk, h->d_tiles + L.itile_off[pi], nt, h->d_err,
                  next);
          }
          if (!tc && next)
            update(p0, 0, rest, (unsigned)((kOuter - kPanel + BT - 1) / BT), kHeadTiles, 1);
          if (next && (e = cudaStreamWaitEvent(st, h->join_ahead, 0)) != cudaSuccess) return e;
        }
        // the outer block into every column after it
        const int64_t rest = L.large_max_m - o0 - 1;
        if (rest <= 0) continue;
        const bool next = o_end < L.large_max_k;
        if (next && (e = look_ahead(o0, 1, o_end)) != cudaSuccess) return e;
        if constexpr (std::is_same<T, float>::value) {
          const int64_t ob = o0 / kOuter;
          const int nt = tc ? (int)L.tile_cnt[ob] : 0;
          if (nt > 0)
            tc_packed_kernel<<<(unsigned)std::min(nt, h->n_sm), kOuterThreads, kPkSmem, st>>>(
                bb, h->dev, front, o0, 1, h->d_pk, h->d_tiles + L.tile_off[ob], nt, h->d_err, next);
        }
        if (!tc) update(o0, 1, rest, ~0u, next ? kHeadTiles : 0, next);
        if (next && (e = cudaStreamWaitEvent(st, h->join_ahead, 0)) != cudaSuccess) return e;
      }
      // the solves' inverses on the side stream
      if (L.inv_cnt[0]) {
        if ((e = cudaEventRecord(h->fork, st)) != cudaSuccess) return e;
        if ((e = cudaStreamWaitEvent(h->side, h->fork, 0)) != cudaSuccess) return e;
        forked = true;
        for (int q = 0; q < kDoublings; q++)
          for (int pass = 0; pass < 2 && L.inv_cnt[q]; pass++)
            inv_join_kernel<T><<<(unsigned)L.inv_cnt[q], kThreads, 0, h->side>>>(
                h->d_inv + L.inv_off[q], bb, h->dev, front, h->d_toff + L.wo_off,
                static_cast<T*>(h->d_work), kPanel << q, pass);
        for (int phase = 0; phase < 3; phase++)
          inv_probe_kernel<T, Dot<T>><<<dim3((unsigned)L.probe_cnt, kInv / 32, 2), 512, 0, h->side>>>(
              h->d_probe + L.probe_off, bb, h->dev, front, h->d_probe_work, phase);
      }
    }
  }
  if (forked) {
    if ((e = cudaEventRecord(h->join, h->side)) != cudaSuccess) return e;
    if ((e = cudaStreamWaitEvent(st, h->join, 0)) != cudaSuccess) return e;
  }
  return cudaGetLastError();
}

template <typename T, typename D>
cudaError_t enqueue_solve_core(nla3d_ldlt* h, const double* b) {
  constexpr int kWarps = kThreads / 32;
  const T* front = static_cast<const T*>(h->d_front);
  cudaStream_t st = h->stream;
  for (const auto& L : h->levels) {
    gather_level_kernel<<<(unsigned)((L.vec1 - L.vec0 + kThreads - 1) / kThreads), kThreads, 0, st>>>(
        L.vec0, L.vec1, h->d_bidx, h->d_gptr, h->d_gsrc, b, h->d_vec);
    if (L.tiny_cnt)
      fwd_tiny_kernel<T><<<(unsigned)((L.tiny_cnt + kWarps - 1) / kWarps), kThreads, 0, st>>>(
          h->d_lists + L.small_off, (int)L.tiny_cnt, h->dev, front, h->d_vec);
    if (L.small_cnt > L.tiny_cnt)
      forward_kernel<T><<<(unsigned)(L.small_cnt - L.tiny_cnt), kThreads, 0, st>>>(
          h->d_lists + L.small_off + L.tiny_cnt, h->dev, front, h->d_vec);
    if (L.narrow_cnt)
      fwd_narrow_kernel<T, D><<<(unsigned)L.narrow_cnt, kThreads, 0, st>>>(
          h->d_lists + L.narrow_off, h->dev, front, h->d_vec);
    const int32_t* wide = h->d_lists + L.wide_off;
    const unsigned nf = (unsigned)L.wide_cnt;
    for (int64_t o0 = 0; nf && o0 < L.wide_max_k; o0 += kInv) {
      const int64_t ob = std::min<int64_t>(kInv, L.wide_max_k - o0);
      fwd_inv_kernel<T, D><<<dim3((unsigned)((ob + kInvRows - 1) / kInvRows), nf), kThreads, 0, st>>>(
          wide, h->dev, front, o0, h->d_vec, h->d_y);
      const int64_t rest = L.wide_max_m - o0 - 1;
      if (rest <= 0) continue;
      const dim3 grid((unsigned)((rest + 31) / 32), nf);
      if (ob > 256)
        fwd_rows_kernel<T, D, 16><<<grid, 512, 0, st>>>(wide, h->dev, front, o0, h->d_y, h->d_vec);
      else
        fwd_rows_kernel<T, D, 8><<<grid, 256, 0, st>>>(wide, h->dev, front, o0, h->d_y, h->d_vec);
    }
  }
  for (auto it = h->levels.rbegin(); it != h->levels.rend(); ++it) {
    const auto& L = *it;
    if (L.tiny_cnt)
      bwd_tiny_kernel<T><<<(unsigned)((L.tiny_cnt + kWarps - 1) / kWarps), kThreads, 0, st>>>(
          h->d_lists + L.small_off, (int)L.tiny_cnt, h->dev, front, h->d_vec, h->d_xf);
    if (L.small_cnt > L.tiny_cnt)
      backward_kernel<T><<<(unsigned)(L.small_cnt - L.tiny_cnt), kThreads, 0, st>>>(
          h->d_lists + L.small_off + L.tiny_cnt, h->dev, front, h->d_vec, h->d_xf);
    if (L.narrow_cnt)
      bwd_narrow_kernel<T, D>
          <<<(unsigned)L.narrow_cnt, kThreads, sizeof(double) * (size_t)L.narrow_max_u, st>>>(
              h->d_lists + L.narrow_off, h->dev, front, h->d_vec, h->d_xf);
    if (!L.wide_cnt) continue;
    const int32_t* wide = h->d_lists + L.wide_off;
    const unsigned nf = (unsigned)L.wide_cnt;
    gather_rest_kernel<T, D>
        <<<dim3((unsigned)((L.wide_max_m + kThreads - 1) / kThreads), nf), kThreads, 0, st>>>(
            wide, h->dev, h->d_vec, h->d_xf);
    bwd_rest_kernel<T, D>
        <<<dim3((unsigned)((L.wide_max_k + kWarps - 1) / kWarps), nf), kThreads, 0, st>>>(
            wide, h->dev, front, h->d_y, h->d_vec);
    for (int64_t o0 = (L.wide_max_k - 1) / kInv * kInv; o0 >= 0; o0 -= kInv) {
      const int64_t ob = std::min<int64_t>(kInv, L.wide_max_k - o0);
      bwd_inv_kernel<T, D><<<dim3((unsigned)((ob + 31) / 32), nf), kColThreads, 0, st>>>(
          wide, h->dev, front, o0, h->d_vec, h->d_xf);
      if (o0 > 0)
        bwd_cols_kernel<T, D><<<dim3((unsigned)((o0 + kWarps - 1) / kWarps), nf), kThreads, 0, st>>>(
            wide, h->dev, front, o0, h->d_xf, h->d_vec);
    }
  }
  return cudaGetLastError();
}

cudaError_t enqueue_residual(nla3d_ldlt* h, const double* A, const double* x, const double* b,
                             double* dr = nullptr) {
  const LdltSymbolic& S = h->S;
  const unsigned blocks = (unsigned)((S.n + kRowsPerBlock - 1) / kRowsPerBlock);
  residual_kernel<<<blocks, kThreads, 0, h->stream>>>(S.n, h->d_fptr, h->d_fcol, h->d_fslot, A, x,
                                                     b, h->d_r, h->d_part, dr, h->d_done,
                                                     h->d_norm);
  return cudaGetLastError();
}

}  // namespace

extern "C" {

int nla3d_ldlt_order(int64_t n, const uint32_t* iofeir, const uint32_t* columns,
                     const double* points, int64_t n_dofs, int32_t* order) {
  const std::string msg = ldlt_nd_order(n, iofeir, columns, points, n_dofs, order);
  return msg.empty() ? NLA3D_OK : NLA3D_ERR_ARG;
}

int nla3d_ldlt_analyze(int64_t n, const uint32_t* iofeir, const uint32_t* columns,
                       const int32_t* perm, double* stats, int32_t* perm_out, int32_t* sn_first_out,
                       int64_t* row_ptr_out, int32_t* rows_out) {
  if (!stats) return NLA3D_ERR_ARG;
  LdltSymbolic S;
  const std::string msg = ldlt_analyze(n, iofeir, columns, perm, &S);
  if (!msg.empty()) return NLA3D_ERR_ARG;
  stats[0] = (double)S.n_sn();
  stats[1] = (double)(S.level_ptr.size() - 1);
  stats[2] = (double)S.max_front;
  stats[3] = (double)S.nnz_L;
  stats[4] = S.flops;
  stats[5] = (double)S.front_off.back();
  stats[6] = (double)S.max_children;
  stats[7] = (double)S.rows.size();
  if (perm_out) std::copy(S.perm.begin(), S.perm.end(), perm_out);
  if (sn_first_out) std::copy(S.sn_first.begin(), S.sn_first.end(), sn_first_out);
  if (row_ptr_out) std::copy(S.row_ptr.begin(), S.row_ptr.end(), row_ptr_out);
  if (rows_out) std::copy(S.rows.begin(), S.rows.end(), rows_out);
  return NLA3D_OK;
}

int nla3d_ldlt_create(int64_t n, const uint32_t* iofeir, const uint32_t* columns,
                      const int32_t* perm, int precision, void* stream, nla3d_ldlt** out) {
  if (!out || precision < 0 || precision > 2) return NLA3D_ERR_ARG;
  *out = nullptr;
  nla3d_ldlt* h = new nla3d_ldlt();
  h->tc = precision == 2;
  if (precision == 2) precision = 1;
  h->prec = precision;
  if (precision == 1) h->pivot_rel = 1e-7;
  const std::string msg = ldlt_analyze(n, iofeir, columns, perm, &h->S);
  if (!msg.empty()) {
    delete h;
    return NLA3D_ERR_ARG;
  }
  const LdltSymbolic& S = h->S;
  h->front_entries = S.front_off.back();
  // the schedule: per level, its small and large fronts
  const int64_t ns = S.n_sn();
  const int nlev = (int)S.level_ptr.size() - 1;
  std::vector<int32_t> lists;
  LdltSolveLists solve_lists;
  if (!ldlt_solve_lists(S, &solve_lists).empty()) {
    delete h;
    return NLA3D_ERR_RANGE;
  }
  std::vector<InvTask> inv_tasks;
  std::vector<uint64_t> toff;
  std::vector<ProbeTask> probes;
  std::vector<int32_t> inv_first(ns, 0);
  size_t n_inv = 0;
  int64_t max_probes = 0;
  uint64_t max_work = 0;
  std::vector<uint64_t> wo, lio, pko;
  std::vector<OuterTile> tiles;
  int64_t max_w = 0, max_large_cnt = 0, max_pk = 0;
  uint64_t max_li = 0;
  h->levels.resize(nlev);
  for (int L = 0; L < nlev; L++) {
    auto& lv = h->levels[L];
    lv.small_off = (int64_t)lists.size();
    // up to kTinyPivots pivots first, those of up to kTinyRows rows before the others
    for (int part = 0; part < 3; part++) {
      for (int32_t q = S.level_ptr[L]; q < S.level_ptr[L + 1]; q++) {
        const int32_t s = S.level_list[q];
        const int of = S.k(s) > kTinyPivots ? 2 : S.m(s) > kTinyRows ? 1 : 0;
        if (S.m(s) > kSmallFront || of != part) continue;
        lists.push_back(s);
        if (part) lv.small_max_m = std::max(lv.small_max_m, S.m(s));
      }
      lv.small_cnt = (int64_t)lists.size() - lv.small_off;
      if (part == 0) lv.warp_cnt = lv.small_cnt;
      if (part == 1) lv.tiny_cnt = lv.small_cnt;
    }
    lv.large_off = (int64_t)lists.size();
    lv.wo_off = (int64_t)wo.size();
    int64_t w = 0, pk = 0;
    uint64_t li = 0;
    for (int32_t q = S.level_ptr[L]; q < S.level_ptr[L + 1]; q++) {
      const int32_t s = S.level_list[q];
      if (S.m(s) > kSmallFront) {
        lists.push_back(s);
        wo.push_back((uint64_t)w);
        w += (int64_t)S.m(s) *
             std::min<int64_t>(kOuter, ((int64_t)S.k(s) + kPanel - 1) / kPanel * kPanel);
        lio.push_back(li);
        pko.push_back((uint64_t)pk);
        pk += ((int64_t)S.m(s) + kTcM - 1) / kTcM * (int64_t)kPkBlock;
        li += (uint64_t)((S.k(s) + kPanel - 1) / kPanel) * kPanel * kPanel;
        lv.large_max_m = std::max<int64_t>(lv.large_max_m, S.m(s));
        lv.large_max_k = std::max<int64_t>(lv.large_max_k, S.k(s));
      }
    }
    lv.large_cnt = (int64_t)lists.size() - lv.large_off;
    // the solves: the large fronts by width, and the joins of the wide ones'
    // inverses (narrow ones have no second 64-pivot block)
    lv.vec0 = solve_lists.level_off[L];
    lv.vec1 = solve_lists.level_off[L + 1];
    for (int wide = 0; wide < 2; wide++) {
      (wide ? lv.wide_off : lv.narrow_off) = (int64_t)lists.size();
      for (int64_t z = 0; z < lv.large_cnt; z++) {
        const int32_t s = lists[lv.large_off + z];
        const int64_t m = S.m(s), k = S.k(s);
        if ((k > kNarrow || m > kNarrowRows) != (wide != 0)) continue;
        lists.push_back(s);
        if (wide) {
          lv.wide_max_m = std::max(lv.wide_max_m, m);
          lv.wide_max_k = std::max(lv.wide_max_k, k);
        } else {
          lv.narrow_max_u = std::max(lv.narrow_max_u, m - k);
        }
      }
    }
    lv.narrow_cnt = lv.wide_off - lv.narrow_off;
    lv.wide_cnt = (int64_t)lists.size() - lv.wide_off;
    uint64_t work = 0;
    for (int64_t z = 0; z < lv.large_cnt; z++) {
      const int64_t k = S.k(lists[lv.large_off + z]);
      toff.push_back(work);
      if (k > kPanel) work += (uint64_t)k * (kInv / 2);
    }
    max_work = std::max(max_work, work);
    lv.probe_off = (int64_t)probes.size();
    for (int64_t z = 0; z < lv.large_cnt; z++) {
      const int32_t s = lists[lv.large_off + z];
      const int64_t k = S.k(s);
      inv_first[s] = (int32_t)n_inv;
      n_inv += (size_t)((k + kInv - 1) / kInv);
      for (int64_t j0 = 0; j0 + kPanel < k; j0 += kInv)
        probes.push_back(ProbeTask{(uint32_t)z, (uint32_t)j0});
    }
    lv.probe_cnt = (int64_t)probes.size() - lv.probe_off;
    max_probes = std::max(max_probes, lv.probe_cnt);
    const int bt = precision ? InvTile<float>::BT : InvTile<double>::BT;
    for (int q = 0; q < kDoublings; q++) {
      const int64_t sz = (int64_t)kPanel << q;
      lv.inv_off[q] = (int64_t)inv_tasks.size();
      for (int64_t z = 0; z < lv.large_cnt; z++) {
        const int64_t k = S.k(lists[lv.large_off + z]);
        for (int64_t j0 = 0; j0 + sz < k; j0 += 2 * sz) {
          const int64_t rows = std::min(sz, k - j0 - sz);
          for (int64_t ct = 0; ct * bt < rows; ct++)
            for (int64_t at = 0; at * bt < sz; at++)
              inv_tasks.push_back(InvTask{(uint32_t)z, (uint32_t)j0, (uint32_t)(ct << 16 | at)});
        }
      }
      lv.inv_cnt[q] = (int64_t)inv_tasks.size() - lv.inv_off[q];
    }
    if (h->tc) {
      // every outer block's update tiles (the rule of update_range, outer):
      // per front with k > o0, rows and columns from jb = min(o0 + kOuter, k)
      for (int64_t o0 = 0; o0 < lv.large_max_k; o0 += kOuter) {
        lv.tile_off.push_back((int64_t)tiles.size());
        for (int64_t z = 0; z < lv.large_cnt; z++) {
          const int32_t s = lists[lv.large_off + z];
          const int64_t k = S.k(s), m = S.m(s);
          if (o0 >= k) continue;
          const int64_t jb = std::min<int64_t>(o0 + kOuter, k);
          if (jb >= m) continue;
          const int64_t b0 = (jb - o0) / kTcM, rb = (m - o0 + kTcM - 1) / kTcM;
          for (int64_t ti = b0; ti < rb; ti++)
            for (int64_t tj = b0; tj <= ti; tj++)
              tiles.push_back(OuterTile{(uint32_t)z, (uint32_t)(ti << 16 | tj)});
        }
        lv.tile_cnt.push_back((int64_t)tiles.size() - lv.tile_off.back());
      }
      // every panel's in-block update (update_range, inner): rows from
      // jb = p0 + pb, columns jb .. min(o0 + kOuter, k)
      for (int64_t p0 = 0; p0 < lv.large_max_k; p0 += kPanel) {
        lv.itile_off.push_back((int64_t)tiles.size());
        const int64_t o0 = p0 - p0 % kOuter;
        for (int64_t z = 0; z < lv.large_cnt; z++) {
          const int32_t s = lists[lv.large_off + z];
          const int64_t k = S.k(s), m = S.m(s);
          if (p0 >= k) continue;
          const int64_t jb = p0 + std::min<int64_t>(kPanel, k - p0);
          const int64_t je = std::min<int64_t>(o0 + kOuter, k);
          if (jb >= je) continue;
          const int64_t b0 = (jb - o0) / kTcM, rb = (m - o0 + kTcM - 1) / kTcM;
          const int64_t cb = (je - o0 + kTcN - 1) / kTcN;
          for (int64_t ti = b0; ti < rb; ti++)
            for (int64_t tj = b0; tj <= ti && tj < cb; tj++)
              tiles.push_back(OuterTile{(uint32_t)z, (uint32_t)(ti << 16 | tj)});
        }
        lv.itile_cnt.push_back((int64_t)tiles.size() - lv.itile_off.back());
      }
    }
    max_w = std::max(max_w, w);
    max_li = std::max(max_li, li);
    max_pk = std::max(max_pk, pk);
    max_large_cnt = std::max(max_large_cnt, lv.large_cnt);
    for (int32_t q = S.level_ptr[L]; q < S.level_ptr[L + 1]; q++) {
      const int32_t s = S.level_list[q];
      lv.has_children |= S.child_ptr[s + 1] > S.child_ptr[s];
    }
  }
  if (lists.size() >= (size_t)INT32_MAX || max_large_cnt > 65535) {
    delete h;
    return NLA3D_ERR_RANGE;
  }
  cudaError_t e = cudaSuccess;
  if (stream) {
    h->stream = (cudaStream_t)stream;
  } else {
    e = cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking);
    if (e != cudaSuccess) {
      delete h;
      return NLA3D_ERR_CUDA;
    }
    h->own_stream = true;
  }
  size_t free_b = 0, total_b = 0;
  e = cudaMemGetInfo(&free_b, &total_b);
  const size_t tsize = precision ? sizeof(float) : sizeof(double);
  const double need = (double)h->front_entries * tsize + (double)S.nnz * 8 + (double)S.n * 64 +
                      (double)S.full_col.size() * 8 + (double)S.rows.size() * 8;
  int rc = NLA3D_OK;
  if (e != cudaSuccess)
    rc = cuda_fail(h, e, "cudaMemGetInfo");
  else if (need > 0.9 * (double)free_b)
    rc = fail(h, NLA3D_ERR_NOMEM, "fronts need more device memory than is free");
#define LCK(x)                                  \
  do {                                          \
    if (rc == NLA3D_OK) {                       \
      cudaError_t _e = (x);                     \
      if (_e != cudaSuccess) rc = cuda_fail(h, _e, #x); \
    }                                           \
  } while (0)
  if (precision)
    LCK(dalloc(h, reinterpret_cast<float**>(&h->d_front), h->front_entries));
  else
    LCK(dalloc(h, reinterpret_cast<double**>(&h->d_front), h->front_entries));
  const size_t nlinv = (size_t)max_li;   // the panels of one level read them, nothing later
  if (precision) {
    // (tensor-core fronts keep the panels' operands packed instead)
    LCK(dalloc(h, reinterpret_cast<float**>(&h->d_W), h->tc ? 1 : (size_t)max_w));
    LCK(dalloc(h, reinterpret_cast<float**>(&h->d_Linv), nlinv));
    LCK(cudaFuncSetAttribute(factor_small_kernel<float>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)(sizeof(float) * kSmallFront * (kSmallFront + 1))));
  } else {
    LCK(dalloc(h, reinterpret_cast<double**>(&h->d_W), (size_t)max_w));
    LCK(dalloc(h, reinterpret_cast<double**>(&h->d_Linv), nlinv));
    LCK(cudaFuncSetAttribute(factor_small_kernel<double>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)(sizeof(double) * kSmallFront * (kSmallFront + 1))));
  }
  LCK(upload(h, &h->d_wo, wo));
  LCK(upload(h, &h->d_lio, lio));
  LCK(dalloc(h, &h->d_vec, S.rows.size()));
  LCK(dalloc(h, &h->d_y, S.rows.size()));
  LCK(upload(h, &h->d_bidx, solve_lists.b_idx));
  LCK(upload(h, &h->d_gptr, solve_lists.ptr));
  LCK(upload(h, &h->d_gsrc, solve_lists.src));
  LCK(upload(h, &h->d_rsn, solve_lists.row_sn));
  LCK(upload(h, &h->d_inv, inv_tasks));
  LCK(upload(h, &h->d_toff, toff));
  LCK(upload(h, &h->d_probe, probes));
  LCK(dalloc(h, &h->d_probe_work, (size_t)max_probes * 4 * kInv));
  h->n_inv = n_inv;
  if (precision)
    LCK(dalloc(h, reinterpret_cast<float**>(&h->d_work), (size_t)max_work));
  else
    LCK(dalloc(h, reinterpret_cast<double**>(&h->d_work), (size_t)max_work));
  LCK(cudaStreamCreateWithFlags(&h->side, cudaStreamNonBlocking));
  LCK(cudaEventCreateWithFlags(&h->fork, cudaEventDisableTiming));
  LCK(cudaEventCreateWithFlags(&h->join, cudaEventDisableTiming));
  LCK(cudaStreamCreateWithFlags(&h->ahead, cudaStreamNonBlocking));
  LCK(cudaEventCreateWithFlags(&h->join_ahead, cudaEventDisableTiming));
  LCK(dalloc(h, &h->d_xf, S.n));
  LCK(dalloc(h, &h->d_rhs, S.n));
  LCK(dalloc(h, &h->d_r, S.n));
  LCK(dalloc(h, &h->d_dx, S.n));
  LCK(dalloc(h, &h->d_part, 2 * ((S.n + kRowsPerBlock - 1) / kRowsPerBlock)));
  LCK(dalloc(h, &h->d_norm, 2));
  LCK(dalloc(h, &h->d_done, 1));
  LCK(cudaMemsetAsync(h->d_done, 0, sizeof(unsigned), h->stream));
  LCK(dalloc(h, &h->d_dot, kDotBlocks));
  if (precision) LCK(dalloc(h, &h->d_dirsum, (size_t)kDirBlocks * kDirSums));
  LCK(dalloc(h, &h->d_maxabs, 1));
  LCK(dalloc(h, &h->d_maxpart, kMaxBlocks));
  LCK(dalloc(h, &h->d_perturbed, 2));
  LCK(dalloc(h, &h->d_err, 1));
  LCK(cudaMemsetAsync(h->d_err, 0, sizeof(int), h->stream));
  if (h->tc) {
    LCK(cudaFuncSetAttribute(tc_packed_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)kPkSmem));
    LCK(upload(h, &h->d_pko, pko));
    LCK(dalloc(h, &h->d_pk, (size_t)std::max<int64_t>(max_pk, 1)));
    LCK(upload(h, &h->d_tiles, tiles));
    int dev = 0;
    LCK(cudaGetDevice(&dev));
    LCK(cudaDeviceGetAttribute(&h->n_sm, cudaDevAttrMultiProcessorCount, dev));
  }
  LCK(upload(h, &h->d_adest, S.a_dest));
  LCK(upload(h, &h->d_perm, S.perm));
  LCK(upload(h, &h->d_lists, lists));
  LCK(upload(h, &h->d_fptr, S.full_ptr));
  LCK(upload(h, &h->d_fcol, S.full_col));
  LCK(upload(h, &h->d_fslot, S.full_slot));
  uint64_t *fo = nullptr, *vo = nullptr;
  int64_t *rp = nullptr, *relp = nullptr;
  int32_t *rw = nullptr, *sf = nullptr;
  uint32_t* rl = nullptr;
  int32_t* inv_first_d = nullptr;
  float* inv_error = nullptr;
  LCK(upload(h, &inv_first_d, inv_first));
  LCK(dalloc(h, &inv_error, n_inv));
  LCK(upload(h, &fo, S.front_off));
  LCK(upload(h, &vo, solve_lists.vec_off));
  LCK(upload(h, &rp, S.row_ptr));
  LCK(upload(h, &rw, S.rows));
  LCK(upload(h, &sf, S.sn_first));
  LCK(upload(h, &relp, S.rel_ptr));
  LCK(upload(h, &rl, S.rel));
  if (precision) {
    // the refinement's directions last, of what the rest has left and with the
    // tenth that `need` leaves free: without them the refinement takes plain steps
    size_t left = 0;
    LCK(cudaMemGetInfo(&left, &total_b));
    const double dirs = 8.0 * (2 * kDirs + 1) * (double)S.n;
    if (rc == NLA3D_OK && dirs <= (double)left - 0.1 * (double)free_b &&
        dalloc(h, &h->d_dirs, ((size_t)2 * kDirs + 1) * S.n) != cudaSuccess)
      cudaGetLastError();
  }
  LCK(cudaStreamSynchronize(h->stream));
#undef LCK
  h->dev = LdltDev{fo, vo, rp, rw, sf, relp, rl, inv_first_d, inv_error};
  if (rc != NLA3D_OK) {
    // keep the handle so that the caller can read the message, then destroy it;
    // what it holds so far is never run
    h->d_front = nullptr;
    *out = h;
    return rc;
  }
  *out = h;
  return NLA3D_OK;
}

const char* nla3d_ldlt_last_error(const nla3d_ldlt* h) { return h ? h->err.c_str() : "null handle"; }

int nla3d_ldlt_info(const nla3d_ldlt* h, double* out) {
  if (!h || !out) return NLA3D_ERR_ARG;
  const LdltSymbolic& S = h->S;
  out[0] = (double)S.n_sn();
  out[1] = (double)h->levels.size();
  out[2] = (double)S.max_front;
  out[3] = (double)S.nnz_L;
  out[4] = S.flops;
  out[5] = (double)h->front_entries * (h->prec ? 4.0 : 8.0);
  out[6] = (double)h->perturbed[0];
  out[7] = (double)h->perturbed[1];
  return NLA3D_OK;
}

int nla3d_ldlt_factor(nla3d_ldlt* h, const double* values) {
  if (!h || !values) return fail(h, NLA3D_ERR_ARG, "ldlt_factor: null argument");
  if (!h->d_front) return fail(h, NLA3D_ERR_ARG, "ldlt_factor: the handle was not set up");
  // the factorisation's kernel sequence is captured once per values array
  // into a CUDA graph and replayed
  cudaError_t e = cudaSuccess;
  if (!h->factor_exec || h->factor_graph_values != values) {
    if (h->factor_exec) cudaGraphExecDestroy(h->factor_exec);
    h->factor_exec = nullptr;
    cudaGraph_t g = nullptr;
    e = cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess) {
      const cudaError_t ec = h->prec ? enqueue_factor<float>(h, values)
                                     : enqueue_factor<double>(h, values);
      e = cudaStreamEndCapture(h->stream, &g);
      if (ec != cudaSuccess) e = ec;
      if (e == cudaSuccess) e = cudaGraphInstantiate(&h->factor_exec, g, 0);
      if (g) cudaGraphDestroy(g);
      if (e != cudaSuccess) h->factor_exec = nullptr;
      h->factor_graph_values = values;
    }
  }
  if (e == cudaSuccess) e = cudaGraphLaunch(h->factor_exec, h->stream);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(h->perturbed, h->d_perturbed, 2 * sizeof(int), cudaMemcpyDeviceToHost,
                        h->stream);
  int tc_err = 0;
  if (e == cudaSuccess && h->tc)
    e = cudaMemcpyAsync(&tc_err, h->d_err, sizeof(int), cudaMemcpyDeviceToHost, h->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
  if (e != cudaSuccess) return cuda_fail(h, e, "ldlt_factor");
  if (tc_err) {
    h->factored = false;
    return fail(h, NLA3D_ERR_CUDA, "ldlt_factor: a tensor-core tile timed out waiting for its MMAs");
  }
  h->factored = true;
  if (h->perturbed[1]) return fail(h, NLA3D_ERR_ELEMENT, "ldlt_factor: a non-finite pivot");
  return NLA3D_OK;
}

}  // extern "C"

namespace {

constexpr int kRestart = 30;

unsigned vec_blocks(int64_t n) {
  return (unsigned)std::min<int64_t>((n + kThreads - 1) / kThreads, 152 * 8);
}

// the solve's kernel sequence (a few thousand launches on large models) is
// captured once into a CUDA graph reading d_rhs and leaving the factor-order
// solution in d_xf; each solve copies its right-hand side in, replays the
// graph and scatters (or adds) the result into `out`
cudaError_t enqueue_solve_any(nla3d_ldlt* h, const double* rhs, double* out, int acc,
                              double* z = nullptr) {
  cudaError_t e = cudaSuccess;
  // FP64 fronts have one mode; FP32 fronts: compensated FP32 products, or
  // FP64 ones in the accurate mode
  const bool accurate = h->prec && h->solve_accurate;
  cudaGraphExec_t& exec = accurate ? h->solve_exec_acc : h->solve_exec;
  if (!exec) {
    cudaGraph_t g = nullptr;
    e = cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) return e;
    const cudaError_t ec =
        !h->prec ? enqueue_solve_core<double, Dot<double>>(h, h->d_rhs)
        : accurate ? enqueue_solve_core<float, DotWide>(h, h->d_rhs)
                   : enqueue_solve_core<float, Dot<float>>(h, h->d_rhs);
    e = cudaStreamEndCapture(h->stream, &g);
    if (ec != cudaSuccess) e = ec;
    if (e == cudaSuccess) e = cudaGraphInstantiate(&exec, g, 0);
    if (g) cudaGraphDestroy(g);
    if (e != cudaSuccess) {
      exec = nullptr;
      return e;
    }
  }
  if (rhs != h->d_rhs)
    e = cudaMemcpyAsync(h->d_rhs, rhs, sizeof(double) * h->S.n, cudaMemcpyDeviceToDevice,
                        h->stream);
  if (e == cudaSuccess) e = cudaGraphLaunch(exec, h->stream);
  if (e != cudaSuccess) return e;
  const unsigned nb = (unsigned)((h->S.n + kThreads - 1) / kThreads);
  solve_finish_kernel<<<nb, kThreads, 0, h->stream>>>(h->S.n, h->d_perm, h->d_xf, out, acc,
                                                     z);
  return cudaGetLastError();
}

// <a, b> with a fixed reduction order (per-block partial sums, summed on the host)
cudaError_t dot(nla3d_ldlt* h, const double* a, const double* b, double* out) {
  double part[kDotBlocks];
  dot_kernel<<<kDotBlocks, kThreads, 0, h->stream>>>(h->S.n, a, b, h->d_dot);
  cudaError_t e = cudaMemcpyAsync(part, h->d_dot, sizeof(part), cudaMemcpyDeviceToHost, h->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
  double acc = 0.0;
  for (int q = 0; q < kDotBlocks; q++) acc += part[q];
  *out = acc;
  return e;
}

// ||b - A x|| and ||b|| (the residual kernel leaves b - A x in d_r)
cudaError_t residual_norms(nla3d_ldlt* h, const double* values, const double* x, const double* b,
                           double* rnorm, double* bnorm, double* dr = nullptr) {
  double sums[2] = {0.0, 0.0};
  cudaError_t e = enqueue_residual(h, values, x, b, dr);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(sums, h->d_norm, sizeof(sums), cudaMemcpyDeviceToHost, h->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
  *rnorm = std::sqrt(sums[0]);
  *bnorm = std::sqrt(sums[1]);
  return e;
}

// the correction after step k: x and d_r corrected; rnorm: ||r|| after it
cudaError_t direction_step(nla3d_ldlt* h, int k, double* x, double* rnorm) {
  const int64_t n = h->S.n;
  double *Q = h->d_dirs, *Z = Q + (size_t)kDirs * n;
  direction_sums_kernel<<<dim3(kDirBlocks, (unsigned)std::max(1, (k + kDirChunk - 1) / kDirChunk)),
                          kThreads, 0, h->stream>>>(n, k, Q, h->d_r, h->d_dirsum);
  direction_step_kernel<<<kDirBlocks, kThreads, 0, h->stream>>>(n, k, Q, Z, h->d_r, x, h->d_dirsum,
                                                               h->d_dot);
  if (!rnorm) return cudaGetLastError();
  double part[kDirBlocks];
  cudaError_t e = cudaMemcpyAsync(part, h->d_dot, sizeof(part), cudaMemcpyDeviceToHost, h->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
  double rr = 0.0;
  for (int q = 0; q < kDirBlocks; q++) rr += part[q];
  *rnorm = std::sqrt(rr);
  return e;
}

// Right-preconditioned restarted GMRES with the factor as the preconditioner
// (GMRES-based iterative refinement), modified Gram-Schmidt, Givens rotations;
// x is improved in place until ||b - A x|| <= tol ||b|| or `budget`
// preconditioner applications are spent.
cudaError_t gmres_refine(nla3d_ldlt* h, const double* values, const double* b, double* x,
                         double tol, int budget, int* apps, double* rel) {
  const LdltSymbolic& S = h->S;
  const int64_t n = S.n;
  cudaStream_t st = h->stream;
  cudaError_t e = cudaSuccess;
  static_assert(2 * kDirs >= kRestart + 1, "the refinement's directions hold the basis");
  if (!h->d_V && h->d_dirs) h->d_V = h->d_dirs;   // done with when this is called
  if (!h->d_V) {
    e = dalloc(h, &h->d_V, (size_t)(kRestart + 1) * n);
    if (e != cudaSuccess) return e;
  }
  const unsigned vb = vec_blocks(n);
  const unsigned mb = (unsigned)((n + kRowsPerBlock - 1) / kRowsPerBlock);
  double rnorm = 0.0, bnorm = 0.0;
  while (true) {
    e = residual_norms(h, values, x, b, &rnorm, &bnorm);
    if (e != cudaSuccess) return e;
    const double scale = bnorm > 0.0 ? bnorm : 1.0;
    *rel = rnorm / scale;
    if (!(*rel > tol) || *apps >= budget) return cudaSuccess;
    double H[kRestart + 1][kRestart] = {};
    double cs[kRestart] = {}, sn[kRestart] = {}, g[kRestart + 1] = {};
    g[0] = rnorm;
    scale_kernel<<<vb, kThreads, 0, st>>>(n, 1.0 / rnorm, h->d_r, h->d_V);
    int j = 0;
    for (; j < kRestart && *apps < budget; j++) {
      double* vj = h->d_V + (size_t)j * n;
      double* w = h->d_V + (size_t)(j + 1) * n;
      e = enqueue_solve_any(h, vj, h->d_dx, 0);   // z = M^-1 v_j
      (*apps)++;
      if (e != cudaSuccess) return e;
      spmv_kernel<<<mb, kThreads, 0, st>>>(n, h->d_fptr, h->d_fcol, h->d_fslot, values, h->d_dx, w);
      for (int i = 0; i <= j; i++) {
        double hij = 0.0;
        e = dot(h, w, h->d_V + (size_t)i * n, &hij);
        if (e != cudaSuccess) return e;
        H[i][j] = hij;
        axpy_kernel<<<vb, kThreads, 0, st>>>(n, -hij, h->d_V + (size_t)i * n, w);
      }
      double ww = 0.0;
      e = dot(h, w, w, &ww);
      if (e != cudaSuccess) return e;
      const double hn = std::sqrt(ww);
      H[j + 1][j] = hn;
      if (hn > 0.0) scale_kernel<<<vb, kThreads, 0, st>>>(n, 1.0 / hn, w, w);
      for (int i = 0; i < j; i++) {
        const double t = cs[i] * H[i][j] + sn[i] * H[i + 1][j];
        H[i + 1][j] = -sn[i] * H[i][j] + cs[i] * H[i + 1][j];
        H[i][j] = t;
      }
      const double a = H[j][j], c = H[j + 1][j];
      const double rho = std::sqrt(a * a + c * c);
      cs[j] = rho > 0.0 ? a / rho : 1.0;
      sn[j] = rho > 0.0 ? c / rho : 0.0;
      H[j][j] = rho;
      H[j + 1][j] = 0.0;
      g[j + 1] = -sn[j] * g[j];
      g[j] = cs[j] * g[j];
      if (std::fabs(g[j + 1]) <= 0.5 * tol * scale || hn == 0.0) {
        j++;
        break;
      }
    }
    // y = H^-1 g, t = V y, x += M^-1 t
    double y[kRestart] = {};
    for (int i = j - 1; i >= 0; i--) {
      double acc = g[i];
      for (int q = i + 1; q < j; q++) acc -= H[i][q] * y[q];
      y[i] = H[i][i] != 0.0 ? acc / H[i][i] : 0.0;
    }
    e = cudaMemsetAsync(h->d_r, 0, sizeof(double) * n, st);
    if (e != cudaSuccess) return e;
    for (int i = 0; i < j; i++)
      axpy_kernel<<<vb, kThreads, 0, st>>>(n, y[i], h->d_V + (size_t)i * n, h->d_r);
    e = enqueue_solve_any(h, h->d_r, x, 1);
    (*apps)++;
    if (e != cudaSuccess) return e;
  }
}

}  // namespace

extern "C" {

int nla3d_ldlt_solve(nla3d_ldlt* h, const double* values, const double* b, double* x,
                     int max_refine, double tol, int* steps, double* rel_residual) {
  if (!h || !values || !b || !x || max_refine < 0)
    return fail(h, NLA3D_ERR_ARG, "ldlt_solve: bad argument");
  if (!h->factored) return fail(h, NLA3D_ERR_ARG, "ldlt_solve: factor first");
  h->solve_accurate = 0;
  cudaError_t e = enqueue_solve_any(h, b, x, 0);
  double rel = 0.0, prev = 0.0, rnorm = 0.0, bnorm = 0.0;
  int it = 0, dirs = 0;
  const size_t n = (size_t)h->S.n;
  if (e == cudaSuccess) e = residual_norms(h, values, x, b, &rnorm, &bnorm);
  if (e != cudaSuccess) return cuda_fail(h, e, "ldlt_solve");
  // Refinement steps.  Plain ones (FP64 fronts) while they converge fast;
  // accelerated ones (FP32 fronts) from the second on, until kDirs are kept,
  // at any rate: they take the least residual over the Krylov space as GMRES
  // does, but x from the steps themselves, so that an inexact factor costs
  // rate and not accuracy, and one application a step instead of FP64 products
  // and one more for x (a 457k-equation bar whose elimination grows: 22 steps in
  // 117 ms, against 27 in 259).  Without a better x for kStalled of them the
  // residual is at its floor or the factor no help.  They apply the factor with
  // the compensated FP32 products (2^-48 per operation): on the same factors FP64
  // products took the same steps to the same residual in each of 1,050 Newton
  // solves of bars of 139k to 1.07M equations, at twice the time a step.
  // GMRES with the same factor after, its preconditioner applied with FP64
  // products.  rel is that of b - A x computed afresh, except between a step's
  // correction and the next.
  const double scale = bnorm > 0.0 ? bnorm : 1.0;
  // the best x of accelerated steps: past the attainable residual their
  // directions are rounding errors
  double* best_x = h->d_dirs ? h->d_dirs + (size_t)2 * kDirs * n : nullptr;
  double best = 0.0;
  int stalled = 0;
  auto restore = [&] {
    if (dirs == 0 || !(rel > best)) return cudaSuccess;
    rel = best;
    return cudaMemcpyAsync(x, best_x, sizeof(double) * n, cudaMemcpyDeviceToDevice, h->stream);
  };
  for (;;) {
    rel = rnorm / scale;
    if (!(rel > tol)) break;
    if (dirs > 0) {
      stalled = dirs == 1 || rel < 0.9 * best ? 0 : stalled + 1;
      if (dirs == 1 || rel < best) {
        best = rel;
        e = cudaMemcpyAsync(best_x, x, sizeof(double) * n, cudaMemcpyDeviceToDevice, h->stream);
        if (e != cudaSuccess) return cuda_fail(h, e, "ldlt_solve");
      }
    }
    if (it >= max_refine) {
      // the copy has ended when the call returns, as on every other way out:
      // the caller may read x on a stream of its own
      e = restore();
      if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
      if (e != cudaSuccess) return cuda_fail(h, e, "ldlt_solve");
      break;
    }
    if (dirs > 0) {
      // the norm after the correction is read only where it can matter
      const bool read = rel < 1e4 * tol;
      e = direction_step(h, dirs - 1, x, read ? &rnorm : nullptr);
      if (e != cudaSuccess) return cuda_fail(h, e, "ldlt_solve");
      if (read && !(rnorm / scale > tol)) {
        e = residual_norms(h, values, x, b, &rnorm, &bnorm);
        if (e != cudaSuccess) return cuda_fail(h, e, "ldlt_solve");
        rel = rnorm / scale;
        if (!(rel > tol)) break;
      }
    }
    // (a plain step that cut less, but whose rate reaches tol with one more, is
    // still cheaper than GMRES, which takes two applications at least)
    if (it > 0 && (dirs > 0 ? dirs == kDirs || stalled == kStalled
                            : !(rel < 0.1 * prev) && !(rel < prev && rel * (rel / prev) <= tol))) {
      h->solve_accurate = 1;
      e = restore();
      if (e == cudaSuccess) e = gmres_refine(h, values, b, x, tol, max_refine, &it, &rel);
      if (e != cudaSuccess) return cuda_fail(h, e, "ldlt_solve (GMRES)");
      break;
    }
    prev = rel;
    // x += A^-1 r with the same factors
    double* q = h->d_dirs ? h->d_dirs + (size_t)dirs * n : nullptr;
    e = enqueue_solve_any(h, h->d_r, x, 1, q ? q + (size_t)kDirs * n : nullptr);
    if (e == cudaSuccess) e = residual_norms(h, values, x, b, &rnorm, &bnorm, q);
    if (e != cudaSuccess) return cuda_fail(h, e, "ldlt_solve");
    if (q) dirs++;
    it++;
  }
  if (steps) *steps = it;
  if (rel_residual) *rel_residual = rel;
  if (!(rel <= tol)) return fail(h, NLA3D_ERR_RANGE, "ldlt_solve: refinement did not reach tol");
  return NLA3D_OK;
}

int nla3d_ldlt_solve_host(nla3d_ldlt* h, const double* values, const double* b_host,
                          double* x_host, int max_refine, double tol, int* steps,
                          double* rel_residual) {
  if (!h || !values || !b_host || !x_host) return fail(h, NLA3D_ERR_ARG, "ldlt_solve_host: bad argument");
  const size_t n = (size_t)h->S.n;
  cudaError_t e = cudaSuccess;
  if (!h->d_hb) e = dalloc(h, &h->d_hb, n);
  if (e == cudaSuccess && !h->d_hx) e = dalloc(h, &h->d_hx, n);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(h->d_hb, b_host, sizeof(double) * n, cudaMemcpyHostToDevice, h->stream);
  if (e != cudaSuccess) return cuda_fail(h, e, "ldlt_solve_host");
  const int rc = nla3d_ldlt_solve(h, values, h->d_hb, h->d_hx, max_refine, tol, steps, rel_residual);
  if (rc != NLA3D_OK && rc != NLA3D_ERR_RANGE) return rc;
  // the refined x also when tol was not reached (the caller reads the residual)
  e = cudaMemcpyAsync(x_host, h->d_hx, sizeof(double) * n, cudaMemcpyDeviceToHost, h->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
  if (e != cudaSuccess) return cuda_fail(h, e, "ldlt_solve_host");
  return rc;
}

int nla3d_ldlt_tc_check(int m, double* out) {
  // one front of m rows whose first kb pivots (one outer block: 256 when
  // m > 512, else 64) are done: the update of rows / columns kb .. m-1 by the
  // FMA kernel and by the tensor cores (operands packed, then bulk-copied by
  // the persistent kernel) from the same random data; out[0] = max
  // |difference|, out[1] = max |update|
  if (m < kPanel + 1 || m > 4096 || !out) return NLA3D_ERR_ARG;
  const int kb = m > 2 * kOuter ? kOuter : kPanel;
  const size_t mm = (size_t)m * m, mw = (size_t)m * kb;
  std::vector<float> F0(mm), W(mw);
  uint64_t x = 88172645463325252ull;   // xorshift, fixed seed
  auto rnd = [&]() {
    x ^= x << 13;
    x ^= x >> 7;
    x ^= x << 17;
    return (float)((double)(x >> 11) / 9007199254740992.0 * 2.0 - 1.0);
  };
  for (auto& v : F0) v = rnd();
  for (auto& v : W) v = rnd();
  std::vector<void*> allocs;
  auto dal = [&](void** p, size_t bytes) {
    cudaError_t e = cudaMalloc(p, bytes);
    if (e == cudaSuccess) allocs.push_back(*p);
    return e;
  };
  float *F1 = nullptr, *F3 = nullptr, *dW = nullptr, *dP = nullptr;
  const size_t mp = (size_t)((m + kTcM - 1) / kTcM) * kPkBlock;
  std::vector<OuterTile> tl;   // the outer update's tiles, as the factorisation lists them
  const int rbk = (m + kTcM - 1) / kTcM, b0 = kb / kTcM;
  for (int ti = b0; ti < rbk; ti++)
    for (int tj = b0; tj <= ti; tj++) tl.push_back(OuterTile{0u, (uint32_t)(ti << 16 | tj)});
  // the operands as the panel kernel packs them (hi: to nearest, ties away)
  std::vector<float> P(mp, 0.0f);
  auto hi = [](float v) {
    uint32_t u;
    std::memcpy(&u, &v, 4);
    u = (u + 0x1000u) & 0xFFFFE000u;
    std::memcpy(&v, &u, 4);
    return v;
  };
  for (int i = 0; i < m; i++)
    for (int c = 0; c < kb; c++) {
      float* t = P.data() + ((size_t)(i / kTcM) * kPkChunks + c / kTcKH) * 4 * kPkTile +
                 (((i % kTcM) >> 3) * (kTcKH / 4) + ((c % kTcKH) >> 2)) * 32 + (i & 7) * 4 + (c & 3);
      const float l = F0[(size_t)i + (size_t)c * m], w = W[(size_t)i + (size_t)c * m];
      t[0] = hi(l);
      t[kPkTile] = l - t[0];
      t[2 * kPkTile] = hi(w);
      t[3 * kPkTile] = w - t[2 * kPkTile];
    }
  OuterTile* dT = nullptr;
  int n_sm = 1, dev = 0;
  int* err = nullptr;
  int32_t* list = nullptr;
  uint64_t *woff = nullptr, *foff = nullptr;
  int64_t* rowp = nullptr;
  int32_t* snf = nullptr;
  cudaError_t e = dal((void**)&F1, mm * 4);
  if (e == cudaSuccess) e = dal((void**)&F3, mm * 4);
  if (e == cudaSuccess) e = dal((void**)&dP, mp * 4);
  if (e == cudaSuccess) e = dal((void**)&dT, tl.size() * sizeof(OuterTile));
  if (e == cudaSuccess)
    e = cudaMemcpy(dT, tl.data(), tl.size() * sizeof(OuterTile), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess) e = dal((void**)&dW, mw * 4);
  if (e == cudaSuccess) e = dal((void**)&err, 4);
  if (e == cudaSuccess) e = dal((void**)&list, 4);
  if (e == cudaSuccess) e = dal((void**)&woff, 8);
  if (e == cudaSuccess) e = dal((void**)&foff, 16);
  if (e == cudaSuccess) e = dal((void**)&rowp, 16);
  if (e == cudaSuccess) e = dal((void**)&snf, 8);
  const int32_t zero32 = 0;
  const uint64_t zero64[2] = {0, (uint64_t)mm};
  const int64_t rp[2] = {0, m};
  const int32_t sf[2] = {0, kb};
  if (e == cudaSuccess) e = cudaMemcpy(F1, F0.data(), mm * 4, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(F3, F0.data(), mm * 4, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(dW, W.data(), mw * 4, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemset(err, 0, 4);
  if (e == cudaSuccess) e = cudaMemcpy(list, &zero32, 4, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(woff, zero64, 8, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(foff, zero64, 16, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(rowp, rp, 16, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(snf, sf, 8, cudaMemcpyHostToDevice);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(tc_packed_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)kPkSmem);
  int tc_err = 0;
  if (e == cudaSuccess) {
    LdltDev d{};
    d.front_off = foff;
    d.row_ptr = rowp;
    d.sn_first = snf;
    const BigBatch bb{list, woff, woff, woff};
    const int64_t rest = m - kb;
    const unsigned t128 = (unsigned)((rest + 127) / 128);
    batched_trailing_kernel<float, 128, 8><<<dim3(t128, t128, 1), kThreads>>>(bb, d, F1, 0, 1,
                                                                               dW, 0, 0);
    e = cudaMemcpy(dP, P.data(), mp * 4, cudaMemcpyHostToDevice);
    tc_packed_kernel<<<(unsigned)std::min<int>((int)tl.size(), n_sm), kOuterThreads, kPkSmem>>>(
        bb, d, F3, 0, 1, dP, dT, (int)tl.size(), err, 0);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e == cudaSuccess) e = cudaMemcpy(&tc_err, err, 4, cudaMemcpyDeviceToHost);
  }
  std::vector<float> R1(mm), R3(mm);
  if (e == cudaSuccess) e = cudaMemcpy(R1.data(), F1, mm * 4, cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) e = cudaMemcpy(R3.data(), F3, mm * 4, cudaMemcpyDeviceToHost);
  for (void* p : allocs) cudaFree(p);
  if (e != cudaSuccess) return NLA3D_ERR_CUDA;
  if (tc_err) return NLA3D_ERR_RANGE;
  double dmax = 0.0, umax = 0.0;
  for (int j = kb; j < m; j++)
    for (int i = j; i < m; i++) {
      const size_t q = (size_t)i + (size_t)j * m;
      dmax = std::max(dmax, (double)std::fabs(R1[q] - R3[q]));
      umax = std::max(umax, (double)std::fabs(R1[q] - F0[q]));
    }
  out[0] = dmax;
  out[1] = umax;
  return NLA3D_OK;
}

int nla3d_ldlt_destroy(nla3d_ldlt* h) {
  if (!h) return NLA3D_OK;
  // a borrowed stream may already be gone: only an owned one is synchronised
  // (cudaFree waits for the device anyway)
  if (h->own_stream && h->stream) cudaStreamSynchronize(h->stream);
  if (h->factor_exec) cudaGraphExecDestroy(h->factor_exec);
  if (h->solve_exec) cudaGraphExecDestroy(h->solve_exec);
  if (h->solve_exec_acc) cudaGraphExecDestroy(h->solve_exec_acc);
  if (h->fork) cudaEventDestroy(h->fork);
  if (h->join) cudaEventDestroy(h->join);
  if (h->side) cudaStreamDestroy(h->side);
  if (h->join_ahead) cudaEventDestroy(h->join_ahead);
  if (h->ahead) cudaStreamDestroy(h->ahead);
  for (void* p : h->allocs) cudaFree(p);
  if (h->own_stream && h->stream) cudaStreamDestroy(h->stream);
  delete h;
  cudaGetLastError();   // leave no error of this teardown to the next caller
  return NLA3D_OK;
}

}  // extern "C"
