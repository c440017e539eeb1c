// Diagonal-block solve / multiply building blocks of the base-case kernels
// (nla_leaf.cu).
//
// All eight (func, side, uplo) forms map onto one canonical problem, a
// LOWER triangle applied from the LEFT:
//   side 'R' becomes side 'L' on transposed operands (X op(A) = B  <=>
//   op(A)^T X^T = B^T), which flips uplo;
//   uplo 'U' becomes lower by reversing the index order of the block
//   (i -> n-1-i on rows and columns of A and on the rows of B).
// Both are pure index maps, so no data is copied.
//
// Here: the index maps and the Float64 solve with one right-hand side per
// thread (many right-hand sides, blocks of at most 128 rows).  Everything
// else runs on strips (nla_leaf_strip.cuh).  Float16 blocks are computed in
// Float32 and rounded once when stored.
#pragma once

#include "nla_common.cuh"

namespace nla {
namespace leafdev {

constexpr int LEAF_THREADS = 128;
constexpr int PANEL = 32;

struct LeafArgs {
  const void* A;
  int64_t lda;
  int tA;
  void* B;
  int64_t ldb;
  int tB;
  int rev;
  int unit;  // unit diagonal: the diagonal of A is taken as 1 and not read
  int cj;    // complex types: read the conjugates of A's elements
  int n;
  int64_t m;
};

template <typename T>
__device__ __forceinline__ int64_t a_off(const LeafArgs& g, int i, int j) {
  int mi = g.rev ? g.n - 1 - i : i, mj = g.rev ? g.n - 1 - j : j;
  return mat_off(mi, mj, g.lda, g.tA);
}

template <typename T>
__device__ __forceinline__ int64_t b_off(const LeafArgs& g, int i, int64_t c) {
  int mi = g.rev ? g.n - 1 - i : i;
  return mat_off(mi, c, g.ldb, g.tB);
}

// Float64 solve with one right-hand side per thread, for n <= COLS_MAX_N and
// CW columns per CTA.  GB300 issues FP64 at two fused multiply-adds per clock
// per SM, and measured time is proportional to the FP64 warp instructions an
// SM issues, whichever sub-partitions issue them (8 warps of independent FMA
// chains take 8/7 of the time of 7).  So a solve over m columns is fastest
// with the fewest columns per CTA that still fit one CTA per SM: 112 for
// m = 16384 (147 CTAs) instead of 128 (128 CTAs, 24 SMs idle).
//
// The kernel works left-looking over 32-row panels.  Each thread keeps its
// panel's 32 values in registers, y, and does two steps:
//   1. Subtract the already solved rows of its column,
//      y -= A[p0:p0+32, 0:p0] x[0:p0]. These are 32 independent FMA chains.
//   2. Solve the panel's triangle column by column, so that y_i gets its
//      update as soon as x_j is known.
// Each thread does n(n-1)/2 FMAs in total. The A rows of the panel are staged
// once per panel in shared memory and read as warp-wide broadcasts. X stays in
// shared memory, one column per thread, so accesses are conflict-free.
constexpr int COLS_MAX_N = 128;
constexpr int LOAD_BATCH = 16;  // loads in flight per thread (one CTA per SM)

// HALVES = 2 runs two threads per right-hand side (256 per CTA): the halves
// split the already-solved rows of each panel's update, so that every SM
// sub-partition has two warps issuing FMAs in that phase; half 1 hands its
// partial sums over through shared memory and half 0 solves the triangle.
__host__ __device__ constexpr size_t leaf_cols_smem_elems(int n, int halves, int cw = LEAF_THREADS) {
  return (size_t)n * cw + (size_t)PANEL * COLS_MAX_N + (size_t)n + (halves > 1 ? (size_t)PANEL * cw : 0);
}

template <int HALVES, int CW>
__device__ __forceinline__ void solve_cols_f64(const LeafArgs& g, int64_t c0, int ncols, unsigned char* smem_raw,
                                               double alpha) {
  static_assert(CW % 8 == 0 && CW <= LEAF_THREADS, "right-hand sides per CTA");
  constexpr int NT = CW * HALVES;  // threads per CTA
  const int n = g.n;
  double* X = reinterpret_cast<double*>(smem_raw);  // n x CW
  double* L = X + (size_t)n * CW;                   // PANEL x COLS_MAX_N: rows p0.., columns 0..
  double* inv_d = L + PANEL * COLS_MAX_N;           // n
  double* Y1 = inv_d + n;                           // PANEL x CW partial sums of half 1
  const double* A = static_cast<const double*>(g.A);
  const double* Bp = static_cast<const double*>(g.B);
  const int t = threadIdx.x, c = t % CW, h = t / CW;

  // Block of B (times alpha), LOAD_BATCH loads in flight per thread.
  const int total = n * CW;
  for (int base = t; base < total; base += NT * LOAD_BATCH) {
    double v[LOAD_BATCH];
#pragma unroll
    for (int u = 0; u < LOAD_BATCH; ++u) {
      const int idx = base + u * NT;
      int i, cc;
      if (!g.tB) { i = idx % n; cc = idx / n; }
      else { cc = idx % CW; i = idx / CW; }
      v[u] = idx < total && cc < ncols ? alpha * Bp[b_off<double>(g, i, c0 + cc)] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < LOAD_BATCH; ++u) {
      const int idx = base + u * NT;
      int i, cc;
      if (!g.tB) { i = idx % n; cc = idx / n; }
      else { cc = idx % CW; i = idx / CW; }
      if (idx < total) X[i * CW + cc] = v[u];
    }
  }
  for (int i = t; i < n; i += NT) inv_d[i] = g.unit ? 1.0 : 1.0 / A[a_off<double>(g, i, i)];
  for (int p0 = 0; p0 < n; p0 += PANEL) {
    const int pw = min(PANEL, n - p0);
    // Columns of A staged for the panel's rows: through the diagonal, rounded
    // up to even for the paired loads (the extra column is zero).
    const int kw = (p0 + pw + 1) & ~1;
    __syncthreads();  // previous panel done with L and Y1 (and X, inv_d ready)
    // Stage A[p0 + i][k], i < PANEL, k < kw; zero on and above the diagonal
    // and below the block.  Threads run along the index contiguous in memory.
    for (int base = t; base < PANEL * kw; base += NT * LOAD_BATCH) {
      double v[LOAD_BATCH];
#pragma unroll
      for (int u = 0; u < LOAD_BATCH; ++u) {
        const int idx = base + u * NT;
        int i, k;
        if (!g.tA) { i = idx % PANEL; k = idx / PANEL; }
        else { k = idx % kw; i = idx / kw; }
        v[u] = idx < PANEL * kw && i < pw && k < p0 + i ? A[a_off<double>(g, p0 + i, k)] : 0.0;
      }
#pragma unroll
      for (int u = 0; u < LOAD_BATCH; ++u) {
        const int idx = base + u * NT;
        int i, k;
        if (!g.tA) { i = idx % PANEL; k = idx / PANEL; }
        else { k = idx % kw; i = idx / kw; }
        if (idx < PANEL * kw) L[i * COLS_MAX_N + k] = v[u];
      }
    }
    __syncthreads();
    double y[PANEL];
#pragma unroll
    for (int i = 0; i < PANEL; ++i) y[i] = h == 0 && i < pw ? X[(p0 + i) * CW + c] : 0.0;
    // Already-solved rows: half h takes k in [h p0 / HALVES, (h+1) p0 / HALVES)
    // (p0 is a multiple of 32, so both ranges have even bounds).  Two k per
    // step with one 16-byte broadcast load of A per row; the two FMAs into
    // each y[i] of a step are PANEL instructions apart.
    const int ka = h * (p0 / HALVES), kb = (h + 1) * (p0 / HALVES);
    for (int k = ka; k < kb; k += 2) {
      const double xk0 = X[k * CW + c], xk1 = X[(k + 1) * CW + c];
      double2 a[PANEL];
#pragma unroll
      for (int i = 0; i < PANEL; ++i) a[i] = *reinterpret_cast<const double2*>(&L[i * COLS_MAX_N + k]);
#pragma unroll
      for (int i = 0; i < PANEL; ++i) y[i] = fma(-a[i].x, xk0, y[i]);
#pragma unroll
      for (int i = 0; i < PANEL; ++i) y[i] = fma(-a[i].y, xk1, y[i]);
    }
    if constexpr (HALVES > 1) {
      if (h == 1) {
#pragma unroll
        for (int i = 0; i < PANEL; ++i) Y1[i * CW + c] = y[i];
      }
      __syncthreads();
      if (h == 0) {
#pragma unroll
        for (int i = 0; i < PANEL; ++i) y[i] += Y1[i * CW + c];
      }
    }
    if (h == 0) {
      if (pw == PANEL) {
        // Full panel: the triangle two columns at a time (x_j, then x_{j+1},
        // then one paired load and two FMAs for each row below).
#pragma unroll
        for (int jj = 0; jj < PANEL / 2; ++jj) {
          const int j = 2 * jj;
          const double xj = y[j] * inv_d[p0 + j];
          const double xj1 = fma(-L[(j + 1) * COLS_MAX_N + p0 + j], xj, y[j + 1]) * inv_d[p0 + j + 1];
          y[j] = xj;
          y[j + 1] = xj1;
#pragma unroll
          for (int i = j + 2; i < PANEL; ++i) {
            const double2 a = *reinterpret_cast<const double2*>(&L[i * COLS_MAX_N + p0 + j]);
            y[i] = fma(-a.x, xj, y[i]);
            y[i] = fma(-a.y, xj1, y[i]);
          }
        }
      } else {
#pragma unroll
        for (int j = 0; j < PANEL; ++j) {
          if (j < pw) {
            const double xj = y[j] * inv_d[p0 + j];
            y[j] = xj;
#pragma unroll
            for (int i = j + 1; i < PANEL; ++i) y[i] = fma(-L[i * COLS_MAX_N + p0 + j], xj, y[i]);
          }
        }
      }
#pragma unroll
      for (int i = 0; i < PANEL; ++i)
        if (i < pw) X[(p0 + i) * CW + c] = y[i];
    }
  }
  __syncthreads();
  double* Bo = static_cast<double*>(g.B);
  for (int idx = t; idx < total; idx += NT) {
    int i, cc;
    if (!g.tB) { i = idx % n; cc = idx / n; }
    else { cc = idx % CW; i = idx / CW; }
    if (cc < ncols) Bo[b_off<double>(g, i, c0 + cc)] = X[i * CW + cc];
  }
}

}  // namespace leafdev
}  // namespace nla
