// Base cases of the recursion on one diagonal block (n <= 1024):
//   func 'S': the triangular solve of LeftLowerTRSM! ... RightUpperTRSM!
//             (src/trsm.jl:5-150);
//   func 'M': the triangular multiply of LeftLowerTRMM! ... RightUpperTRMM!
//             (src/trmm.jl:43-389).
// The canonical-form mapping and the column-per-thread Float64 solve are in
// nla_leaf.cuh, the strip kernel that runs every other block in
// nla_leaf_strip.cuh.
#include <algorithm>
#include <cstdlib>
#include <mutex>
#include <type_traits>

#include "nla_leaf.cuh"
#include "nla_leaf_strip.cuh"

namespace nla {
namespace {

using namespace leafdev;

template <int HALVES, int CW>
__global__ void __launch_bounds__(CW * HALVES, 1) leaf_solve_cols_kernel(LeafArgs g) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int64_t c0 = (int64_t)blockIdx.x * CW;
  const int ncols = (int)(g.m - c0 < CW ? g.m - c0 : CW);
  solve_cols_f64<HALVES, CW>(g, c0, ncols, smem_raw, 1.0);
}

// Threads per right-hand side of the Float64 column-per-thread leaf:
// NLA_LEAF_COLS = 0 (use the strip kernel), 1 or 2 (default 2).
int leaf_cols_mode() {
  static const int mode = [] {
    const char* v = getenv("NLA_LEAF_COLS");
    if (v && (v[0] == '0' || v[0] == '1' || v[0] == '2') && v[1] == 0) return v[0] - '0';
    return 2;
  }();
  return mode;
}

template <int HALVES, int CW>
int launch_leaf_cols(const LeafArgs& g, cudaStream_t s) {
  const size_t smem = leaf_cols_smem_elems(g.n, HALVES, CW) * sizeof(double);
  const int64_t grid = (g.m + CW - 1) / CW;
  if (g.n > COLS_MAX_N || smem > 200 * 1024) return fail(NLA_ERR_UNSUPPORTED, "leaf: shared memory plan too large");
  if (grid > 2147483647LL) return fail(NLA_ERR_UNSUPPORTED, "leaf: too many right-hand sides");
  static std::once_flag once;
  static cudaError_t st = cudaSuccess;
  std::call_once(once, [] {
    st = cudaFuncSetAttribute(leaf_solve_cols_kernel<HALVES, CW>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              200 * 1024);
  });
  if (st != cudaSuccess) return cuda_status(st, "cudaFuncSetAttribute(leaf_solve_cols_kernel)");
  TraceScope trace(NLA_K_LEAF_SOLVE, s, (double)g.n * g.n * (double)g.m,
                   8.0 * ((double)g.n * (g.n + 1) / 2 + 2.0 * (double)g.n * g.m));
  leaf_solve_cols_kernel<HALVES, CW><<<(unsigned)grid, CW * HALVES, smem, s>>>(g);
  NLA_CHECK_LAUNCH("leaf_solve_cols_kernel");
  return NLA_OK;
}

// Right-hand sides per CTA of the two-threads-per-column leaf: the fewest of
// 128, 112, 96 and 64 that keep every CTA in one wave of one CTA per SM
// (NLA_LEAF_CW forces one of them).
int leaf_cols_width(int64_t m) {
  const char* v = getenv("NLA_LEAF_CW");  // read per launch, so tests can pin each width
  const int forced = v ? atoi(v) : 0;
  if (forced == 128 || forced == 112 || forced == 96 || forced == 64 || forced == 56) return forced;
  const int64_t sms = num_sms();
  for (int cw : {64, 96, 112})
    if ((m + cw - 1) / cw <= sms) return cw;
  return 128;
}

int launch_leaf_cols2(const LeafArgs& g, cudaStream_t s) {
  switch (leaf_cols_width(g.m)) {
    case 56: return launch_leaf_cols<2, 56>(g, s);
    case 64: return launch_leaf_cols<2, 64>(g, s);
    case 96: return launch_leaf_cols<2, 96>(g, s);
    case 112: return launch_leaf_cols<2, 112>(g, s);
    default: return launch_leaf_cols<2, 128>(g, s);
  }
}

template <typename T, int PB, int NC, int WC, bool SOLVE, int NW = 8>
__global__ void __launch_bounds__(32 * NW) leaf_strip_kernel(const LeafArgs g) {
  chain_begin();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  strip_block<T, PB, NC, WC, NW, SOLVE>(g, smem_raw);
}

constexpr size_t STRIP_SMEM_MAX = 200 * 1024;

template <typename T, int PB, int NC, int WC, bool SOLVE, int NW = 8>
int launch_strip(const LeafArgs& g, cudaStream_t s) {
  using Tc = typename Elem<T>::compute;
  const size_t smem = strip_smem_elems<Tc>(g.n, PB, NC, WC, NW) * sizeof(Tc);
  constexpr int CW = 32 / PB * NC * WC;
  const int64_t grid = (g.m + CW - 1) / CW;
  if (grid > 2147483647LL) return fail(NLA_ERR_UNSUPPORTED, "leaf: too many right-hand sides");
  if (smem > STRIP_SMEM_MAX) return fail(NLA_ERR_UNSUPPORTED, "leaf: shared memory plan too large");
  static std::once_flag once;
  static cudaError_t st = cudaSuccess;
  std::call_once(once, [] {
    st = cudaFuncSetAttribute(leaf_strip_kernel<T, PB, NC, WC, SOLVE, NW>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)STRIP_SMEM_MAX);
  });
  if (st != cudaSuccess) return cuda_status(st, "cudaFuncSetAttribute(leaf_strip_kernel)");
  // n^2 m flops per solve or multiply (the benchmark's convention); bytes:
  // the triangle once plus B read and written.
  TraceScope trace(SOLVE ? NLA_K_LEAF_SOLVE : NLA_K_LEAF_MULT, s, (double)g.n * g.n * (double)g.m,
                   (double)sizeof(T) * ((double)g.n * (g.n + 1) / 2 + 2.0 * (double)g.n * g.m));
  leaf_strip_kernel<T, PB, NC, WC, SOLVE, NW><<<(unsigned)grid, 32 * NW, smem, s>>>(g);
  NLA_CHECK_LAUNCH("leaf_strip_kernel");
  return NLA_OK;
}

// Blocks of few rows with very many right-hand sides: one right-hand side per
// thread, its column in shared memory, four rows at a time in registers.  Every
// FMA is one of the triangle's (a strip's lanes each form a whole panel, which
// for few rows is mostly wasted), and rows are formed with k increasing.
constexpr int COL_T = 64;  // right-hand sides and threads per CTA
constexpr int COL_P = COL_T + 1;
// The block in packed rows of four: L(i, k), k <= i | 3, at col_at(i, k).
__host__ __device__ constexpr int col_at(int i, int k) { return 8 * (i >> 2) * ((i >> 2) + 1) + 4 * k + (i & 3); }
constexpr size_t column_smem_elems(int n) {
  const int nr = (n + 3) & ~3;
  return (size_t)col_at(nr, 0) + (size_t)nr * COL_P + 2 * nr;  // the block, X, the diagonal, its reciprocals
}

template <typename T, bool SOLVE>
__global__ void __launch_bounds__(COL_T) leaf_column_kernel(const LeafArgs g) {
  using Tc = typename Elem<T>::compute;
  using Vec = typename StripTraits<Tc>::Vec;
  using Mx = StripMath<Tc>;
  constexpr int VK = StripTraits<Tc>::VK;
  chain_begin();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int n = g.n, nr = (n + 3) & ~3, t = threadIdx.x;
  Tc* L = reinterpret_cast<Tc*>(smem_raw);
  Tc* X = L + col_at(nr, 0);  // X(i, c) at X[i COL_P + c]
  Tc* dia = X + nr * COL_P;
  Tc* inv = dia + nr;
  const int64_t c0 = (int64_t)blockIdx.x * COL_T;
  const int ncols = (int)(g.m - c0 < COL_T ? g.m - c0 : COL_T);
  const int64_t sk = (g.tA ? 1 : g.lda) * (g.rev ? -1 : 1), si = (g.tA ? g.lda : 1) * (g.rev ? -1 : 1);
  const T* A = static_cast<const T*>(g.A) + (g.rev ? (int64_t)(n - 1) * (g.lda + 1) : 0);
  const int64_t bi = (g.tB ? g.ldb : 1) * (g.rev ? -1 : 1), bc = g.tB ? 1 : g.ldb;
  T* B = static_cast<T*>(g.B) + (g.rev ? (int64_t)(n - 1) * (g.tB ? g.ldb : 1) : 0) + c0 * bc;

  for (int idx = t; idx < nr * nr; idx += COL_T) {
    const int i = g.tA ? idx / nr : idx % nr, k = g.tA ? idx % nr : idx / nr;
    if (k <= (i | 3)) L[col_at(i, k)] = i < n && k < i ? Mx::conj_if(Elem<T>::load(A + i * si + k * sk), g.cj) : Mx::zero();
  }
  for (int i = t; i < nr; i += COL_T) {
    const Tc d = g.unit || i >= n ? Mx::one() : Mx::conj_if(Elem<T>::load(A + i * (si + sk)), g.cj);
    dia[i] = d;
    inv[i] = Mx::inverse(d);
  }
  // B along its contiguous index, eight loads in flight per thread.
  constexpr int BATCH = 8;
  auto at = [&](int idx, int& i, int& c) { g.tB ? (i = idx / COL_T, c = idx % COL_T) : (c = idx / nr, i = idx % nr); };
  for (int i0 = t; i0 < nr * COL_T; i0 += COL_T * BATCH) {
    T v[BATCH];
#pragma unroll
    for (int u = 0; u < BATCH; ++u) {
      int i, c;
      at(i0 + COL_T * u, i, c);
      v[u] = i < n && c < ncols ? B[i * bi + c * bc] : raw_zero<T>();
    }
#pragma unroll
    for (int u = 0; u < BATCH; ++u) {
      int i, c;
      at(i0 + COL_T * u, i, c);
      if (i0 + COL_T * u < nr * COL_T) X[i * COL_P + c] = Elem<T>::load(&v[u]);
    }
  }
  __syncthreads();
  Tc* x = X + t;
  for (int b = 0; b < nr; b += 4) {
    const int r0 = SOLVE ? b : nr - 4 - b;
    Tc z[4], y[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      y[i] = x[(r0 + i) * COL_P];
      z[i] = Mx::zero();
    }
#pragma unroll 4
    for (int k = 0; k < r0; ++k) {
      Tc l[4];
#pragma unroll
      for (int i = 0; i < 4; i += VK) st_unpack(*reinterpret_cast<const Vec*>(L + col_at(r0, k) + i), l + i);
      const Tc xk = x[k * COL_P];
#pragma unroll
      for (int i = 0; i < 4; ++i) z[i] = Mx::fma_(l[i], xk, z[i]);
    }
    // The sum from zero and then subtracted: chained onto b it would round at
    // b's size at every step (Float32 error of 50 rows 1.29e-7 against 1.0e-7).
    if (SOLVE) {
#pragma unroll
      for (int i = 0; i < 4; ++i) z[i] = y[i] - z[i];
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (SOLVE) y[j] = Mx::divided(z[j], inv[r0 + j], dia[r0 + j]);
#pragma unroll
      for (int i = j + 1; i < 4; ++i) {
        const Tc l = L[col_at(r0 + i, r0 + j)];
        z[i] = SOLVE ? Mx::fms_(l, y[j], z[i]) : Mx::fma_(l, y[j], z[i]);
      }
      x[(r0 + j) * COL_P] = SOLVE ? y[j] : Mx::fma_(dia[r0 + j], y[j], z[j]);
    }
  }
  __syncthreads();
  for (int idx = t; idx < nr * COL_T; idx += COL_T) {
    int i, c;
    at(idx, i, c);
    if (i < n && c < ncols) Elem<T>::store(B + i * bi + c * bc, X[i * COL_P + c]);
  }
}

template <typename T, bool SOLVE>
int launch_column(const LeafArgs& g, cudaStream_t s) {
  using Tc = typename Elem<T>::compute;
  const size_t smem = column_smem_elems(g.n) * sizeof(Tc);
  const int64_t grid = (g.m + COL_T - 1) / COL_T;
  if (grid > 2147483647LL) return fail(NLA_ERR_UNSUPPORTED, "leaf: too many right-hand sides");
  static std::once_flag once;
  static cudaError_t st = cudaSuccess;
  std::call_once(once, [] {
    st = cudaFuncSetAttribute(leaf_column_kernel<T, SOLVE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)STRIP_SMEM_MAX);
  });
  if (st != cudaSuccess) return cuda_status(st, "cudaFuncSetAttribute(leaf_column_kernel)");
  TraceScope trace(SOLVE ? NLA_K_LEAF_SOLVE : NLA_K_LEAF_MULT, s, (double)g.n * g.n * (double)g.m,
                   (double)sizeof(T) * ((double)g.n * (g.n + 1) / 2 + 2.0 * (double)g.n * g.m));
  leaf_column_kernel<T, SOLVE><<<(unsigned)grid, COL_T, smem, s>>>(g);
  NLA_CHECK_LAUNCH("leaf_column_kernel");
  return NLA_OK;
}

// Right-hand sides per SM from which a block of n rows is faster one column
// per thread: a CTA of columns takes its time whether or not the others are
// there, until they fill the SMs, while strips' time grows with their number.
// Blocks of more rows stay on strips, whose products reuse A.  Measured on 152
// SMs, strips against columns, us (solve): Float64 n = 16 28 / 24 at m = 6000,
// 137 / 45 at 100000, n = 48 65 / 73 at 8000, 84 / 73 at 12000; Float32 n = 32
// 22 / 26 at 8000, 33 / 26 at 20000, 71 / 34 at 100000; ComplexF32 n = 32
// 37 / 41 at 12000, 163 / 73 at 100000; ComplexF64 n = 16 56 / 76 at 4000,
// 83 / 77 at 6000, 900 / 278 at 100000, n = 64 502 / 483 at 12000, 4114 / 2666
// at 100000.
template <typename Tc, bool SOLVE>
int64_t column_from(int64_t n) {
  constexpr bool CX = !std::is_floating_point<Tc>::value;
  constexpr bool F64 = sizeof(Tc) == (CX ? 16 : 8);
  const int64_t never = INT32_MAX;
  if (CX && F64) return SOLVE ? (n <= 64 ? 14 + n : never) : n <= 56 ? 40 + n * 5 / 4 : never;
  if (CX) return n > 56 ? never : SOLVE ? std::min<int64_t>(5 + 3 * n, 105) : std::min<int64_t>(35 + n * 3 / 2, 85);
  if (F64) return SOLVE ? (n <= 64 ? 22 + n * 15 / 16 : never) : n <= 32 ? 30 + 3 * n : never;
  return n > 56 ? never : SOLVE ? 45 + n * 3 / 2 : 75 + n * 9 / 8;
}

// Right-hand sides per CTA: the width with the least ceil(CTAs / SMs) *
// (width + c), where c is a strip's fixed time (the triangles' chains and
// the staging of A) in columns' worth of its product: about one column in
// Float64, whose product is bound by the DFMA pipe, and about 32 in Float32.
// Float64 solves of 4 and 2 columns count as 6 and 5, for their 32-row
// triangles (n = 128, m = 3000: 4, 8 and 16 columns 139, 117 and 112 us, n = 64
// in ComplexF64 271, 189 and 209).
// Float64 takes 16-row panels from 8 columns on (32-row triangles cost the
// DFMA pipe more than the steps they save), Float32 always 32-row panels.
// Measured against one warp-group CTA per 16 or 32 columns with 32-row
// panels solved by one warp: Float64 96 x 24 97 -> 13 us, 256 x 256 560 ->
// 54 us; Float32 256 x 8192 110 -> 44 us; Float16 256 x 4096 98 -> 32 us;
// Float64 multiply 64 x 6144 115 -> 36 us.
template <typename T, bool SOLVE>
int launch_strips(const LeafArgs& g, cudaStream_t s) {
  using Tc = typename Elem<T>::compute;
  constexpr bool CX = !std::is_floating_point<Tc>::value;
  constexpr bool F64 = sizeof(Tc) == (CX ? 16 : 8);
  constexpr int WIDEST = F64 ? (CX ? 16 : 32) : (CX ? 32 : 64);
  const int64_t sms = num_sms(), c = F64 ? 1 : CX ? 8 : 32;
  if (g.m > sms * column_from<Tc, SOLVE>(g.n)) return launch_column<T, SOLVE>(g, s);
  // Warps on 32 and 64 columns.  Float32 products wait for shared memory with
  // two warps per scheduler; a second K group gives it four (and costs one
  // sum through shared memory per panel): solve 256 x 8192 47.9 -> 44.4 us,
  // multiply 128 x 8192 16.3 -> 14.3 us (15.2 since multiplies stop at
  // the diagonal), 64 x 6144 8.4 -> 7.3 us.  On 8 and
  // 16 columns, where the triangles' chains bound, it gave nothing (25.2 us
  // at 256 x 1000 either way).
  constexpr int NWW = CX || F64 ? 8 : 16;
  int best = 0;
  int64_t cost = 0;
  for (int w : {64, 32, 16, 8, 4, 2}) {
    if (w > WIDEST) continue;
    if (strip_smem_elems<Tc>(g.n, 32, w < 8 ? 1 : w / 8, w < 8 ? w : 8, w < 32 ? 8 : NWW) * sizeof(Tc) > STRIP_SMEM_MAX && w > 2) continue;
    const int eff = F64 && SOLVE && w < 8 ? w / 2 + 4 : w;
    const int64_t grid = (g.m + w - 1) / w, k = (grid + sms - 1) / sms * (eff + c);
    if (best == 0 || k < cost) best = w, cost = k;
  }
  switch (best) {
    case 64:
      if constexpr (WIDEST >= 64) return launch_strip<T, 32, 8, 8, SOLVE, NWW>(g, s);
    case 32:
      if constexpr (WIDEST >= 32)
        return F64 ? launch_strip<T, 16, 2, 8, SOLVE>(g, s) : launch_strip<T, 32, 4, 8, SOLVE, NWW>(g, s);
    case 16: return F64 ? launch_strip<T, 16, 1, 8, SOLVE>(g, s) : launch_strip<T, 32, 2, 8, SOLVE>(g, s);
    case 8: return F64 ? launch_strip<T, 16, 1, 4, SOLVE>(g, s) : launch_strip<T, 32, 1, 8, SOLVE>(g, s);
    case 4: return launch_strip<T, 32, 1, 4, SOLVE>(g, s);
    default: return launch_strip<T, 32, 1, 2, SOLVE>(g, s);
  }
}

// The canonical form of a diagonal block (side R as side L on transposed
// views, uplo U as lower with the index order reversed).
LeafArgs leaf_args(char side, char uplo, int64_t n, int64_t m, const Mat& A, const Mat& B, bool unit) {
  LeafArgs g;
  g.A = A.p;
  g.lda = A.ld;
  g.tA = A.t;
  g.B = B.p;
  g.ldb = B.ld;
  g.tB = 0;
  g.unit = unit ? 1 : 0;
  g.cj = A.c;
  g.n = (int)n;
  g.m = m;
  if (side == 'R') {  // X op(A) = B  <=>  op(A)^T X^T = B^T
    g.tA = !g.tA;
    g.tB = 1;
    uplo = uplo == 'L' ? 'U' : 'L';
  }
  g.rev = uplo == 'U';
  return g;
}

}  // namespace

int launch_leaf_strips_complex(char func, char side, char uplo, int dtype, int64_t n, int64_t m, const Mat& A,
                               const Mat& B, cudaStream_t s, bool unit) {
  const LeafArgs g = leaf_args(side, uplo, n, m, A, B, unit);
  if (dtype == NLA_C64)
    return func == 'S' ? launch_strips<cx::cpx<double>, true>(g, s) : launch_strips<cx::cpx<double>, false>(g, s);
  return func == 'S' ? launch_strips<cx::cpx<float>, true>(g, s) : launch_strips<cx::cpx<float>, false>(g, s);
}

int launch_leaf(char func, char side, char uplo, int dtype, int64_t n, int64_t m, const Mat& A, const Mat& B,
                cudaStream_t s, bool unit) {
  if (is_complex(dtype)) return launch_leaf_complex(func, side, uplo, dtype, n, m, A, B, s, unit);
  if (n <= 0 || m <= 0) return NLA_OK;
  if (n > 1024) return fail(NLA_ERR_ARG, "diag block: n must be <= 1024");
  if (B.t) return fail(NLA_ERR_UNSUPPORTED, "diag block: transposed B view");
  const LeafArgs g = leaf_args(side, uplo, n, m, A, B, unit);
  if (func == 'S') {
    // Float64 blocks of 49 to 128 rows where one wave of wide CTAs fits and
    // strips of 32 columns would leave the last wave short: one right-hand
    // side per thread, or two threads per right-hand side; from 113 rows also
    // where several waves are three quarters full.  Measured at n = 64 (128)
    // on 152 SMs, strips against columns, us: m = 8192 88 (219) against 86
    // (229), 12000 111 (300) against 92 (265), 16000 144 (391) against 98 (290),
    // 20000 162 (484) against 187 (617), 30000 235 (675) against 188 (616),
    // 100000 662 (1961) against 534 (1822); at 64 rows the kernel of one thread
    // per right-hand side and 64 to a CTA takes the last two (168 and 480).
    // (NLA_LEAF_COLS=0 turns it off, NLA_LEAF_CW pins a width from m = 1024.)
    const int64_t sms = num_sms(), wave = 128 * sms, waves = (m + wave - 1) / wave;
    const bool pinned = m >= 8 * LEAF_THREADS && getenv("NLA_LEAF_CW") != nullptr;
    const bool full = waves == 1 ? n > 48 && m > 68 * sms : n > 112 && 4 * m > 3 * wave * waves;
    if (dtype == NLA_F64 && n <= COLS_MAX_N && (full || pinned) && leaf_cols_mode() != 0)
      return leaf_cols_mode() == 1 ? launch_leaf_cols<1, LEAF_THREADS>(g, s) : launch_leaf_cols2(g, s);
  }
  const bool S = func == 'S';
  switch (dtype) {
    case NLA_F64: return S ? launch_strips<double, true>(g, s) : launch_strips<double, false>(g, s);
    case NLA_F32: return S ? launch_strips<float, true>(g, s) : launch_strips<float, false>(g, s);
    case NLA_F16: return S ? launch_strips<__half, true>(g, s) : launch_strips<__half, false>(g, s);
    default: return fail(NLA_ERR_DTYPE, "diag block: unknown dtype");
  }
}

}  // namespace nla
