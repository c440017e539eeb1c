// Base cases of the recursion on one diagonal block (n <= 1024):
//   func 'S': the triangular solve of LeftLowerTRSM! ... RightUpperTRSM!
//             (src/trsm.jl:5-150);
//   func 'M': the triangular multiply of LeftLowerTRMM! ... RightUpperTRMM!
//             (src/trmm.jl:43-389).
// The canonical-form mapping and the column-per-thread Float64 solve are in
// nla_leaf.cuh, the strip kernel that runs every other block in
// nla_leaf_strip.cuh.
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

// Right-hand sides per CTA: the width with the least ceil(CTAs / SMs) *
// (width + c), where c is a strip's fixed time (the triangles' chains and
// the staging of A) in columns' worth of its product: about one column in
// Float64, whose product is bound by the DFMA pipe, and about 32 in Float32.
// Float64 takes 16-row panels from 8 columns on (32-row triangles cost the
// DFMA pipe more than the steps they save), Float32 always 32-row panels.
// Measured against one warp-group CTA per 16 or 32 columns with 32-row
// panels solved by one warp: Float64 96 x 24 97 -> 13 us, 256 x 256 560 ->
// 42 us; Float32 256 x 8192 110 -> 44 us; Float16 256 x 4096 98 -> 32 us;
// Float64 multiply 64 x 6144 115 -> 36 us.
template <typename T, bool SOLVE>
int launch_strips(const LeafArgs& g, cudaStream_t s) {
  using Tc = typename Elem<T>::compute;
  constexpr bool CX = !std::is_floating_point<Tc>::value;
  constexpr bool F64 = sizeof(Tc) == (CX ? 16 : 8);
  constexpr int WIDEST = F64 ? (CX ? 16 : 32) : (CX ? 32 : 64);
  const int64_t sms = num_sms(), c = F64 ? 1 : CX ? 8 : 32;
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
    const int64_t grid = (g.m + w - 1) / w, k = (grid + sms - 1) / sms * (w + c);
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
    // Float64 blocks of up to 128 rows where one wave of wide CTAs fits and
    // strips of 32 columns would leave the last wave short: one right-hand
    // side per thread, or two threads per right-hand side.  Measured at
    // n = 64 (128) on 152 SMs, strips against columns: m = 8192 58 (174)
    // against 70 (214) us, 14336 73 (235) against 78 (250), 16384 97 (315)
    // against 83 (276), 20000 116 (383) against 174 (600).
    // (NLA_LEAF_COLS=0 turns it off, NLA_LEAF_CW pins a width from m = 1024.)
    const int64_t sms = num_sms();
    const bool pinned = getenv("NLA_LEAF_CW") != nullptr && m >= 8 * LEAF_THREADS;
    if (dtype == NLA_F64 && n <= COLS_MAX_N && ((m > 96 * sms && m <= 128 * sms) || pinned) && leaf_cols_mode() != 0)
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
