// Complex element types (ComplexF32, ComplexF64) for the plain path: the
// diagonal-block solve and multiply, the off-diagonal update and the alpha
// scaling that the recursion of unified_rec (src/rectrxm.jl:101-198) calls.
//
// The reference's unified_rec is restricted to real element types
// (src/rectrxm.jl:101), though its base-case docstrings list complex ones
// (src/trsm.jl:180-183).  These kernels run the same recursion on complex
// data: trans 'T' reads A transposed, 'C' reads its conjugate transpose (the
// Adjoint wrapper), and the arithmetic is ordinary complex arithmetic
// (nla_cplx.cuh).  Diagonal blocks run on the strip kernel of the real types
// (nla_leaf_strip.cuh).
//
// Values are interleaved (re, im) pairs, column-major, as Julia and torch
// store them.
#include <mutex>

#include "nla_common.cuh"
#include "nla_cplx.cuh"

namespace nla {
namespace cx {

// C (N x M) += alpha * op(A) (N x K) * op(B) (K x M), alpha real (+-1 in
// the recursion).  64 x 64 tiles, 256 threads, each a 4 x 4 register tile;
// K in chunks of 16 staged in shared memory; conjugation applied as the
// operands are staged.
constexpr int GK = 16;
template <typename R, int GT>
__global__ void __launch_bounds__(256) cplx_gemm_kernel(int64_t N, int64_t M, int64_t K, R alpha, const cpx<R>* A,
                                                        int64_t lda, int tA, int cA, const cpx<R>* B, int64_t ldb,
                                                        int tB, int cB, cpx<R>* C, int64_t ldc) {
  chain_begin();
  __shared__ cpx<R> As[GK][GT + 1], Bs[GK][GT + 1];
  const int t = threadIdx.x, tr = t % 16, tc = t / 16;
  const int64_t i0 = (int64_t)blockIdx.x * GT, j0 = (int64_t)blockIdx.y * GT;
  constexpr int RT = GT / 16;  // rows and columns per thread
  cpx<R> acc[RT][RT];
#pragma unroll
  for (int a = 0; a < RT; ++a)
#pragma unroll
    for (int b = 0; b < RT; ++b) acc[a][b] = zero<R>();
  for (int64_t k0 = 0; k0 < K; k0 += GK) {
    for (int idx = t; idx < GK * GT; idx += 256) {
      // op(A)(i, k): threads along i for a plain view, along k for a transposed one.
      int i, k;
      if (!tA) { i = idx % GT; k = idx / GT; }
      else { k = idx % GK; i = idx / GK; }
      const int64_t gi = i0 + i, gk = k0 + k;
      As[k][i] = gi < N && gk < K ? conj_if(A[mat_off(gi, gk, lda, tA)], cA != 0) : zero<R>();
      int j, kb;
      if (!tB) { kb = idx % GK; j = idx / GK; }
      else { j = idx % GT; kb = idx / GT; }
      const int64_t gj = j0 + j, gkb = k0 + kb;
      Bs[kb][j] = gj < M && gkb < K ? conj_if(B[mat_off(gkb, gj, ldb, tB)], cB != 0) : zero<R>();
    }
    __syncthreads();
#pragma unroll 4
    for (int k = 0; k < GK; ++k) {
      cpx<R> av[RT], bv[RT];
#pragma unroll
      for (int a = 0; a < RT; ++a) av[a] = As[k][tr + 16 * a];
#pragma unroll
      for (int b = 0; b < RT; ++b) bv[b] = Bs[k][tc + 16 * b];
#pragma unroll
      for (int a = 0; a < RT; ++a)
#pragma unroll
        for (int b = 0; b < RT; ++b) acc[a][b] = fma_c(av[a], bv[b], acc[a][b]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int a = 0; a < RT; ++a) {
    const int64_t i = i0 + tr + 16 * a;
    if (i >= N) continue;
#pragma unroll
    for (int b = 0; b < RT; ++b) {
      const int64_t j = j0 + tc + 16 * b;
      if (j >= M) continue;
      cpx<R>* p = C + i + j * ldc;
      const cpx<R> c = *p;
      *p = mk(fma(alpha, acc[a][b].re, c.re), fma(alpha, acc[a][b].im, c.im));
    }
  }
}

// B .= alpha .* B with the product formed in ComplexF64 and rounded to the
// element type (src/rectrxm.jl:64, :72).
template <typename R>
__global__ void cplx_scale_kernel(int64_t rows, int64_t cols, double are, double aim, cpx<R>* B, int64_t ldb, int tB) {
  const int64_t total = rows * cols;
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    int64_t i, j;
    if (!tB) { i = idx % rows; j = idx / rows; }
    else { j = idx % cols; i = idx / cols; }
    cpx<R>* p = B + mat_off(i, j, ldb, tB);
    const double br = (double)p->re, bi = (double)p->im;
    *p = mk((R)(are * br - aim * bi), (R)(are * bi + aim * br));
  }
}

}  // namespace cx

bool is_complex(int dtype) { return dtype == NLA_C32 || dtype == NLA_C64; }

constexpr int64_t CPLX_LEAF_MAX = 128;  // rows of a complex diagonal block

int launch_leaf_complex(char func, char side, char uplo, int dtype, int64_t n, int64_t m, const Mat& A, const Mat& B,
                        cudaStream_t s, bool unit) {
  if (n <= 0 || m <= 0) return NLA_OK;
  if (n > 1024) return fail(NLA_ERR_ARG, "diag block: n must be <= 1024");
  if (B.t) return fail(NLA_ERR_UNSUPPORTED, "diag block: transposed B view");
  if (n > CPLX_LEAF_MAX) {
    // A larger block (the reference's 256-row solve leaves, or a direct
    // nla_diag_block call) runs the recursion itself down to blocks that fit.
    RecPlan c{func, side, uplo, dtype, m, CPLX_LEAF_MAX, s, GEMM_PLAIN, 1, false};
    c.unit = unit;
    return recurse(c, A, n, B);
  }
  return launch_leaf_strips_complex(func, side, uplo, dtype, n, m, A, B, s, unit);
}

int launch_gemm_complex(int dtype, int64_t N, int64_t M, int64_t K, double alpha, const Mat& A, const Mat& B,
                        const Mat& C, cudaStream_t s) {
  if (N <= 0 || M <= 0) return NLA_OK;
  if (C.t) return fail(NLA_ERR_UNSUPPORTED, "gemm: transposed output view");
  // Tiles as in the real update: 64 x 64, or 32 x 32 where that divides the
  // output more evenly over the SMs (measured for ComplexF32 1000 x 128 x 128,
  // 32 against 128 CTAs).
  const int64_t sms = num_sms();
  auto tiles = [&](int64_t t) { return ((N + t - 1) / t) * ((M + t - 1) / t); };
  const int64_t w64 = (tiles(64) + sms - 1) / sms * (64 * 64), w32 = (tiles(32) + sms - 1) / sms * (32 * 32 * 3 / 2);
  const int gt = w32 < w64 && M <= 65535 * 32ll ? 32 : 64;
  const int64_t gx = (N + gt - 1) / gt, gy = (M + gt - 1) / gt;
  if (gx > 2147483647LL || gy > 65535) return fail(NLA_ERR_UNSUPPORTED, "gemm: matrix too large for one launch");
  const size_t es = dtype == NLA_C64 ? 16 : 8;
  TraceScope trace(NLA_K_GEMM_SIMT, s, 8.0 * (double)N * (double)M * (double)K,
                   (double)es * ((double)N * K + (double)K * M + 2.0 * (double)N * M));
  const dim3 grid((unsigned)gx, (unsigned)gy);
  auto run = [&](auto kernel, auto one) {
    using R = decltype(one);
    kernel<<<grid, 256, 0, s>>>(N, M, K, (R)alpha, static_cast<const cx::cpx<R>*>(A.p), A.ld, A.t, A.c,
                                static_cast<const cx::cpx<R>*>(B.p), B.ld, B.t, B.c, static_cast<cx::cpx<R>*>(C.p),
                                C.ld);
  };
  if (dtype == NLA_C64) gt == 64 ? run(cx::cplx_gemm_kernel<double, 64>, 1.0) : run(cx::cplx_gemm_kernel<double, 32>, 1.0);
  else gt == 64 ? run(cx::cplx_gemm_kernel<float, 64>, 1.0f) : run(cx::cplx_gemm_kernel<float, 32>, 1.0f);
  NLA_CHECK_LAUNCH("cplx_gemm_kernel");
  return NLA_OK;
}

int launch_scale_complex(int dtype, int64_t rows, int64_t cols, double alpha_re, double alpha_im, const Mat& B,
                         cudaStream_t s) {
  if (rows <= 0 || cols <= 0 || (alpha_re == 1.0 && alpha_im == 0.0)) return NLA_OK;
  const int64_t total = rows * cols;
  int64_t blocks = (total + 255) / 256;
  const int64_t cap = (int64_t)num_sms() * 8;
  if (blocks > cap) blocks = cap;
  TraceScope trace(NLA_K_SCALE, s, 6.0 * (double)total, 2.0 * (double)total * (double)dtype_size(dtype));
  if (dtype == NLA_C64)
    cx::cplx_scale_kernel<double><<<(unsigned)blocks, 256, 0, s>>>(rows, cols, alpha_re, alpha_im,
                                                                    static_cast<cx::cpx<double>*>(B.p), B.ld, B.t);
  else
    cx::cplx_scale_kernel<float><<<(unsigned)blocks, 256, 0, s>>>(rows, cols, alpha_re, alpha_im,
                                                                   static_cast<cx::cpx<float>*>(B.p), B.ld, B.t);
  NLA_CHECK_LAUNCH("cplx_scale_kernel");
  return NLA_OK;
}

}  // namespace nla
