// Float32 off-diagonal update on the tensor cores (tcgen05):
//   C (M x N) += alpha * op(A) (M x K) * op(B) (K x N)
// in tiles of 128 rows and 128, 64 or 32 columns.
//
// Each Float32 value is the sum of three BF16 values, x = h + m + l exactly
// (24 bits of significand as 8 + 8 + 8, each rounded to nearest; the split
// into BF16 terms is that of Henry, Tang and Heinecke, "Leveraging the
// bfloat16 artificial intelligence datatype for higher-precision
// computations", ARITH 2019).  Unlike the scaled integer slices of the
// Float64 update, the terms carry their own exponents, so small elements of
// a row keep their full precision (down to 2^-100, see careful()).  Of the nine products the six of weight
// up to 2^-16 are formed (h h; h m, m h; m m, h l, l h); the three left out
// are below 2^-26 of |a||b| each, under the rounding of one Float32 FMA.
//
// Tensor-core accumulators do not round to nearest (their sums are biased
// towards zero), so no sum stays in them for long: chunks of 64 values of K
// are accumulated in TMEM (h h in one accumulator, the five smaller products
// in another), and the drain warps add each chunk to Float32 registers with
// ordinary rounded additions.  That leaves fewer roundings per element than
// the FMA chain of the CUDA-core update, whose error grows with K.
//
// ComplexF32 updates are the same product on real views: the complex C is
// a real matrix of 2 M rows (re, im interleaved), op(B) one of 2 K rows, and
// op(A) is staged as 2 M x 2 K, each a as the block (re, -im; im, re).
//
// What bounds it: shared memory (per 64 values of K and 128 x 128 outputs the
// six products read 176 KiB of operands from it, and TMA writes 96 KiB;
// stages of 32 values of K were slower, fewer drains hardly faster):
// 1190 TFLOP/s of executed products, 199 of the
// update's, at 4096 x 4096 x 8192 (FFMA update: 39.9).  Warps: 0 loads A, 1 issues MMAs, 2 loads B,
// 3-10 drain (two TMEM buffers of 256 columns) and update C.
//
// Rows of A and columns of B that hold Inf or NaN, or values so small or
// large that low terms or sums would leave Float32's normal range, are
// marked when they are staged; a tile with outputs that they touch forms
// those outputs from the original operands by a tiled loop of FMAs after its
// products (plain_tile), or instead of them when that is all of its outputs.
#include <cudaTypedefs.h>

#include <mutex>

#include "nla_common.cuh"
#include "nla_umma.cuh"

namespace nla {
namespace {

constexpr int BM = 128, BN = 128, BK = 64;
constexpr int TILE_BYTES = BM * BK * 2;
constexpr int SL = 3;
constexpr int F32_THREADS = 352;
// Tiles of 128 rows and TN (128, 64 or 32) columns: two or three stages.
constexpr int f32_stages(int TN) { return TN == 128 ? 2 : 3; }
constexpr int f32_stage_bytes(int TN) { return SL * (BM + TN) * BK * 2; }
constexpr int f32_smem(int TN) { return f32_stages(TN) * f32_stage_bytes(TN) + 1024 + 256; }
static_assert(f32_smem(128) + 1056 <= 232448 && f32_smem(64) + 1056 <= 232448, "shared memory above the per-block limit");

// Row marks: 0 for a row of zeros, else the largest exponent field plus one
// (1 .. 256, 256 for Inf and NaN), so that the row's largest value lies in
// [2^(mark - 128), 2^(mark - 127)); MARK_TINY more when the row holds a
// nonzero value below 2^-100, whose low terms would be subnormal.  An output
// is left to the plain product when its row or column is not finite or has
// such a value, or when the largest products leave [2^-90, 2^106] (their low
// terms, or sums of up to 2^20 of them, would leave the normal range).
constexpr int MARK_LOW = 28, MARK_TINY = 512;  // the mark of 2^-100
__device__ __forceinline__ bool careful(int ma, int mb) {
  if (ma >= 256 || mb >= 256) return true;
  if (ma == 0 || mb == 0) return false;
  return ma + mb < 166 || ma + mb > 360;
}

struct F32Params {
  int M, N, K;
  int num_kb;
  int tiles_m, tiles_n;
  const float* A;  // element (i, k) at A[i * asi + k * ask]
  int64_t asi, ask;
  const float* B;  // element (k, j) at B[k * bsk + j * bsj]
  int64_t bsk, bsj;
  const int* mark_a;  // per 64-wide block of K and row: the block's mark at [kb * rows_pad + row]
  const int* mark_b;
  int rows_a, rows_b;  // padded
  float* C;
  int64_t ldc;
  float alpha;
  int* err;
  int cplx;       // operands are complex (strides in complex elements), M and K count real rows
  float ima, imb;  // -1 where the operand is conjugated, else 1
};

// The careful outputs of a tile by FMAs with k increasing (the order of the
// CUDA-core update), the whole tile formed by the 256 threads of the drain
// warps: 8 x TN / 16 outputs each, K slabs of 8 double-buffered in the ring's
// shared memory with the next slab in registers.  Bound by the FMA pipe with
// two warps per scheduler.  Measured at 2048^3, where the tensor cores take
// 136 us and the CUDA-core update 531: one row of A that is not finite 381 us,
// every output outside the range 688 us.  (One serial sum per output, 64 of
// them in the lane of such a row, took 4670 and 8420 us.)  At 4096 x 4096 x
// 8192: 1.41 ms, 6.92, 1.61 and 8.37 ms.
constexpr int PK = 8;
template <int TN>
__device__ __noinline__ void plain_tile(const F32Params& p, float* smem, const int* mark, int m0, int n0) {
  constexpr int CPT = TN / 16, CV = CPT < 4 ? CPT : 4;  // columns per thread, adjacent ones
  constexpr int LDA = BM + 4, LDB = TN + 4, LA = BM * PK / 256, LB = TN * PK / 256;
  float* As = smem;                 // [2][PK][LDA]
  float* Bs = smem + 2 * PK * LDA;  // [2][PK][LDB]
  const int t = (int)threadIdx.x - 96, tx = t & 15, ty = t >> 4;
  // Slot e of a slab is element (ai + e ai_step, ak + e ak_step) of op(A), likewise
  // (bk + .., bj + ..) of op(B), threads along the index that is
  // contiguous in memory.  In the real view of complex operands (re, -im; im,
  // re) and (re; im) those steps are even, so a thread stays on one part.
  const bool ka = p.ask == 1, kb = p.bsk == 1, cx = p.cplx != 0;
  const int ai = ka ? t / PK : t % BM, ak = ka ? t % PK : t / BM;
  const int bj = kb ? t / PK : t % TN, bk = kb ? t % PK : t / TN;
  const int ai_step = ka ? 256 / PK : 0, ak_step = ka ? 0 : 256 / BM;
  const int bj_step = kb ? 256 / PK : 0, bk_step = kb ? 0 : 256 / TN;
  const int64_t sa = ai_step * p.asi + ak_step * p.ask, sb = (cx ? 2 : 1) * bj_step * p.bsj + bk_step * p.bsk;
  const int i0 = m0 + ai, j0 = n0 + bj;
  const float* pa = p.A + (cx ? 2 * ((i0 >> 1) * p.asi + (ak >> 1) * p.ask) + ((i0 ^ ak) & 1) : i0 * p.asi + ak * p.ask);
  const float* pb = p.B + (cx ? 2 * ((bk >> 1) * p.bsk + j0 * p.bsj) + (bk & 1) : bk * p.bsk + j0 * p.bsj);
  const float fa = cx && ((i0 ^ ak) & 1) ? (i0 & 1 ? p.ima : -p.ima) : 1.0f, fb = cx && (bk & 1) ? p.imb : 1.0f;
  const int64_t slab_a = PK * p.ask, slab_b = PK * p.bsk;
  const int ni = p.M - i0, nj = p.N - j0, K = p.K;
  float ra[LA], rb[LB];
  auto load = [&](int k0) {
#pragma unroll
    for (int e = 0; e < LA; ++e) ra[e] = e * ai_step < ni && k0 + ak + e * ak_step < K ? pa[e * sa] : 0.0f;
#pragma unroll
    for (int e = 0; e < LB; ++e) rb[e] = e * bj_step < nj && k0 + bk + e * bk_step < K ? pb[e * sb] : 0.0f;
    pa += slab_a;
    pb += slab_b;
  };
  auto store = [&](int buf) {
#pragma unroll
    for (int e = 0; e < LA; ++e) As[(buf * PK + ak + e * ak_step) * LDA + ai + e * ai_step] = fa * ra[e];
#pragma unroll
    for (int e = 0; e < LB; ++e) Bs[(buf * PK + bk + e * bk_step) * LDB + bj + e * bj_step] = fb * rb[e];
  };
  // Local row of slot r and column of slot c.
  auto row = [&](int r) { return (r >> 2) * 64 + 4 * tx + (r & 3); };
  auto col = [&](int c) { return (c / CV) * 64 + CV * ty + c % CV; };
  float acc[8][CPT];
#pragma unroll
  for (int r = 0; r < 8; ++r)
#pragma unroll
    for (int c = 0; c < CPT; ++c) acc[r][c] = 0.0f;
  load(0);
  store(0);
  asm volatile("bar.sync 1, 256;" ::: "memory");
  const int nk = (K + PK - 1) / PK;
  for (int kt = 0; kt < nk; ++kt) {
    const int buf = kt & 1;
    if (kt + 1 < nk) load((kt + 1) * PK);
#pragma unroll
    for (int k = 0; k < PK; ++k) {
      const float* ar = As + (buf * PK + k) * LDA + 4 * tx;
      const float* br = Bs + (buf * PK + k) * LDB + CV * ty;
      float a[8], b[CPT];
      *reinterpret_cast<float4*>(a) = *reinterpret_cast<const float4*>(ar);
      *reinterpret_cast<float4*>(a + 4) = *reinterpret_cast<const float4*>(ar + 64);
#pragma unroll
      for (int c = 0; c < CPT; c += CV) {
        if constexpr (CV == 4) *reinterpret_cast<float4*>(b + c) = *reinterpret_cast<const float4*>(br + c / CV * 64);
        else *reinterpret_cast<float2*>(b) = *reinterpret_cast<const float2*>(br);
      }
#pragma unroll
      for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int c = 0; c < CPT; ++c) acc[r][c] = fmaf(a[r], b[c], acc[r][c]);
    }
    if (kt + 1 < nk) store(buf ^ 1);
    asm volatile("bar.sync 1, 256;" ::: "memory");
  }
#pragma unroll
  for (int c = 0; c < CPT; ++c) {
    const int j = n0 + col(c), mb = mark[BM + col(c)];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const int i = m0 + row(r);
      if (i < p.M && j < p.N && careful(mark[row(r)], mb)) {
        float* cp = p.C + i + (int64_t)j * p.ldc;
        *cp = fmaf(p.alpha, acc[r][c], *cp);
      }
    }
  }
}

template <int TN>
__global__ void __launch_bounds__(F32_THREADS, 1)
    umma_f32_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                    const __grid_constant__ F32Params p) {
  constexpr int F32_STAGES = f32_stages(TN), F32_STAGE_BYTES = f32_stage_bytes(TN);
  constexpr int B_BYTES = TN * BK * 2;  // one term's tile of B
  constexpr int HALF = TN / 2;          // columns per drain warp
  constexpr int CB = HALF < 32 ? HALF : 32;  // columns of C per batch of loads
  chain_begin();
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* fullA = reinterpret_cast<uint64_t*>(smem + F32_STAGES * F32_STAGE_BYTES);
  uint64_t* fullB = fullA + F32_STAGES;
  uint64_t* empty = fullB + F32_STAGES;
  uint64_t* cfull = empty + F32_STAGES;
  uint64_t* cempty = cfull + 2;
  uint64_t* drain = cempty + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
  __shared__ volatile int s_abort;
  __shared__ int s_mark[2 * BM];  // marks of the tile's rows and columns
  __shared__ int s_lo[8], s_hi[8];  // their extremes by drain warp (of nonzero marks): rows, then columns
  __shared__ int s_careful, s_tensor;  // whether the tile has outputs for the plain product, and for the tensor cores

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // Output tiles are rasterised in groups of 8 tile rows for L2 reuse.
  constexpr int group = 8;
  const int per_group = group * p.tiles_n;
  const int g = blockIdx.x / per_group;
  const int first_m = g * group;
  const int gsize = min(p.tiles_m - first_m, group);
  const int local = blockIdx.x % per_group;
  const int m0 = (first_m + local % gsize) * BM, n0 = (local / gsize) * TN;

  if (threadIdx.x == 0) {
    s_abort = 0;
    s_careful = s_tensor = 0;
    for (int s = 0; s < F32_STAGES; ++s) {
      umma::mbar_init(umma::smem_u32(&fullA[s]), 1);
      umma::mbar_init(umma::smem_u32(&fullB[s]), 1);
      umma::mbar_init(umma::smem_u32(&empty[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      umma::mbar_init(umma::smem_u32(&cfull[b]), 1);
      umma::mbar_init(umma::smem_u32(&cempty[b]), 8);
    }
    umma::mbar_init(umma::smem_u32(drain), 1);
    umma::fence_barrier_init();
    umma::prefetch_tmap(&tmA);
    umma::prefetch_tmap(&tmB);
  }
  if (warp == 1) umma::tmem_alloc(umma::smem_u32(tmem_slot), 512);
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0 || warp == 2) {
    const bool is_a = warp == 0;
    if (lane == 0) {
      uint64_t* own = is_a ? fullA : fullB;
      int kb = 0;
      for (; kb < p.num_kb; ++kb) {
        const int s = kb % F32_STAGES;
        if (!umma::mbar_wait(umma::smem_u32(&empty[s]), ((uint32_t)(kb / F32_STAGES) & 1u) ^ 1u, &s_abort, p.err, 51))
          break;
        const uint32_t fb = umma::smem_u32(&own[s]);
        uint8_t* st = smem + (size_t)s * F32_STAGE_BYTES + (is_a ? 0 : SL * TILE_BYTES);
        const int bytes = is_a ? TILE_BYTES : B_BYTES, row0 = is_a ? m0 * SL : n0 / BN * BN * SL + n0 % BN;
        umma::mbar_arrive_expect_tx(fb, (uint32_t)(SL * bytes));
        for (int sl = 0; sl < SL; ++sl)
          umma::tma_load_2d(umma::smem_u32(st + sl * bytes), is_a ? &tmA : &tmB, fb, kb * BK, row0 + sl * BM);
      }
      umma::producer_quiesce(own, F32_STAGES, kb, &s_abort, p.err, 52);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t id1 = umma::idesc_f16(BM, TN, true), id2 = umma::idesc_f16(BM, 2 * TN, true);
      for (int kb = 0; kb < p.num_kb; ++kb) {
        const int s = kb % F32_STAGES, b = kb & 1;
        if (!umma::mbar_wait(umma::smem_u32(&cempty[b]), ((uint32_t)(kb >> 1) & 1u) ^ 1u, &s_abort, p.err, 53) ||
            !umma::mbar_wait(umma::smem_u32(&fullA[s]), (uint32_t)(kb / F32_STAGES) & 1u, &s_abort, p.err, 54) ||
            !umma::mbar_wait(umma::smem_u32(&fullB[s]), (uint32_t)(kb / F32_STAGES) & 1u, &s_abort, p.err, 54))
          break;
        umma::fence_after_sync();
        const uint32_t a0 = umma::smem_u32(smem + (size_t)s * F32_STAGE_BYTES), b0 = a0 + SL * TILE_BYTES;
        const uint32_t d0 = tmem + (uint32_t)(b * 2 * TN), d1 = d0 + (uint32_t)TN;
        // A_h against (B_h, B_m), adjacent in shared memory: one MMA of
        // N = 2 TN into both accumulators.
#pragma unroll
        for (int kk = 0; kk < BK / 16; ++kk)
          umma::mma_f16(d0, umma::desc_kmajor_sw128(a0 + kk * 32), umma::desc_kmajor_sw128(b0 + kk * 32), id2,
                        kk == 0 ? 0u : 1u);
        constexpr int qa[4] = {1, 1, 0, 2}, qb[4] = {0, 1, 2, 0};  // m h, m m, h l, l h
#pragma unroll
        for (int pr = 0; pr < 4; ++pr)
#pragma unroll
          for (int kk = 0; kk < BK / 16; ++kk)
            umma::mma_f16(d1, umma::desc_kmajor_sw128(a0 + qa[pr] * TILE_BYTES + kk * 32),
                          umma::desc_kmajor_sw128(b0 + qb[pr] * B_BYTES + kk * 32), id1, 1u);
        umma::mma_commit(umma::smem_u32(&empty[s]));
        umma::mma_commit(umma::smem_u32(&cfull[b]));
      }
      umma::mma_commit(umma::smem_u32(drain));
      umma::mbar_wait(umma::smem_u32(drain), 0, &s_abort, p.err, 55, false);
    }
  } else {
    const int q = warp & 3;
    const int h = (warp - 3) >> 2;  // column half: 0 (warps 3-6) or 1 (warps 7-10)
    const int i = m0 + q * 32 + lane, c0 = n0 + h * HALF;
    {
      // The marks of the tile's rows (threads 0-127) and columns (128-255).
      const int t = (int)threadIdx.x - 96, r = t & (BM - 1);
      const int* mk = t < BM ? p.mark_a + m0 + r : p.mark_b + n0 + r;
      const int step = t < BM ? p.rows_a : p.rows_b;
      int m = 0;
#pragma unroll 4
      for (int kb = 0; kb < p.num_kb; ++kb) m = max(m, t < BM + TN ? mk[(int64_t)kb * step] : 0);
      s_mark[t] = m;
      const int lo = __reduce_min_sync(0xffffffffu, m ? m : 1024), hi = __reduce_max_sync(0xffffffffu, m);
      if (lane == 0) s_lo[t >> 5] = lo, s_hi[t >> 5] = hi;
      asm volatile("bar.sync 1, 256;" ::: "memory");
    }
    // Outputs that are left to the plain product, if any: usually the extremes
    // exclude them.  When they are all of the tile, nothing else is formed.
    const int lo_a = min(min(s_lo[0], s_lo[1]), min(s_lo[2], s_lo[3])), lo_b = min(min(s_lo[4], s_lo[5]), min(s_lo[6], s_lo[7]));
    const int hi_a = max(max(s_hi[0], s_hi[1]), max(s_hi[2], s_hi[3])), hi_b = max(max(s_hi[4], s_hi[5]), max(s_hi[6], s_hi[7]));
    const bool looked = hi_a >= 256 || hi_b >= 256 || lo_a + lo_b < 166 || hi_a + hi_b > 360;
    if (looked) {
      bool some = false, others = false;
      if (i < p.M)
        for (int j = 0; j < min(HALF, p.N - c0); ++j) {
          const bool c = careful(s_mark[q * 32 + lane], s_mark[BM + h * HALF + j]);
          some |= c;
          others |= !c;
        }
      if (some) s_careful = 1;
      if (others) s_tensor = 1;
      asm volatile("bar.sync 1, 256;" ::: "memory");
      if (!s_tensor) s_abort = 1;  // the other warps stop: nothing of what they form is used
    }
    float acc[HALF];
#pragma unroll
    for (int j = 0; j < HALF; ++j) acc[j] = 0.0f;
    bool ok = !looked || s_tensor;
    for (int kb = 0; kb < p.num_kb && ok; ++kb) {
      const int b = kb & 1;
      ok = __all_sync(0xffffffffu, umma::mbar_wait(umma::smem_u32(&cfull[b]), (uint32_t)(kb >> 1) & 1u, &s_abort, p.err, 56));
      if (!ok) break;
      umma::fence_after_sync();
      const uint32_t ta = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * 2 * TN + h * HALF);
#pragma unroll
      for (int j0 = 0; j0 < HALF; j0 += 16) {
        uint32_t r0[16], r1[16];
        umma::tmem_ld16(ta + (uint32_t)j0, r0);
        umma::tmem_ld16(ta + (uint32_t)(TN + j0), r1);
#pragma unroll
        for (int j = 0; j < 16; ++j) acc[j0 + j] += __uint_as_float(r0[j]) + __uint_as_float(r1[j]);
      }
      umma::fence_before_sync();
      __syncwarp();
      if (lane == 0) umma::mbar_arrive(umma::smem_u32(&cempty[b]));
    }
    if (ok) {
      const int ma = s_mark[q * 32 + lane];
      const int* mb = s_mark + BM + h * HALF;
      float* C = p.C + i;
#pragma unroll
      for (int j0 = 0; j0 < HALF; j0 += CB) {
        // All loads of C before the first store (a store may alias a later load).
        float cv[CB];
        uint32_t skip = 0;
#pragma unroll
        for (int j = 0; j < CB; ++j) {
          const int col = c0 + j0 + j;
          const bool in = i < p.M && col < p.N;
          cv[j] = in ? C[(int64_t)col * p.ldc] : 0.0f;
          if (!in || (looked && careful(ma, mb[j0 + j]))) skip |= 1u << j;
        }
#pragma unroll
        for (int j = 0; j < CB; ++j)
          if (!(skip >> j & 1u)) C[(int64_t)(c0 + j0 + j) * p.ldc] = fmaf(p.alpha, acc[j0 + j], cv[j]);
      }
    }
  }

  umma::fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    umma::fence_after_sync();
    umma::tmem_dealloc(tmem, 512);
  }
  // No load or MMA is in flight any more: the ring is free.
  if (s_careful && warp >= 3) plain_tile<TN>(p, reinterpret_cast<float*>(smem), s_mark, m0, n0);
}

// ---------------------------------------------------------------------------
// Staging: the three BF16 terms of both operands in one launch, K-major,
// rows padded to 128 and K to 64 with zeros; the terms of one 128-row tile
// adjacent (row (t * 3 + term) * 128 + r for row t * 128 + r), and a mark per
// row.  One 32 x 64 tile per CTA.
// ---------------------------------------------------------------------------
struct F32Job {
  const float* X;  // element (row, k) at X[row * si + k * sk]
  int64_t si, sk;
  int rows, K;
  int cplx;  // 1: rows and K are pairs (re, im) of complex elements, as op(A); 2: only K, as op(B)
  float im;  // sign of the imaginary parts
  __nv_bfloat16* out;
  int64_t k_pad;
  int* mark;   // the block of K's marks at mark[kb * rows_pad + row]
  int blocks;  // 32-row blocks
};

// Rounded to BF16; values that would round to infinity stay finite (the next
// term takes up the rest).
__device__ __forceinline__ float bf16_near(float x) {
  const float y = __bfloat162float(__float2bfloat16_rn(x));
  return isinf(y) && !isinf(x) ? copysignf(__uint_as_float(0x7f7f0000u), x) : y;
}

__global__ void __launch_bounds__(256) stage_f32_kernel(const F32Job a, const F32Job b) {
  chain_begin();
  __shared__ float tile[32][66];
  const bool first = (int)blockIdx.x < a.blocks;
  const F32Job j = first ? a : b;
  const int i0 = (int)(first ? blockIdx.x : blockIdx.x - a.blocks) * 32, k0 = (int)blockIdx.y * 64;
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  // Threads along the index that is contiguous in memory; loads all in flight.
  const bool kfast = j.sk == 1;
  float v[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const int idx = t + 256 * e;
    const int i = i0 + (kfast ? idx >> 6 : idx & 31), k = k0 + (kfast ? idx & 63 : idx >> 5);
    const bool in = i < j.rows && k < j.K;
    if (j.cplx == 0) {
      v[e] = in ? j.X[i * j.si + k * j.sk] : 0.0f;
    } else {
      const bool pair = j.cplx == 1;
      const int part = pair ? (i ^ k) & 1 : k & 1;  // 0: real part, 1: imaginary
      const float x = in ? j.X[2 * ((pair ? i >> 1 : i) * j.si + (k >> 1) * j.sk) + part] : 0.0f;
      v[e] = part ? (pair && !(i & 1) ? -j.im : j.im) * x : x;
    }
  }
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const int idx = t + 256 * e;
    const int i = kfast ? idx >> 6 : idx & 31, k = kfast ? idx & 63 : idx >> 5;
    tile[i][k] = v[e];
  }
  __syncthreads();
#pragma unroll
  for (int pass = 0; pass < 4; ++pass) {
    const int i = warp + 8 * pass, gi = i0 + i;
    const float2 x = *reinterpret_cast<const float2*>(&tile[i][2 * lane]);
    uint32_t* o = reinterpret_cast<uint32_t*>(j.out + ((int64_t)(gi >> 7) * SL * 128 + (gi & 127)) * j.k_pad + k0 + 2 * lane);
    float r0 = x.x, r1 = x.y;
#pragma unroll
    for (int sl = 0; sl < SL; ++sl) {
      const float h0 = bf16_near(r0), h1 = bf16_near(r1);
      o[sl * (128 * j.k_pad / 2)] = (__float_as_uint(h0) >> 16) | (__float_as_uint(h1) & 0xffff0000u);
      r0 -= h0;
      r1 -= h1;
    }
    const uint32_t u0 = __float_as_uint(x.x) << 1, u1 = __float_as_uint(x.y) << 1;  // magnitude bits
    const uint32_t um = max(u0, u1);
    int mk = um ? (int)(um >> 24) + 1 : 0;
    mk = __reduce_max_sync(0xffffffffu, mk);
    const bool tiny = (u0 && (int)(u0 >> 24) + 1 < MARK_LOW) || (u1 && (int)(u1 >> 24) + 1 < MARK_LOW);
    if (__any_sync(0xffffffffu, tiny)) mk |= MARK_TINY;
    if (lane == 0) j.mark[(int64_t)blockIdx.y * (j.blocks * 32) + gi] = mk;
  }
}

int64_t pad_to(int64_t x, int64_t m) { return (x + m - 1) / m * m; }
size_t terms_bytes(int64_t rows, int64_t K) {
  return (size_t)SL * (size_t)pad_to(rows, BM) * (size_t)pad_to(K, BK) * 2;  // a multiple of 1024
}
size_t marks_bytes(int64_t rows, int64_t K) { return (size_t)pad_to(rows, BM) * (size_t)(pad_to(K, BK) / BK) * sizeof(int); }

// Columns of C per tile: the narrowest whose tiles still are one wave, since
// with few tiles a launch's time is one tile's loads, products and C update.
// Measured (rows x K x columns, 128 columns against the rule, with staging):
// 512^3 24.4 -> 17.7 us, 476 x 1024 x 900 38.3 -> 27.6, 1024^3 38.6 -> 30.6;
// the same bits.  Beyond one wave wide tiles read their operands fewer times.
int f32_tile_cols(int64_t M, int64_t N) {
  const int64_t tm = (M + BM - 1) / BM;
  int tn = BN;
  while (tn > 32 && tm * ((N + tn / 2 - 1) / (tn / 2)) <= num_sms()) tn /= 2;
  return tn;
}

}  // namespace

size_t f32_update_bytes(int64_t M, int64_t N, int64_t K) {
  return terms_bytes(M, K) + terms_bytes(N, K) + marks_bytes(M, K) + marks_bytes(N, K) + 1024;
}

// cplx: ComplexF32 operands, with M and K counting their real rows (twice the
// complex ones).
int launch_gemm_f32_umma(int64_t M, int64_t N, int64_t K, double alpha, const Mat& A, const Mat& B, const Mat& C,
                         void* ws, bool cplx, cudaStream_t s) {
  const int64_t Mp = pad_to(M, BM), Np = pad_to(N, BN), Kp = pad_to(K, BK);
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(ws) + 1023) & ~uintptr_t(1023));
  auto* ta = reinterpret_cast<__nv_bfloat16*>(base);
  auto* tb = reinterpret_cast<__nv_bfloat16*>(base + terms_bytes(M, K));
  int* marks = reinterpret_cast<int*>(base + terms_bytes(M, K) + terms_bytes(N, K));
  int* err = device_error_word();
  if (!err) return fail(NLA_ERR_UNSUPPORTED, "Float32 tensor-core update: no device error word");

  F32Params p{};
  p.M = (int)M;
  p.N = (int)N;
  p.K = (int)K;
  p.num_kb = (int)(Kp / BK);
  p.tiles_m = (int)(Mp / BM);
  const int tn = f32_tile_cols(M, N);
  p.tiles_n = (int)((N + tn - 1) / tn);
  p.A = static_cast<const float*>(A.p);
  p.asi = A.t ? A.ld : 1;
  p.ask = A.t ? 1 : A.ld;
  p.B = static_cast<const float*>(B.p);
  p.bsk = B.t ? B.ld : 1;
  p.bsj = B.t ? 1 : B.ld;
  p.mark_a = marks;
  p.mark_b = marks + Mp * (Kp / BK);
  p.rows_a = (int)Mp;
  p.rows_b = (int)Np;
  p.C = static_cast<float*>(C.p);
  p.ldc = cplx ? 2 * C.ld : C.ld;
  p.alpha = (float)alpha;
  p.err = err;
  p.cplx = cplx ? 1 : 0;
  p.ima = A.c ? -1.0f : 1.0f;
  p.imb = B.c ? -1.0f : 1.0f;
  {
    TraceScope trace(NLA_K_SPLIT, s, 0.0, (double)(M + N) * (double)K * 4.0 + (double)(Mp + Np) * Kp * 2.0 * SL);
    const F32Job ja{p.A, p.asi, p.ask, (int)M, (int)K, p.cplx, p.ima, ta, Kp, marks, (int)(Mp / 32)};
    const F32Job jb{p.B, p.bsj, p.bsk, (int)N, (int)K, 2 * p.cplx, p.imb, tb, Kp, marks + Mp * (Kp / BK), (int)(Np / 32)};
    launch_chained(stage_f32_kernel, dim3((unsigned)((Mp + Np) / 32), (unsigned)(Kp / 64)), 256, 0, s, ja, jb);
    NLA_CHECK_LAUNCH("stage_f32_kernel");
  }
  CUtensorMap mA, mB;
  NLA_TRY(staged_map(&mA, ta, (uint64_t)Kp, (uint64_t)(SL * Mp)));
  NLA_TRY(staged_map(&mB, tb, (uint64_t)Kp, (uint64_t)(SL * Np), (uint32_t)tn));
  static std::once_flag once;
  static cudaError_t st = cudaSuccess;
  std::call_once(once, [] {
    st = cudaFuncSetAttribute(umma_f32_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, f32_smem(128));
    if (st == cudaSuccess)
      st = cudaFuncSetAttribute(umma_f32_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, f32_smem(64));
    if (st == cudaSuccess)
      st = cudaFuncSetAttribute(umma_f32_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, f32_smem(32));
  });
  if (st != cudaSuccess) return cuda_status(st, "cudaFuncSetAttribute(umma_f32_kernel)");
  TraceScope trace(NLA_K_GEMM_UMMA, s, 6.0 * 2.0 * (double)M * (double)N * (double)K,
                   (double)SL * 2.0 * (double)(Mp + Np) * Kp + 8.0 * (double)M * (double)N);
  launch_chained(tn == 128 ? umma_f32_kernel<128> : tn == 64 ? umma_f32_kernel<64> : umma_f32_kernel<32>,
                 (unsigned)((int64_t)p.tiles_m * p.tiles_n), F32_THREADS, f32_smem(tn), s, mA, mB, p);
  NLA_CHECK_LAUNCH("umma_f32_kernel");
  return NLA_OK;
}

}  // namespace nla
