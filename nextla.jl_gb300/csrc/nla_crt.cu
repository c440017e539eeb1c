// Exact FP64 products on the tensor cores from residues:
//   C (M x N) += alpha * A (M x K) * B (K x N), Float64,
// by the Chinese remainder theorem (Ozaki, Uchino and Imamura, "Ozaki Scheme
// II: a GEMM-oriented emulation of floating-point matrix multiplication using
// an integer modular technique", 2025).
//
// Every row of op(A) and column of op(B) is scaled by a power of two and
// rounded to integers |y| <= 2^(t-1), t = 56 (55 for K > 14336).  The integer
// product's sums are below K 2^(2t-2) in magnitude, so they are known exactly
// from their residues modulo 16 pairwise coprime moduli of at most 253, whose
// product is P = 2^125.09.  Balanced residues are below 128 in magnitude:
// exact in BF16, and the FP32 sums of 1024 of their products stay below 2^24,
// so the tensor cores form them exactly.  One product per modulus, 16 in
// all, where digit slices of the same accuracy take 28 (umma_exact kernels,
// 7 slices of 8 bits, pairs p + q <= 6).  The only roundings are those of the
// operands to t bits (at most 2^-56 of the row's largest value, below the
// pairs that the slices leave out) and the final one to FP64.
//
//   crt_exp_kernel / crt_split_kernel   row exponents, then the 16 residues
//                        of every element, K-major (one kernel for short K);
//   crt_gemm_kernel      persistent: items (modulus, 256 x 128 tile), TMA
//                        ring, two TMEM accumulators, 16 drain warps that
//                        reduce each chunk modulo p and leave one byte per
//                        element and modulus;
//   crt_finish_kernel    16 bytes -> 128-bit integer -> FP64, and C's update
//                        (or the residual C - P - d x, rounded once).
#include <cudaTypedefs.h>

#include <mutex>

#include "nla_common.cuh"
#include "nla_umma.cuh"

namespace nla {
namespace {

constexpr int L = 16;
constexpr int BU = 128, BV = 256, BK = 64;
constexpr int U_BYTES = BU * BK * 2, V_BYTES = BV * BK * 2;
constexpr int RING_BYTES = 4 * (U_BYTES + V_BYTES);  // four stages, or six of 128 + 128 rows
constexpr int MAX_STAGES = RING_BYTES / (2 * U_BYTES);
constexpr int DRAIN_WARPS = 16, THREADS = (3 + DRAIN_WARPS) * 32;
constexpr int CHUNK = 16;  // K blocks of 64 per exact FP32 sum: 1024 x 2^14 = 2^24
constexpr int SMEM = RING_BYTES + 1024 + 256;
static_assert(SMEM + 64 <= 232448, "shared memory above the per-block limit");
constexpr int SENTINEL_EXP = -2139062144;  // 0x80808080: "no element seen"
constexpr int NONFINITE_EXP = 0x7fffffff;
constexpr float MAGIC = 12582912.0f;  // 1.5 * 2^23: rounds a float to an integer when added and subtracted
constexpr int64_t MAX_K = 57344;      // integer headroom: K 2^(2 t - 2) < 0.45 P

// Number of bits t of the scaled operands.
__host__ __device__ constexpr int operand_bits(int64_t K) { return K <= 14336 ? 56 : 55; }

// The reconstruction sums y_l P / p_l group by group (three moduli, the last
// group one), inner sums in 32 bits: sum_g (sum_l y_l P_g / p_l) (P / P_g).
constexpr int GROUPS = (L + 2) / 3;

struct Tables {
  float p[L], inv_p[L];      // modulus and its reciprocal
  float k[2][L][4];  // 2^(14 i) f mod p, balanced; f = 1, or (P / p)^-1 for C's row operand
  uint32_t in[L];            // P_g / p
  uint32_t m[GROUPS][4];     // P / P_g, 32-bit limbs
  uint32_t q[GROUPS];        // round(2^54 / P_g)
  uint32_t P[4];
  // Starting values of the sums.  The planes hold z + 128 after a sign flip,
  // so 128 times the sums of the constants above are taken off.  q0 makes
  // the quotient's sum positive (QB too many, plus a half to round), and
  // m0 takes QB P off for adding (QB - quotient) P; every limb starts
  // 2^62 higher, which its successor takes back, so that all stay positive.
  unsigned long long m0[4], q0;
};
constexpr unsigned QB = 64;

// Pairwise coprime, and small enough that a balanced residue that is off by
// one from rounding (p / 2 + 1) is still a signed byte.
constexpr uint32_t MODULI[L] = {253, 251, 249, 247, 245, 241, 239, 233, 229, 227, 223, 211, 199, 197, 193, 191};

constexpr Tables make_tables() {
  Tables T{};
  unsigned __int128 P = 1;
  for (int l = 0; l < L; ++l) P *= MODULI[l];
  for (int i = 0; i < 4; ++i) T.P[i] = (uint32_t)(P >> (32 * i));
  for (int l = 0; l < L; ++l) {
    const uint32_t p = MODULI[l], r = (uint32_t)(P / p % p);
    uint32_t w = 1;
    while (w * r % p != 1) ++w;
    T.p[l] = (float)p;
    T.inv_p[l] = 1.0f / (float)p;
    for (int o = 0; o < 2; ++o) {
      uint32_t f = o ? w : 1;
      for (int i = 0; i < 4; ++i) {
        T.k[o][l][i] = f > p / 2 ? (float)f - (float)p : (float)f;
        f = f * (16384u % p) % p;
      }
    }
  }
  for (int g = 0; g < GROUPS; ++g) {
    uint32_t Pg = 1;
    for (int l = 3 * g; l < 3 * g + 3 && l < L; ++l) Pg *= MODULI[l];
    for (int l = 3 * g; l < 3 * g + 3 && l < L; ++l) T.in[l] = Pg / MODULI[l];
    const unsigned __int128 M = P / Pg;
    for (int i = 0; i < 4; ++i) T.m[g][i] = (uint32_t)(M >> (32 * i));
    // The last group's quotient (one modulus) would not fit 32 bits at 2^54:
    // it is taken at 2^31 and its products (at most 254 / 191 of that, 32
    // bits) shifted up by 23.
    T.q[g] = (uint32_t)(((g + 1 < GROUPS ? 1ull << 54 : 1ull << 31) + Pg / 2) / Pg);
    for (int l = 3 * g; l < 3 * g + 3 && l < L; ++l) {
      for (int i = 0; i < 4; ++i) T.m0[i] += 128ull * T.in[l] * T.m[g][i];
      T.q0 += g + 1 < GROUPS ? 128ull * T.in[l] * T.q[g] : (128ull * T.in[l] * T.q[g]) << 23;
    }
  }
  for (int i = 0; i < 4; ++i)
    T.m0[i] = 0 - T.m0[i] - (unsigned long long)QB * T.P[i] + (1ull << 62) - (i > 0 ? 1ull << 30 : 0);
  T.q0 = ((unsigned long long)QB << 54) + (1ull << 53) - T.q0;
  return T;
}
__constant__ const Tables c_t = make_tables();

// r = v mod p, balanced (|r| <= p / 2 up to the rounding of v / p, so at most
// p / 2 + 1), for an integer |v| <= 2^24: every step is exact but the choice
// of the quotient.
__device__ __forceinline__ float mod_balanced(float v, float p, float inv_p) {
  const float q = __fadd_rn(__fmaf_rn(v, inv_p, MAGIC), -MAGIC);
  return __fmaf_rn(-p, q, v);
}

// ---------------------------------------------------------------------------
// Staging.
// ---------------------------------------------------------------------------
struct Job {
  const double* X;  // element (row, k) at X[row * si + k * sk]
  int64_t si, sk;
  int64_t rows, K;
  int tri;    // 0 all, 1 k <= row, 2 k >= row, 3 k < row, 4 k > row: the rest counts as zero
  int bits;
  int f;      // 1: residues times (P / p)^-1 (C's row operand)
  int* e;     // row exponents
  uint16_t* out;  // L planes of rows_pad x K_pad BF16
  int64_t rows_pad, K_pad;
};

__device__ __forceinline__ bool in_tri(int tri, int64_t i, int64_t k) {
  switch (tri) {
    case 1: return k <= i;
    case 2: return k >= i;
    case 3: return k < i;
    case 4: return k > i;
    default: return true;
  }
}

// frexp-style exponent of |x| plus one (x 2^-e lies in [1/4, 1/2) for the
// largest element of a row), from the bit pattern.
__device__ __forceinline__ int exp_of(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const int biased = (int)((b >> 52) & 0x7FF);
  if (biased == 0x7FF) return NONFINITE_EXP;
  if (biased == 0) return (b << 12) == 0 ? SENTINEL_EXP : -1021;
  return biased - 1021;
}

// x 2^(bits - ex) rounded to an integer (0 for zeros, non-finite values and
// rows that hold one).
__device__ __forceinline__ long long fixed_of(double x, int ex, int bits) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const int biased = (int)((b >> 52) & 0x7FF);
  if (biased == 0x7FF || ex == NONFINITE_EXP || ex == SENTINEL_EXP) return 0;
  const unsigned long long mant = b & ((1ull << 52) - 1);
  const unsigned long long m = biased ? (mant | (1ull << 52)) : mant;
  const int sh = (biased ? biased : 1) - 1075 - ex + bits;  // m 2^sh
  long long y = 0;
  if (sh >= 0) y = (long long)(m << sh);
  else if (sh > -63) y = (long long)((m + (1ull << (-sh - 1))) >> (-sh));
  return b >> 63 ? -y : y;
}

// One 32 x 64 tile (rows i0.., K k0..): eight loads per thread, all in
// flight, along the index that is contiguous in memory (slot e at row
// i + e di, K k + e dk of the thread's first).
__device__ __forceinline__ void load_tile(const Job& j, int64_t i0, int64_t k0, double (&v)[8]) {
  const bool kfast = j.sk == 1;
  const int t = threadIdx.x, ti = kfast ? t >> 6 : t & 31, tk = kfast ? t & 63 : t >> 5;
  const int di = kfast ? 4 : 0, dk = kfast ? 0 : 8;
  const double* p = j.X + (i0 + ti) * j.si + (k0 + tk) * j.sk;
  const int64_t step = kfast ? 4 * j.si : 8 * j.sk;
  const int ni = (int)min((int64_t)64, j.rows - i0) - ti, nk = (int)min((int64_t)64, j.K - k0) - tk;
  if (j.tri == 0) {
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = e * di < ni && e * dk < nk ? p[e * step] : 0.0;
  } else {
#pragma unroll
    for (int e = 0; e < 8; ++e)
      v[e] = e * di < ni && e * dk < nk && in_tri(j.tri, i0 + ti + e * di, k0 + tk + e * dk) ? p[e * step] : 0.0;
  }
}

__device__ __forceinline__ void tile_to_smem(const Job& j, double (*tile)[65], const double (&v)[8]) {
  const bool kfast = j.sk == 1;
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const int idx = threadIdx.x + 256 * e;
    tile[kfast ? idx >> 6 : idx & 31][kfast ? idx & 63 : idx >> 5] = v[e];
  }
}

// Largest exponents of the tile's rows into sred: with sk == 1 thread e-slots
// lie in rows (t >> 6) + 4 e, else in row t & 31.
__device__ __forceinline__ void tile_row_max(const Job& j, int (*sred)[32], int (&m)[8]) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (j.sk != 1) {
    int x = m[0];
#pragma unroll
    for (int e = 1; e < 8; ++e) x = max(x, m[e]);
    sred[warp][lane] = x;
  } else {
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int r = __reduce_max_sync(0xffffffffu, m[e]);
      if (lane == 0) sred[warp][e] = r;  // row (warp >> 1) + 4 e
    }
  }
}
__device__ __forceinline__ int row_max_of(const Job& j, int (*sred)[32], int r) {
  if (j.sk == 1) return max(sred[2 * (r & 3)][r >> 2], sred[2 * (r & 3) + 1][r >> 2]);
  int x = SENTINEL_EXP;
#pragma unroll
  for (int w = 0; w < 8; ++w) x = max(x, sred[w][r]);
  return x;
}

// The residues of the tile.  y is cut into 14-bit pieces (the top one
// signed), whose products with 2^(14 i) mod p and their sum stay below 2^23:
// exact in Float32, on the FMA pipe rather than the integer one (four dot
// products of bytes, the form before, took 276 instructions per element and
// 1.4 times as long).  C's row operand carries the factor (P / p)^-1 of the
// reconstruction in the same constants.  Two adjacent K values per lane, one
// 32-bit store per modulus.
__device__ __forceinline__ void pieces14(long long y, float (&c)[4]) {
  const uint32_t lo = (uint32_t)y, hi = (uint32_t)((unsigned long long)y >> 32);
  c[0] = __uint_as_float(0x4B000000u | (lo & 0x3FFFu)) - 8388608.0f;
  c[1] = __uint_as_float(0x4B000000u | ((lo >> 14) & 0x3FFFu)) - 8388608.0f;
  c[2] = __uint_as_float(0x4B000000u | (__funnelshift_r(lo, hi, 28) & 0x3FFFu)) - 8388608.0f;
  c[3] = __int_as_float(0x4B400000 + ((int)hi >> 10)) - MAGIC;
}

template <int F>
__device__ __forceinline__ void split_tile_f(const Job& j, const double (*tile)[65], const int* ex_rows, int64_t i0,
                                             int64_t k0) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t plane = j.rows_pad * j.K_pad / 2;  // 32-bit words
#pragma unroll 1
  for (int pass = 0; pass < 4; ++pass) {
    const int i = warp + 8 * pass;
    const int ex = ex_rows[i];
    float c0[4], c1[4];
    pieces14(fixed_of(tile[i][2 * lane], ex, j.bits), c0);
    pieces14(fixed_of(tile[i][2 * lane + 1], ex, j.bits), c1);
    uint32_t* o = reinterpret_cast<uint32_t*>(j.out) + ((i0 + i) * j.K_pad + k0) / 2 + lane;
#pragma unroll
    for (int l = 0; l < L; ++l) {
      const float* k = c_t.k[F][l];
      const float s0 = fmaf(c0[3], k[3], fmaf(c0[2], k[2], fmaf(c0[1], k[1], c0[0] * k[0])));
      const float s1 = fmaf(c1[3], k[3], fmaf(c1[2], k[2], fmaf(c1[1], k[1], c1[0] * k[0])));
      const float r0 = mod_balanced(s0, c_t.p[l], c_t.inv_p[l]), r1 = mod_balanced(s1, c_t.p[l], c_t.inv_p[l]);
      // An integer of at most 8 bits: its BF16 pattern is the float's upper half.
      *o = __byte_perm(__float_as_uint(r0), __float_as_uint(r1), 0x7632);
      o += plane;
    }
  }
}

__device__ __forceinline__ void split_tile(const Job& j, const double (*tile)[65], const int* ex_rows, int64_t i0,
                                           int64_t k0) {
  if (j.f) split_tile_f<1>(j, tile, ex_rows, i0, k0);
  else split_tile_f<0>(j, tile, ex_rows, i0, k0);
}

// Row exponents of both operands, one 32 x 64 tile per CTA (e preset to
// SENTINEL_EXP).
__global__ void __launch_bounds__(256) crt_exp_kernel(const Job a, const Job b, int blocks_a) {
  chain_begin();
  __shared__ int sred[8][32];
  const bool first = (int)blockIdx.x < blocks_a;
  const Job j = first ? a : b;
  const int64_t i0 = (int64_t)(first ? blockIdx.x : blockIdx.x - blocks_a) * 32, k0 = (int64_t)blockIdx.y * 64;
  if (k0 >= j.K) return;
  double v[8];
  load_tile(j, i0, k0, v);
  int m[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) m[e] = exp_of(v[e]);
  tile_row_max(j, sred, m);
  __syncthreads();
  if (threadIdx.x < 32 && i0 + threadIdx.x < j.rows) {
    const int x = row_max_of(j, sred, threadIdx.x);
    if (x != SENTINEL_EXP) atomicMax(j.e + i0 + threadIdx.x, x);
  }
}

__global__ void __launch_bounds__(256) crt_split_kernel(const Job a, const Job b, int blocks_a) {
  chain_begin();
  __shared__ double tile[32][65];
  __shared__ int sexp[32];
  const bool first = (int)blockIdx.x < blocks_a;
  const Job j = first ? a : b;
  const int64_t i0 = (int64_t)(first ? blockIdx.x : blockIdx.x - blocks_a) * 32, k0 = (int64_t)blockIdx.y * 64;
  if (k0 >= j.K_pad) return;
  if (threadIdx.x < 32) sexp[threadIdx.x] = i0 + threadIdx.x < j.rows ? j.e[i0 + threadIdx.x] : SENTINEL_EXP;
  double v[8];
  load_tile(j, i0, k0, v);
  tile_to_smem(j, tile, v);
  __syncthreads();
  split_tile(j, tile, sexp, i0, k0);
}

// Short K: exponents and residues of 32 rows by one CTA (the second pass over
// its rows reads L2), so one launch stages both operands.
__global__ void __launch_bounds__(256) crt_stage_kernel(const Job a, const Job b, int blocks_a) {
  chain_begin();
  __shared__ double tile[2][32][65];
  __shared__ int sred[8][32];
  __shared__ int sexp[32];
  const bool first = (int)blockIdx.x < blocks_a;
  const Job j = first ? a : b;
  const int64_t i0 = (int64_t)(first ? blockIdx.x : blockIdx.x - blocks_a) * 32;
  const int64_t ktiles = j.K_pad / 64;
  int m[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) m[e] = SENTINEL_EXP;
  double v[8];
  for (int64_t kt = 0; kt < ktiles; ++kt) {
    load_tile(j, i0, kt * 64, v);
#pragma unroll
    for (int e = 0; e < 8; ++e) m[e] = max(m[e], exp_of(v[e]));
  }
  tile_row_max(j, sred, m);
  __syncthreads();
  if (threadIdx.x < 32) {
    const int x = row_max_of(j, sred, threadIdx.x);
    sexp[threadIdx.x] = x;
    if (i0 + threadIdx.x < j.rows) j.e[i0 + threadIdx.x] = x;
  }
  for (int64_t kt = 0; kt < ktiles; ++kt) {
    if (ktiles > 1) load_tile(j, i0, kt * 64, v);
    tile_to_smem(j, tile[kt & 1], v);
    __syncthreads();
    split_tile(j, tile[kt & 1], sexp, i0, kt * 64);
  }
}

// ---------------------------------------------------------------------------
// The products.
// ---------------------------------------------------------------------------
// C's columns (the operand U, 128 per tile) lie along TMEM lanes and its rows
// (V, 256 or 128 per tile) along TMEM columns, so that a drain thread holds
// consecutive rows of one column: one 16-byte store per 16 of them.
struct GemmArgs {
  int M, N, K;          // rows and columns of C
  int tiles_u, tiles_v, items;
  int bv;               // rows of C per tile: 256, or 128 when C has no more
  int stages, stage_bytes;
  int rows_u, rows_v;   // padded: modulus l's plane starts at row l * rows
  int tri_u, tri_v;
  uint8_t* planes;      // byte (i, j) of modulus l at l * plane + i + j * ldp
  int64_t plane, ldp;
  int* err;
};

// K range of the staged triangle that meets rows [r0, r0 + span).
__device__ __forceinline__ void tri_k_range(int tri, int r0, int span, int K, int& lo, int& hi) {
  lo = 0;
  hi = K - 1;
  if (tri == 1 || tri == 3) hi = min(K - 1, r0 + span - 1);
  else if (tri == 2 || tri == 4) lo = r0;
}

struct Item {
  int l, u0, v0, kb0, kb1;
};
__device__ __forceinline__ Item item_at(const GemmArgs& p, int w) {
  // Moduli outermost; a modulus' tiles in groups of 8 along U for L2 reuse.
  const int tiles = p.tiles_u * p.tiles_v;
  Item it;
  it.l = w / tiles;
  const int t = w - it.l * tiles, per_group = 8 * p.tiles_v;
  const int first = t / per_group * 8, local = t % per_group;
  const int gsize = min(p.tiles_u - first, 8);
  it.u0 = (first + local % gsize) * BU;
  it.v0 = local / gsize * p.bv;
  int alo, ahi, blo, bhi;
  tri_k_range(p.tri_u, it.u0, BU, p.K, alo, ahi);
  tri_k_range(p.tri_v, it.v0, p.bv, p.K, blo, bhi);
  const int klo = max(alo, blo), khi = min(ahi, bhi);
  it.kb0 = klo / BK;
  it.kb1 = khi >= klo ? khi / BK + 1 : it.kb0;  // empty when the triangles miss each other
  return it;
}

// 16 integers |z| < 128 as signed bytes.
__device__ __forceinline__ uint4 signed_bytes(const float (&z)[16]) {
  uint32_t y[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) y[j] = __float_as_uint(z[j] + MAGIC);
  uint4 v;
  v.x = __byte_perm(__byte_perm(y[0], y[1], 0x0040), __byte_perm(y[2], y[3], 0x0040), 0x5410);
  v.y = __byte_perm(__byte_perm(y[4], y[5], 0x0040), __byte_perm(y[6], y[7], 0x0040), 0x5410);
  v.z = __byte_perm(__byte_perm(y[8], y[9], 0x0040), __byte_perm(y[10], y[11], 0x0040), 0x5410);
  v.w = __byte_perm(__byte_perm(y[12], y[13], 0x0040), __byte_perm(y[14], y[15], 0x0040), 0x5410);
  return v;
}

__global__ void __launch_bounds__(THREADS, 1)
    crt_gemm_kernel(const __grid_constant__ CUtensorMap tmU, const __grid_constant__ CUtensorMap tmV, const GemmArgs p) {
  chain_begin();
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* fullU = reinterpret_cast<uint64_t*>(smem + RING_BYTES);
  uint64_t* fullV = fullU + MAX_STAGES;
  uint64_t* empty = fullV + MAX_STAGES;
  uint64_t* cfull = empty + MAX_STAGES;
  uint64_t* cempty = cfull + 2;
  uint64_t* drain = cempty + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
  __shared__ volatile int s_abort;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    s_abort = 0;
    for (int s = 0; s < MAX_STAGES; ++s) {
      umma::mbar_init(umma::smem_u32(&fullU[s]), 1);
      umma::mbar_init(umma::smem_u32(&fullV[s]), 1);
      umma::mbar_init(umma::smem_u32(&empty[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      umma::mbar_init(umma::smem_u32(&cfull[b]), 1);
      umma::mbar_init(umma::smem_u32(&cempty[b]), DRAIN_WARPS);
    }
    umma::mbar_init(umma::smem_u32(drain), 1);
    umma::fence_barrier_init();
    umma::prefetch_tmap(&tmU);
    umma::prefetch_tmap(&tmV);
  }
  if (warp == 1) umma::tmem_alloc(umma::smem_u32(tmem_slot), 512);
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  bool ok = true;

  if (warp == 0 || warp == 2) {
    const bool is_u = warp == 0;
    if (lane == 0) {
      uint64_t* own = is_u ? fullU : fullV;
      const uint32_t bytes = (uint32_t)(is_u ? U_BYTES : p.bv * BK * 2);
      int n = 0, s = 0;
      uint32_t par = 1;  // of the empty barriers: the first round passes
      for (int w = blockIdx.x; w < p.items && ok; w += gridDim.x) {
        const Item it = item_at(p, w);
        const int y = it.l * (is_u ? p.rows_u : p.rows_v) + (is_u ? it.u0 : it.v0);
        for (int kb = it.kb0; kb < it.kb1; ++kb, ++n) {
          if (!umma::mbar_wait(umma::smem_u32(&empty[s]), par, &s_abort, p.err, 61)) {
            ok = false;
            break;
          }
          const uint32_t fb = umma::smem_u32(&own[s]);
          umma::mbar_arrive_expect_tx(fb, bytes);
          umma::tma_load_2d(umma::smem_u32(smem + s * p.stage_bytes + (is_u ? 0 : U_BYTES)), is_u ? &tmU : &tmV, fb,
                            kb * BK, y);
          if (++s == p.stages) s = 0, par ^= 1;
        }
      }
      umma::producer_quiesce(own, p.stages, n, &s_abort, p.err, 62);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc = umma::idesc_f16(BU, p.bv, true);
      int s = 0, ch = 0;
      uint32_t par = 0;
      for (int w = blockIdx.x; w < p.items && ok; w += gridDim.x) {
        const Item it = item_at(p, w);
        for (int c0 = it.kb0; c0 < it.kb1 && ok; c0 += CHUNK, ++ch) {
          const int b = ch & 1;
          if (!umma::mbar_wait(umma::smem_u32(&cempty[b]), ((uint32_t)(ch >> 1) & 1u) ^ 1u, &s_abort, p.err, 63)) {
            ok = false;
            break;
          }
          umma::fence_after_sync();
          const uint32_t d = tmem + (uint32_t)(b * BV);
          for (int kb = c0; kb < min(c0 + CHUNK, it.kb1); ++kb) {
            if (!umma::mbar_wait(umma::smem_u32(&fullU[s]), par, &s_abort, p.err, 64) ||
                !umma::mbar_wait(umma::smem_u32(&fullV[s]), par, &s_abort, p.err, 64)) {
              ok = false;
              break;
            }
            umma::fence_after_sync();
            const uint32_t a0 = umma::smem_u32(smem + s * p.stage_bytes), b0 = a0 + U_BYTES;
#pragma unroll
            for (int kk = 0; kk < BK / 16; ++kk)
              umma::mma_f16(d, umma::desc_kmajor_sw128(a0 + kk * 32), umma::desc_kmajor_sw128(b0 + kk * 32), idesc,
                            (kb > c0 || kk > 0) ? 1u : 0u);
            umma::mma_commit(umma::smem_u32(&empty[s]));
            if (++s == p.stages) s = 0, par ^= 1;
          }
          if (ok) umma::mma_commit(umma::smem_u32(&cfull[b]));
        }
      }
      umma::mma_commit(umma::smem_u32(drain));
      umma::mbar_wait(umma::smem_u32(drain), 0, &s_abort, p.err, 65, false);
    }
  } else {
    // Drain warps: TMEM lane quarter warp % 4 (a lane is a column of C), a
    // quarter of the tile's rows of C each.
    const int q = warp & 3, per = p.bv / 4, r0 = ((warp - 3) >> 2) * per;
    int ch = 0;
    for (int w = blockIdx.x; w < p.items && ok; w += gridDim.x) {
      const Item it = item_at(p, w);
      const float pf = c_t.p[it.l], ip = c_t.inv_p[it.l];
      const int col = it.u0 + q * 32 + lane, row = it.v0 + r0;
      const bool store = col < p.N && row < p.rows_v;
      uint4* o = reinterpret_cast<uint4*>(p.planes + it.l * p.plane + row + (int64_t)col * p.ldp);
      const int nch = (it.kb1 - it.kb0 + CHUNK - 1) / CHUNK;
      if (nch == 1) {
        // One chunk: straight from TMEM to bytes.
        const int b = ch & 1;
        ok = __all_sync(0xffffffffu,
                        umma::mbar_wait(umma::smem_u32(&cfull[b]), (uint32_t)(ch >> 1) & 1u, &s_abort, p.err, 66));
        if (!ok) break;
        umma::fence_after_sync();
        const uint32_t ta = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * BV + r0);
        uint4 bytes[4];
#pragma unroll
        for (int j0 = 0; j0 < 64; j0 += 32) {
          if (j0 < per) {
            uint32_t r[32];
            umma::tmem_ld32(ta + (uint32_t)j0, r);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              float z[16];
#pragma unroll
              for (int j = 0; j < 16; ++j) z[j] = mod_balanced(__uint_as_float(r[16 * h + j]), pf, ip);
              bytes[j0 / 16 + h] = signed_bytes(z);
            }
          }
        }
        umma::fence_before_sync();
        __syncwarp();
        if (lane == 0) umma::mbar_arrive(umma::smem_u32(&cempty[b]));
        ++ch;
        if (store) {
#pragma unroll
          for (int j0 = 0; j0 < 64; j0 += 16)
            if (j0 < per) o[j0 / 16] = bytes[j0 / 16];
        }
        continue;
      }
      float acc[64];
#pragma unroll
      for (int j = 0; j < 64; ++j) acc[j] = 0.0f;
      for (int c = 0; c < nch; ++c, ++ch) {
        const int b = ch & 1;
        ok = __all_sync(0xffffffffu,
                        umma::mbar_wait(umma::smem_u32(&cfull[b]), (uint32_t)(ch >> 1) & 1u, &s_abort, p.err, 66));
        if (!ok) break;
        umma::fence_after_sync();
        const uint32_t ta = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * BV + r0);
#pragma unroll
        for (int j0 = 0; j0 < 64; j0 += 16) {
          if (j0 < per) {
            uint32_t r[16];
            umma::tmem_ld16(ta + (uint32_t)j0, r);
#pragma unroll
            for (int j = 0; j < 16; ++j) acc[j0 + j] += mod_balanced(__uint_as_float(r[j]), pf, ip);
          }
        }
        umma::fence_before_sync();
        __syncwarp();
        if (lane == 0) umma::mbar_arrive(umma::smem_u32(&cempty[b]));
      }
      if (ok && store) {
#pragma unroll
        for (int j0 = 0; j0 < 64; j0 += 16) {
          if (j0 < per) {
            float z[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) z[j] = mod_balanced(acc[j0 + j], pf, ip);  // |sum| <= 56 x 128
            o[j0 / 16] = signed_bytes(z);
          }
        }
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
}

// ---------------------------------------------------------------------------
// Reconstruction and update.
// ---------------------------------------------------------------------------
struct FinishArgs {
  const uint8_t* planes;
  int64_t plane, ldp;
  int M, N;
  const int* ea;
  const int* eb;
  int e_bias;  // -2 t
  double* C;
  int64_t ldc;
  double alpha;
  // Residual (res_x set): C := C - P - d x, d of the row (or column) of C.
  const double* res_x;
  int64_t res_ldx;
  const double* res_d;
  int64_t res_dstride;
  int d_col;
};

struct Wide {  // a signed 128-bit integer as sign and magnitude
  unsigned long long hi, lo;
  bool neg;
};

__device__ __noinline__ double pow2_slow(double m, int e) { return ldexp(m, e); }

// The magnitude's leading 53 bits, rounded to nearest even: value = m 2^k
// (m <= 2^53; 0 for 0).
__device__ __forceinline__ unsigned long long leading53(const Wide& x, int& k) {
  const int lz = x.hi ? __clzll((long long)x.hi) : 64 + __clzll((long long)x.lo);
  if (lz == 128) {
    k = 0;
    return 0;
  }
  // Normalised: the leading bit at bit 63 of `top`, the rest below it.
  unsigned long long top, rest;
  if (lz >= 64) {
    top = x.lo << (lz - 64);
    rest = 0;
  } else {
    top = lz ? (x.hi << lz) | (x.lo >> (64 - lz)) : x.hi;
    rest = x.lo << lz;
  }
  k = 64 - lz + 11;
  unsigned long long m = top >> 11;
  const unsigned long long rem = top & 2047ull;
  if (rem > 1024 || (rem == 1024 && (rest != 0 || (m & 1)))) ++m;
  return m;
}

// (-1)^neg m 2^e for an integer m <= 2^53.
__device__ __forceinline__ double to_f64(unsigned long long m, int e, bool neg) {
  if (m == 0) return 0.0;
  // m is normalised (leading bit 52, or 2^53 after rounding up) except for
  // integers of fewer bits, which come left-aligned as well.
  const int up = (int)(m >> 53);
  const int biased = 52 + up + e + 1023;
  if (biased <= 0 || biased >= 2047) return pow2_slow(neg ? -(double)m : (double)m, e);
  const unsigned long long bits = ((unsigned long long)biased << 52) | ((m >> up) & 0xFFFFFFFFFFFFFull);
  return __longlong_as_double((long long)(bits | (neg ? 1ull << 63 : 0ull)));
}

// The general case of round_wide, out of line.
__device__ __noinline__ double round_wide_slow(unsigned long long hi, unsigned long long lo, bool neg, int e) {
  const Wide x{hi, lo, neg};
  int k;
  const unsigned long long m = leading53(x, k);
  return to_f64(m, k + e, neg);
}

// (-1)^(sign != 0) (u3 : u2 : u1 : u0) 2^e to nearest even, in 32-bit steps.
__device__ __forceinline__ double round_wide(uint32_t u3, uint32_t u2, uint32_t u1, uint32_t u0, uint32_t sign, int e) {
  // The three limbs from the leading one on, and whether any bit follows.
  const bool top = u3 != 0;
  const uint32_t a = top ? u3 : u2, b = top ? u2 : u1, c = top ? u1 : u0;
  const uint32_t rest = top ? u0 : 0u;
  const int lz = __clz((int)a);
  const uint32_t n2 = __funnelshift_l(b, a, lz), n1 = __funnelshift_l(c, b, lz), n0 = c << lz;
  const int biased = 1023 + (top ? 127 : 95) - lz + e;
  if (a == 0 || biased <= 0 || biased >= 2046)
    return round_wide_slow(((unsigned long long)u3 << 32) | u2, ((unsigned long long)u1 << 32) | u0, sign != 0, e);
  const uint32_t ml = __funnelshift_r(n1, n2, 11);  // mantissa: n2 : n1 without its last 11 bits
  const uint32_t up = ((n1 & 0x7FFu) + 0x3FFu + ((ml & 1u) | (uint32_t)((n0 | rest) != 0))) >> 11;
  // The leading bit adds one to the exponent field, as does a carry.
  const unsigned long long bits =
      (((unsigned long long)(((uint32_t)(biased - 1) << 20) + (n2 >> 11)) << 32) | ml) + up;
  return __longlong_as_double((long long)(bits | ((unsigned long long)(sign & 0x80000000u) << 32)));
}

__device__ __forceinline__ void two_sum(double a, double b, double& s, double& e) {
  s = a + b;
  const double bp = s - a;
  e = (a - (s - bp)) + (b - bp);
}

constexpr int FIN_PITCH = 36;    // four rows of 32 lanes, staggered over the banks
// A warp takes 128 rows of one column: each lane reads 4 rows'
// bytes of every plane as one word, forms their integers, and the results
// pass through shared memory so that C is read and written along its rows.
__global__ void __launch_bounds__(256, 4) crt_finish_kernel(const FinishArgs p) {
  chain_begin();
  __shared__ double buf[8][4 * FIN_PITCH];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i0 = blockIdx.x * 128;
  const int ib = i0 + 4 * lane;
  int er[4];  // row exponents with the bias (at least -4200: far below any sum that matters)
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    er[r] = ib + r < p.M ? p.ea[ib + r] : 0;
    if (er[r] != NONFINITE_EXP) er[r] = max(er[r], -4000) + p.e_bias;
  }
  const int64_t col = (int64_t)blockIdx.y * 8 + warp;
  if (col >= p.N) return;
  uint32_t w[L];
#pragma unroll
  for (int l = 0; l < L; ++l)
    w[l] = *reinterpret_cast<const uint32_t*>(p.planes + l * p.plane + ib + col * p.ldp) ^ 0x80808080u;
  double cv[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int i = i0 + lane + 32 * r;
    cv[r] = i < p.M ? p.C[i + col * p.ldc] : 0.0;
  }
  int ejc = p.eb[col];
  if (ejc != NONFINITE_EXP) ejc = max(ejc, -4000);
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    // x = sum_l y_l (P / p_l) - round(sum_l y_l / p_l) P, |x| < 0.45 P.
    // The leading limb needs only its value modulo 2^32.
    unsigned long long a0 = c_t.m0[0], a1 = c_t.m0[1], a2 = c_t.m0[2], qs = c_t.q0;
    uint32_t a3 = (uint32_t)c_t.m0[3];
#pragma unroll
    for (int g = 0; g < GROUPS; ++g) {
      uint32_t sg = 0;
#pragma unroll
      for (int l = 3 * g; l < 3 * g + 3 && l < L; ++l) sg += __byte_perm(w[l], 0, 0x4440 + r) * c_t.in[l];
      if (g + 1 < GROUPS) qs += (unsigned long long)sg * c_t.q[g];
      else qs += (unsigned long long)(sg * c_t.q[g]) << 23;
      a0 += (unsigned long long)sg * c_t.m[g][0];
      a1 += (unsigned long long)sg * c_t.m[g][1];
      a2 += (unsigned long long)sg * c_t.m[g][2];
      a3 += sg * c_t.m[g][3];
    }
    const uint32_t nq = 2 * QB - (uint32_t)(qs >> 54);  // 2 QB - (quotient + QB)
    a0 += (unsigned long long)nq * c_t.P[0];
    a1 += (unsigned long long)nq * c_t.P[1] + (a0 >> 32);
    a2 += (unsigned long long)nq * c_t.P[2] + (a1 >> 32);
    a3 += nq * c_t.P[3] + (uint32_t)(a2 >> 32);
    uint32_t u0 = (uint32_t)a0, u1 = (uint32_t)a1, u2 = (uint32_t)a2, u3 = a3;
    const uint32_t sign = (uint32_t)((int)u3 >> 31);
    {
      // |x|
      const unsigned long long lo = (((unsigned long long)(u1 ^ sign) << 32) | (u0 ^ sign)) + (sign & 1u);
      const unsigned long long hi =
          (((unsigned long long)(u3 ^ sign) << 32) | (u2 ^ sign)) + ((sign & 1u) && lo == 0 ? 1ull : 0ull);
      u0 = (uint32_t)lo;
      u1 = (uint32_t)(lo >> 32);
      u2 = (uint32_t)hi;
      u3 = (uint32_t)(hi >> 32);
    }
    const int e = er[r] + ejc;
    const bool bad = er[r] == NONFINITE_EXP || ejc == NONFINITE_EXP;
    double v;
    Wide x{};
    unsigned long long m = 0;
    int k = 0;
    if (p.res_x == nullptr) {
      v = round_wide(u3, u2, u1, u0, sign, e);
    } else {
      x.hi = ((unsigned long long)u3 << 32) | u2;
      x.lo = ((unsigned long long)u1 << 32) | u0;
      x.neg = sign != 0;
      m = leading53(x, k);
      v = to_f64(m, k + e, x.neg);
    }
    if (bad) v = __longlong_as_double(0x7ff8000000000000ll);
    if (p.res_x != nullptr && ib + r < p.M) {
      // The rest of the exact product below its leading 53 bits.
      unsigned __int128 u = ((unsigned __int128)x.hi << 64) | x.lo;
      const unsigned __int128 head = k >= 0 ? (unsigned __int128)m << k : (unsigned __int128)m >> -k;
      const __int128 rest = (__int128)(u - head);
      const unsigned __int128 ra = rest < 0 ? (unsigned __int128)-rest : (unsigned __int128)rest;
      const Wide rw{(unsigned long long)(ra >> 64), (unsigned long long)ra, (rest < 0) != x.neg};
      int k2;
      const unsigned long long m2 = leading53(rw, k2);
      const double lo = to_f64(m2, k2 + e, rw.neg);
      const int64_t at = ib + r + col * p.res_ldx;
      const double dg = p.res_d[(p.d_col ? col : (int64_t)(ib + r)) * p.res_dstride];
      const double xv = p.res_x[at];
      const double c = p.C[ib + r + col * p.ldc];
      const double pr = dg * xv, pe = fma(dg, xv, -pr);
      double t1, e1, t2, e2;
      two_sum(c, -v, t1, e1);
      two_sum(t1, -pr, t2, e2);
      if (!bad) v = t2 + (((e1 + e2) - pe) - lo);
    }
    buf[warp][r * FIN_PITCH + lane] = v;
  }
  __syncwarp();
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int ri = lane + 32 * r;
    const double v = buf[warp][(ri & 3) * FIN_PITCH + (ri >> 2)];
    if (i0 + ri < p.M) p.C[i0 + ri + col * p.ldc] = p.res_x != nullptr ? v : fma(p.alpha, v, cv[r]);
  }
}

// ---------------------------------------------------------------------------
// Host side.
// ---------------------------------------------------------------------------
int64_t pad_to(int64_t x, int64_t m) { return (x + m - 1) / m * m; }
size_t plane_bytes(int64_t rows, int64_t K) { return (size_t)pad_to(rows, BU) * (size_t)pad_to(K, BK) * 2; }

void stage_job(const Mat& X, const CrtStaged& st, Job* j) {
  j->X = static_cast<const double*>(X.p);
  j->si = X.t ? X.ld : 1;
  j->sk = X.t ? 1 : X.ld;
  j->rows = st.rows;
  j->K = st.K;
  j->tri = st.tri;
  j->bits = operand_bits(st.K);
  j->f = st.row_operand ? 1 : 0;
  j->e = st.e;
  j->out = static_cast<uint16_t*>(st.res);
  j->rows_pad = st.rows_pad;
  j->K_pad = st.K_pad;
}

}  // namespace

// With short K the residues' planes and their reconstruction outweigh the
// products that they save, once C is large: slices against residues, us, K = 64,
// 128, 192, 256: 4000 x 4000 219 / 293, 262 / 317, 307 / 331, 351 / 345, 128 x 100000
// 240 / 303, 322 / 360, 412 / 444, 491 / 523; but 2000 x 2000 78 / 90, 94 / 98, 113 /
// 106 and 20000 x 64 74 / 57, 98 / 74.
bool crt_wanted(int64_t M, int64_t N, int64_t K) {
  const double c = (double)pad_to(M, BU) * (double)pad_to(N, BU);
  return K >= 256 || c <= 3e6 || c <= 31250.0 * (double)K;
}

// Sizes that the residues' integers, grids and maps hold.
bool crt_usable(int64_t M, int64_t N, int64_t K) {
  return K <= MAX_K && M <= (1 << 24) && N <= (1 << 24) && L * pad_to(M, BU) < INT32_MAX && L * pad_to(N, BU) < INT32_MAX &&
         pad_to(M, BU) / BU * (pad_to(N, BU) / BU) * L < INT32_MAX && N <= (int64_t)65535 * 8;
}

size_t crt_staged_bytes(int64_t rows, int64_t K) {
  return L * plane_bytes(rows, K) + (((size_t)pad_to(rows, BU) * sizeof(int) + 1023) & ~(size_t)1023);
}
size_t crt_planes_bytes(int64_t M, int64_t N) { return (size_t)L * (size_t)pad_to(M, BU) * (size_t)N; }

// Residues take 32 bytes per element and the planes 16 per element of C,
// against the slices' 14 and 8, and the workspaces are kept between calls: a
// whole 16384 x 16384 solve held 8.6 GB instead of 3.9.  So residues are
// formed in panels within what slices would take (or the stream holds already,
// or 1 GiB).  That solve takes 72.0 ms whole and 72.4 in panels.
constexpr int64_t PANEL_MIN = 1024;
CrtPanels crt_panels(bool cols, int64_t M, int64_t N, int64_t K, size_t budget) {
  const int64_t dim = cols ? N : M;
  const size_t fixed = crt_staged_bytes(cols ? M : N, K) + 1024;
  auto need = [&](int64_t w) {
    return fixed + crt_staged_bytes(w, K) + (cols ? crt_planes_bytes(M, w) : crt_planes_bytes(w, N));
  };
  if (dim <= PANEL_MIN || need(dim) <= budget) return {cols, dim, need(dim)};
  int64_t w = PANEL_MIN;
  while (w + PANEL_MIN < dim && need(w + PANEL_MIN) <= budget) w += PANEL_MIN;
  const int64_t panels = (dim + w - 1) / w;
  w = pad_to((dim + panels - 1) / panels, 256);  // of about equal width
  return {cols, w, need(w)};
}

size_t crt_budget(size_t slices_bytes, size_t held) {
  constexpr size_t FLOOR = (size_t)1 << 30;
  const size_t b = slices_bytes > held ? slices_bytes : held;
  return b > FLOOR ? b : FLOOR;
}

CrtStaged crt_layout(void* buf, int64_t rows, int64_t K, int tri, bool row_operand) {
  CrtStaged st;
  st.res = buf;
  st.e = reinterpret_cast<int*>(static_cast<uint8_t*>(buf) + L * plane_bytes(rows, K));
  st.rows = rows;
  st.rows_pad = pad_to(rows, BU);
  st.K = K;
  st.K_pad = pad_to(K, BK);
  st.tri = tri;
  st.row_operand = row_operand;
  return st;
}

// Stages one or two operands (Y may be null) in as few launches as K allows.
int crt_stage(const Mat& X, const CrtStaged& sx, const Mat* Y, const CrtStaged* sy, cudaStream_t s) {
  Job a{}, b{};
  stage_job(X, sx, &a);
  if (Y) stage_job(*Y, *sy, &b);
  const int ba = (int)(sx.rows_pad / 32), bb = Y ? (int)(sy->rows_pad / 32) : 0;
  const int64_t kmax = Y ? (sx.K_pad > sy->K_pad ? sx.K_pad : sy->K_pad) : sx.K_pad;
  double elems = (double)sx.rows * (double)sx.K;
  if (Y) elems += (double)sy->rows * (double)sy->K;
  TraceScope trace(NLA_K_SPLIT, s, 0.0, elems * (16.0 + 2.0 * L));
  if (kmax <= 256) {
    launch_chained(crt_stage_kernel, (unsigned)(ba + bb), 256, 0, s, a, b, ba);
    NLA_CHECK_LAUNCH("crt_stage_kernel");
    return NLA_OK;
  }
  cudaMemsetAsync(sx.e, 0x80, (size_t)sx.rows_pad * sizeof(int), s);
  if (Y) cudaMemsetAsync(sy->e, 0x80, (size_t)sy->rows_pad * sizeof(int), s);
  const dim3 grid((unsigned)(ba + bb), (unsigned)(kmax / 64));
  launch_chained(crt_exp_kernel, grid, 256, 0, s, a, b, ba);
  NLA_CHECK_LAUNCH("crt_exp_kernel");
  launch_chained(crt_split_kernel, grid, 256, 0, s, a, b, ba);
  NLA_CHECK_LAUNCH("crt_split_kernel");
  trace_kernels(1);
  return NLA_OK;
}

// C (A.rows x B.rows) += alpha A B^T, or with res the residual form; planes
// holds crt_planes_bytes.  One of A and B was staged as the row operand (the
// factor of the reconstruction; products commute, so either may be).  d_col:
// the residual's diagonal belongs to C's columns (B is the staged triangle).
int crt_gemm(const CrtStaged& A, const CrtStaged& B, double alpha, const Mat& C, uint8_t* planes, cudaStream_t s,
             const ResidualTerm* res, bool d_col) {
  if (A.row_operand == B.row_operand) return fail(NLA_ERR_ARG, "exact update: operands not staged for each other");
  GemmArgs g{};
  g.M = (int)A.rows;
  g.N = (int)B.rows;
  g.K = (int)A.K;
  g.bv = A.rows_pad > 128 ? BV : 128;
  g.stage_bytes = U_BYTES + g.bv * BK * 2;
  g.stages = RING_BYTES / g.stage_bytes;
  g.tiles_u = (int)(B.rows_pad / BU);
  g.tiles_v = (int)((A.rows_pad + g.bv - 1) / g.bv);
  g.items = L * g.tiles_u * g.tiles_v;
  g.rows_u = (int)B.rows_pad;
  g.rows_v = (int)A.rows_pad;
  g.tri_u = B.tri;
  g.tri_v = A.tri;
  g.planes = planes;
  g.ldp = A.rows_pad;
  g.plane = A.rows_pad * B.rows;
  g.err = device_error_word();
  if (!g.err) return fail(NLA_ERR_UNSUPPORTED, "exact update: no device error word");
  CUtensorMap mU, mV;
  NLA_TRY(staged_map(&mU, B.res, (uint64_t)B.K_pad, (uint64_t)(L * B.rows_pad), BU));
  // A 256-row box past a plane's padding reads the next plane (or zeros past
  // the last one): those rows of C are not stored.
  NLA_TRY(staged_map(&mV, A.res, (uint64_t)A.K_pad, (uint64_t)(L * A.rows_pad), (uint32_t)g.bv));
  static std::once_flag once;
  static cudaError_t st = cudaSuccess;
  std::call_once(once, [] {
    st = cudaFuncSetAttribute(crt_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
  });
  if (st != cudaSuccess) return cuda_status(st, "cudaFuncSetAttribute(crt_gemm_kernel)");
  const double tri_frac = A.tri != 0 || B.tri != 0 ? 0.5 : 1.0;
  TraceScope trace(NLA_K_GEMM_UMMA, s, 2.0 * (double)g.M * g.N * (double)g.K * L * tri_frac,
                   2.0 * L * (double)(A.rows_pad + B.rows_pad) * A.K_pad + (2.0 * L + 16.0) * (double)g.M * g.N);
  const int sms = num_sms();
  launch_chained(crt_gemm_kernel, (unsigned)(g.items < sms ? g.items : sms), THREADS, SMEM, s, mU, mV, g);
  NLA_CHECK_LAUNCH("crt_gemm_kernel");
  FinishArgs f{};
  f.planes = planes;
  f.plane = g.plane;
  f.ldp = g.ldp;
  f.M = g.M;
  f.N = g.N;
  f.ea = A.e;
  f.eb = B.e;
  f.e_bias = -2 * operand_bits(A.K);
  f.C = static_cast<double*>(C.p);
  f.ldc = C.ld;
  f.alpha = alpha;
  if (res) {
    f.res_x = res->x;
    f.res_ldx = res->ldx;
    f.res_d = res->d;
    f.res_dstride = res->dstride;
    f.d_col = d_col ? 1 : 0;
  }
  const dim3 grid((unsigned)(A.rows_pad / 128), (unsigned)((g.N + 7) / 8));
  launch_chained(crt_finish_kernel, grid, 256, 0, s, f);
  NLA_CHECK_LAUNCH("crt_finish_kernel");
  trace_kernels(1);
  return NLA_OK;
}

}  // namespace nla
