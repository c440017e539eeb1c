// Diagonal-block solve / multiply on strips of right-hand sides: one CTA of
// NW (8 or 16) warps takes CW right-hand sides through the whole n x n block
// (canonical lower-left form, nla_leaf.cuh).
//
// What bounds it.  Float64: the DFMA pipe (2 per clock per SM, one warp
// instruction per 16 clocks) once every SM has a strip; Float32 and Float16
// (computed in Float32): shared-memory operand reads.  With few right-hand
// sides it is the serial chain of the triangle.  So the strip is as narrow
// as it takes to give every SM one (2 columns at least), and where strips
// are narrower than the CTA's warps, the warps split the K range of the
// product (KG groups) instead of the columns.
//
// Layout.  The block is walked in panels of PB = 16 or 32 rows,
// left-looking: a lane holds one row (lane % PB) of NC columns, the halves
// of a warp different columns when PB = 16.
//   1. acc = A[p0:p0+PB, 0:p0] X[0:p0, :], A staged through shared memory in
//      chunks of KC columns, loaded into registers one chunk ahead, both
//      operands read from shared memory as 16-byte vectors along K;
//   2. y = X[p0+row] - acc, then the panel's triangle, each of its PB - 1
//      steps one product with the row's reciprocal, one shuffle and one FMA.
//      (Scaling the rows by their reciprocals first, as src/trsm.jl:15-27
//      does, would leave the shuffle and the FMA, but rounds every
//      coefficient once more: 1.4 times the Float64 error at 96 rows.)
//      32-row panels have half the fixed steps (staging, barriers, sums),
//      16-row panels half the idle lanes of the triangle, which count on the
//      DFMA pipe.
// With KG = 1 a warp owns its columns: only the staging of A needs a
// barrier, one per chunk.  X stays in shared memory (column-major), so the
// right-hand sides are read and written once.
#pragma once

#include <type_traits>

#include "nla_cplx.cuh"
#include "nla_leaf.cuh"

namespace nla {
namespace leafdev {

constexpr int ST_ROWS = 32;  // the strip's rows are padded to a multiple of this

template <typename Tc> struct StripTraits;
// VK: elements of a 16-byte vector.
template <> struct StripTraits<double> {
  using Vec = double2;
  static constexpr int VK = 2;
};
template <> struct StripTraits<float> {
  using Vec = float4;
  static constexpr int VK = 4;
};
template <> struct StripTraits<cx::cpx<float>> {
  using Vec = float4;
  static constexpr int VK = 2;
};
template <> struct StripTraits<cx::cpx<double>> {
  using Vec = double2;
  static constexpr int VK = 1;
};
constexpr int ST_KC = 128;  // columns of A per chunk
__device__ __forceinline__ void st_unpack(const double2& v, double* o) { o[0] = v.x; o[1] = v.y; }
__device__ __forceinline__ void st_unpack(const float4& v, float* o) { o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w; }

__device__ __forceinline__ void st_unpack(const float4& v, cx::cpx<float>* o) {
  o[0] = cx::mk(v.x, v.y);
  o[1] = cx::mk(v.z, v.w);
}
__device__ __forceinline__ void st_unpack(const double2& v, cx::cpx<double>* o) { o[0] = cx::mk(v.x, v.y); }

// The arithmetic of the strip, real and complex.
template <typename Tc> struct StripMath {
  __device__ static Tc zero() { return Tc(0); }
  __device__ static Tc one() { return Tc(1); }
  __device__ static Tc conj_if(Tc a, int) { return a; }
  __device__ static Tc fma_(Tc a, Tc x, Tc c) { return fma(a, x, c); }
  __device__ static Tc fms_(Tc a, Tc x, Tc c) { return fma(-a, x, c); }
  __device__ static Tc shfl(Tc v, int src) { return __shfl_sync(0xffffffffu, v, src); }
  __device__ static Tc inverse(Tc d) { return Tc(1) / d; }
  // z / d with inv = 1 / d.
  __device__ static Tc quotient(Tc z, Tc inv, Tc) { return z * inv; }
  __device__ static Tc divided(Tc z, Tc inv, Tc) { return z * inv; }
};
template <typename R> struct StripMath<cx::cpx<R>> {
  using Tc = cx::cpx<R>;
  __device__ static Tc zero() { return cx::zero<R>(); }
  __device__ static Tc one() { return cx::mk(R(1), R(0)); }
  __device__ static Tc conj_if(Tc a, int c) { return cx::conj_if(a, c != 0); }
  __device__ static Tc fma_(Tc a, Tc x, Tc c) { return cx::fma_c(a, x, c); }
  __device__ static Tc fms_(Tc a, Tc x, Tc c) { return cx::fms_c(a, x, c); }
  __device__ static Tc shfl(Tc v, int src) {
    return cx::mk(__shfl_sync(0xffffffffu, v.re, src), __shfl_sync(0xffffffffu, v.im, src));
  }
  __device__ static Tc inverse(Tc d) { return cx::div(one(), d); }
  // The product with the reciprocal, corrected once by the remainder: as
  // accurate as the quotient itself (a complex reciprocal carries several
  // roundings), without a division in the triangle's chain.  Where the
  // reciprocal or the quotient overflows it is not finite; strip_block then
  // solves the panel again by divisions.
  __device__ static Tc quotient(Tc z, Tc inv, Tc d) {
    const Tc q = cx::fma_c(z, inv, zero());
    return cx::fma_c(cx::fms_c(q, d, z), inv, q);
  }
  __device__ static bool finite(Tc a) { return isfinite(a.re) && isfinite(a.im); }
  __device__ __noinline__ static Tc divided(Tc z, Tc, Tc d) { return cx::div(z, d); }
};

template <typename T> __device__ __forceinline__ T raw_zero() { return T(0.0f); }
template <> __device__ __forceinline__ cx::cpx<float> raw_zero() { return cx::zero<float>(); }
template <> __device__ __forceinline__ cx::cpx<double> raw_zero() { return cx::zero<double>(); }

// Column pitch of X: a multiple of the vector, at least n.
template <typename Tc> __host__ __device__ constexpr int st_ldx(int n) {
  constexpr int VK = StripTraits<Tc>::VK;
  return ((n + ST_ROWS - 1) / ST_ROWS * ST_ROWS) + VK;  // panels are stored whole; the pad staggers the banks
}
template <typename Tc> __host__ __device__ constexpr int st_lda() { return ST_KC + StripTraits<Tc>::VK; }

// PB rows per panel, NW warps, WC of them across the columns with 32 / PB NC
// columns each.
template <typename Tc> __host__ __device__ constexpr size_t strip_smem_elems(int n, int PB, int NC, int WC, int NW) {
  return (size_t)(32 / PB) * NC * WC * st_ldx<Tc>(n)              // X
         + (size_t)2 * PB * st_lda<Tc>()                          // A chunks
         + (size_t)2 * PB * (PB + 1)                              // panel triangles
         + (size_t)2 * ((n + ST_ROWS - 1) / ST_ROWS * ST_ROWS)    // the diagonal and its reciprocals
         + (WC < NW ? (size_t)NW * NC * 32 : 0);                  // partial sums of the K groups
}

// CW = (32 / PB) NC WC columns per CTA: WC warps across them, KG = NW / WC across K.
template <typename T, int PB, int NC, int WC, int NW, bool SOLVE>
__device__ __forceinline__ void strip_block(const LeafArgs& g, unsigned char* smem_raw) {
  using Tc = typename Elem<T>::compute;
  using Tr = StripTraits<Tc>;
  using Vec = typename Tr::Vec;
  using Mx = StripMath<Tc>;
  constexpr int ST_THREADS = 32 * NW;
  constexpr int KC = ST_KC, VK = Tr::VK, KG = NW / WC, SUBS = 32 / PB, CW = SUBS * NC * WC;
  constexpr int DPER = (PB * PB + ST_THREADS - 1) / ST_THREADS;  // triangle elements per thread
  constexpr int LDA = st_lda<Tc>();
  constexpr int PER = PB * KC / ST_THREADS;  // chunk elements per thread
  const int n = g.n, ldx = st_ldx<Tc>(n), nr = (n + ST_ROWS - 1) / ST_ROWS * ST_ROWS;
  Tc* X = reinterpret_cast<Tc*>(smem_raw);          // CW columns of ldx
  Tc* As = X + (size_t)CW * ldx;                    // 2 x PB x LDA
  Tc* Dg = As + 2 * PB * LDA;                    // 2 x PB x (PB + 1)
  Tc* inv = Dg + 2 * PB * (PB + 1);           // nr
  Tc* dia = inv + nr;                               // nr
  Tc* part = dia + nr;                              // KG > 1: NW warps x NC x 32
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int row = lane & (PB - 1), sub = lane / PB;
  const int wc = warp % WC, kg = warp / WC;
  const int col0 = wc * SUBS * NC + sub * NC;  // this lane's columns col0 .. col0 + NC - 1
  const int64_t c0 = (int64_t)blockIdx.x * CW;
  const int ncols = (int)(g.m - c0 < CW ? g.m - c0 : CW);
  // Canonical element (i, k) of A at A[i si + k sk], (i, c) of the strip at
  // Bs[i bi + c bc]: strides once, so that an address is one multiply-add.
  const int64_t sk = (g.tA ? 1 : g.lda) * (g.rev ? -1 : 1), si = (g.tA ? g.lda : 1) * (g.rev ? -1 : 1);
  const T* A = static_cast<const T*>(g.A) + (g.rev ? (int64_t)(n - 1) * (g.lda + 1) : 0);
  const int64_t bi = (g.tB ? g.ldb : 1) * (g.rev ? -1 : 1), bc = g.tB ? 1 : g.ldb;
  T* B = static_cast<T*>(g.B) + (g.rev ? (int64_t)(n - 1) * (g.tB ? g.ldb : 1) : 0) + c0 * bc;

  // A chunk of the panel's rows, K columns k0 ..: slot e of a thread is
  // element (fi + e ei, fk + e ek), threads along the index that is
  // contiguous in memory.
  T ra[PER];  // as stored: converted when they go to shared memory, so that the loads stay together
  T rd[DPER];
  const int fi = g.tA ? t / KC : t & (PB - 1), fk = g.tA ? t & (KC - 1) : t / PB;
  const int ei = g.tA ? ST_THREADS / KC : 0, ek = g.tA ? 0 : ST_THREADS / PB;
  const int64_t es = g.tA ? ei * si : ek * sk;
  // Triangle slot e: element (di + e de, dk) for a transposed A, (di, dk + e de) otherwise.
  constexpr int de = ST_THREADS / PB;
  const int di = g.tA ? t / PB : t & (PB - 1), dk = g.tA ? t & (PB - 1) : t / PB;
  auto fetch = [&](int p0, int k0, int kend, bool diag) {
    const T* p = A + (p0 + fi) * si + (k0 + fk) * sk;
    const int ni = n - p0 - fi, nk = kend - k0 - fk;  // slots inside: e ei < ni, e ek < nk
#pragma unroll
    for (int e = 0; e < PER; ++e) ra[e] = e * ei < ni && e * ek < nk ? p[e * es] : raw_zero<T>();
    if (diag) {
#pragma unroll
      for (int e = 0; e < DPER; ++e) {
        const int i = g.tA ? di + e * de : di, k = g.tA ? dk : dk + e * de;
        rd[e] = p0 + i < n && k < i ? A[(p0 + i) * si + (p0 + k) * sk] : raw_zero<T>();
      }
    }
  };

  // Panels in order (SOLVE) with ceil(p0 / KC) chunks each, at least one step.
  // Multiplies take the panel's own columns into the chunks (K < p0 + PB).
  const int npan = (n + PB - 1) / PB;
  auto kend_of = [&](int p) { return SOLVE ? p * PB : min((p + 1) * PB, n); };
  auto chunks_of = [&](int p) { const int ke = kend_of(p); return ke > KC ? (ke + KC - 1) / KC : 1; };

  fetch(0, 0, kend_of(0), SOLVE && chunks_of(0) == 1);
  // The strip of B, several loads in flight per thread; zeros past the block.
  // Along the rows a warp takes columns warp, warp + NW, ...; along the
  // columns consecutive threads take consecutive columns.
  constexpr int BATCH = 8;
  if (!g.tB) {
    for (int c = warp; c < CW; c += NW)
      for (int i0 = lane; i0 < nr; i0 += 32 * BATCH) {
        T v[BATCH];
#pragma unroll
        for (int u = 0; u < BATCH; ++u) {
          const int i = i0 + 32 * u;
          v[u] = i < n && c < ncols ? B[i * bi + c * bc] : raw_zero<T>();
        }
#pragma unroll
        for (int u = 0; u < BATCH; ++u)
          if (i0 + 32 * u < nr) X[(size_t)c * ldx + i0 + 32 * u] = Elem<T>::load(&v[u]);
      }
  } else {
    constexpr int RS = ST_THREADS / CW;  // rows per pass
    const int c = t % CW;
    for (int i0 = t / CW; i0 < nr; i0 += RS * BATCH) {
      T v[BATCH];
#pragma unroll
      for (int u = 0; u < BATCH; ++u) {
        const int i = i0 + RS * u;
        v[u] = i < n && c < ncols ? B[i * bi + c] : raw_zero<T>();
      }
#pragma unroll
      for (int u = 0; u < BATCH; ++u)
        if (i0 + RS * u < nr) X[(size_t)c * ldx + i0 + RS * u] = Elem<T>::load(&v[u]);
    }
  }
  for (int i = t; i < nr; i += ST_THREADS) {
    const Tc d = g.unit || i >= n ? Mx::one() : Mx::conj_if(Elem<T>::load(A + i * (si + sk)), g.cj);
    dia[i] = d;
    if (SOLVE) inv[i] = Mx::inverse(d);
  }
  __syncthreads();

  Tc acc[NC];
  int step = 0;
  for (int p = 0; p < npan; ++p) {
    const int p0 = p * PB, kend = kend_of(p), nch = chunks_of(p);
#pragma unroll
    for (int q = 0; q < NC; ++q) acc[q] = Mx::zero();
    for (int ch = 0; ch < nch; ++ch, ++step) {
      const int k0 = ch * KC;
      Tc* Ab = As + (step & 1) * PB * LDA;
      Tc* Db = Dg + (step & 1) * PB * (PB + 1);
#pragma unroll
      for (int e = 0; e < PER; ++e) {
        const int i = fi + e * ei, k = fk + e * ek;
        Tc v = Mx::conj_if(Elem<T>::load(&ra[e]), g.cj);
        if (!SOLVE && k0 + k >= p0 + i) v = Mx::zero();  // strictly below the diagonal
        Ab[i * LDA + k] = v;
      }
      const bool last = ch + 1 == nch;
      if (SOLVE && last) {
#pragma unroll
        for (int e = 0; e < DPER; ++e) {
          const int i2 = g.tA ? di + e * de : di, k2 = g.tA ? dk : dk + e * de;
          Db[i2 * (PB + 1) + k2] = Mx::conj_if(Elem<T>::load(&rd[e]), g.cj);
        }
      }
      __syncthreads();
      if (!last) fetch(p0, k0 + KC, kend, SOLVE && ch + 2 == nch);
      else if (p + 1 < npan) fetch(p0 + PB, 0, kend_of(p + 1), SOLVE && chunks_of(p + 1) == 1);

      // Product: K units of one vector, dealt to the K groups in turn.
      const int kw = min(KC, kend - k0);
      const int units = kw > 0 ? (kw + VK - 1) / VK : 0;  // A is staged as zeros past kend, X holds zeros past n
      const Tc* ar = Ab + row * LDA;
      const Tc* xr = X + (size_t)col0 * ldx + k0;
      // Multiplies: units of the panel's own rows (from `own` on) take X only
      // left of the diagonal, so that no Inf or NaN from past it is used.
      const int own = SOLVE ? units : min(units, max(0, (p0 - k0) / VK));
      auto unit = [&](int u, bool mask) {
        Tc a[VK];
        st_unpack(*reinterpret_cast<const Vec*>(ar + u * VK), a);
#pragma unroll
        for (int q = 0; q < NC; ++q) {
          Tc x[VK];
          st_unpack(*reinterpret_cast<const Vec*>(xr + (size_t)q * ldx + u * VK), x);
#pragma unroll
          for (int v = 0; v < VK; ++v) {
            if (mask && k0 + u * VK + v >= p0 + row) x[v] = Mx::zero();
            acc[q] = Mx::fma_(a[v], x[v], acc[q]);
          }
        }
      };
      int u = kg;
#pragma unroll 4
      for (; u < own; u += KG) unit(u, false);
      if (!SOLVE)
#pragma unroll 2
        for (; u < units; u += KG) unit(u, true);
      if (last) {
        if constexpr (KG > 1) {
          if (kg > 0) {
#pragma unroll
            for (int q = 0; q < NC; ++q) part[(warp * NC + q) * 32 + lane] = acc[q];
          }
          __syncthreads();
        }
        if (kg == 0) {
          if constexpr (KG > 1) {
#pragma unroll
            for (int q = 0; q < NC; ++q) {
              Tc s[KG];
              s[0] = acc[q];
#pragma unroll
              for (int h = 1; h < KG; ++h) s[h] = part[((h * WC + wc) * NC + q) * 32 + lane];
#pragma unroll
              for (int w = 1; w < KG; w *= 2)
#pragma unroll
                for (int h = 0; h + w < KG; h += 2 * w) s[h] = s[h] + s[h + w];
              acc[q] = s[0];
            }
          }
          if constexpr (SOLVE) {
            const Tc iv = inv[p0 + row], dr = dia[p0 + row];
            Tc z[NC], d[PB - 1];
#pragma unroll
            for (int j = 0; j < PB - 1; ++j) d[j] = Db[row * (PB + 1) + j];  // zero on and above the diagonal
#pragma unroll
            for (int q = 0; q < NC; ++q) z[q] = X[(size_t)(col0 + q) * ldx + p0 + row] - acc[q];
#pragma unroll
            for (int j = 0; j < PB - 1; ++j)
#pragma unroll
              for (int q = 0; q < NC; ++q) {
                const Tc xj = Mx::shfl(Mx::quotient(z[q], iv, dr), (lane & ~(PB - 1)) | j);
                if (row > j) z[q] = Mx::fms_(d[j], xj, z[q]);
              }
            if constexpr (std::is_floating_point<Tc>::value) {
#pragma unroll
              for (int q = 0; q < NC; ++q) X[(size_t)(col0 + q) * ldx + p0 + row] = Mx::quotient(z[q], iv, dr);
            } else {
#pragma unroll
              for (int q = 0; q < NC; ++q) z[q] = Mx::quotient(z[q], iv, dr);
              // The chain's time is in its steps, so the test for results that
              // are not finite (a pivot without a finite reciprocal, a quotient
              // that overflows) comes once per panel; the divisions then give
              // what is finite, and infinities where there is none.
              bool again = false;
#pragma unroll
              for (int q = 0; q < NC; ++q) again |= !Mx::finite(z[q]);
              if (__any_sync(0xffffffffu, again)) {
#pragma unroll
                for (int q = 0; q < NC; ++q) z[q] = X[(size_t)(col0 + q) * ldx + p0 + row] - acc[q];
#pragma unroll 1
                for (int j = 0; j < PB - 1; ++j) {
                  const Tc dj = Db[row * (PB + 1) + j];
#pragma unroll
                  for (int q = 0; q < NC; ++q) {
                    const Tc xj = Mx::shfl(Mx::divided(z[q], iv, dr), (lane & ~(PB - 1)) | j);
                    if (row > j) z[q] = Mx::fms_(dj, xj, z[q]);
                  }
                }
#pragma unroll
                for (int q = 0; q < NC; ++q) z[q] = Mx::divided(z[q], iv, dr);
              }
#pragma unroll
              for (int q = 0; q < NC; ++q) X[(size_t)(col0 + q) * ldx + p0 + row] = z[q];
            }
            if constexpr (KG == 1) __syncwarp();
          } else {
#pragma unroll
            for (int q = 0; q < NC; ++q) {
              // The diagonal's product last, on the whole sum: usually the
              // largest term, so the row is rounded at its size once.
              const Tc y = Mx::fma_(dia[p0 + row], X[(size_t)(col0 + q) * ldx + p0 + row], acc[q]);
              if (p0 + row < n && col0 + q < ncols) Elem<T>::store(B + (p0 + row) * bi + (col0 + q) * bc, y);
            }
          }
        }
      }
    }
  }
  if (SOLVE) {
    __syncthreads();
    if (!g.tB) {
      for (int c = warp; c < ncols; c += NW)
        for (int i = lane; i < n; i += 32) Elem<T>::store(B + i * bi + c * bc, X[(size_t)c * ldx + i]);
    } else if (t % CW < ncols) {
      for (int i = t / CW; i < n; i += ST_THREADS / CW)
        Elem<T>::store(B + i * bi + t % CW, X[(size_t)(t % CW) * ldx + i]);
    }
  }
}

}  // namespace leafdev
}  // namespace nla
