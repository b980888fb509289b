// Shared-memory building blocks for nb x nb diagonal blocks (nb <= 128):
// blocked Cholesky, triangular inverse and register-blocked mini-GEMMs.
#pragma once
#include "internal.h"

namespace egpu {

// ---------------------------------------------------------------------------
// Diagonal-block kernels.  The nb x nb block (nb <= 128) lives in shared
// memory with leading dimension kLDS = 132 (4 mod 16: the 8-byte DMMA
// fragment loads, rows g + 8.. x columns t + 4.., hit 16 distinct bank pairs
// per half warp; even, so every column starts on a 16-byte boundary for
// 16-byte copies), always as a LOWER triangle (an upper triangle is
// handled as the lower triangle of its transpose: UVar3Unb and LVar3Unb
// perform the same operations on A and A^T).
//
// What bounds them: dependent chains run by one warp (the 16-column leaves),
// so the leaf loops are written for a short chain per column and for few
// instructions: rolled, with the registers rotating by one column per step as
// part of the update itself.  Unrolled leaves (170 KB of code in one kernel)
// spent their time fetching instructions.
constexpr int kLDS = 132;
constexpr int kDiagSmemBase = (128 * kLDS + 128) * (int)sizeof(double);

template <typename T>
__device__ __forceinline__ T& SE(T* S, int r, int c) { return S[r + c * kLDS]; }

// ------------------------------------------------------------ pivot search --
constexpr int kNoPos = 0x7fffffff;  // "no row": a lane that does not take part

// |a| as a key whose unsigned order is the order of |a| (non-negative doubles)
__device__ __forceinline__ unsigned long long abs_key(double v) {
  return (unsigned long long)__double_as_longlong(fabs(v));
}

// The rare part of warp_argmax, out of line (the column loops are short of
// instruction-cache room): the upper halves tie.
static __device__ __noinline__ unsigned warp_argmax_tie(bool c, unsigned lo, int pos) {
  const unsigned ml = __reduce_max_sync(0xffffffffu, c ? lo : 0u);
  const unsigned r = __reduce_min_sync(0xffffffffu, c && lo == ml ? (unsigned)pos : (unsigned)kNoPos);
  return __ballot_sync(0xffffffffu, c && lo == ml && (unsigned)pos == r);
}

// Lane of the first maximal key over the lanes with pos != kNoPos, ties to
// the lowest position; -1 when no lane takes part.
__device__ __forceinline__ int warp_argmax(unsigned long long key, int pos) {
  const bool in = pos != kNoPos;
  const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
  const unsigned mh = __reduce_max_sync(0xffffffffu, in ? hi : 0u);
  unsigned m = __ballot_sync(0xffffffffu, in && hi == mh);
  if (__popc(m) > 1) m = warp_argmax_tie(in && hi == mh, lo, pos);  // warp-uniform
  return __ffs(m) - 1;
}

// ---------------------------------------------------------------------------
// Building blocks on shared-memory operands (all column-major).

// Columns [J0, J0 + 8) of warp_chol16 (NW: the columns after the current one
// that can still be needed, 15 or 7).
template <int NW>
__device__ __forceinline__ void warp_chol16_cols(double (&z)[16], double& d, double& mine, int& fail, int j0, bool inv,
                                                 int i, double* Sd, int lds, double* Xd, double* buf) {
#pragma unroll 1
  for (int j = j0; j < j0 + 8; ++j) {
    double* cb = buf + (j & 1) * 16;  // two slots: a slow lane may still read the other one
    if (!inv && i > j) cb[i - j - 1] = z[0];
    const double dn = __shfl_sync(0xffffffffu, z[1], (j + 1) & 15);
    __syncwarp();
    double c[NW + 1];  // a_{j+1+k, j}; entries past the block are stale and only reach columns past it
#pragma unroll
    for (int q = 0; q < (NW + 1) / 2; ++q) {
      const double2 v = *reinterpret_cast<const double2*>(cb + 2 * q);
      c[2 * q] = v.x;
      c[2 * q + 1] = v.y;
    }
    const double rs = rsqrt(d);
    if (fail == 0 && d <= 0.0) fail = j + 1;
    if (i == j) mine = d;
    c[0] *= rs;
    d = fma(-c[0], c[0], dn);
    const double m = z[0] * rs;
#pragma unroll
    for (int k = 1; k < NW; ++k) c[k] *= rs;
#pragma unroll
    for (int k = 0; k < NW; ++k) z[k] = fma(-m, c[k], z[k + 1]);
    if (inv) Xd[j] = m;
    else if (i > j) Sd[j * lds] = m;
  }
}

// Cholesky of one 16 x 16 lower block at S[o.., o..] (LVar3Unb,
// Cholesky/LVar3.hpp:19-49) and the inverse of its factor (into X, 16 x 16, ld
// ldx, zero above the diagonal) by one warp, in one loop over the columns.
// Lane i < 16 holds row i of the block, lane 16 + c column c of the identity;
// register 0 is the current column.  Step j, with the raw column a_kj
// broadcast through shared memory and d = a_jj, is the same for both halves:
// m = z_0 / sqrt(d) is the finished entry of the factor (of its inverse), and
// z_k -= m l_kj, l_kj = a_kj / sqrt(d) formed by every lane for itself, is the
// update of A22 (the forward substitution with the factor).  The chain per
// column is one reciprocal square root, one multiply and one FMA (55 + 23 + 23
// cycles here): the broadcast precedes the square root, and the next pivot is
// formed by every lane from a copy of a_{j+1,j+1} fetched beforehand.  The
// diagonal keeps the pivots: who stores the factor takes their roots, all of a
// block's side by side (here, one root per leaf, 230 cycles).  d times the
// reciprocal root would be up to an ulp off, and NaN for an infinite pivot
// (whose column is 0 and whose row of the inverse is 0).
// Measured per block, alone on the SM: 7000 cycles with the reciprocal, the
// root and the failure test in the chain one after the other.
// buf: 32 doubles of shared memory, 16-byte aligned, of this warp.
// Returns 0 or the 1-based column of a non-positive pivot (warp-uniform).
__device__ inline int warp_chol16(double* S, int lds, int o, double* X, int ldx, double* buf) {
  const int lane = threadIdx.x & 31, i = lane & 15;
  const bool inv = lane >= 16;
  double* Sd = S + (o + i) + o * lds;
  double z[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) z[k] = inv ? (k == i ? 1.0 : 0.0) : (k <= i ? Sd[k * lds] : 0.0);
  double d = __shfl_sync(0xffffffffu, z[0], 0), mine = 1.0;
  int fail = 0;
  warp_chol16_cols<15>(z, d, mine, fail, 0, inv, i, Sd, lds, X + i * ldx, buf);
  warp_chol16_cols<7>(z, d, mine, fail, 8, inv, i, Sd, lds, X + i * ldx, buf);
  if (!inv) Sd[i * lds] = mine;
  __syncwarp();
  return fail;
}

// Inverse of one 16 x 16 lower block at S[o.., o..] (unit: diagonal taken as
// 1) by one warp, into X (ld ldx): lane c < 16 forms column c by forward
// substitution, x_j = z_0 / l_jj, z_k -= l_kj x_j, register 0 the current row.
// The 16 reciprocals of the diagonal are formed in parallel, one per lane.
__device__ inline void warp_trinv16(const double* S, int lds, int o, int unit, double* X, int ldx) {
  const int lane = threadIdx.x & 31;
  const double rinv = (unit || lane >= 16) ? 1.0 : 1.0 / S[(o + lane) + (o + lane) * lds];
  double z[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) z[k] = (k == lane) ? 1.0 : 0.0;
#pragma unroll 1
  for (int j = 0; j < 16; ++j) {
    const double* col = S + (o + j + 1) + (o + j) * lds;  // rows past the block only reach rows past it
    const double x = z[0] * __shfl_sync(0xffffffffu, rinv, j);
#pragma unroll
    for (int k = 0; k < 15; ++k) z[k] = fma(-col[k], x, z[k + 1]);
    z[15] = 0.0;
    if (lane < 16) X[j + lane * ldx] = x;
  }
}

// Temporary area of the DMMA diagonal kernels: 8 leaf inverses and
// one 64 x 64 product buffer (ld 68).
constexpr int kLeafLD = 20;  // 4 mod 16, as the block itself
constexpr int kTmpLD = 68;
constexpr int kDiagTmpDoubles = 8 * 16 * kLeafLD + 64 * kTmpLD;
constexpr int kDiagSmem = kDiagSmemBase + kDiagTmpDoubles * (int)sizeof(double);

// Flat (one pass, all copies in flight) transfers of a b x b triangle between
// global memory and S; a column-by-column loop costs one memory round trip
// per column.  `upper`: the global block holds the triangle transposed
// (S(r, c) = G[c + r ld]); consecutive threads always take consecutive
// global addresses.
__device__ inline void tri_load_async(double* S, const double* G, long long ld, int b, bool upper) {
  // a warp per column j, lanes over rows; 16-byte copies when G's columns are
  // 16-byte aligned (the copy may start one row above the diagonal: S's
  // strict upper triangle is never read)
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const bool vec = !upper && (ld % 2 == 0) && (reinterpret_cast<uintptr_t>(G) % 16 == 0);
  for (int j = warp; j < b; j += nw) {
    const double* g = G + (long long)j * ld;
    if (vec) {
      for (int i = (j & ~1) + 2 * lane; i < b; i += 64) {
        if (i + 1 < b) cp_async16_cg(&S[i + j * kLDS], &g[i]);
        else cp_async8(&S[i + j * kLDS], &g[i]);
      }
    } else if (!upper) {
      for (int i = j + lane; i < b; i += 32) cp_async8(&S[i + j * kLDS], &g[i]);
    } else {
      for (int i = lane; i <= j; i += 32) cp_async8(&S[j + i * kLDS], &g[i]);  // G(i, j), i <= j
    }
  }
}
// Lower triangle of S (r >= c) into G; the other triangle of the b x b block
// is written as zero when `zero_other`, else left alone.
__device__ inline void tri_store(const double* S, double* G, long long ld, int b, bool upper, bool zero_other) {
  // a warp per column j of G, lanes over rows i; 16-byte stores when aligned
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const bool vec = !upper && (ld % 2 == 0) && (reinterpret_cast<uintptr_t>(G) % 16 == 0);
  for (int j = warp; j < b; j += nw) {
    double* g = G + (long long)j * ld;
    if (vec) {
      const double* s = S + j * kLDS;
      for (int i = (zero_other ? 0 : (j & ~1)) + 2 * lane; i < b; i += 64) {
        const double v0 = i >= j ? s[i] : 0.0;
        if (i + 1 < b && (i >= j || zero_other)) {
          *reinterpret_cast<double2*>(&g[i]) = make_double2(v0, i + 1 >= j ? s[i + 1] : 0.0);
        } else {
          if (i >= j || zero_other) g[i] = v0;
          if (i + 1 < b) g[i + 1] = s[i + 1];  // i + 1 == j: on the diagonal
        }
      }
    } else {
      for (int i = lane; i < b; i += 32) {
        const int r = upper ? j : i, c = upper ? i : j;  // S coordinates
        if (r >= c) g[i] = S[r + c * kLDS];
        else if (zero_other) g[i] = 0.0;
      }
    }
  }
}

// Pad the lower b x b triangle in S to bp = round_up(b, 16) with identity.
__device__ inline int pad16_identity(double* S, int b) {
  const int bp = (b + 15) & ~15;
  for (int e = threadIdx.x; e < (bp - b) * bp; e += blockDim.x) {
    const int r = b + e / bp, c = e % bp;  // rows b..bp-1, all columns
    if (r >= c) S[r + c * kLDS] = (r == c) ? 1.0 : 0.0;
  }
  return bp;
}

// One 16 x 16 tile (two 16 x 8 DMMA columns) of a product of shared-memory
// operands by one warp, k in [kbeg, kend): C = alpha A op(B).  A_LOWER /
// B_LOWER: A (B) is zero above its diagonal and what is stored there is not
// used.  B_TRANS: op(B) = B^T.  C may be A (this tile's rows and k columns):
// every lane has read before any writes.
template <bool A_LOWER, bool B_LOWER, bool B_TRANS = false>
__device__ __forceinline__ void smem_dmma_tile16(const double* A, int lda, const double* B, int ldb, double* C,
                                                 int ldc, int r0, int c0, int kbeg, int kend, double alpha) {
  static_assert(!(B_LOWER && B_TRANS), "not needed");
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  double acc0[4] = {0.0, 0.0, 0.0, 0.0}, acc1[4] = {0.0, 0.0, 0.0, 0.0};
  const int ra = r0 + g, rb = r0 + g + 8, ca = c0 + g, cb = c0 + g + 8;
#pragma unroll 2
  for (int k0 = kbeg; k0 < kend; k0 += 8) {
    const int ka = k0 + t, kb = k0 + t + 4;
    double a[4], b0[2], b1[2];
    a[0] = (!A_LOWER || ka <= ra) ? A[ra + ka * lda] : 0.0;
    a[1] = (!A_LOWER || ka <= rb) ? A[rb + ka * lda] : 0.0;
    a[2] = (!A_LOWER || kb <= ra) ? A[ra + kb * lda] : 0.0;
    a[3] = (!A_LOWER || kb <= rb) ? A[rb + kb * lda] : 0.0;
    b0[0] = (!B_LOWER || ca <= ka) ? (B_TRANS ? B[ca + ka * ldb] : B[ka + ca * ldb]) : 0.0;
    b0[1] = (!B_LOWER || ca <= kb) ? (B_TRANS ? B[ca + kb * ldb] : B[kb + ca * ldb]) : 0.0;
    b1[0] = (!B_LOWER || cb <= ka) ? (B_TRANS ? B[cb + ka * ldb] : B[ka + cb * ldb]) : 0.0;
    b1[1] = (!B_LOWER || cb <= kb) ? (B_TRANS ? B[cb + kb * ldb] : B[kb + cb * ldb]) : 0.0;
    dmma_16x8x8(acc0, a, b0);
    dmma_16x8x8(acc1, a, b1);
  }
  __syncwarp();
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int r = r0 + g + ((q >= 2) ? 8 : 0), c = c0 + 2 * t + (q & 1);
    C[r + c * ldc] = alpha * acc0[q];
    C[r + (c + 8) * ldc] = alpha * acc1[q];
  }
}

// In-place inverse of the lower bp x bp triangle in S (bp a multiple of 16,
// padded with identity), given the inverses of its 16 x 16 diagonal blocks in
// Xl (block q at Xl + q*16*kLeafLD).  Levels of doubling block size:
//   inv([[A, 0], [B, C]]) = [[Ai, 0], [-Ci B Ai, Ci]],  T = B Ai, X21 = -Ci T.
// All pairs of a level run side by side (their T's, s x s with ld s + 4, fit
// the 64 x 68 buffer at every level), so the inverse of a 128 block costs six
// CTA barriers.
__device__ inline void smem_trinv_dmma(double* S, int bp, const double* Xl, double* T) {
  const int warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  // leaves into place
  const int nleaf = bp / 16;
  for (int e = threadIdx.x; e < nleaf * 256; e += blockDim.x) {
    const int q = e >> 8, i = (e >> 4) & 15, k = e & 15;
    if (i >= k) S[(16 * q + i) + (16 * q + k) * kLDS] = Xl[q * 16 * kLeafLD + i + k * kLeafLD];
  }
  __syncthreads();
  for (int s = 16; s < bp; s *= 2) {
    const int n16 = s / 16, per = n16 * n16, ldt = s + 4;
    const int pairs = (bp + s - 1) / (2 * s);  // blocks at o = 2 s i with o + s < bp
#pragma unroll 1
    for (int e = warp; e < pairs * per; e += nw) {
      const int i = e / per, f = e - i * per, r0 = (f % n16) * 16, c0 = (f / n16) * 16, o = 2 * s * i;
      if (o + s + r0 >= bp) continue;
      // T = B * Ai, B = S[o+s.., o..], Ai = S[o.., o..] lower
      smem_dmma_tile16<false, true>(S + (o + s) + o * kLDS, kLDS, S + o + o * kLDS, kLDS, T + i * s * ldt, ldt, r0,
                                    c0, c0, s, 1.0);
    }
    __syncthreads();
#pragma unroll 1
    for (int e = warp; e < pairs * per; e += nw) {
      const int i = e / per, f = e - i * per, r0 = (f % n16) * 16, c0 = (f / n16) * 16, o = 2 * s * i;
      if (o + s + r0 >= bp) continue;
      // X21 = -Ci * T, Ci = S[o+s.., o+s..] lower
      smem_dmma_tile16<true, false>(S + (o + s) + (o + s) * kLDS, kLDS, T + i * s * ldt, ldt,
                                    S + (o + s) + o * kLDS, kLDS, r0, c0, 0, r0 + 16, -1.0);
    }
    __syncthreads();
  }
}

// C(r0.., c0..) -= A(r0.., 0..15) A(c0.., 0..15)^T on one 16 x 16 tile (both ld
// LD); on the diagonal (r0 == c0) only the lower triangle is written.  The
// products are summed before they meet C: adding them to C one by one rounds
// at C's size sixteen times (backward error of a factorization 3.0e-16 instead
// of 1.8e-16 at n = 100).
template <int LD = kLDS>
__device__ __forceinline__ void smem_syrk_tile16(const double* A, double* C, int r0, int c0) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  double acc[2][4], cc[2][4];
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      cc[h][q] = C[(r0 + g + ((q >= 2) ? 8 : 0)) + (c0 + 8 * h + 2 * t + (q & 1)) * LD];
      acc[h][q] = 0.0;
    }
  double a[2][4], b[2][2][2];
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const double* ak = A + (8 * u + t) * LD + g;
    a[u][0] = -ak[r0];
    a[u][1] = -ak[r0 + 8];
    a[u][2] = -ak[r0 + 4 * LD];
    a[u][3] = -ak[r0 + 8 + 4 * LD];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      b[u][h][0] = ak[c0 + 8 * h];
      b[u][h][1] = ak[c0 + 8 * h + 4 * LD];
    }
  }
#pragma unroll
  for (int u = 0; u < 2; ++u)
#pragma unroll
    for (int h = 0; h < 2; ++h) dmma_16x8x8(acc[h], a[u], b[u][h]);
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int r = r0 + g + ((q >= 2) ? 8 : 0), c = c0 + 8 * h + 2 * t + (q & 1);
      if (r0 != c0 || r >= c) C[r + c * LD] = cc[h][q] + acc[h][q];
    }
}

// L21 := A21 * X11^T in place (A21: m2 x 16 at P, ld kLDS, m2 % 16 == 0;
// X11: 16 x 16, ld kLeafLD): warp w takes 16-row tiles w, w + nw, ...; both
// 8-column halves stay in registers until the whole row tile is read.
__device__ inline void smem_l21_inplace(double* P, int m2, const double* X11) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  for (int rt = warp; rt < m2 / 16; rt += nw) {
    const int r0 = rt * 16;
    double acc0[4] = {0.0, 0.0, 0.0, 0.0}, acc1[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int k0 = 0; k0 < 16; k0 += 8) {
      double a[4], b0[2], b1[2];
      a[0] = P[(r0 + g) + (k0 + t) * kLDS];
      a[1] = P[(r0 + g + 8) + (k0 + t) * kLDS];
      a[2] = P[(r0 + g) + (k0 + t + 4) * kLDS];
      a[3] = P[(r0 + g + 8) + (k0 + t + 4) * kLDS];
      b0[0] = X11[g + (k0 + t) * kLeafLD];  // op(B)[k][c] = X11[c][k]
      b0[1] = X11[g + (k0 + t + 4) * kLeafLD];
      b1[0] = X11[(g + 8) + (k0 + t) * kLeafLD];
      b1[1] = X11[(g + 8) + (k0 + t + 4) * kLeafLD];
      dmma_16x8x8(acc0, a, b0);
      dmma_16x8x8(acc1, a, b1);
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int r = r0 + g + ((q >= 2) ? 8 : 0), c = 2 * t + (q & 1);
      P[r + c * kLDS] = acc0[q];
      P[r + (c + 8) * kLDS] = acc1[q];
    }
  }
}

// Lower Cholesky of the bp x bp block in S (bp a multiple of 16; the caller
// pads with identity) in 16-column steps, the diagonal 16 x 16 leaves
// factored and inverted by one warp (X11 into Xl), L21 = A21 X11^T and the
// trailing update A22 -= L21 L21^T on the tensor cores.  Look-ahead: while
// warps 1.. update the rest of A22, warp 0 updates the next diagonal leaf
// first and factors it.  The diagonal keeps the pivots (see warp_chol16).
// Returns 0 or the 1-based column of a non-positive pivot (uniform).
__device__ inline int smem_chol_dmma(double* S, int bp, double* Xl) {
  __shared__ int s_fail;
  __shared__ __align__(16) double s_col[32];
  const int warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  if (warp == 0) {
    const int f = warp_chol16(S, kLDS, 0, Xl, kLeafLD, s_col);
    if (threadIdx.x == 0) s_fail = f;
  }
  __syncthreads();
  for (int o = 0; o < bp; o += 16) {
    if (s_fail) return s_fail;
    const int m2 = bp - o - 16;
    if (m2 <= 0) break;
    double* L21 = S + (o + 16) + o * kLDS;
    double* A22 = S + (o + 16) + (o + 16) * kLDS;
    smem_l21_inplace(L21, m2, Xl + (o / 16) * 16 * kLeafLD);
    __syncthreads();
    if (warp == 0) {
      smem_syrk_tile16(L21, A22, 0, 0);
      __syncwarp();
      const int f = warp_chol16(S, kLDS, o + 16, Xl + ((o + 16) / 16) * 16 * kLeafLD, kLeafLD, s_col);
      if (threadIdx.x == 0) s_fail = f ? o + 16 + f : 0;
    } else {
      const int nt = m2 / 16;
#pragma unroll 1
      for (int e = warp; e < nt * (nt + 1) / 2; e += nw - 1) {  // tile 0 is warp 0's
        int ti = (int)((sqrtf(8.0f * e + 1.0f) - 1.0f) * 0.5f);  // e = ti (ti + 1) / 2 + tj, ti >= tj
        while ((ti + 1) * (ti + 2) / 2 <= e) ++ti;
        while (ti * (ti + 1) / 2 > e) --ti;
        smem_syrk_tile16(L21, A22, 16 * ti, 16 * (e - ti * (ti + 1) / 2));
      }
    }
    __syncthreads();
  }
  return s_fail;
}

}  // namespace egpu
