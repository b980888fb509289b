// FP64 tensor-core GEMM / SYRK engine for sm_100a.
//
// C[MxN] = alpha * op(A)[MxK] * op(B)[KxN] + beta * C, optionally restricted
// to the lower (tri=1) or upper (tri=2) triangle of C.  This single engine
// carries every level-3 call of the factor-and-solve path:
//   * Herk/Syrk trailing update of Cholesky  (Cholesky/LVar3.hpp:114,
//     UVar3.hpp:113; dsyrk_ at src/core/imports/blas.cpp:1043)
//   * Gemm trailing update of LU             (LU.hpp:203; dgemm_ at blas.cpp:930)
//   * Trsm panel / row-panel solves, run as a multiply by the explicitly
//     inverted diagonal block                 (LVar3.hpp:113, LU.hpp:202)
//
// Operands are staged global->shared by TMA (cp.async.bulk.tensor, one
// elected thread, mbarrier completion), 4-stage ring, BK = 16.  The math is
// FP64 DMMA (mma.sync m16n8k8 f64): Blackwell's tcgen05 has no f64 kind, and
// DMMA reaches the FP64 peak (37.2 TFLOP/s measured, DFMA 34.1).
//
// Shared-memory layouts (no bank conflicts on any fragment load but K-major
// A's, whose even rows meet two to a bank, which the DMMA pipe hides):
//   MN-major operand (m or n contiguous in global): BM/16 boxes of 16 m x
//     16 k, each [16 k][16 m] (128 B per k row) with the 128B swizzle (16-byte
//     chunk c of row k at chunk c ^ (k & 7)); one 16-byte load gives two
//     adjacent rows -> feeds two m16 tiles (row-interleaved tile pairs).  The
//     four lanes of a quad read k rows 2t (+1) of the same chunk, which the
//     swizzle spreads over distinct banks (plain [16 k][BM] rows, 8 BM bytes
//     apart, would put all four in the same banks).
//   K-major operand (k contiguous in global): smem [BM][16 k], 128B swizzle;
//     one 16-byte load gives the k pair (2t, 2t+1) of one row.
// The k index inside each k8 step is permuted (logical t <-> physical 2t,
// t+4 <-> 2t+1) identically for A and B, which leaves the product unchanged.
#pragma once
#include "common.cuh"

namespace egpu {

struct GemmParams {
  double* C;
  long long ldc;
  int M, N, K;
  double alpha, beta;
  int tri;  // 0 full, 1 lower (row >= col), 2 upper (row <= col)
  int tiles_m, tiles_n;
  int cvec;  // C base 16-byte aligned and ldc even: paired 16-byte epilogue
  DevStatus* status;
};

constexpr int kBK = 16;
constexpr int kStages = 4;

// Warps of (16 MI) x 32, two CTAs per SM, one tile per CTA.  MI = 2: eight
// warps, so that a CTA alone on its SM (a small product, or the other CTA in
// its epilogue) still fills the DMMA pipe; MI = 4: four warps with fewer
// fragment loads per DMMA, the better one for long k loops on a full chip
// (launch_dgemm chooses).  C full, n = 8192, K = 128 (NT): 0.72 ms with MI = 4, 0.58
// with MI = 2 (0.80 of the DMMA rate; n = 16384 2.27 ms, 0.82); K = 2048 (NN): 8.00 and
// 8.13 ms (0.92, 0.91).  Several tiles per CTA with the next tile's loads under
// the epilogue measured slower (0.67 with four, 0.66 with eight at K = 128): the
// two CTAs of an SM then stay in step, both in the main loop and both in the
// epilogue, where one tile per CTA lets them drift apart; two groups of four
// warps taking turns in one CTA 0.51.
template <int WARPS_M, int WARPS_N, int MI>
struct GemmShape {
  static constexpr int BM = 16 * MI * WARPS_M;
  static constexpr int BN = 32 * WARPS_N;
  static constexpr int kThreads = 32 * WARPS_M * WARPS_N;
  static constexpr int kStageBytes = (BM + BN) * kBK * 8;
  static constexpr int kSmemBytes = kStages * kStageBytes + 1024 /*align*/ + 16 * kStages /*barriers*/;
};

// Map a linear CTA index onto (tile_m, tile_n) for the triangular modes with
// BM = 2*BN (tile-row i covers rows [BM i, BM i + BM), tile-col j covers
// [BN j, BN j + BN)).  Lower: column j needs rows i >= j/2 (count
// max(0, MT - j/2)); upper: rows i <= j/2 (count min(j/2 + 1, MT)).
// cum(j) = number of tiles in columns < j.
__device__ __forceinline__ long long tri_S(long long j) {  // sum_{j'<j} floor(j'/2)
  const long long a = j / 2;
  return (j & 1) ? a * a : a * (a - 1);
}
__device__ __forceinline__ long long tri_cum_lower(int j, int MT) {
  const long long jj = min((long long)j, 2ll * MT);
  return jj * MT - tri_S(jj);
}
__device__ __forceinline__ long long tri_cum_upper(int j, int MT) {
  const long long J0 = 2ll * MT;
  if (j <= J0) return tri_S(j) + j;
  return tri_S(J0) + J0 + (j - J0) * MT;
}

__device__ __forceinline__ bool map_tile(const GemmParams& p, int& ti, int& tj) {
  const int L = (int)blockIdx.x;
  if (p.tri == 0) {
    ti = L % p.tiles_m;
    tj = L / p.tiles_m;
    return tj < p.tiles_n;
  }
  int lo = 0, hi = p.tiles_n;  // find largest j with cum(j) <= L
  while (hi - lo > 1) {
    int mid = (lo + hi) >> 1;
    long long c = p.tri == 1 ? tri_cum_lower(mid, p.tiles_m) : tri_cum_upper(mid, p.tiles_m);
    if (c <= L) lo = mid; else hi = mid;
  }
  tj = lo;
  if (p.tri == 1) {
    ti = tj / 2 + (int)(L - tri_cum_lower(tj, p.tiles_m));
  } else {
    ti = (int)(L - tri_cum_upper(tj, p.tiles_m));
  }
  return ti < p.tiles_m && tj < p.tiles_n;
}

template <bool AK, bool BK, int WARPS_M, int WARPS_N, int MI>
__global__ void __launch_bounds__(32 * WARPS_M * WARPS_N, 2)
    dgemm_tma_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                     const GemmParams p) {
  using S = GemmShape<WARPS_M, WARPS_N, MI>;
  constexpr int BM = S::BM, BN = S::BN;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + kStages * S::kStageBytes);
  uint64_t* empty = full + kStages;  // one arrival per warp when it is done with a stage
  __shared__ int s_go, s_row, s_col;
  __shared__ int s_issued;  // k-tiles whose loads have been issued
  const int KT = (p.K + kBK - 1) / kBK;

  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int wm = warp % WARPS_M, wn = warp / WARPS_M;

  if (tid == 32) {  // beside warp 0's set-up
    int ti, tj;
    const bool in = map_tile(p, ti, tj);
    s_row = in ? ti * BM : -1;
    s_col = tj * BN;
  }
  if (tid == 0) {
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], S::kThreads / 32);
    }
    fence_mbar_init();
    s_issued = min(kStages, KT);
    // an earlier step failed: the CTA takes one thread's reading
    s_go = p.status == nullptr || ((volatile DevStatus*)p.status)->code == 0;
  }
  __syncthreads();
  if (!s_go || s_row < 0) return;
  const int row0 = s_row, col0 = s_col;

  auto issue = [&](int kt) {
    const int s = kt % kStages;
    double* sA = reinterpret_cast<double*>(smem + s * S::kStageBytes);
    double* sB = sA + BM * kBK;
    mbar_expect_tx(&full[s], S::kStageBytes);
    if (AK) {
      tma_load_2d(sA, &tmA, &full[s], kt * kBK, row0);
    } else {
#pragma unroll
      for (int b = 0; b < BM / 16; ++b) tma_load_2d(sA + b * 256, &tmA, &full[s], row0 + 16 * b, kt * kBK);
    }
    if (BK) {
      tma_load_2d(sB, &tmB, &full[s], kt * kBK, col0);
    } else {
#pragma unroll
      for (int b = 0; b < BN / 16; ++b) tma_load_2d(sB + b * 256, &tmB, &full[s], col0 + 16 * b, kt * kBK);
    }
  };
  if (tid == 0)
    for (int kt = 0; kt < kStages && kt < KT; ++kt) issue(kt);
  // Pull this tile of C into L2 while the main loop runs, so the epilogue's
  // read-modify-write does not wait on HBM (one bulk prefetch per column).
  if (p.beta != 0.0 && p.cvec) {
    const int nrow = min(BM, p.M - row0);
    const int ncol = min(BN, p.N - col0);
    const unsigned bytes = (unsigned)((nrow * 8) & ~15);  // never past the column's end
    for (int c = tid; c < ncol && bytes > 0; c += S::kThreads) {
      const double* src = p.C + (long long)(col0 + c) * p.ldc + row0;
      asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes) : "memory");
    }
  }

  double acc[MI][4][4];
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int r = 0; r < 4; ++r) acc[i][j][r] = 0.0;

  bool ok = true;
  for (int kt = 0; kt < KT; ++kt) {
    const int s = kt % kStages;
    const uint32_t parity = (uint32_t)(kt / kStages) & 1u;
    // warp-uniform outcome: the DMMAs below need the whole warp converged
    // (with MI = 4 the loop is left only at its end: a branch out of it here
    // costs the NORMAL, NORMAL product 6% at K = 4096, n = 6000 8.99 ms instead of
    // 8.45; with MI = 2 it gains up to 6% there, n = 1000)
    ok = __all_sync(0xffffffffu, ok && mbar_wait_bounded(&full[s], parity));
    if (MI < 4 && !ok) break;
    const double* sA = reinterpret_cast<const double*>(smem + s * S::kStageBytes);
    const double* sB = sA + BM * kBK;
#pragma unroll
    for (int ks = 0; ks < 2; ++ks) {
      double af[MI][4], bf[4][2];
      const int ke = ks * 8 + 2 * t;  // physical k pair (ke, ke+1)
      if (AK) {
#pragma unroll
        for (int i = 0; i < MI; ++i) {
          // the same row interleaving as for MN-major A (a thread's rows 2g, 2g + 1
          // are adjacent, for the 16-byte epilogue); its even rows meet two to a
          // bank, which the DMMA pipe hides
          const int r0 = wm * 16 * MI + (i >> 1) * 32 + 2 * g + (i & 1);
          const int r1 = r0 + 16;
          const int ch = ks * 4 + t;
          const double2 v0 = *reinterpret_cast<const double2*>(sA + r0 * 16 + ((ch ^ (r0 & 7)) << 1));
          const double2 v1 = *reinterpret_cast<const double2*>(sA + r1 * 16 + ((ch ^ (r1 & 7)) << 1));
          af[i][0] = v0.x; af[i][2] = v0.y; af[i][1] = v1.x; af[i][3] = v1.y;
        }
      } else {
        // boxes wm * MI + 2 pr and + 1 (rows +16), chunk g of rows ke, ke + 1
        const int c0 = (g ^ (ke & 7)) << 1, c1 = (g ^ ((ke + 1) & 7)) << 1;
#pragma unroll
        for (int pr = 0; pr < MI / 2; ++pr) {
          const double* bx = sA + (wm * MI + 2 * pr) * 256;
          const double2 v00 = *reinterpret_cast<const double2*>(bx + ke * 16 + c0);
          const double2 v01 = *reinterpret_cast<const double2*>(bx + (ke + 1) * 16 + c1);
          const double2 v10 = *reinterpret_cast<const double2*>(bx + 256 + ke * 16 + c0);
          const double2 v11 = *reinterpret_cast<const double2*>(bx + 256 + (ke + 1) * 16 + c1);
          af[2 * pr][0] = v00.x; af[2 * pr][1] = v10.x; af[2 * pr][2] = v01.x; af[2 * pr][3] = v11.x;
          af[2 * pr + 1][0] = v00.y; af[2 * pr + 1][1] = v10.y; af[2 * pr + 1][2] = v01.y; af[2 * pr + 1][3] = v11.y;
        }
      }
      if (BK) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int n = wn * 32 + j * 8 + g;
          const int ch = ks * 4 + t;
          const double2 v = *reinterpret_cast<const double2*>(sB + n * 16 + ((ch ^ (n & 7)) << 1));
          bf[j][0] = v.x; bf[j][1] = v.y;
        }
      } else {
        const int c0 = (g ^ (ke & 7)) << 1, c1 = (g ^ ((ke + 1) & 7)) << 1;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const double* bx = sB + (wn * 2 + q) * 256;  // box of n rows wn * 32 + q * 16 ..
          const double2 v0 = *reinterpret_cast<const double2*>(bx + ke * 16 + c0);
          const double2 v1 = *reinterpret_cast<const double2*>(bx + (ke + 1) * 16 + c1);
          bf[2 * q][0] = v0.x; bf[2 * q][1] = v1.x;
          bf[2 * q + 1][0] = v0.y; bf[2 * q + 1][1] = v1.y;
        }
      }
#pragma unroll
      for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) dmma_16x8x8(acc[i][j], af[i], bf[j]);
    }
    // This warp is done with stage s.  The refill is a TMA write into the
    // same bytes, and an mbarrier release alone does not order this warp's
    // generic-proxy reads before an async-proxy write: lane 0 fences (after
    // the warp has converged) and arrives.  Warp 0 refills the stage for
    // k-tile kt + kStages once every warp has arrived (the whole warp waits,
    // lane 0 issues, so warp 0 stays converged); the other warps run ahead
    // into the stages already loaded instead of meeting at a CTA barrier.
    __syncwarp();
    if (lane == 0) {
      fence_proxy_async_smem();
      mbar_arrive(&empty[s]);
    }
    if (warp == 0 && kt + kStages < KT) {
      ok = __all_sync(0xffffffffu, ok && mbar_wait_bounded(&empty[s], parity));
      if (MI < 4 && !ok) break;
      if (ok && lane == 0) issue(kt + kStages);
      if (ok && (MI == 4 || lane == 0)) s_issued = kt + kStages + 1;
      __syncwarp();
    }
    if (!ok) break;
  }

  // a warp that gave up (bounded wait) leaves early; all meet here
  if (!__syncthreads_and(ok)) {
    if (tid == 0) {
      set_status(p.status, kTimeout, 100);
      // Drain copies still in flight before the CTA's shared memory goes away.
      for (int r = max(0, s_issued - kStages); r < s_issued; ++r)
        (void)mbar_wait_bounded(&full[r % kStages], (uint32_t)(r / kStages) & 1u);
    }
    __syncthreads();
    return;
  }

  // Epilogue: C = alpha * acc + beta * C on the valid (and triangle) region.
  // A thread's loads of a group are all in flight before the first is used:
  // with a test around each load they ran one after the other, 27 K cycles per
  // tile against 31 K for the main loop at K = 128 (two CTAs on the SM).
  const double alpha = p.alpha, beta = p.beta;
  auto row_of = [&](int i, int r) -> int {
    return row0 + wm * 16 * MI + (i >> 1) * 32 + 2 * g + (i & 1) + ((r >= 2) ? 16 : 0);
  };
  auto col_of = [&](int j, int r) -> int {
    const int c = 2 * t + (r & 1);
    if (BK) return col0 + wn * 32 + j * 8 + c;
    return col0 + wn * 32 + (j >> 1) * 16 + 2 * c + (j & 1);
  };
  auto valid = [&](int row, int col) -> bool {
    if (row >= p.M || col >= p.N) return false;
    if (p.tri == 1 && row < col) return false;
    if (p.tri == 2 && row > col) return false;
    return true;
  };
  double* cbase = p.C + (long long)col_of(0, 0) * p.ldc + row_of(0, 0);
  // element (i, j, r) lies at cbase + off(i, j, r)
  auto off = [&](int i, int j, int r) -> long long {
    const int dc = BK ? j * 8 + (r & 1) : (j >> 1) * 16 + 2 * (r & 1) + (j & 1);
    return (long long)dc * p.ldc + (i >> 1) * 32 + (i & 1) + ((r >= 2) ? 16 : 0);
  };
  // a tile wholly inside C (and its triangle) takes no test per element; the
  // row tiles 2 pr and 2 pr + 1 hold rows (2g, 2g + 1): one 16-byte access
  const bool inside = row0 + BM <= p.M && col0 + BN <= p.N && !(p.tri == 1 && row0 < col0 + BN - 1) &&
                      !(p.tri == 2 && row0 + BM - 1 > col0);
  if (inside && p.cvec) {
#pragma unroll
    for (int pr = 0; pr < MI / 2; ++pr)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        double2 cc[4];
#pragma unroll
        for (int r = 0; r < 4; ++r)
          cc[r] = beta != 0.0 ? *reinterpret_cast<const double2*>(cbase + off(2 * pr, j, r)) : make_double2(0.0, 0.0);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          cc[r].x = fma(beta, cc[r].x, alpha * acc[2 * pr][j][r]);
          cc[r].y = fma(beta, cc[r].y, alpha * acc[2 * pr + 1][j][r]);
          *reinterpret_cast<double2*>(cbase + off(2 * pr, j, r)) = cc[r];
        }
      }
    return;
  }
#pragma unroll
  for (int pr = 0; pr < MI / 2; ++pr)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      double c0[4], c1[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        c0[r] = beta != 0.0 && valid(row_of(2 * pr, r), col_of(j, r)) ? cbase[off(2 * pr, j, r)] : 0.0;
        c1[r] = beta != 0.0 && valid(row_of(2 * pr + 1, r), col_of(j, r)) ? cbase[off(2 * pr + 1, j, r)] : 0.0;
      }
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        if (valid(row_of(2 * pr, r), col_of(j, r)))
          cbase[off(2 * pr, j, r)] = fma(beta, c0[r], alpha * acc[2 * pr][j][r]);
        if (valid(row_of(2 * pr + 1, r), col_of(j, r)))
          cbase[off(2 * pr + 1, j, r)] = fma(beta, c1[r], alpha * acc[2 * pr + 1][j][r]);
      }
    }
}

}  // namespace egpu
