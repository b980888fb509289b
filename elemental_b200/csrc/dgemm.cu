// Host side of the FP64 GEMM engine: tensor-map encoding and launch.
#include <cudaTypedefs.h>

#include <mutex>

#include "dgemm.cuh"
#include "internal.h"

namespace egpu {

static PFN_cuTensorMapEncodeTiled_v12000 g_encode = nullptr;
static std::once_flag g_encode_once;

static PFN_cuTensorMapEncodeTiled_v12000 encoder() {
  std::call_once(g_encode_once, [] {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      g_encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
  });
  return g_encode;
}

// 2-D tensor map over a column-major FP64 view: `inner` contiguous elements,
// `outer` columns `ld` elements apart.
static bool make_map(CUtensorMap* m, const double* base, uint64_t inner, uint64_t outer, uint64_t ld,
                     uint32_t box_inner, uint32_t box_outer, bool swz128) {
  auto enc = encoder();
  if (!enc) return false;
  cuuint64_t dims[2] = {inner, outer};
  cuuint64_t strides[1] = {ld * sizeof(double)};
  cuuint32_t box[2] = {box_inner, box_outer};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 2, const_cast<double*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE,
                   swz128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

bool make_tma_2d(CUtensorMap* m, int dtype, const void* base, uint64_t inner, uint64_t outer,
                 uint64_t ld_bytes, uint32_t box_inner, uint32_t box_outer, bool swz128) {
  auto enc = encoder();
  if (!enc) return false;
  cuuint64_t dims[2] = {inner, outer};
  cuuint64_t strides[1] = {ld_bytes};
  cuuint32_t box[2] = {box_inner, box_outer};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(m, (CUtensorMapDataType)dtype, 2, const_cast<void*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE,
                   swz128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

static int sm_count_of_current_device() {
  static int cache[32] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 32 && cache[dev] > 0) return cache[dev];
  int n = 0;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
  if (dev >= 0 && dev < 32) cache[dev] = n;
  return n;
}

bool tma_compatible(const void* p, long long ld) {
  return (reinterpret_cast<uintptr_t>(p) % 16 == 0) && (ld % 2 == 0) && ld > 0;
}

template <bool AK, bool BK, int WM, int WN, int MI>
static cudaError_t launch_variant(cudaStream_t st, const CUtensorMap& ma, const CUtensorMap& mb,
                                  const GemmParams& p, long long nblocks) {
  using S = GemmShape<WM, WN, MI>;
  auto kern = dgemm_tma_kernel<AK, BK, WM, WN, MI>;
  static unsigned attr_mask = 0;  // per template instance, one bit per device
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 32 || !(attr_mask & (1u << dev))) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kSmemBytes);
    if (e != cudaSuccess) return e;
    if (dev < 32) attr_mask |= (1u << dev);
  }
  kern<<<(unsigned)nblocks, S::kThreads, S::kSmemBytes, st>>>(ma, mb, p);
  count_launch();
  return cudaGetLastError();
}


// ---- small products ------------------------------------------------------
// A product with few tiles (a panel multiply or the next block column's update
// of a small factorization) is bound by latencies, not by the DMMA rate: the
// engine's 128 x 64 x 128 tile takes 8 us on one SM however idle the rest is.
// Here a CTA of eight warps takes a small tile of C (32 x 32, or 16 or 32 rows
// by all columns, or all rows by 16 columns) with the whole of K: A's and B's
// parts are copied to shared memory by 16-byte cp.async, all in flight at
// once together with the tile of C, so the chain is one round trip to L2, the
// products and the store.  C may be A when the CTA covers every column of C,
// or B when it covers every row: all of it is in shared memory before any
// store.  (Warps that read their operands from L2 sixteen k at a time, one
// round trip each: 22 us per launch at M = 2048, N = K = 128; now 8 to 10.)
struct SmallParams {
  const double* A;
  const double* B;
  double* C;
  long long lda, ldb, ldc;
  int M, N, K, tri;
  double alpha, beta;
  const DevStatus* status;
};

// 16-byte cp.async of which the first `bytes` are read and the rest is zero
__device__ __forceinline__ void cp_async16_zfill(void* smem_dst, const void* gmem_src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(smem_dst)), "l"(gmem_src), "r"(bytes)
               : "memory");
}

constexpr int small_ld(int tile) { return tile + 4; }  // MN-major parts: 4 mod 16, conflict-free fragment loads

// Copy rows [r0, r0 + T) of an operand, k in [0, KP) (zero past R rows and K),
// to shared memory: MN-major as [k][T + 4], K-major as [row][KP + 4].
template <bool KM, int T>
__device__ __forceinline__ void small_stage(double* S, const double* G, long long ld, int r0, int R, int K, int KP) {
  if (!KM) {
    constexpr int CH = T / 2;  // chunks per k
    for (int e = threadIdx.x; e < KP * CH; e += 256) {
      const int k = e / CH, r = 2 * (e % CH), left = R - (r0 + r);
      const int bytes = k < K ? (left >= 2 ? 16 : left == 1 ? 8 : 0) : 0;
      cp_async16_zfill(S + k * small_ld(T) + r, bytes ? G + (long long)k * ld + r0 + r : G, bytes);
    }
  } else {
    const int ch = KP / 2, lds = KP + 4;
    for (int e = threadIdx.x; e < T * ch; e += 256) {
      const int r = e / ch, k = 2 * (e - r * ch), left = K - k;
      const int bytes = r0 + r < R ? (left >= 2 ? 16 : left == 1 ? 8 : 0) : 0;
      cp_async16_zfill(S + r * lds + k, bytes ? G + (long long)(r0 + r) * ld + k : G, bytes);
    }
  }
}

// U: the k loop's unrolling.  2 takes up to 70 registers, three CTAs to an SM,
// which is what the operands leave room for from K = 128 on (us, U = 1 / 2, NORMAL,
// NORMAL, 768^2 14.5 / 12.4, 1216^2 24.7 / 22.7); with K <= 64 and U = 1 there are five
// (8.3 / 10.4 at 768^2, K = 64).
template <bool AK, bool BK, int TM, int TN, int U>
__global__ void __launch_bounds__(256) dgemm_small_kernel(const SmallParams p) {
  extern __shared__ __align__(16) double ss[];
  constexpr int TILES = (TM / 16) * (TN / 8), PER = TILES / 8;  // 16 x 8 DMMA tiles per warp
  static_assert(TILES % 8 == 0, "eight warps");
  // an earlier step failed: the CTA takes one thread's reading (another stream
  // may set the status meanwhile), which comes in with the copies.  (Through a
  // shared word it cost 10 to 30% of 500 CTAs and more at K = 128.)
  bool bad = false;
  if (threadIdx.x == 0) bad = p.status != nullptr && ((const volatile DevStatus*)p.status)->code != 0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int row0 = blockIdx.x * TM, col0 = blockIdx.y * TN;
  if ((p.tri == 1 && row0 + TM - 1 < col0) || (p.tri == 2 && row0 > col0 + TN - 1)) return;
  const int KP = (p.K + 7) & ~7;
  double* sA = ss;
  double* sB = ss + (AK ? TM * (KP + 4) : KP * small_ld(TM));
  small_stage<AK, TM>(sA, p.A, p.lda, row0, p.M, p.K, KP);
  small_stage<BK, TN>(sB, p.B, p.ldb, col0, p.N, p.K, KP);
  // this warp's tiles: row tile rt, column tiles ct, ct + 1, ..
  const int rt = (warp * PER) / (TN / 8), ct = (warp * PER) % (TN / 8);
  double acc[PER][4], cc[PER][4];
#pragma unroll
  for (int j = 0; j < PER; ++j)
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int m = row0 + 16 * rt + g + (r >= 2 ? 8 : 0), n = col0 + 8 * (ct + j) + 2 * t + (r & 1);
      const bool v = p.beta != 0.0 && m < p.M && n < p.N && !(p.tri == 1 && m < n) && !(p.tri == 2 && m > n);
      cc[j][r] = v ? p.C[m + (long long)n * p.ldc] : 0.0;
      acc[j][r] = 0.0;
    }
  cp_async_wait_all();
  if (__syncthreads_or(bad)) return;
  const int as = AK ? 1 : small_ld(TM), am = AK ? KP + 4 : 1;  // k and row strides
  const int bs = BK ? 1 : small_ld(TN), bn = BK ? KP + 4 : 1;
  const double* pa = sA + (16 * rt + g) * am + t * as;
  const double* pb = sB + (8 * ct + g) * bn + t * bs;
  double acc2[PER][4];  // two chains per tile
#pragma unroll
  for (int j = 0; j < PER; ++j)
#pragma unroll
    for (int r = 0; r < 4; ++r) acc2[j][r] = 0.0;
  auto step = [&](double (&d)[PER][4], int k0) {
    const double a[4] = {pa[k0 * as], pa[k0 * as + 8 * am], pa[(k0 + 4) * as], pa[(k0 + 4) * as + 8 * am]};
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      const double b[2] = {pb[k0 * bs + 8 * j * bn], pb[(k0 + 4) * bs + 8 * j * bn]};
      dmma_16x8x8(d[j], a, b);
    }
  };
  int k0 = 0;
#pragma unroll U
  for (; k0 + 8 < KP; k0 += 16) {
    step(acc, k0);
    step(acc2, k0 + 8);
  }
  if (k0 < KP) step(acc, k0);
#pragma unroll
  for (int j = 0; j < PER; ++j)
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int m = row0 + 16 * rt + g + (r >= 2 ? 8 : 0), n = col0 + 8 * (ct + j) + 2 * t + (r & 1);
      const bool v = m < p.M && n < p.N && !(p.tri == 1 && m < n) && !(p.tri == 2 && m > n);
      const double x = acc[j][r] + acc2[j][r];
      if (v) p.C[m + (long long)n * p.ldc] = p.beta == 0.0 ? p.alpha * x : fma(p.beta, cc[j][r], p.alpha * x);
    }
}

template <bool AK, bool BK, int TM, int TN, int U>
static cudaError_t launch_small_variant(cudaStream_t st, const SmallParams& p) {
  auto kern = dgemm_small_kernel<AK, BK, TM, TN, U>;
  constexpr int kMax = 200 * 1024;
  static unsigned attr_mask = 0;  // per template instance, one bit per device
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 32 || !(attr_mask & (1u << dev))) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMax);
    if (e != cudaSuccess) return e;
    if (dev < 32) attr_mask |= (1u << dev);
  }
  const int KP = (p.K + 7) & ~7;
  const size_t smem = sizeof(double) * ((size_t)(AK ? TM * (KP + 4) : KP * small_ld(TM)) +
                                        (size_t)(BK ? TN * (KP + 4) : KP * small_ld(TN)));
  if (smem > kMax) return cudaErrorInvalidValue;
  const dim3 grid((p.M + TM - 1) / TM, (p.N + TN - 1) / TN);
  kern<<<grid, 256, smem, st>>>(p);
  count_launch();
  return cudaGetLastError();
}

template <int TM, int TN, int U = 2>
static cudaError_t launch_small_tile(cudaStream_t st, bool ak, bool bk, const SmallParams& p) {
  if (ak && bk) return launch_small_variant<true, true, TM, TN, U>(st, p);
  if (ak) return launch_small_variant<true, false, TM, TN, U>(st, p);
  if (bk) return launch_small_variant<false, true, TM, TN, U>(st, p);
  return launch_small_variant<false, false, TM, TN, U>(st, p);
}

// Do two column-major views share an element?  Views with the same leading
// dimension are compared as blocks of one matrix (a panel's row block and the
// block below it interleave in memory without sharing anything); others by the
// memory they span.
static bool views_overlap(const double* a, long long rows_a, long long cols_a, long long lda, const double* b,
                          long long rows_b, long long cols_b, long long ldb) {
  const intptr_t bytes = reinterpret_cast<intptr_t>(a) - reinterpret_cast<intptr_t>(b);
  if (lda == ldb && bytes % 8 == 0 && rows_a <= lda && rows_b <= ldb) {
    const long long diff = bytes / 8, dc = diff >= 0 ? diff / lda : -((-diff + lda - 1) / lda), dr = diff - dc * lda;
    // a's element (0, 0) is b's (dr, dc), 0 <= dr < ld; its rows past the end
    // of b's column are those of (dr - ld, dc + 1)
    auto meet = [&](long long r, long long c) { return r < rows_b && r + rows_a > 0 && c < cols_b && c + cols_a > 0; };
    return meet(dr, dc) || meet(dr - lda, dc + 1);
  }
  const uintptr_t a0 = reinterpret_cast<uintptr_t>(a), a1 = a0 + 8 * ((cols_a - 1) * lda + rows_a);
  const uintptr_t b0 = reinterpret_cast<uintptr_t>(b), b1 = b0 + 8 * ((cols_b - 1) * ldb + rows_b);
  return a0 < b1 && b0 < a1;
}

// The small form when it applies; else EGPU_ERR_UNSUPPORTED (then the TMA
// engine runs).
static int launch_dgemm_small(cudaStream_t st, bool a_kmajor, bool b_kmajor, int M, int N, int K, double alpha,
                              const double* A, long long lda, const double* B, long long ldb, double beta, double* C,
                              long long ldc, int tri, DevStatus* status) {
  if (K > 256) return EGPU_ERR_UNSUPPORTED;
  const bool alias_a = views_overlap(C, M, N, ldc, A, a_kmajor ? K : M, a_kmajor ? M : K, lda);
  const bool alias_b = views_overlap(C, M, N, ldc, B, b_kmajor ? K : N, b_kmajor ? N : K, ldb);
  if (alias_a && alias_b) return EGPU_ERR_UNSUPPORTED;
  // in place only as the drivers use it: C is A (the same rows) or C is B
  // (column n of C is column n of op(B)^T)
  if (alias_a && !(C == A && ldc == lda && !a_kmajor && N <= 128 && K <= 128)) return EGPU_ERR_UNSUPPORTED;
  if (alias_b && !(C == B && ldc == ldb && b_kmajor && M <= 128 && K <= 128)) return EGPU_ERR_UNSUPPORTED;
  const int sms = sm_count_of_current_device();
  const long long t32 = (long long)((M + 31) / 32) * ((N + 31) / 32);
  // Out of place up to where the engine, whose tiles need half the operand
  // traffic, catches up.  This form's time over the engine's, 148 SMs, best and
  // worst layout (MN-major both, K-major both): K = 64, 1444 tiles of 32 x 32
  // (1216^2) 0.82 and 0.84, 1936 1.00 and 1.11; K = 128, 1444 0.72 and 0.90, 1764 0.86 and
  // 1.04, 2304 1.06 and 1.32; K = 256, MN-major, 784 0.88, 1444 0.98.  K-major operands
  // cost more with K, and the engine has one CTA to an SM up to 148 of its tiles:
  // both K-major 576 tiles 0.84 at K = 192 and 1.01 at 256, 1024 1.32 and 1.69, 1444 1.00
  // and 1.36; one K-major, K = 256, 576 0.78, 784 1.12, 1444 1.10.  At most 64 rows or
  // 32 columns leave half of the engine's 128 x 64 tile empty: K = 256, 64 x 16384
  // 0.68 to 1.00 (16384 x 64, which do not, 1.40 with both K-major).
  // In place one wave of CTAs (M = 2048: 22 us in the engine, 10 here; the
  // Cholesky at n = 16384 0.6% slower with the whole range of M here).
  const bool long_k = a_kmajor && b_kmajor ? K > 128 : (a_kmajor || b_kmajor) && K > 192;
  const int per_sm = long_k && M > 64 && N > 32 ? 4 : 10;
  if (!alias_a && !alias_b && t32 / (tri ? 2 : 1) > (long long)per_sm * sms) return EGPU_ERR_UNSUPPORTED;
  if (alias_a && M > 32 * sms) return EGPU_ERR_UNSUPPORTED;
  if (alias_b && N > 32 * sms) return EGPU_ERR_UNSUPPORTED;
  SmallParams p;
  p.A = A; p.B = B; p.C = C; p.lda = lda; p.ldb = ldb; p.ldc = ldc;
  p.M = M; p.N = N; p.K = K; p.tri = tri; p.alpha = alpha; p.beta = beta; p.status = status;
  const double lo_n = std::min(M, N), rect = tri == 1 ? std::max(0, M - N) : std::max(0, N - M);
  const double entries = tri == 0 ? (double)M * N : lo_n * (lo_n + 1) / 2 + rect * lo_n;
  TraceMark tm(st, beta == 0.0 ? kTraceTrsm : kTraceUpdate, 2.0 * entries * K,
               8.0 * ((double)M * K + (double)N * K + (beta == 0.0 ? 1.0 : 2.0) * entries));
  cudaError_t e;
  if (alias_a && M <= 16 * sms) e = launch_small_tile<16, 128>(st, a_kmajor, b_kmajor, p);
  else if (alias_a) e = launch_small_tile<32, 128>(st, a_kmajor, b_kmajor, p);
  else if (alias_b && N <= 16 * sms) e = launch_small_tile<128, 16>(st, a_kmajor, b_kmajor, p);
  else if (alias_b) e = launch_small_tile<128, 32>(st, a_kmajor, b_kmajor, p);
  else if (K <= 64) e = launch_small_tile<32, 32, 1>(st, a_kmajor, b_kmajor, p);
  else e = launch_small_tile<32, 32>(st, a_kmajor, b_kmajor, p);
  if (e != cudaSuccess) {
    set_last_error(e, "dgemm_small launch", __FILE__, __LINE__);
    return EGPU_ERR_CUDA;
  }
  return EGPU_OK;
}

// C = alpha * op(A) * op(B) + beta * C (tri: 0 full, 1 lower, 2 upper).
//   a_kmajor = false: A stored M x K column-major (op = NORMAL)
//   a_kmajor = true : A stored K x M column-major (op = TRANSPOSE)
//   b_kmajor = true : B stored K x N column-major (op = NORMAL)
//   b_kmajor = false: B stored N x K column-major (op = TRANSPOSE)
// wide = true (MN-major A) selects a 64 x 128 tile, which keeps whole 128-wide
// row panels inside one CTA (in-place multiply by an inverted triangle).
int launch_dgemm(cudaStream_t st, bool a_kmajor, bool b_kmajor, int M, int N, int K, double alpha,
                 const double* A, long long lda, const double* B, long long ldb, double beta, double* C,
                 long long ldc, int tri, bool wide, DevStatus* status) {
  if (M <= 0 || N <= 0) return EGPU_OK;
  if (K <= 0) return launch_scale(st, M, N, beta, C, ldc, tri);
  if (!tma_compatible(A, lda) || !tma_compatible(B, ldb)) return EGPU_ERR_ALIGN;
  if (wide && (tri != 0 || a_kmajor)) return EGPU_ERR_ARG;
  {
    const int rc = launch_dgemm_small(st, a_kmajor, b_kmajor, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, tri,
                                      status);
    if (rc != EGPU_ERR_UNSUPPORTED) return rc;
  }
  const int BM = wide ? 64 : 128, BN = wide ? 128 : 64;
  CUtensorMap ma, mb;
  // K-major: one {16 k, BM} box per stage; MN-major: BM / 16 boxes of
  // {16 m, 16 k} (both 128B-swizzled, see dgemm.cuh)
  bool ok = a_kmajor ? make_map(&ma, A, K, M, lda, kBK, BM, true) : make_map(&ma, A, M, K, lda, 16, kBK, true);
  ok = ok && (b_kmajor ? make_map(&mb, B, K, N, ldb, kBK, BN, true) : make_map(&mb, B, N, K, ldb, 16, kBK, true));
  if (!ok) return EGPU_ERR_TMA;
  GemmParams p;
  p.C = C; p.ldc = ldc; p.M = M; p.N = N; p.K = K; p.alpha = alpha; p.beta = beta; p.tri = tri;
  p.tiles_m = (M + BM - 1) / BM;
  p.tiles_n = (N + BN - 1) / BN;
  p.status = status;
  p.cvec = (reinterpret_cast<uintptr_t>(C) % 16 == 0) && (ldc % 2 == 0);
  long long nblocks;
  if (tri == 0) {
    nblocks = (long long)p.tiles_m * p.tiles_n;
  } else {
    nblocks = 0;
    for (int j = 0; j < p.tiles_n; ++j) {
      int lo = tri == 1 ? j / 2 : 0;
      int hi = tri == 1 ? p.tiles_m : std::min(j / 2 + 1, p.tiles_m);
      nblocks += std::max(0, hi - lo);
    }
  }
  if (nblocks > 0x3fffffff) return EGPU_ERR_UNSUPPORTED;
  // entries of C the product touches: the whole M x N block, or the lower
  // (tri 1) / upper (tri 2) trapezoid -- a launch over rows [c0, n) of block
  // columns [c0, c1) is a triangle on top of a rectangle
  const double lo_n = std::min(M, N), rect = tri == 1 ? std::max(0, M - N) : std::max(0, N - M);
  const double entries = tri == 0 ? (double)M * N : lo_n * (lo_n + 1) / 2 + rect * lo_n;
  const double flops = 2.0 * entries * K;
  const double bytes = 8.0 * ((double)M * K + (double)N * K + (beta == 0.0 ? 1.0 : 2.0) * entries);
  TraceMark tm(st, beta == 0.0 ? kTraceTrsm : kTraceUpdate, flops, bytes);
  cudaError_t e;
  // Warps of 64 x 32 for long k loops whose last wave leaves most SMs with two
  // CTAs (the main loop counts); of 32 x 32 for short ones (the epilogue counts)
  // and where the last wave leaves one CTA to an SM, which four of the larger
  // warps do not fill.  C full, NT, time with 64 x 32 over that with 32 x 32, 296 CTAs
  // at once: n = 1500 (288 CTAs) K = 128 1.01, 384 0.92, 4096 0.89; n = 2048 (512) K =
  // 256 0.98, 384 0.96, 4096 0.92; n = 3000 (1128) K = 384 1.04, 512 1.01, 4096 0.94; n =
  // 8192 K = 128 1.23, 512 1.02, 2048 1.01; but n = 1000 (128) 1.09, n = 1800 (435)
  // 1.17 and n = 3500 (1540) 1.05 to 1.08 at every K >= 512
  const long long slots = 2ll * sm_count_of_current_device(), last = nblocks % slots;
  const bool big = K >= (nblocks <= 2 * slots ? 384 : 512) && (last == 0 || 2 * last > slots);
  if (wide) {
    if (!b_kmajor) e = launch_variant<false, false, 2, 4, 2>(st, ma, mb, p, nblocks);
    else e = launch_variant<false, true, 2, 4, 2>(st, ma, mb, p, nblocks);
  } else if (big) {
    if (!a_kmajor && !b_kmajor) e = launch_variant<false, false, 2, 2, 4>(st, ma, mb, p, nblocks);
    else if (!a_kmajor && b_kmajor) e = launch_variant<false, true, 2, 2, 4>(st, ma, mb, p, nblocks);
    else if (a_kmajor && !b_kmajor) e = launch_variant<true, false, 2, 2, 4>(st, ma, mb, p, nblocks);
    else e = launch_variant<true, true, 2, 2, 4>(st, ma, mb, p, nblocks);
  } else {
    if (!a_kmajor && !b_kmajor) e = launch_variant<false, false, 4, 2, 2>(st, ma, mb, p, nblocks);
    else if (!a_kmajor && b_kmajor) e = launch_variant<false, true, 4, 2, 2>(st, ma, mb, p, nblocks);
    else if (a_kmajor && !b_kmajor) e = launch_variant<true, false, 4, 2, 2>(st, ma, mb, p, nblocks);
    else e = launch_variant<true, true, 4, 2, 2>(st, ma, mb, p, nblocks);
  }
  if (e != cudaSuccess) {
    set_last_error(e, "dgemm launch", __FILE__, __LINE__);
    return EGPU_ERR_CUDA;
  }
  return EGPU_OK;
}

// C := beta * C on the (tri) region; used for K == 0 products.
__global__ void scale_kernel(int M, int N, double beta, double* C, long long ldc, int tri) {
  const long long total = (long long)M * N;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const int r = (int)(idx % M), c = (int)(idx / M);
    if (tri == 1 && r < c) continue;
    if (tri == 2 && r > c) continue;
    double* p = C + (long long)c * ldc + r;
    *p = (beta == 0.0) ? 0.0 : beta * *p;
  }
}

int launch_scale(cudaStream_t st, int M, int N, double beta, double* C, long long ldc, int tri) {
  if (M <= 0 || N <= 0 || beta == 1.0) return EGPU_OK;
  long long total = (long long)M * N;
  int blocks = (int)std::min<long long>((total + 255) / 256, 148 * 16);
  scale_kernel<<<blocks, 256, 0, st>>>(M, N, beta, C, ldc, tri);
  count_launch();
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_last_error(e, "scale launch", __FILE__, __LINE__);
    return EGPU_ERR_CUDA;
  }
  return EGPU_OK;
}

}  // namespace egpu
