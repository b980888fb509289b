// Register-resident LU panel (lu::Panel, lapack-like/LU/Panel.hpp:19-89).
//
// One thread-block cluster of P <= 16 CTAs of 256 threads; CTA c owns rows
// [c R, c R + R) (R a multiple of 16), the first CT = 32 CW threads of the CTA
// (its column threads) own local rows t, t + CT, ... (RT of them); the other
// warps help between the sub-panels.  The panel is processed in 16-column
// sub-panels; a column thread keeps its rows' sub-panel entries in registers,
// and each column step rotates them by one as part of its rank-1 update,
// v[k] := v[k + 1] - l u[k], so that register 0 is always the current
// column, the column loop stays rolled, and the columns already done have
// rotated out as zeros (the winner's u needs no masking).
//
// What bounds it: the chain of column steps (one CTA barrier, one exchange
// over the cluster each), so what counts is the length of one step in
// instructions as well as in latencies (here: a warp reduction 56 cycles, a
// CTA barrier 25, with an OR over the CTA 100, an asynchronous store into
// another CTA and the wait for it about 600).  An unrolled column loop
// (column t = register t) made 330 KB of straight-line code, every
// instruction of it fetched anew in every sub-panel; the rolled form is 85 KB
// in all.  One 128-column panel, before (unrolled, interchanges in the
// messages, register FMAs for the trailing columns) and now: m = 128 0.36 ->
// 0.162 ms, m = 2048 0.354 -> 0.195 ms, m = 8192 0.459 -> 0.308 ms.
//
// Pivoting inside a sub-panel is logical: a chosen row is marked done where
// it is, and every thread tracks the position its rows would have under the
// reference's interchanges (position j <-> position p_j), which also breaks
// ties (lowest position: the strict '>' scan of Panel.hpp:52-63).
//
// Per column:
//  1. each warp finds its first maximal |a| (the upper 32 bits of |a| by
//     redux.sync; the lower bits and the position only on a tie); the lane
//     that owns the candidate stages it with 1 / pivot in shared memory;
//  2. after the barrier of the column threads every warp picks the CTA's
//     candidate from the warps' and the threads store it into every CTA's
//     shared memory (st.async, 16-byte units, counted in bytes on the
//     destination's mbarrier for this column; each CTA arms its own mbarrier
//     with the byte count).  A panel of one CTA skips the exchange;
//  3. every thread waits (bounded) on its own CTA's mbarrier, picks the winner
//     from the P messages, scales (by the sender's correctly rounded
//     1 / pivot, Panel.hpp:78-79), stores the finished column entry to the
//     shared-memory copy of the sub-panel, and rank-1 updates (Panel.hpp:80).
// The message buffers alternate between two slots by column parity: a CTA
// writes slot s for column j + 2 only after it has received every CTA's
// column j + 1 message, which each CTA sends after all its threads are done
// with column j's slot, and a CTA re-arms slot s for column j + 2 before it
// sends column j + 1.  Stopping (an exact zero pivot, seen by every CTA in
// the same column, or a wait that ran out, which is broadcast to every CTA)
// is made CTA-uniform (a lost wait through a shared flag read after the next
// barrier; slots by column parity, so no thread can see it earlier than
// another), and every CTA executes
// the same number of cluster barriers (one per sub-panel, one at the end)
// whatever happens, so a stop cannot strand a CTA at a barrier.
// After a sub-panel: every thread writes its rows' entries to their new
// positions, the interchanges are applied to the panel's other columns (row
// moves by the CTA that owns each destination row, all sources read before
// the cluster barrier), every CTA solves the 16 x (b - c1) block
// U12 = inv(L11) A12 itself (CTA 0 stores it), and updates its rows of the
// remaining panel columns, A[r, c1:b) -= L[r, c0:c1) U12, with DMMA (L from the
// shared-memory copy, 32 x 32 warp tiles of C straight from and to L2).  The
// result equals lu::Panel's: the same pivots, and the panel's trailing columns
// updated in 16-column blocks.  Last, CTA 0 forms the composed interchanges
// (ComposePivots.hpp:81-125) from the tracked rows and inv(unit lower L11) of
// the panel's top block (16 x 16 diagonal-block inverses, then DMMA doubling).
#include "diag_common.cuh"
#include "internal.h"

namespace egpu {

namespace {

constexpr int kRpThreads = 256;
constexpr int kRpWarps = kRpThreads / 32;  // also the most column warps
constexpr int kRpW = 16;         // sub-panel width
constexpr int kRpMsg = 10;       // double2 per candidate: {|a|, position : row}, {1 / pivot, pivot}, u[0..14]
constexpr int kRpMaxCl = 16;
constexpr int kRpLdU = 132;      // 4 mod 16: conflict-free DMMA fragment loads

// shared-memory layout (in doubles); the sub-panel copy Lb is [16][R + 4] at the end
constexpr int kRpOffMsg = 0;                                          // [2][kRpMaxCl][kRpMsg] double2
constexpr int kRpOffCand = kRpOffMsg + 2 * kRpMaxCl * kRpMsg * 2;     // [2][kRpWarps][kRpMsg] double2
constexpr int kRpOffL11 = kRpOffCand + 2 * kRpWarps * kRpMsg * 2;     // 16 x 16 (ld 17)
constexpr int kRpOffU12 = kRpOffL11 + 16 * 17;                        // [16][kRpLdU]
constexpr int kRpOffMv = kRpOffU12 + 16 * kRpLdU;                     // [2 * 16][128] row moves
constexpr int kRpOffLb = kRpOffMv + 2 * kRpW * 128;
constexpr int kRpInvDoubles = 128 * kLDS + 128 + kDiagTmpDoubles;  // the final inv(L11)
constexpr uint32_t kRpColBytes(int P) { return (uint32_t)(P * kRpMsg * 16); }
constexpr int rp_smem_doubles(int R) {
  const int work = kRpOffLb + kRpW * (R + 4) + 32;  // + the last tile's rows past R (read, not stored)
  return work > kRpInvDoubles ? work : kRpInvDoubles;
}

// 32-bit shared::cluster address of the same object in CTA `rank`
__device__ __forceinline__ uint32_t map_rank(const void* p, unsigned rank) {
  uint32_t out;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(out) : "r"(smem_u32(p)), "r"(rank));
  return out;
}
__device__ __forceinline__ void st_cluster(uint32_t addr, int v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
// asynchronous 16-byte store into another CTA of the cluster, counted (bytes)
// on the mbarrier `bar` of that CTA
__device__ __forceinline__ void st_async(uint32_t addr, double2 v, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];" ::"r"(addr),
               "d"(v.x), "d"(v.y), "r"(bar)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait_cluster(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Barrier of the CT column threads.
template <int CT>
__device__ __forceinline__ void column_sync() {
  asm volatile("barrier.cta.sync 1, %0;" ::"n"(CT) : "memory");
}

}  // namespace

template <int CW, int RT>
__global__ void __launch_bounds__(kRpThreads, 1) lu_panel_rp_kernel(int m, int b, double* A, long long lda, int* p,
                                                                     int offset, int* image, int* preimage,
                                                                     double* W, int ldw, DevStatus* st, int R) {
  constexpr int CT = 32 * CW;  // column threads
  extern __shared__ __align__(16) double sm[];
  double2* MSG = reinterpret_cast<double2*>(sm + kRpOffMsg);
  double2* CANDB = reinterpret_cast<double2*>(sm + kRpOffCand);
  double* L11 = sm + kRpOffL11;
  double* U12 = sm + kRpOffU12;
  double* MV = sm + kRpOffMv;
  double* Lb = sm + kRpOffLb;  // the sub-panel's finished entries, [16][ldl] by local row
  const int ldl = R + 4;       // 4 mod 16
  __shared__ int s_piv[128], s_inv[128];
  __shared__ int s_msrc[2 * kRpW], s_mdst[2 * kRpW];  // the sub-panel's row moves (dst -1: none here)
  __shared__ int s_skip, s_abort, s_lost[2];
  __shared__ __align__(8) uint64_t s_bar[2];

  const int P = gridDim.x;
  const unsigned cta = cluster_ctarank();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int r0 = (int)cta * R;
  const int rows = max(0, min(R, m - r0));

  // a failed earlier step: every CTA takes CTA 0's reading of the status
  if (tid == 0) {
    s_skip = (st != nullptr && ((volatile DevStatus*)st)->code != 0);
    s_abort = s_lost[0] = s_lost[1] = 0;
    // one phase per column: this CTA's arrival with the byte count of every
    // CTA's candidate
    mbar_init(&s_bar[0], 1);
    mbar_init(&s_bar[1], 1);
    fence_mbar_init();
    mbar_expect_tx(&s_bar[0], kRpColBytes(P));
    mbar_expect_tx(&s_bar[1], kRpColBytes(P));
  }
  __syncthreads();
  cluster_arrive_release();
  cluster_wait_acquire();
  const int skip = *cluster_map(&s_skip, 0u);
  cluster_arrive_release();
  cluster_wait_acquire();
  if (skip) return;

  const int ncols = min(b, m);
  bool stop = false;  // CTA-uniform
  int jdone = 0;      // columns whose pivot is known
  // the exchange: this thread's units of the CTA's message, by destination
  constexpr int kSend = (kRpMaxCl * kRpMsg + CT - 1) / CT;
  uint32_t send_dst[kSend], send_bar[kSend];
  int send_q[kSend];
  if (tid < CT)
#pragma unroll
    for (int i = 0; i < kSend; ++i) {
      const int e = tid + i * CT, d = e / kRpMsg, q = e - d * kRpMsg;
      send_q[i] = d < P ? q : -1;
      send_dst[i] = d < P ? map_rank(&MSG[(int)cta * kRpMsg + q], (unsigned)d) : 0u;
      send_bar[i] = d < P ? map_rank(&s_bar[0], (unsigned)d) : 0u;
    }
  int gpos = tid;     // where the panel's original row tid (< ncols) is now
  for (int c0 = 0; c0 < ncols; c0 += kRpW) {
    const int c1 = min(ncols, c0 + kRpW), w = c1 - c0;
    int tpos = c0 + (lane & 15);  // where the sub-panel's original row c0 + lane is now (lanes < 16)
    if (!stop && tid < CT) {
      // ---- load the sub-panel rows into registers (own rows >= c0; .cg: no stale L1)
      double v[RT][kRpW];
      int pos[RT];      // the row's position; kNoPos: not a row of the sub-panel
      bool done[RT];    // already a pivot row
#pragma unroll
      for (int s = 0; s < RT; ++s) {
        const int lr = s * CT + tid;
        const bool act = lr < rows && r0 + lr >= c0;
        pos[s] = act ? r0 + lr : kNoPos;
        done[s] = !act;
      }
      {
        const double* src = A + (long long)c0 * lda + r0 + tid;
#pragma unroll
        for (int k = 0; k < kRpW; ++k) {
#pragma unroll
          for (int s = 0; s < RT; ++s) v[s][k] = (!done[s] && k < w) ? __ldcg(src + s * CT) : 0.0;
          src += lda;
        }
      }
      bool stop_after = false;  // this warp lost a wait
      // ---- column loop
#pragma unroll 1
      for (int t = 0; t < w; ++t) {
        const int j = c0 + t, par = j & 1;
        const uint32_t phase = (uint32_t)(j >> 1) & 1u;
        double2* CAND = CANDB + par * kRpWarps * kRpMsg;
        // 1. the warp's candidate; its owner stages it
        unsigned long long key = 0ull;
        int kpos = kNoPos, ks = 0;
        double pv0 = 1.0;
#pragma unroll
        for (int s = 0; s < RT; ++s) {  // branch-free: a row that is done counts as |a| = 0 at no position
          const unsigned long long kk = done[s] ? 0ull : abs_key(v[s][0]);
          const int kp = done[s] ? kNoPos : pos[s];
          const bool better = kk > key || (kk == key && kp < kpos);
          key = better ? kk : key;
          kpos = better ? kp : kpos;
          ks = better ? s : ks;
          pv0 = better ? v[s][0] : pv0;
        }
        const double pinv = __drcp_rn(pv0);  // the correctly rounded 1 / pivot
        const int wl = warp_argmax(key, kpos);
        double2* cw = &CAND[warp * kRpMsg];
        if (wl < 0) {
          if (lane == 0) cw[0] = make_double2(0.0, __hiloint2double(kNoPos, 0));
        } else if (lane == wl) {
          cw[0] = make_double2(__longlong_as_double((long long)key),
                               __hiloint2double(kpos, r0 + ks * CT + tid));
          cw[1] = make_double2(pinv, pv0);
#pragma unroll
          for (int s = 0; s < RT; ++s)
            if (s == ks) {
#pragma unroll
              for (int q = 0; q < 8; ++q)
                cw[2 + q] = make_double2(v[s][2 * q + 1], q < 7 ? v[s][2 * q + 2] : 0.0);
            }
        }
        column_sync<CT>();
        // a wait of this CTA that ran out in the last column (written before
        // this barrier; the slot of this column is another one)
        const int lost = *(volatile int*)&s_lost[par ^ 1];
        // 2. the CTA's candidate, sent to every CTA
        const double2* cand;  // the P (or CW) candidates to choose the winner from
        int wc;
        if (P > 1) {
          {
            unsigned long long ck = 0ull;
            int cpos = kNoPos;
            if (lane < CW) {
              const double2 h = CAND[lane * kRpMsg];
              ck = (unsigned long long)__double_as_longlong(h.x);
              cpos = __double2hiint(h.y);
            }
            const int wsrc = max(0, warp_argmax(ck, cpos));
#pragma unroll
            for (int i = 0; i < kSend; ++i)
              if (send_q[i] >= 0)
                st_async(send_dst[i] + (uint32_t)(par * kRpMaxCl * kRpMsg * 16), CAND[wsrc * kRpMsg + send_q[i]],
                         send_bar[i] + 8u * (uint32_t)par);
          }
          // 3. every CTA's message (bounded wait; a wait that runs out stops the cluster)
          bool got = false;
          for (long long it = 0; it < kSpinLimit; ++it) {
            if (mbar_try_wait_cluster(&s_bar[par], phase)) {
              got = true;
              break;
            }
            if (*(volatile int*)&s_abort) break;
            if (it > 64) __nanosleep(64);
          }
          // re-arm this slot for column j + 2: no CTA can send that column
          // before every CTA has sent column j + 1, which this CTA does after this
          if (got && tid == 0) mbar_expect_tx(&s_bar[par], kRpColBytes(P));
          if (!got) {
            s_lost[par] = 1;
            set_status(st, kTimeout, 41);
            for (int d = 0; d < P; ++d) st_cluster(map_rank(&s_abort, (unsigned)d), 1);
          }
          // the warp goes on together: one lane's lost wait ends the column for all
          if (__any_sync(0xffffffffu, !got || lost)) {
            if (lost) {  // CTA-uniform: known to every column thread since the barrier
              stop = true;
              break;
            }
            stop_after = true;
            continue;
          }
          cand = MSG + par * kRpMaxCl * kRpMsg;
        } else {
          cand = CAND;
        }
        // the winner (first maximal |a|, lowest position on ties)
        {
          unsigned long long gk = 0ull;
          int gp = kNoPos;
          if (lane < (P > 1 ? P : CW)) {
            const double2 h = cand[lane * kRpMsg];
            gk = (unsigned long long)__double_as_longlong(h.x);
            gp = __double2hiint(h.y);
          }
          wc = warp_argmax(gk, gp);
        }
        const double2* wm = cand + max(wc, 0) * kRpMsg;
        const double whd = wm[0].y;
        const int wpos = __double2hiint(whd), wrow = __double2loint(whd);
        const double2 wi = wm[1];
        if (wc < 0 || wi.y == 0.0) {  // exact zero pivot: SingularMatrixException (Panel.hpp:76-77)
          if (cta == 0 && tid == 0) set_status(st, kSingular, offset + j + 1);
          stop = true;  // the same messages in every CTA: cluster-uniform
          break;
        }
        jdone = j + 1;
        if (tid == 0) {
          s_piv[j] = wpos;
          s_msrc[kRpW + t] = wrow;
        }
        // interchange of positions j and wpos (Panel.hpp:66-72)
        if (tpos == j) tpos = wpos;
        else if (tpos == wpos) tpos = j;
        if (gpos == j) gpos = wpos;
        else if (gpos == wpos) gpos = j;
        double u[kRpW];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const double2 x = wm[2 + q];
          u[2 * q] = x.x;
          u[2 * q + 1] = x.y;
        }
        // the winner's row is final: its entries go to the copy as they are
#pragma unroll
        for (int s = 0; s < RT; ++s) {
          const int lr = s * CT + tid;
          if (pos[s] == j) pos[s] = wpos;
          if (r0 + lr == wrow && pos[s] != kNoPos) {
            pos[s] = j;
            done[s] = true;
#pragma unroll
            for (int k = 0; k < kRpW; ++k)
              if (t + k < kRpW) Lb[(t + k) * ldl + lr] = v[s][k];
          }
        }
        // scale (Panel.hpp:78-79) and rank-1 update (Geru, :80); what rows
        // that are done (or no rows) compute here is not used
#pragma unroll
        for (int s = 0; s < RT; ++s) {
          const double l = v[s][0] * wi.x;
          if (!done[s]) Lb[t * ldl + s * CT + tid] = l;
#pragma unroll
          for (int k = 0; k < kRpW - 1; ++k) v[s][k] = fma(-l, u[k], v[s][k + 1]);
          v[s][kRpW - 1] = 0.0;
        }
      }
      stop = stop || stop_after;
      if (!stop) {
        // ---- write the sub-panel back, every row to its new position
#pragma unroll
        for (int s = 0; s < RT; ++s) {
          if (pos[s] != kNoPos) {
            double* dst = A + (long long)c0 * lda + pos[s];
            const double* from = Lb + s * CT + tid;
#pragma unroll 4
            for (int k = 0; k < w; ++k) dst[k * lda] = from[k * ldl];
          }
        }
        // The sub-panel's row moves: move i takes row c0 + i to where it is
        // now; move 16 + i takes the row chosen as pivot i to c0 + i when it
        // came from below the sub-panel.  A move is kept when this CTA owns
        // its destination.
        if (warp == 0) {
          __syncwarp();  // lane 0's s_msrc
          const int i = lane & 15;
          if (lane < kRpW) {
            s_msrc[i] = c0 + i;
            s_mdst[i] = (i < w && tpos != c0 + i && tpos >= r0 && tpos < r0 + rows) ? tpos : -1;
          } else {
            const int d = c0 + i;
            s_mdst[kRpW + i] = (i < w && s_msrc[kRpW + i] >= c1 && d >= r0 && d < r0 + rows) ? d : -1;
          }
        }
      }
    }
    stop = __syncthreads_or(stop);
    // The moves apply to the panel's other columns [0, c0) and [c1, b); rows
    // c0..c1-1 of columns [c1, b) become U12 and are not moved; U12's input
    // row i is the old row of pivot i.
    const int nout = b - w;
    const int ntr = b - c1;  // trailing panel columns
    constexpr int kMvPer = 2 * kRpW * 128 / kRpThreads, kU12Per = kRpW * 128 / kRpThreads;
    const int mcol = tid & 127, mq = tid >> 7;  // this thread's column and first move of the moves
    if (!stop) {
      // all of a thread's gathers are issued before any is stored, so their
      // L2 latencies overlap
      double g[kMvPer], gu[kU12Per];
#pragma unroll
      for (int q = 0; q < kMvPer; ++q) {
        const int mv = q * (kRpThreads / 128) + mq, d = s_mdst[mv];
        g[q] = 0.0;
        if (d >= 0 && mcol < nout) {
          const int col = mcol < c0 ? mcol : mcol + w;
          if (!(col >= c1 && d < c1)) g[q] = __ldcg(&A[(long long)col * lda + s_msrc[mv]]);
        }
      }
#pragma unroll
      for (int q = 0; q < kU12Per; ++q) {
        const int i = q * (kRpThreads / 128) + mq;
        gu[q] = (i < w && mcol < ntr) ? __ldcg(&A[(long long)(c1 + mcol) * lda + s_msrc[kRpW + i]]) : 0.0;
      }
#pragma unroll
      for (int q = 0; q < kMvPer; ++q) MV[(q * (kRpThreads / 128) + mq) * 128 + mcol] = g[q];
#pragma unroll
      for (int q = 0; q < kU12Per; ++q) {
        const int i = q * (kRpThreads / 128) + mq;
        if (i < w && mcol < ntr) U12[i * kRpLdU + mcol] = gu[q];
      }
    }
    // every source read and every sub-panel row written, cluster-wide
    cluster_arrive_release();
    cluster_wait_acquire();
    if (!stop) {
#pragma unroll
      for (int q = 0; q < kMvPer; ++q) {
        const int mv = q * (kRpThreads / 128) + mq, d = s_mdst[mv];
        if (d >= 0 && mcol < nout) {
          const int col = mcol < c0 ? mcol : mcol + w;
          if (!(col >= c1 && d < c1)) A[(long long)col * lda + d] = MV[mv * 128 + mcol];
        }
      }
      if (ntr > 0) {  // a trailing block follows only a full sub-panel: w = 16
        // L11 from the pivot rows, and the shared-memory copy of the rows that
        // were moved into this CTA's part
        const int i = tid >> 4, k = tid & 15, d = s_mdst[i];
        const double x = __ldcg(&A[(long long)(c0 + k) * lda + c0 + i]);
        if (d >= c1) Lb[k * ldl + d - r0] = __ldcg(&A[(long long)(c0 + k) * lda + d]);
        L11[i + k * 17] = x;
      }
    }
    __syncthreads();
    if (!stop && ntr > 0) {
      // U12 := inv(unit lower L11) A12, one column per thread, in shared memory
      if (tid < ntr) {
        double u[kRpW];
#pragma unroll
        for (int i = 0; i < kRpW; ++i) u[i] = U12[i * kRpLdU + tid];
#pragma unroll
        for (int i = 0; i < kRpW - 1; ++i)
#pragma unroll
          for (int k = i + 1; k < kRpW; ++k) u[k] = fma(-L11[k + i * 17], u[i], u[k]);
#pragma unroll
        for (int i = 0; i < kRpW; ++i) U12[i * kRpLdU + tid] = u[i];
        if (cta == 0)
#pragma unroll
          for (int i = 0; i < kRpW; ++i) A[(long long)(c1 + tid) * lda + c0 + i] = u[i];
      } else if (tid < 128) {
#pragma unroll
        for (int i = 0; i < kRpW; ++i) U12[i * kRpLdU + tid] = 0.0;
      }
    }
    __syncthreads();
    if (!stop && ntr > 0) {
      // A[r, c1:b) -= L[r, c0:c1) U12 for own rows r >= c1: 32 x 32 warp tiles
      const int lr1 = max(0, c1 - r0);  // a multiple of 16
      const int g = lane >> 2, t4 = lane & 3;
      const int trow = (rows - lr1 + 31) / 32, tcol = (ntr + 31) / 32;
      const int ntile = trow * tcol;
      auto row_col = [&](int tile, int& lr, int& cb) {
        lr = lr1 + (tile % trow) * 32;
        cb = (tile / trow) * 32;
      };
      // element (i, jn, q) of a tile: row 16 i + g (+ 8), column 8 jn + 2 t4 (+ 1)
      auto load = [&](double (&acc)[2][4][4], int tile) {
        int lr, cb;
        row_col(tile, lr, cb);
        const double* C = A + (long long)(c1 + cb + 2 * t4) * lda + r0 + lr + g;
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int jn = 0; jn < 4; ++jn)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const int rr = 16 * i + ((q >= 2) ? 8 : 0), cc = 8 * jn + (q & 1);
              acc[i][jn][q] =
                  (lr + g + rr < rows && cb + 2 * t4 + cc < ntr) ? __ldcg(&C[(long long)cc * lda + rr]) : 0.0;
            }
      };
      auto update = [&](double (&acc)[2][4][4], int tile) {
        int lr, cb;
        row_col(tile, lr, cb);
#pragma unroll
        for (int k0 = 0; k0 < kRpW; k0 += 8) {
          double af[2][4], bf[4][2];
          const double* la = &Lb[(k0 + t4) * ldl + lr + g];
#pragma unroll
          for (int i = 0; i < 2; ++i) {  // rows past the CTA's end are computed and not stored
            af[i][0] = -la[16 * i];
            af[i][1] = -la[16 * i + 8];
            af[i][2] = -la[4 * ldl + 16 * i];
            af[i][3] = -la[4 * ldl + 16 * i + 8];
          }
          const double* ub = &U12[(k0 + t4) * kRpLdU + cb + g];
#pragma unroll
          for (int jn = 0; jn < 4; ++jn) {
            bf[jn][0] = ub[8 * jn];
            bf[jn][1] = ub[4 * kRpLdU + 8 * jn];
          }
#pragma unroll
          for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int jn = 0; jn < 4; ++jn) dmma_16x8x8(acc[i][jn], af[i], bf[jn]);
        }
        double* C = A + (long long)(c1 + cb + 2 * t4) * lda + r0 + lr + g;
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int jn = 0; jn < 4; ++jn)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const int rr = 16 * i + ((q >= 2) ? 8 : 0), cc = 8 * jn + (q & 1);
              if (lr + g + rr < rows && cb + 2 * t4 + cc < ntr) C[(long long)cc * lda + rr] = acc[i][jn][q];
            }
      };
      // the next tile's loads are in flight while the current one is updated
      double xa[2][4][4], xb[2][4][4];
      if (warp < ntile) load(xa, warp);
#pragma unroll 1
      for (int tile = warp; tile < ntile; tile += 2 * kRpWarps) {
        if (tile + kRpWarps < ntile) load(xb, tile + kRpWarps);
        update(xa, tile);
        if (tile + kRpWarps < ntile) {
          if (tile + 2 * kRpWarps < ntile) load(xa, tile + 2 * kRpWarps);
          update(xb, tile + kRpWarps);
        }
      }
    }
    __syncthreads();
  }
  // all CTAs done with each other's shared memory and with the panel
  cluster_arrive_release();
  cluster_wait_acquire();
  if (cta != 0) return;
  if (tid < jdone) p[tid] = s_piv[tid] + offset;
  if (stop) return;
  // ComposePivots (ComposePivots.hpp:81-125) over the whole panel: original
  // row i is now at gpos; position i holds the original row that is there now,
  // or the row its pivot was first taken from
  if (tid < 128) s_inv[tid] = -1;
  __syncthreads();
  if (tid < ncols) {
    image[tid] = gpos;
    if (gpos < ncols) s_inv[gpos] = tid;
  }
  __syncthreads();
  if (tid < ncols) preimage[tid] = s_inv[tid] >= 0 ? s_inv[tid] : s_piv[tid];
  if (W == nullptr) return;
  // inv(unit lower L11) of the panel's top bb x bb block, by CTA 0: 16 x 16
  // diagonal-block inverses by warps, then the DMMA doubling steps
  const int bb = ncols;
  double* S = sm;
  tri_load_async(S, A, lda, bb, false);  // rows written by other CTAs: not read through L1 before
  cp_async_wait_all();
  __syncthreads();
  double* Xl = S + 128 * kLDS + 128;
  double* T = Xl + 8 * 16 * kLeafLD;
  const int bp = pad16_identity(S, bb);
  __syncthreads();
  for (int q = warp; q < bp / 16; q += kRpThreads / 32) warp_trinv16(S, kLDS, 16 * q, 1, Xl + q * 16 * kLeafLD, kLeafLD);
  __syncthreads();
  smem_trinv_dmma(S, bp, Xl, T);
  tri_store(S, W, ldw, bb, false, true);  // the leaves hold the unit diagonal
}

// Launch the register-resident panel when m fits one cluster (b <= m <= 16 x
// 1024 rows with a 16-CTA cluster) and b <= 128.  Returns EGPU_ERR_UNSUPPORTED
// when it does not apply.  The fewest rows per CTA, from 128 on, that fit one
// cluster: the trailing updates inside the panel get shorter with every CTA,
// the exchange only a little longer.  128 columns, us, with at most 16, 8 and 4
// CTAs: m = 1000 191 / 190 / 254, 2048 195 / 251 / 303, 8192 308 / 443 / 847.  Four column
// warps up to 256 rows a CTA and eight above: four warps with four rows a
// thread measured 0.36 ms at m = 8192.
int launch_lu_panel_rp(cudaStream_t st, int m, int b, double* A, long long lda, int* p, int offset, int* image,
                       int* preimage, double* W, int ldw, DevStatus* status, int cluster_max) {
  if (b > 128 || b < 1 || m < b || cluster_max < 1) return EGPU_ERR_UNSUPPORTED;
  using Kern = void (*)(int, int, double*, long long, int*, int, int*, int*, double*, int, DevStatus*, int);
  struct Config {
    Kern kern;
    int rmax;    // rows per CTA
    int cl_max;  // largest cluster it can be scheduled with (-1: not asked yet)
  };
  static Config configs[4] = {{lu_panel_rp_kernel<4, 1>, 128, -1}, {lu_panel_rp_kernel<4, 2>, 256, -1},
                              {lu_panel_rp_kernel<8, 2>, 512, -1}, {lu_panel_rp_kernel<8, 4>, 1024, -1}};
  Kern kern = nullptr;
  size_t smem = 0;
  int P = 0, R = 0;
  for (Config& c : configs) {  // the fewest rows per CTA that fit one cluster
    smem = sizeof(double) * rp_smem_doubles(c.rmax);
    if (c.cl_max < 0) {
      int fits = 0;
      if (cudaFuncSetAttribute(c.kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) == cudaSuccess &&
          cudaFuncSetAttribute(c.kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) {
        for (int n : {16, 8}) {
          cudaLaunchConfig_t cfg = {};
          cfg.gridDim = dim3(n);
          cfg.blockDim = dim3(kRpThreads);
          cfg.dynamicSmemBytes = smem;
          cudaLaunchAttribute attr[1];
          attr[0].id = cudaLaunchAttributeClusterDimension;
          attr[0].val.clusterDim.x = n;
          attr[0].val.clusterDim.y = 1;
          attr[0].val.clusterDim.z = 1;
          cfg.attrs = attr;
          cfg.numAttrs = 1;
          int ncl = 0;
          if (cudaOccupancyMaxActiveClusters(&ncl, c.kern, &cfg) == cudaSuccess && ncl > 0) {
            fits = n;
            break;
          }
        }
      }
      cudaGetLastError();
      c.cl_max = fits;
    }
    const int cmax = std::min(std::min(c.cl_max, kRpMaxCl), cluster_max);
    if (cmax < 1 || (m + c.rmax - 1) / c.rmax > cmax) continue;
    kern = c.kern;
    R = std::max(128, ((m + cmax - 1) / cmax + 15) / 16 * 16);
    P = (m + R - 1) / R;
    break;
  }
  if (kern == nullptr) return EGPU_ERR_UNSUPPORTED;
  TraceMark tm(st, kTracePanel, (double)m * b * b, 16.0 * m * b);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(P);
  cfg.blockDim = dim3(kRpThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = P;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, m, b, A, lda, p, offset, image, preimage, W, ldw, status, R);
  count_launch();
  if (e != cudaSuccess) {
    set_last_error(e, "lu_panel_rp launch", __FILE__, __LINE__);
    return EGPU_ERR_CUDA;
  }
  return EGPU_OK;
}

}  // namespace egpu
