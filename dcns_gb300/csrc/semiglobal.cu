// Two-piece affine semi-global DP with z-drop and band (SemiGlobal_no_avx, impl/sequenceAlignment3.cpp:681-928)
// and its traceback.
//
// Rows are processed in stripes of 128: lane l owns the four consecutive rows 128s+1+4l .. 128s+4+4l of stripe s as
// an anti-diagonal wavefront: at step t lane l computes column j = jstart + t - l for its four rows top to bottom,
// receiving the cell above its first row (M, both vertical-gap states, and the query code) from lane l-1 through
// __shfl_up_sync; rows inside a lane pass the cell above in registers.  Lane 0 takes the row above the stripe from
// the stripe before, through a boundary row in global memory staged into shared memory (with the query codes) 32-63
// steps ahead of use.  The horizontal gap states stay in registers of the lane that owns the row.  Each cell's
// priority chain (diag > F1 > E1 > F2 > E2) and gap updates use the DPX max-with-predicate instruction, which yields
// the maximum and the reference's comparison bit at once.
//
// Two schedules of the stripes.  The batched path runs every stripe of every DP as an independent unit of one
// persistent grid (sg_flow_kernel: a long DP spreads over as many warps as it has stripes; the weighted drivers' DPs
// too).  The one-pair entry point without allocation keeps a whole DP on one CTA whose warps take its stripes in turn
// on a barrier schedule (sg_kernel), which needs only one CTA's boundary rows.
//
// A direction code is one byte per cell (state 0..4 in bits 0-2, gap-continuation flags in bits 3-6): the reference's
// traceback needs all seven bits to stay bit-exact.  sg_kernel stores them for every cell; the flow's DPs store
// checkpoints, and the traceback computes the codes again in the tiles its path goes through.  Layout of the stored
// codes: stripe-major, then step, then lane, one 32-bit word per
// lane and step holding its four rows, so the 32 lanes of a step write 128 consecutive bytes.  Cells the reference
// never writes (outside the band and the band's last column) are never read: the traceback's bounds test returns 255
// for them.
//
// Row-level decisions (running maximum, z-drop, empty row) depend on all earlier rows, so each stripe is computed
// first and its 128 rows are then evaluated in order; rows after a stop are discarded.  Rows past n2 + w have an empty
// band: the reference then scores only the last column from a stale cell of column n2-1, which is replayed exactly
// from the two values the DP left there.
#include <algorithm>
#include <climits>
#include <type_traits>

#include "device_common.cuh"

namespace dcns {

constexpr int kSgD = 2;              // super-steps between the starts of consecutive stripes
constexpr int kSgR = 4;              // rows per lane
constexpr int kSgRows = 32 * kSgR;  // rows per stripe

// Wavefront steps of one stripe (columns its rows span, plus the 31-step lane skew), an upper bound for every stripe.
// Computed in 64 bits: 2w + kSgRows does not fit an int for bands near 2^30.
__host__ __device__ inline int64_t sg_stride_steps(int n2, int w) {
  const int64_t span = 2 * (int64_t)w + kSgRows;
  return (n2 < span ? (int64_t)n2 : span) + 32;
}

int64_t sg_tb_bytes(int n1, int n2, int w) {
  if (n1 <= 0 || n2 <= 0) return 0;
  return (int64_t)((n1 + kSgRows - 1) / kSgRows) * sg_stride_steps(n2, w) * 32 * kSgR;
}

// Super-step length K (wavefront steps between CTA barriers) for a DP whose stripes take at most smax steps, on a CTA
// of nw warps:
//  * a warp finishes stripe s before stripe s+nw starts:   kSgD * nw * K >= smax
//  * every boundary cell is written at least one barrier before the consumer stages it 32-63 steps ahead of use.
//    Stripe s writes column j at its step j - jstart_s + 31; stripe s+1, which starts kSgD super-steps later, stages
//    it at step j - jstart_{s+1} - 63 or later, and jstart_{s+1} - jstart_s <= kSgRows; so the producer is at most
//    kSgRows + 94 steps ahead of that read, which must be at most (kSgD - 1) * K:  K >= kSgRows + 96
__host__ __device__ inline int sg_superstep(int n2, int w, int nw) {
  const int64_t span = 2 * (int64_t)w + kSgRows;
  const int smax = (int)(n2 < span ? (int64_t)n2 : span) + 31;
  const int k = (smax + kSgD * nw - 1) / (kSgD * nw);
  static_assert(kSgD == 2, "the lower bound below assumes two super-steps between stripe starts");
  return k > kSgRows + 96 ? k : kSgRows + 96;
}

// One CTA of NW warps per DP (stripe s on warp s mod NW), on a fixed schedule: stripe s runs steps
// [(g - 2s) K, (g - 2s + 1) K) in super-step g, and all warps meet at a barrier after every super-step, so every cross-warp dependency (the row above a stripe, the row
// evaluation order, the stop decision) crosses at least one __syncthreads.  There are no flag waits.
//   bnd   global scratch of this CTA: per stripe slot (s mod 8), the stripe's last row (M, F1, F2) by column
template <int NW>
__global__ void __launch_bounds__(32 * NW) sg_kernel(SgTask *__restrict__ tasks, const int *__restrict__ idx, int n,
                                                      Arena ar, Params P, uint8_t *__restrict__ tb,
                                                      SgRec *__restrict__ bnd_all, int64_t bnd_stride,
                                                      int *__restrict__ counter) {
  __shared__ SgRec stage[NW][2][32];  // per warp: boundary cells of the next two 32-column chunks
  __shared__ int stage_c[NW][2][32];  // and the query codes of those columns
  __shared__ int row_best[NW][kSgRows], row_bestj[NW][kSgRows];
  __shared__ int done_stripe[NW];
  __shared__ int s_max, s_end1, s_end2, s_rows, s_next_eval, s_stop, s_stale_last, s_stale_prev, s_task;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int o1 = P.open1, x1 = P.ext1, o2 = P.open2, x2 = P.ext2, w = P.bandwidth;
  SgRec *bnd = bnd_all + (int64_t)blockIdx.x * NW * bnd_stride;
  for (;;) {
    if (threadIdx.x == 0) s_task = atomicAdd(counter, 1);
    __syncthreads();
    const int q = s_task;
    if (q >= n) break;
    if (threadIdx.x < NW) done_stripe[threadIdx.x] = -1;
    if (threadIdx.x == 0) {
      // ends are 1-based rows/columns and stay -1 while no cell is positive: the reference then reports -2 (0-based)
      s_max = 0, s_end1 = -1, s_end2 = -1, s_rows = 0, s_next_eval = 0, s_stop = 0;
      s_stale_last = kOut, s_stale_prev = kOut;
    }
    __syncthreads();
    SgTask &T = tasks[idx[q]];
    const int n1 = T.n1, n2 = T.n2;
    const SeqView s1{T.base1, T.a1, T.dir}, s2{T.base2, T.a2, T.dir};
    const bool codes = T.want_codes != 0;
    const int r_last = n2 - 1 + w;
    const int n1_eff = (n1 <= 0 || n2 <= 0) ? 0 : min(n1, n2 + w);  // rows with a non-empty band
    const int nstripes = (n1_eff + kSgRows - 1) / kSgRows;
    const int64_t stride = sg_stride_steps(n2, w);
    const int K = sg_superstep(n2, w, NW);
    // per-warp stripe state (registers persist across super-steps)
    int cs = warp;  // this warp's current stripe
    int i0 = 0, jstart = 0, nsteps = 0, upB = 0, tdone = 0;
    bool live = false, produce = false;
    int ci[kSgR], c0[kSgR], c1[kSgR], e1[kSgR], e2[kSgR], best[kSgR], bestj[kSgR], prevM[kSgR];
    bool liver[kSgR];
    int diag = kOut, outM = kOut, outF1 = kOut, outF2 = kOut, outC = 0;
    SgRec *bup = nullptr, *bdown = nullptr;
    uint32_t *trow = nullptr;
    auto stage_chunk = [&](int chunk) {  // columns jstart + 32*chunk + lane of the row above, into stage[chunk & 1]
      const int j = jstart + 32 * chunk + lane;
      SgRec r{kOut, kOut, kOut};
      if (cs > 0 && j >= 1 && j <= upB) r = bup[j];
      stage[warp][chunk & 1][lane] = r;
      stage_c[warp][chunk & 1][lane] = (j >= 1 && j <= n2) ? s2.at(ar, j - 1) : 0;
    };
    auto begin_stripe = [&]() {
      const int s = cs;
      i0 = kSgRows * s + 1 + kSgR * lane;
      live = i0 <= n1_eff;
#pragma unroll
      for (int k = 0; k < kSgR; ++k) {
        const int i = i0 + k;
        liver[k] = i <= n1_eff;
        c0[k] = max(i - w, 1);
        c1[k] = min(i + w, n2);
        ci[k] = liver[k] ? s1.at(ar, i - 1) : 0;
        e1[k] = kOut, e2[k] = kOut, best[k] = 0, bestj[k] = 0, prevM[k] = kOut;
      }
      const int r0 = kSgRows * s + 1, rl = min(kSgRows * s + kSgRows, n1_eff);
      jstart = max(r0 - w, 1);
      nsteps = min(rl + w, n2) - jstart + 1 + 31;
      upB = min(kSgRows * s + w, n2);  // the row above (128s) holds columns [max(128s - w, 1), upB]
      produce = s + 1 < nstripes;
      trow = reinterpret_cast<uint32_t *>(tb + T.tb_off) + (int64_t)s * stride * 32;
      bup = bnd + (int64_t)((s + NW - 1) % NW) * bnd_stride;
      bdown = bnd + (int64_t)(s % NW) * bnd_stride;
      diag = (lane == 0 && s > 0 && jstart > 1) ? bup[jstart - 1].m : kOut;
      outM = kOut, outF1 = kOut, outF2 = kOut, outC = 0;
      tdone = 0;
      stage_chunk(0);
      stage_chunk(1);
      __syncwarp();
    };
    const int nsuper = nstripes > 0 ? kSgD * (nstripes - 1) + (int)((stride + K - 1) / K) + 1 : 0;
    bool started = false;
    for (int g = 0; g < nsuper; ++g) {
      // ---- compute: the warp's current stripe, if it is scheduled in this super-step
      if (cs < nstripes && g >= kSgD * cs) {
        if (!started) {
          begin_stripe();
          started = true;
        }
        const int tend = min(nsteps, (g - kSgD * cs + 1) * K);
        for (int t = tdone; t < tend; ++t) {
          int upM = __shfl_up_sync(0xFFFFFFFFu, outM, 1);
          int upF1 = __shfl_up_sync(0xFFFFFFFFu, outF1, 1);
          int upF2 = __shfl_up_sync(0xFFFFFFFFu, outF2, 1);
          int cj = __shfl_up_sync(0xFFFFFFFFu, outC, 1);
          if ((t & 31) == 0 && t > 0) {
            __syncwarp();
            stage_chunk((t >> 5) + 1);  // two chunks ahead of lane 0's reads
          }
          const int j = jstart + t - lane;
          if (lane == 0) {
            const SgRec r = stage[warp][(t >> 5) & 1][t & 31];
            upM = r.m, upF1 = r.f1, upF2 = r.f2;
            cj = stage_c[warp][(t >> 5) & 1][t & 31];
          }
          // the lane's rows top to bottom; (aM, aF1, aF2) = the cell above, dg = the diagonal cell
          int aF1 = upF1, aF2 = upF2, dg = diag;
          uint32_t word = 0xFFFFFFFFu;
#pragma unroll
          for (int k = 0; k < kSgR; ++k) {
            const int i = i0 + k;
            int cM = kOut, cF1 = kOut, cF2 = kOut;
            if (liver[k] && j >= c0[k] && j <= c1[k]) {
              const int dgv = (j == 1) ? (i == 1 ? 0 : kOut) : dg;
              const bool last = (j == c1[k]);
              const int fin1 = last ? kOut : aF1, fin2 = last ? kOut : aF2;
              int v = score_of(ci[k], cj, P.match, P.mismatch) + dgv;
              int d = 0;
              bool pr;
              v = __vibmax_s32(fin1, v, &pr);  // pr: !(v > fin1)
              d = pr ? 1 : d;
              v = __vibmax_s32(e1[k], v, &pr);
              d = pr ? 2 : d;
              v = __vibmax_s32(fin2, v, &pr);
              d = pr ? 3 : d;
              v = __vibmax_s32(e2[k], v, &pr);
              d = pr ? 4 : d;
              cM = v;
              if (v > best[k]) best[k] = v, bestj[k] = j;
              if (j == n2 - 1) {
                if (i == r_last) s_stale_last = v;
                if (i == r_last - 1) s_stale_prev = v;
              }
              if (!last) {
                const int h = v + o1, h2 = v + o2;
                cF1 = __vibmax_s32(fin1 + x1, h, &pr);
                d |= pr ? 8 : 0;
                e1[k] = __vibmax_s32(e1[k] + x1, h, &pr);
                d |= pr ? 16 : 0;
                cF2 = __vibmax_s32(fin2 + x2, h2, &pr);
                d |= pr ? 32 : 0;
                e2[k] = __vibmax_s32(e2[k] + x2, h2, &pr);
                d |= pr ? 64 : 0;
                word = (word & ~(0xFFu << (8 * k))) | ((uint32_t)d << (8 * k));
              }
              if (k == kSgR - 1 && lane == 31 && produce) bdown[j] = SgRec{cM, cF1, cF2};
            }
            dg = prevM[k];  // row k at column j - 1: the diagonal of row k + 1
            prevM[k] = cM;
            aF1 = cF1, aF2 = cF2;
            if (k == kSgR - 1) outM = cM;
          }
          if (codes && live) trow[(int64_t)t * 32 + lane] = word;
          diag = upM;
          outF1 = aF1, outF2 = aF2, outC = cj;
        }
        tdone = tend;
        if (tdone == nsteps) {  // stripe complete: publish its rows for the in-order evaluation
#pragma unroll
          for (int k = 0; k < kSgR; ++k) {
            row_best[cs % NW][kSgR * lane + k] = best[k];
            row_bestj[cs % NW][kSgR * lane + k] = bestj[k];
          }
          __syncwarp();
          if (lane == 0) done_stripe[cs % NW] = cs;
          cs += NW;
          started = false;
        }
      }
      __syncthreads();
      // ---- evaluate finished stripes in row order (warp 0, lane 0)
      if (threadIdx.x == 0 && !s_stop) {
        int mx = s_max, e1r = s_end1, e2r = s_end2, rows = s_rows, ne = s_next_eval;
        bool stop = false;
        while (!stop && ne < nstripes && done_stripe[ne % NW] == ne) {
          for (int r = 0; r < kSgRows && !stop; ++r) {
            const int ii = kSgRows * ne + 1 + r;
            if (ii > n1_eff) break;
            const int tm = row_best[ne % NW][r], tj = row_bestj[ne % NW][r];
            if (tm > mx) mx = tm, e1r = ii, e2r = tj;
            int l = (ii - e1r) - (tj - e2r);
            l = l > 0 ? l : -l;
            rows = ii;
            if (mx - tm > P.zdrop + l * x2)
              stop = true;
            else if (tj <= 0)
              stop = true;
          }
          ++ne;
        }
        s_max = mx, s_end1 = e1r, s_end2 = e2r, s_rows = rows, s_next_eval = ne;
        if (stop) s_stop = 1;
      }
      __syncthreads();
      if (s_stop || s_next_eval >= nstripes) break;  // uniform: every thread reads the same shared values
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      int mx = s_max, e1r = s_end1, e2r = s_end2, rows = s_rows;
      bool stop = s_stop != 0;
      if (!stop && n1 > n1_eff && n2 >= 1 && n1_eff > 0) {
        // empty-band rows: only the last column, from the stale column n2-1 of the row with the same parity
        const int c2 = s2.at(ar, n2 - 1);
        for (int ii = n1_eff + 1; ii <= n1 && !stop; ++ii) {
          const int dg = (n2 == 1) ? (int)kOut : (((ii - 1 - r_last) % 2 == 0) ? s_stale_last : s_stale_prev);
          int v = score_of(s1.at(ar, ii - 1), c2, P.match, P.mismatch) + dg;
          if (!(v > kOut)) v = kOut;
          const int tm = v > 0 ? v : 0, tj = v > 0 ? n2 : 0;
          if (tm > mx) mx = tm, e1r = ii, e2r = tj;
          int l = (ii - e1r) - (tj - e2r);
          l = l > 0 ? l : -l;
          rows = ii;
          if (mx - tm > P.zdrop + l * x2)
            stop = true;
          else if (tj <= 0)
            stop = true;
        }
      }
      T.score = mx;
      T.end1 = e1r;
      T.end2 = e2r;
      T.rows = rows;
      T.status = 0;
    }
    __syncthreads();
  }
}

// Resident CTAs per SM of the NW-warp kernel.
int sg_ctas_per_sm(int nw) {
  int nb = 0;
  cudaError_t e = nw == 2 ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, sg_kernel<2>, 64, 0)
                  : nw == 4 ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, sg_kernel<4>, 128, 0)
                            : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, sg_kernel<kSgNW>, 32 * kSgNW, 0);
  if (e != cudaSuccess) {
    (void)cudaGetLastError();
    nb = 1;
  }
  return nb > 0 ? nb : 1;
}

int64_t sg_bnd_bytes(int grid, int max_n2, int nw) {
  return (int64_t)grid * nw * ((int64_t)max_n2 + 2) * sizeof(SgRec);
}

void launch_semiglobal(SgTask *tasks, const int *idx, int n, Arena ar, Params p, uint8_t *tb, void *bnd,
                       int max_n2, int *work_counter, int grid, int nw, cudaStream_t st) {
  if (n <= 0) return;
  const int64_t stride = (int64_t)max_n2 + 2;
  if (nw == 2)
    sg_kernel<2><<<grid, 64, 0, st>>>(tasks, idx, n, ar, p, tb, (SgRec *)bnd, stride, work_counter);
  else if (nw == 4)
    sg_kernel<4><<<grid, 128, 0, st>>>(tasks, idx, n, ar, p, tb, (SgRec *)bnd, stride, work_counter);
  else
    sg_kernel<kSgNW><<<grid, 32 * kSgNW, 0, st>>>(tasks, idx, n, ar, p, tb, (SgRec *)bnd, stride, work_counter);
}

// ------------------------------------------------------------------ stripes as a flow of independent warp units
// The DPs of a launch are cut into their 128-row stripes (units), handed out by one atomic counter in the order of
// SgFlow::order; every warp of a persistent grid takes the next unit, computes it and takes the next.  The host orders
// the units stripe-major within groups of consecutive DPs (queue order: largest DPs first): stripe 0 of every DP of
// the group, then stripe 1, ... so that when a warp takes stripe s its stripe s - 1 has been running for a while, even
// when a few DPs of 200,000 rows make up the whole launch (in DP order the late stripes of one long DP would wait for
// its wavefront to reach them).  Stripe s of a DP depends only on stripe s - 1, whose last row reaches it through
// global memory: one boundary row per DP (stripe s reads a column before it overwrites it with its own last row), or,
// for DPs with a path, a row per stripe that stays as a checkpoint.  A boundary cell carries the number of the stripe
// that wrote it, in the same 128-bit store, so the consumer sees by the cell itself that it is there: no fence, no
// progress counter.  So a long DP runs on as many warps as it has stripes, each a few chunks behind the stripe above
// it.  Each DP's stripes are handed out in increasing order and a stripe waits only on lower stripes of its own DP,
// which are held by running warps, so the waits always end; each still has an iteration limit, after which the warp
// flags a device error (SgFlow::err) and abandons the DP.
//
// Row-level decisions (running maximum, z-drop, non-positive row maximum) are taken in row order: after computing
// stripe s, its warp waits until s - 1 is evaluated, evaluates its 128 rows from the DP's running state and
// publishes it; the stripe whose rows stop the DP, or its last stripe, writes the DP's result.  Stripes computed past
// the stop are abandoned at their next chunk (their checkpoints lie past the DP's last row and are never read).
// Iteration limit of every wait: each iteration is an L2 load and a 100-200 ns sleep, so a wait gives up after about
// a second or more; the longest legitimate wait (a stripe of 200,000 columns while its SM is shared) is some tens of
// ms.
constexpr int kSgSpin = 1 << 22;

__device__ __forceinline__ int sg_ld_acquire(const int *p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void sg_st_release(int *p, int v) {
  asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ int sg_ld_relaxed(const int *p) {
  int v;
  asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// A boundary cell and the tag that says which stripe wrote it, in one 128-bit access: the consumer of a column knows by
// the tag that the values beside it are the ones it waits for, without a fence and a counter between the two.
__device__ __forceinline__ void sg_st_cell(SgCell *p, int m, int f1, int f2, int tag) {
  const uint64_t lo = (uint64_t)(uint32_t)m | (uint64_t)(uint32_t)f1 << 32;
  const uint64_t hi = (uint64_t)(uint32_t)f2 | (uint64_t)(uint32_t)tag << 32;
  asm volatile("{\n .reg .b128 t;\n mov.b128 t, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], t;\n}" ::"l"(p), "l"(lo),
               "l"(hi)
               : "memory");
}
__device__ __forceinline__ SgCell sg_ld_cell(const SgCell *p) {
  uint64_t lo, hi;
  asm volatile("{\n .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}"
               : "=l"(lo), "=l"(hi)
               : "l"(p)
               : "memory");
  return SgCell{(int)(uint32_t)lo, (int)(lo >> 32), (int)(uint32_t)hi, (int)(hi >> 32)};
}

// Waits until *flag >= need, or until *stop_flag != 0; every lane polls (one broadcast load).  Returns 1 when the
// flag is reached, 0 when the DP stopped, -1 when the iteration limit ran out or another warp already flagged an
// error (*err), so that after one failed wait the whole grid winds down instead of timing out wait after wait.
__device__ __forceinline__ int sg_wait_at_least(const int *flag, int need, const int *stop_flag, const int *err) {
  for (int it = 0; it < kSgSpin; ++it) {
    const bool ok = sg_ld_acquire(flag) >= need;
    if (__all_sync(0xFFFFFFFFu, ok)) return 1;
    if (__any_sync(0xFFFFFFFFu, sg_ld_relaxed(stop_flag) != 0)) return 0;
    if ((it & 63) == 63 && __any_sync(0xFFFFFFFFu, sg_ld_relaxed(err) != 0)) return -1;
    __nanosleep(200);
  }
  return -1;
}

constexpr int kSgFlowWarps = 4;   // warps per block of the flow kernel
constexpr int kSgFlowBlocks = 2;  // blocks per SM that its registers must allow
constexpr int kSgChunk = 16;      // steps between two looks at the stripe above
constexpr int kSgUnroll = 8;      // of them unrolled

// ---- traceback checkpoints
// A DP whose path is wanted keeps no direction code per cell.  It keeps what is needed to compute any 128 x 128 tile
// of itself again: the row above every stripe (M, F1, F2 by column, what the stripes pass to each other anyway) and,
// for every stripe, each column that is a multiple of 128 (M and the two horizontal states behind it, by row): 28
// bytes per 128 cells instead of one per cell, and a forward pass of 12 integer operations a cell instead of about
// 26.  The traceback computes the tiles that its path goes through again, with codes, in shared memory.
constexpr int kSgTile = 128;  // columns between two column checkpoints

__host__ __device__ inline int64_t sg_ck_row_stride(int n2, int w) { return (n2 < 2 * (int64_t)w ? n2 : 2 * (int64_t)w) + 2; }
__host__ __device__ inline int64_t sg_ck_cols(int n2, int w) {
  const int64_t span = 2 * (int64_t)w + kSgRows;
  return (n2 < span ? n2 : span) / kSgTile + 2;
}
__host__ __device__ inline int64_t sg_ck_stripes(int n1, int n2, int w) {
  if (n1 <= 0 || n2 <= 0) return 0;
  const int64_t n1_eff = n1 < (int64_t)n2 + w ? n1 : (int64_t)n2 + w;
  return (n1_eff + kSgRows - 1) / kSgRows;
}
int64_t sg_ck_row_bytes(int n1, int n2, int w) {
  return sg_ck_stripes(n1, n2, w) * sg_ck_row_stride(n2, w) * (int64_t)sizeof(SgCell);
}
int64_t sg_ck_col_bytes(int n1, int n2, int w) {
  return sg_ck_stripes(n1, n2, w) * sg_ck_cols(n2, w) * 3 * kSgRows * (int64_t)sizeof(int);
}

// The row above stripe s as an array by column j (columns from jstart - 1 on exist).
__device__ __forceinline__ SgCell *sg_ck_row(uint8_t *tb, const SgTask &T, int w, int s) {
  const int jstart = max(kSgRows * s + 1 - w, 1);
  return reinterpret_cast<SgCell *>(tb + T.tb_off) + (int64_t)s * sg_ck_row_stride(T.n2, w) - (jstart - 1);
}
// Column j (a multiple of kSgTile, at least jstart) of stripe s: M, then E1, then E2, each by row.
__device__ __forceinline__ int *sg_ck_col(uint8_t *tb, const SgTask &T, int w, int s, int j) {
  const int jstart = max(kSgRows * s + 1 - w, 1);
  const int64_t q = (int64_t)s * sg_ck_cols(T.n2, w) + (j / kSgTile - jstart / kSgTile);
  return reinterpret_cast<int *>(tb + T.ck_off) + q * 3 * kSgRows;
}

// ---- scoring of a lane's rows.  KIND 0: the same parameters everywhere; 1, 2: the weighted drivers with one or two
// gap pieces (SemiGlobal_single_gap_penalty and SemiGlobal with weights, impl/sequenceAlignment3.cpp:1483-1890): row i
// takes the category of its seq1 base for the substitution, the horizontal gap states and the z-drop, and the
// category of the next base for the vertical gap states it leaves (a row at the end of seq1 keeps its own).
__device__ __forceinline__ int sgw_cat(const SgTask &T, const int16_t *__restrict__ wt, int i) {
  // category of DP row i (1-based): forward rows follow seq1 from a1, reverse rows go down from a1
  const int64_t pos = T.dir == 0 ? (int64_t)T.a1 + i - 1 : (int64_t)T.a1 - (i - 1);
  return wt[T.wbase + pos];
}

__device__ __forceinline__ int sgw_next_cat(const SgTask &T, const int16_t *__restrict__ wt, int i, int own) {
  const int64_t pos = T.dir == 0 ? (int64_t)T.a1 + i : (int64_t)T.a1 - i;
  return (pos < 0 || pos >= T.wlen) ? own : wt[T.wbase + pos];
}

template <int KIND>
struct SgRowParams {  // one row's: horizontal and vertical gap pieces, substitution scores
  int o1h, x1h, o2h, x2h, o1v, x1v, o2v, x2v, mt, mm;
  __device__ __forceinline__ void load(const SgTask &T, const SgWeights &W, int i, bool live) {
    const int rc = live ? sgw_cat(T, W.weights, i) : 0;
    const int nc = live ? sgw_next_cat(T, W.weights, i, rc) : 0;
    const int32_t *a = W.cats + 7 * rc, *b = W.cats + 7 * nc;
    mt = __ldg(a), mm = __ldg(a + 1), o1h = __ldg(a + 2), x1h = __ldg(a + 3), o2h = __ldg(a + 4), x2h = __ldg(a + 5);
    o1v = __ldg(b + 2), x1v = __ldg(b + 3), o2v = __ldg(b + 4), x2v = __ldg(b + 5);
  }
};
template <>
struct SgRowParams<0> {};

// Scores of one row against a column, from the column's selector: byte 0..3 of `prof` is the score against the 2-bit
// code 0..3, and a column N selects the zero bytes behind it; a row N has prof = 0 (Scorei: N scores 0).  A selector
// repeats the byte's sign into the upper bytes.
__device__ __forceinline__ uint32_t sg_selector(int code) {
  const uint32_t k = code == 2 ? 4u : (uint32_t)(code - (code >> 1) + (code >> 2));  // 0 1 3 4 -> 0 1 2 3
  return k == 4u ? 0x4444u : k | (k | 8u) * 0x1110u;
}
__device__ __forceinline__ uint32_t sg_profile(int ci, int match, int mismatch) {
  if (ci == 2) return 0u;
  uint32_t r = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) r |= (uint32_t)(uint8_t)(int8_t)(ci == k + (k >> 1) ? match : mismatch) << (8 * k);
  return r;
}
__device__ __forceinline__ int sg_score(uint32_t prof, uint32_t sel) {
  uint32_t d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(prof), "r"(0u), "r"(sel));
  return (int)d;
}
template <int KIND>
__device__ __forceinline__ int sg_row_score(uint32_t prof, const SgRowParams<KIND> &r, uint32_t sel) {
  if constexpr (KIND == 0) {
    return sg_score(prof, sel);
  } else {  // prof: 1 in the byte of the row's own code, so the selected byte says match; categories score in 32 bits
    const int same = sg_score(prof, sel);
    return (prof == 0u || sel == 0x4444u) ? 0 : (same != 0 ? r.mt : r.mm);
  }
}

// One cell: (aF1, aF2) = the vertical gap states of the cell above, dg = the diagonal cell, sc its score.  INSIDE:
// the cell is in the band, off the band's last column.  Otherwise cells outside the band leave kOut in M and both F
// and reset the row's horizontal states to kOut (the reference starts a row with them OUT).  The band's last column
// takes no vertical gap from above; under KIND 0 it takes the cell's maximum but leaves kOut in both F (its gap
// states are not updated, and the row's horizontal states are not read again), so that the row below reads kOut
// there by itself; the weighted DPs update every column and drop the states on reading.  With CODES, *d gets the
// cell's direction code: the winning state (priority order diag, F1, E1, F2, E2, a later state winning ties) and the
// four gap-continuation flags; codes of cells outside the band are never read by the traceback, nor is the last
// column's under KIND 0.
template <bool CODES, int KIND, bool INSIDE>
__device__ __forceinline__ int sg_cell(int sc, int dg, int aF1, int aF2, int &e1, int &e2, bool valid, bool last,
                                       const SgRowParams<KIND> &r, const Params &P, int &cF1, int &cF2, uint32_t *d) {
  int o1h, x1h, o2h, x2h, o1v, x1v, o2v, x2v;
  if constexpr (KIND == 0) {
    o1h = o1v = P.open1, x1h = x1v = P.ext1, o2h = o2v = P.open2, x2h = x2v = P.ext2;
  } else {
    o1h = r.o1h, x1h = r.x1h, o2h = r.o2h, x2h = r.x2h, o1v = r.o1v, x1v = r.x1v, o2v = r.o2v, x2v = r.x2v;
    if (!INSIDE && last) aF1 = kOut, aF2 = kOut;
  }
  int v, nF1, nF2 = kOut, nE1, nE2 = kOut;
  if constexpr (CODES) {
    bool pr, p1, p2, p3 = false, p4 = false;
    uint32_t c = 0;
    v = __vibmax_s32(aF1, sc + dg, &pr);  // pr: !(v > F1)
    c = pr ? 1u : c;
    v = __vibmax_s32(e1, v, &pr);
    c = pr ? 2u : c;
    if constexpr (KIND != 1) {
      v = __vibmax_s32(aF2, v, &pr);
      c = pr ? 3u : c;
      v = __vibmax_s32(e2, v, &pr);
      c = pr ? 4u : c;
      nF2 = __vibmax_s32(aF2 + x2v, v + o2v, &p3);
      nE2 = __vibmax_s32(e2 + x2h, v + o2h, &p4);
    }
    nF1 = __vibmax_s32(aF1 + x1v, v + o1v, &p1);
    nE1 = __vibmax_s32(e1 + x1h, v + o1h, &p2);
    *d = c | (p1 ? 8u : 0u) | (p2 ? 16u : 0u) | (p3 ? 32u : 0u) | (p4 ? 64u : 0u);
  } else {
    v = __viaddmax_s32(dg, sc, aF1);
    if constexpr (KIND != 1) {
      v = max(__vimax3_s32(v, e1, aF2), e2);
      nF2 = __viaddmax_s32(aF2, x2v, v + o2v);
      nE2 = __viaddmax_s32(e2, x2h, v + o2h);
    } else {
      v = max(v, e1);
    }
    nF1 = __viaddmax_s32(aF1, x1v, v + o1v);
    nE1 = __viaddmax_s32(e1, x1h, v + o1h);
  }
  if constexpr (INSIDE) {
    cF1 = nF1, cF2 = nF2, e1 = nE1, e2 = nE2;
    return v;
  } else {
    const bool upd = valid && (KIND != 0 || !last);
    cF1 = upd ? nF1 : kOut;
    cF2 = upd ? nF2 : kOut;
    e1 = valid ? nE1 : kOut;
    e2 = valid ? nE2 : kOut;
    return valid ? v : kOut;
  }
}

// A column of the row above, as a lane-0 cell reads it, with the column's selector in the place of the padding.
struct __align__(16) SgFeed {
  int m, f1, f2;
  uint32_t sel;
};

// CK: the DPs keep traceback checkpoints.
//
// Steps run in chunks of 16 of one of four kinds.  Inside: the columns of all lanes lie in the band of every row of the
// stripe, off the band's last column and the stale column: no band test (9 of 22 operations a cell).  Left: some rows
// have not reached their band's first column.  What lies left of a row's band feeds only cells left of the next rows'
// bands, but for its horizontal states and the row's maximum: those alone are masked.  Right: some rows are past
// their band's last column.  What lies right of it feeds only cells right of the next rows' bands, but for the
// vertical states that reach the next row's last column, which takes none: those and the maximum are masked.  Any:
// both ends in one chunk, and the stripes that hold a stale column.
//
// Bound: the latency of a step (185-215 cycles for 81 instructions without checkpoints, 230 with them) times the chain
// of stripes.  A stripe starts 31 + 2 chunks of steps behind the one above, and under a sliding band 128 columns more
// at its left end, and again ends so much later at its right end: with the full band tests there, 2.3 times the
// instructions, a chunk's wait was passed back along the band and all stripes went at half speed.  Two blocks per SM:
// a stripe slowed by its neighbours on the scheduler slows the chain behind it, so more warps than the DPs can use at
// a time cost more than they give.
//
// Measured on one GB300: one DP of 20,000 more rows under bands of 2,000 and 20,000: 6.2 -> 3.0 ms, 35 -> 19 us a
// stripe.  Of it the chunk looked ahead one instead of two chunks 0.5 ms, the left kind 0.3, the right kind 2.0.
// 30 DPs of a 200 kb pair 497 (direction codes for every cell, band tests in every cell, progress counters with
// release and acquire, 5 blocks per SM) -> 159 (codes computed again from checkpoints, tests only at the ends,
// tagged cells) -> 78 ms; 2,715 DPs of the 500-pair batch 39.9 -> 16.8 -> 13.6 ms; 400 DPs of 3 kb with a path
// 14.3 -> 4.85 -> 3.65 ms; the weighted drivers' 1,072 DPs 128.5 (one warp each, 32 rows at a time) -> 4.2 -> 3.0 ms.
// Blocks per SM, 2 / 3 / 4 (the last before the right kind): 78 / 102 / 142 ms on the long DPs, 13.6 / 13.8 / 15.9 on
// the batch.  Steps unrolled 1 / 4 / 8 / 16: 15.4 / 14.2 / 13.8 / 14.3 ms on the batch.  The checkpoints' address
// computed once per stripe and their test left out of chunks without such a column: 101 -> 83 instructions a step.
enum SgEdge { kSgInside, kSgLeft, kSgRight, kSgAny };
template <bool CK, int KIND>
__global__ void __launch_bounds__(32 * kSgFlowWarps, kSgFlowBlocks) sg_flow_kernel(SgFlow F, Arena ar, Params P,
                                                                                      SgWeights W,
                                                                                      uint8_t *__restrict__ tb) {
  __shared__ SgFeed stage[kSgFlowWarps][2][kSgChunk];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int w = P.bandwidth;
  for (;;) {
    long long u = 0;
    if (lane == 0) u = (long long)atomicAdd(F.unit_counter, 1ull);
    u = __shfl_sync(0xFFFFFFFFu, u, 0);
    if (u >= F.total_units) break;
    if (__any_sync(0xFFFFFFFFu, sg_ld_relaxed(F.err) != 0)) break;  // a wait ran out: the launch fails as a whole
    const int2 qs = F.order[u];  // the u-th unit handed out: stripe qs.y of DP qs.x
    const int q = qs.x, s = qs.y;
    SgTask &T = F.tasks[F.idx[q]];
    SgFlowDP &D = F.dps[q];
    const int n1 = T.n1, n2 = T.n2;
    const int n1_eff = (n1 <= 0 || n2 <= 0) ? 0 : min(n1, n2 + w);
    const int nstripes = (n1_eff + kSgRows - 1) / kSgRows;
    if (nstripes == 0) {  // nothing to align: the reference reports score 0 and ends -2 (0-based)
      if (lane == 0) T.score = 0, T.end1 = -1, T.end2 = -1, T.rows = 0, T.status = 0;
      continue;
    }
    if (__any_sync(0xFFFFFFFFu, sg_ld_relaxed(&D.stop) != 0)) continue;
    const SeqView s1{T.base1, T.a1, T.dir}, s2{T.base2, T.a2, T.dir};
    const int r_last = n2 - 1 + w;
    const bool produce = s + 1 < nstripes;
    // the row above and the row this stripe leaves, by column
    const SgCell *const bin = CK ? sg_ck_row(tb, T, w, s) : F.bnd + D.bnd_off;
    SgCell *const bout = CK ? sg_ck_row(tb, T, w, s + 1) : F.bnd + D.bnd_off;
    const int i0 = kSgRows * s + 1 + kSgR * lane;
    // per row of the lane: band [c0, c0 + span] (rows past the DP: an empty band), scores, running states
    uint32_t prof[kSgR];
    SgRowParams<KIND> rp[kSgR];
    int e1[kSgR], e2[kSgR], best[kSgR], bestj[kSgR], prevM[kSgR];
    int stale_rows = 0;  // bit k: row k is row r_last (bit 4 + k: row r_last - 1)
#pragma unroll
    for (int k = 0; k < kSgR; ++k) {
      const int i = i0 + k;
      const bool lv = i <= n1_eff;
      const int ci = lv ? s1.at(ar, i - 1) : 2;
      prof[k] = KIND == 0 ? sg_profile(ci, P.match, P.mismatch) : sg_profile(ci, 1, 0);
      if constexpr (KIND != 0) rp[k].load(T, W, i, lv);
      if (KIND == 0 && lv && i == r_last) stale_rows |= 1 << k;
      if (KIND == 0 && lv && i == r_last - 1) stale_rows |= 16 << k;
      e1[k] = kOut, e2[k] = kOut, best[k] = 0, bestj[k] = 0, prevM[k] = kOut;
    }
    const int r0 = kSgRows * s + 1, rl = min(kSgRows * s + kSgRows, n1_eff);
    const int jstart = max(r0 - w, 1), jend = min(rl + w, n2);
    const int nsteps = jend - jstart + 1 + 31;
    const int upB = min(kSgRows * s + w, n2);  // the row above (128s) holds columns [max(128s - w, 1), upB]
    // steps [in_lo, in_hi) have every lane's column in [max(r0 + 127 - w, 1), min(r0 + w, n2 - 1)): inside the band of
    // all rows, off the last and the stale column (rows past the DP compute what nobody reads)
    const int in_lo = max(r0 + kSgRows - 1 - w, 1) - jstart + 31;
    const int in_hi = min(r0 + w, n2 - 1) - jstart;
    const bool plain_right = KIND != 0 || rl < r_last - 1;  // no row of the stripe passes its stale column on
    int abandon = 0;  // 0 computing, 1 the DP stopped, -1 a wait ran out
    // column jstart + kSgChunk * chunk + lane of the row above, as it is now, and whether stripe s - 1 has written it
    // (tag s; the columns past row 128s's band hold kOut)
    auto look = [&](int chunk, SgCell &v) {  // the load alone, so that nothing waits for it: see `there`
      v = sg_ld_cell(bin + min(jstart + kSgChunk * chunk + (lane & (kSgChunk - 1)), upB));
    };
    auto there = [&](int chunk, SgCell &v) {
      const bool need = s > 0 && lane < kSgChunk && jstart + kSgChunk * chunk + lane <= upB;
      const bool ok = !need || v.tag == s;
      if (!need) v = SgCell{kOut, kOut, kOut, s};
      return __all_sync(0xFFFFFFFFu, ok) != 0;
    };
    // the words that hold those columns' symbols (loaded a chunk before they are staged)
    auto look_syms = [&](int chunk) {
      const int j = jstart + kSgChunk * chunk + lane;
      uint2 r{0u, 0u};
      if (lane < kSgChunk && j <= n2) {
        const int64_t k = s2.base + s2.a + (s2.dir == 0 ? j - 1 : 1 - j);
        r = uint2{__ldg(ar.pk + (k >> 4)), __ldg(ar.nm + (k >> 5))};
      }
      return r;
    };
    auto stage_cells = [&](int chunk, const SgCell &v, const uint2 &sy) {
      const int j = jstart + kSgChunk * chunk + lane;
      if (lane < kSgChunk) {
        const uint32_t k = (uint32_t)(s2.base + s2.a + (s2.dir == 0 ? j - 1 : 1 - j));
        const uint32_t two = (sy.x >> (2u * (k & 15u))) & 3u, n = (sy.y >> (k & 31u)) & 1u;
        const uint32_t code = s2.dir == 0 ? two : 3u - two;
        stage[warp][chunk & 1][lane] =
            SgFeed{v.m, v.f1, v.f2, j <= n2 && n == 0u ? code | (code | 8u) * 0x1110u : 0x4444u};
      }
    };
    // Looks until stripe s - 1 has written the chunk's columns (every wait ends or runs out of iterations, as
    // sg_wait_at_least).
    auto wait_cells = [&](int chunk, SgCell &v) {
      for (int it = 0;; ++it) {
        look(chunk, v);
        if (there(chunk, v)) return;
        if (__any_sync(0xFFFFFFFFu, sg_ld_relaxed(&D.stop) != 0)) {
          abandon = 1;
          return;
        }
        if (it >= kSgSpin || ((it & 63) == 63 && __any_sync(0xFFFFFFFFu, sg_ld_relaxed(F.err) != 0))) {
          abandon = -1;
          return;
        }
        __nanosleep(100);
      }
    };
    SgCell ahead;
    uint2 syms = look_syms(0);
    wait_cells(0, ahead);
    stage_cells(0, ahead, syms);
    // the diagonal of the stripe's first row at column jstart: cell (0, 0) = 0 for the DP's first row, else the
    // row above at jstart - 1 (kOut at column 0), written before column jstart
    int diag = kOut;
    if (s == 0) diag = lane == 0 ? 0 : kOut;
    if (s > 0 && jstart > 1 && abandon == 0) {
      SgCell d{kOut, kOut, kOut, 0};
      for (int it = 0; it < kSgSpin && d.tag != s; ++it) d = sg_ld_cell(bin + (jstart - 1));
      if (lane == 0) diag = d.m;
      if (__any_sync(0xFFFFFFFFu, d.tag != s)) abandon = -1;
    }
    __syncwarp();
    int outM = kOut, outF1 = kOut, outF2 = kOut;
    uint32_t outS = 0x4444u;
    const int cl = i0 - w;  // the lane's first row's first column, or less than 1
    const bool lane0 = lane == 0, write_bnd = lane == 31 && produce;
    // the lane's part of column checkpoint j: 3 kSgRows ints each, kSgTile columns apart
    static_assert(kSgTile == kSgRows, "");
    int *const ckp = CK ? sg_ck_col(tb, T, w, s, jstart / kSgTile * kSgTile) - (int64_t)3 * (jstart / kSgTile * kSgTile) +
                              kSgR * lane
                        : nullptr;

    auto step = [&](int t, const SgFeed *srow, auto edge, auto cks) {
      constexpr bool CKS = decltype(cks)::value;
      constexpr SgEdge EDGE = decltype(edge)::value;
      int upM = __shfl_up_sync(0xFFFFFFFFu, outM, 1);
      int aF1 = __shfl_up_sync(0xFFFFFFFFu, outF1, 1);
      int aF2 = KIND == 1 ? kOut : __shfl_up_sync(0xFFFFFFFFu, outF2, 1);
      uint32_t sel = __shfl_up_sync(0xFFFFFFFFu, outS, 1);
      const SgFeed rec = srow[t & (kSgChunk - 1)];  // every lane reads it, lane 0 uses it
      upM = lane0 ? rec.m : upM;
      aF1 = lane0 ? rec.f1 : aF1;
      if (KIND != 1) aF2 = lane0 ? rec.f2 : aF2;
      sel = lane0 ? rec.sel : sel;
      const int j = jstart + t - lane;
      int dg = diag;
      const bool stale_col = EDGE == kSgAny && KIND == 0 && stale_rows != 0 && j == n2 - 1;
#pragma unroll
      for (int k = 0; k < kSgR; ++k) {
        bool valid = true, last = false, end = false;
        if constexpr (EDGE == kSgLeft) valid = j >= max(cl + k, 1);
        if constexpr (EDGE == kSgRight) {
          const int c1 = min(cl + k + 2 * w, n2);
          valid = j <= c1;
          if (KIND != 0 && j == c1) aF1 = kOut, aF2 = kOut;
          end = j >= c1;
        }
        if constexpr (EDGE == kSgAny) {
          const int i = i0 + k, c0 = max(i - w, 1), c1 = min(i + w, n2);
          valid = i <= n1_eff && j >= c0 && j <= c1;
          last = j == c1;
        }
        int cF1, cF2;
        const int cM =
            sg_cell<false, KIND, EDGE != kSgAny>(sg_row_score<KIND>(prof[k], rp[k], sel), dg, aF1, aF2, e1[k], e2[k],
                                                 valid, last, rp[k], P, cF1, cF2, nullptr);
        if constexpr (EDGE == kSgRight && KIND == 0) {
          cF1 = end ? kOut : cF1;
          cF2 = end ? kOut : cF2;
        }
        if constexpr (EDGE == kSgLeft) {
          e1[k] = valid ? e1[k] : kOut;
          if (KIND != 1) e2[k] = valid ? e2[k] : kOut;
        }
        bool keep;  // !(cM > best): the first maximum of the row stays
        best[k] = __vibmax_s32(best[k], (EDGE == kSgLeft || EDGE == kSgRight) && !valid ? kOut : cM, &keep);
        bestj[k] = keep ? bestj[k] : j;
        if (stale_col && valid) {
          if ((stale_rows >> k) & 1) D.stale_last = cM;
          if ((stale_rows >> (4 + k)) & 1) D.stale_prev = cM;
        }
        if (k == kSgR - 1 && write_bnd && valid) sg_st_cell(bout + j, cM, cF1, cF2, s + 1);
        dg = prevM[k];  // row k at column j - 1: the diagonal of row k + 1
        prevM[k] = cM;
        aF1 = cF1, aF2 = cF2;
        if (k == kSgR - 1) outM = cM;
      }
      if constexpr (CKS) {
        if ((j & (kSgTile - 1)) == 0 && (EDGE == kSgInside || (j >= jstart && j <= jend))) {
          int *const c = ckp + (int64_t)3 * j;
          *reinterpret_cast<int4 *>(c) = make_int4(prevM[0], prevM[1], prevM[2], prevM[3]);
          *reinterpret_cast<int4 *>(c + kSgRows) = make_int4(e1[0], e1[1], e1[2], e1[3]);
          if (KIND != 1) *reinterpret_cast<int4 *>(c + 2 * kSgRows) = make_int4(e2[0], e2[1], e2[2], e2[3]);
        }
      }
      diag = upM;
      outF1 = aF1, outF2 = aF2, outS = sel;
    };

    // Chunks of kSgChunk steps.  At a chunk's start the warp looks at the columns of the next one (and at the DP's
    // stop flag); at its end they are staged if they were all there, so the steps hide the round trip to L2, and a
    // warp that runs too close behind its producer waits there.
    for (int tc = 0; tc < nsteps && abandon == 0; tc += kSgChunk) {
      const int chunk = tc / kSgChunk;
      const SgFeed *const srow = stage[warp][chunk & 1];
      const int stopped = sg_ld_relaxed(&D.stop);
      look(chunk + 1, ahead);
      syms = look_syms(chunk + 1);
      auto run = [&](auto edge, auto cks) {
#pragma unroll kSgUnroll
        for (int t = tc; t < tc + kSgChunk; ++t) step(t, srow, edge, cks);
      };
      const std::integral_constant<SgEdge, kSgInside> inside{};
      const std::integral_constant<SgEdge, kSgLeft> left{};
      const std::integral_constant<SgEdge, kSgRight> right{};
      const std::integral_constant<SgEdge, kSgAny> any{};
      const std::bool_constant<CK> ck{};
      const int tend = min(tc + kSgChunk, nsteps);
      if (tc >= in_lo && tc + kSgChunk <= in_hi) {
        // the chunk's columns end at j1 and begin 31 + kSgChunk - 1 before it: a column checkpoint among them?
        const int j1 = jstart + tc + kSgChunk - 1;
        if (CK && (j1 & (kSgTile - 1)) <= 31 + kSgChunk - 1)
          run(inside, ck);
        else
          run(inside, std::false_type{});
      } else if (tc + kSgChunk <= in_hi) {
        run(left, ck);
      } else if (tc >= in_lo && plain_right) {
        if (tend == tc + kSgChunk)
          run(right, ck);
        else
          for (int t = tc; t < tend; ++t) step(t, srow, right, ck);
      } else {
        for (int t = tc; t < tend; ++t) step(t, srow, any, ck);
      }
      if (__any_sync(0xFFFFFFFFu, stopped != 0)) abandon = 1;  // the DP ended
      if (abandon == 0 && !there(chunk + 1, ahead)) wait_cells(chunk + 1, ahead);
      __syncwarp();
      stage_cells(chunk + 1, ahead, syms);
      __syncwarp();
    }
    if (abandon < 0 && lane == 0) {
      atomicExch(F.err, 1);
      atomicExch(&D.stop, 1);
      T.status = 4;
    }
    if (abandon != 0) continue;
    // ---- the stripe's rows in order, from the DP's running state after stripe s - 1
    if (s > 0) {
      const int r = sg_wait_at_least(&D.evaluated, s, &D.stop, F.err);
      if (r <= 0) {
        if (r < 0 && lane == 0) {
          atomicExch(F.err, 1);
          atomicExch(&D.stop, 1);
          T.status = 4;
        }
        continue;
      }
      if (__any_sync(0xFFFFFFFFu, sg_ld_relaxed(&D.stop) != 0)) continue;  // an earlier stripe ended the DP
    }
    int mx = 0, e1r = -1, e2r = -1, rows = 0;  // ends are 1-based and stay -1 while no cell is positive
    if (s > 0) mx = sg_ld_relaxed(&D.mx), e1r = sg_ld_relaxed(&D.e1r), e2r = sg_ld_relaxed(&D.e2r),
               rows = sg_ld_relaxed(&D.rows);
    int zd[kSgR];  // the rows' z-drop, per category
    if constexpr (KIND != 0) {
#pragma unroll
      for (int k = 0; k < kSgR; ++k)
        zd[k] = i0 + k <= n1_eff ? __ldg(W.cats + 7 * sgw_cat(T, W.weights, i0 + k) + 6) : 0;
    }
    bool stop = false;
    for (int ol = 0; ol < 32; ++ol) {  // row 128s + 1 + 4 ol + k is lane ol's row k
#pragma unroll
      for (int k = 0; k < kSgR; ++k) {
        const int tm = __shfl_sync(0xFFFFFFFFu, best[k], ol), tj = __shfl_sync(0xFFFFFFFFu, bestj[k], ol);
        int z = P.zdrop, x = P.ext2;
        if constexpr (KIND != 0) {
          z = __shfl_sync(0xFFFFFFFFu, zd[k], ol);
          x = KIND == 1 ? 0 : __shfl_sync(0xFFFFFFFFu, rp[k].x2h, ol);
        }
        const int ii = r0 + kSgR * ol + k;
        if (!stop && ii <= n1_eff) {
          if (tm > mx) mx = tm, e1r = ii, e2r = tj;
          int l = (ii - e1r) - (tj - e2r);
          l = l > 0 ? l : -l;
          rows = ii;
          if (mx - tm > z + l * x)
            stop = true;
          else if (tj <= 0)
            stop = true;
        }
      }
    }
    if (lane == 0) {
      if (KIND == 0 && !stop && s == nstripes - 1 && n1 > n1_eff && n2 >= 1) {
        // empty-band rows: only the last column, from the stale column n2-1 of the row with the same parity
        const int c2 = s2.at(ar, n2 - 1);
        const int st_last = sg_ld_relaxed(&D.stale_last), st_prev = sg_ld_relaxed(&D.stale_prev);
        for (int ii = n1_eff + 1; ii <= n1 && !stop; ++ii) {
          const int dg = (n2 == 1) ? (int)kOut : (((ii - 1 - r_last) % 2 == 0) ? st_last : st_prev);
          int v = score_of(s1.at(ar, ii - 1), c2, P.match, P.mismatch) + dg;
          if (!(v > kOut)) v = kOut;
          const int tm = v > 0 ? v : 0, tj = v > 0 ? n2 : 0;
          if (tm > mx) mx = tm, e1r = ii, e2r = tj;
          int l = (ii - e1r) - (tj - e2r);
          l = l > 0 ? l : -l;
          rows = ii;
          if (mx - tm > P.zdrop + l * P.ext2)
            stop = true;
          else if (tj <= 0)
            stop = true;
        }
      }
      // the weighted DPs end at their first row with an empty band
      if (KIND != 0 && !stop && s == nstripes - 1 && n1 > n1_eff) rows = n1_eff + 1;
      if (stop || s == nstripes - 1) {
        T.score = mx;
        T.end1 = e1r;
        T.end2 = e2r;
        T.rows = rows;
        T.status = 0;
        if (stop) atomicExch(&D.stop, 1);
      } else {
        D.mx = mx, D.e1r = e1r, D.e2r = e2r, D.rows = rows;
      }
      __threadfence();
      sg_st_release(&D.evaluated, s + 1);
    }
    __syncwarp();
  }
}

int64_t sg_flow_units(int n1, int n2, int w) {
  const int64_t n1_eff = (n1 <= 0 || n2 <= 0) ? 0 : std::min<int64_t>(n1, (int64_t)n2 + w);
  return std::max<int64_t>(1, (n1_eff + kSgRows - 1) / kSgRows);
}

int64_t sg_flow_grid_warps(int nsm, int blocks) { return (int64_t)nsm * blocks * kSgFlowWarps; }

void launch_semiglobal_flow(const SgFlow &f, Arena ar, Params p, const SgWeights *wt, uint8_t *tb, bool path, int nsm,
                            int blocks_per_sm, cudaStream_t st) {
  if (f.total_units <= 0) return;
  const int64_t warps = std::min<int64_t>(f.total_units, sg_flow_grid_warps(nsm, blocks_per_sm));
  const int blocks = (int)((warps + kSgFlowWarps - 1) / kSgFlowWarps), threads = 32 * kSgFlowWarps;
  auto run = [&](auto kernel) { kernel<<<blocks, threads, 0, st>>>(f, ar, p, wt ? *wt : SgWeights{}, tb); };
  if (wt && wt->pieces == 1)
    path ? run(sg_flow_kernel<true, 1>) : run(sg_flow_kernel<false, 1>);
  else if (wt)
    path ? run(sg_flow_kernel<true, 2>) : run(sg_flow_kernel<false, 2>);
  else
    path ? run(sg_flow_kernel<true, 0>) : run(sg_flow_kernel<false, 0>);
}

// ------------------------------------------------------------------ traceback of the flow's DPs: tiles computed again
// The walk of sg_traceback_warp_kernel below (the same state machine, ends, padding and reversal), over the tiles of
// 128 rows x 128 columns that the path goes through, computed again from the checkpoints around them with their
// direction codes in shared memory.  One block of NT warps per DP: each warp computes one of the next NT tiles in the
// direction of the walk's state (a diagonal; a row or a column inside a gap, since the second gap piece may run over
// thousands of cells), because a tile takes one warp some 15 us whatever else the SM does; then the first warp walks
// them until the path leaves them all.  The walk takes a run at a time: the lanes look at the next 32 cells in the
// current direction, and a ballot says how far the state holds.  NT = 8 where the DPs leave SMs idle anyway (one
// block per SM), else 4 (three blocks per SM).
//
// Bound: the steps of a tile (159 of them, two warps to a scheduler: five sixths of the time), then the walk's chain of
// shared-memory reads and votes (520 cycles a run).  Half the tiles ahead are on the path; the others lie past a gap
// that moved it across a tile's corner.  Steps that all lanes take without a test of it, the last operation of the
// CIGAR in registers, tests of the band only in tiles that need them, and the reversal by all threads: 30 DPs of a
// 200 kb pair 28.4 -> 24.8 ms, 2,715 DPs of the 500-pair batch 2.16 -> 1.90 ms, 400 DPs of 3 kb 0.84 -> 0.66 ms.

struct SgTile {
  int s, ja, jb, tr;  // stripe, columns [ja, jb], rows up to tr
  int inside;         // whether its cells lie in every row's band, off the last column
};

template <int KIND, bool INSIDE>
__device__ __forceinline__ void sg_tile_codes(const SgTask &T, const Arena &ar, const Params &P, const SgWeights &W,
                                              uint8_t *__restrict__ tb, const SgTile &X, uint32_t (*code)[32],
                                              SgFeed *feed, int lane) {
  const int w = P.bandwidth, n2 = T.n2, n1_eff = min(T.n1, n2 + w);
  const SeqView s1{T.base1, T.a1, T.dir}, s2{T.base2, T.a2, T.dir};
  const int ts = X.s, ja = X.ja, jb = X.jb;
  const int jstart = max(kSgRows * ts + 1 - w, 1), upB = min(kSgRows * ts + w, n2);
  const int left = (jb - 1) / kSgTile * kSgTile;  // the column checkpoint left of the tile
  const SgCell *const bin = sg_ck_row(tb, T, w, ts);
  for (int c = lane; c <= jb - ja; c += 32) {
    const int j = ja + c;
    SgFeed rec{kOut, kOut, kOut, sg_selector(s2.at(ar, j - 1))};
    if (ts > 0 && j <= upB) rec.m = bin[j].m, rec.f1 = bin[j].f1, rec.f2 = bin[j].f2;
    feed[c] = rec;
  }
  const int i0 = kSgRows * ts + 1 + kSgR * lane;
  uint32_t prof[kSgR];
  SgRowParams<KIND> rp[kSgR];
  int e1[kSgR], e2[kSgR], prevM[kSgR];
  const bool from = left >= jstart;
  const int *const col = from ? sg_ck_col(tb, T, w, ts, left) + kSgR * lane : nullptr;
#pragma unroll
  for (int k = 0; k < kSgR; ++k) {
    const int i = i0 + k;
    const bool lv = i <= n1_eff;
    const int ci = lv ? s1.at(ar, i - 1) : 2;
    prof[k] = KIND == 0 ? sg_profile(ci, P.match, P.mismatch) : sg_profile(ci, 1, 0);
    if constexpr (KIND != 0) rp[k].load(T, W, i, lv);
    prevM[k] = from ? col[k] : kOut;
    const bool in = from && left >= i - w;  // left of its band a row has no horizontal gap
    e1[k] = in ? col[kSgRows + k] : kOut;
    e2[k] = (in && KIND != 1) ? col[2 * kSgRows + k] : kOut;
  }
  // the diagonal of the lane's first row at column ja: lanes above 0 take the lane above's checkpoint by shuffle
  int diag = kOut;
  if (lane == 0) diag = ts == 0 ? (ja == 1 ? 0 : kOut) : (ja > 1 && ja - 1 <= upB) ? bin[ja - 1].m : kOut;
  int outM = prevM[kSgR - 1], outF1 = kOut, outF2 = kOut;
  __syncwarp();
  const int nsteps = jb - ja + 1 + (X.tr - 1 - kSgRows * ts) / kSgR;
  auto step = [&](int t, auto all) {  // all: every lane is in the tile
    constexpr bool ALL = decltype(all)::value;
    int upM = __shfl_up_sync(0xFFFFFFFFu, outM, 1);
    int aF1 = __shfl_up_sync(0xFFFFFFFFu, outF1, 1);
    int aF2 = __shfl_up_sync(0xFFFFFFFFu, outF2, 1);
    const int c = t - lane, j = ja + c;
    const bool on = ALL || (c >= 0 && j <= jb);
    const SgFeed rec = feed[on ? c : 0];
    if (lane == 0) upM = rec.m, aF1 = rec.f1, aF2 = rec.f2;
    if (on) {
      int dg = diag;
      uint32_t word = 0;
#pragma unroll
      for (int k = 0; k < kSgR; ++k) {
        bool valid = true, last = false;
        if constexpr (!INSIDE) {
          const int i = i0 + k, c0 = max(i - w, 1), c1 = min(i + w, n2);
          valid = i <= n1_eff && j >= c0 && j <= c1;
          last = j == c1;
        }
        int cF1, cF2;
        uint32_t d = 0;
        const int cM = sg_cell<true, KIND, INSIDE>(sg_row_score<KIND>(prof[k], rp[k], rec.sel), dg, aF1, aF2, e1[k],
                                                   e2[k], valid, last, rp[k], P, cF1, cF2, &d);
        word |= d << (8 * k);
        dg = prevM[k];
        prevM[k] = cM;
        aF1 = cF1, aF2 = cF2;
      }
      outM = prevM[kSgR - 1];
      code[c][lane] = word;
      outF1 = aF1, outF2 = aF2;
    }
    diag = upM;
  };
  int t = 0;
  const int full = min(nsteps, jb - ja + 1);
  for (; t < min(nsteps, 31); ++t) step(t, std::false_type{});
#pragma unroll 2
  for (; t < full; ++t) step(t, std::true_type{});
  for (; t < nsteps; ++t) step(t, std::false_type{});
  __syncwarp();
}

template <int KIND, int NT>
__global__ void __launch_bounds__(32 * NT) sg_retrace_kernel(SgTask *__restrict__ tasks,
                                                                   const int *__restrict__ idx, Arena ar, Params P,
                                                                   SgWeights W, uint8_t *__restrict__ tb,
                                                                   uint32_t *__restrict__ cig) {
  extern __shared__ uint4 rt_smem[];  // per warp: codes [column][lane] (a lane's four rows a word), then the feed
  __shared__ SgTile tile[NT];
  __shared__ int more, nops;
  const int lane = threadIdx.x & 31, wb = threadIdx.x >> 5;
  auto codes_of = [&](int k) { return reinterpret_cast<uint32_t(*)[32]>(rt_smem) + k * kSgTile; };
  SgFeed *const feed = reinterpret_cast<SgFeed *>(reinterpret_cast<uint32_t(*)[32]>(rt_smem) + NT * kSgTile) +
                       wb * kSgTile;
  const int w = P.bandwidth;
  SgTask &T = tasks[idx[blockIdx.x]];
  const int n1 = T.n1, n2 = T.n2, n1_eff = (n1 <= 0 || n2 <= 0) ? 0 : min(n1, n2 + w), rows = T.rows;
  // the walk's state: the same in every lane of the first warp
  int ii = T.end1, jj = T.end2, state = 0, nc = 0;
  uint32_t *const out = cig + T.cig_off;
  const int cap = T.cig_cap;
  uint32_t last = 0xFFFFFFFFu;
  int len = 0;
  bool full = false;
  auto push = [&](uint32_t op, int n) {  // the last operation stays in registers until another follows
    if (op == last) {
      len += n;
      return;
    }
    if (len > 0) {
      if (nc >= cap) {
        full = true;
        return;
      }
      if (lane == 0) out[nc] = ((uint32_t)len << 4) | last;
      ++nc;
    }
    last = op;
    len = n;
  };
  auto in_band = [&](int i, int j) {
    return i > 0 && j > 0 && i <= rows && j >= max(i - w, 1) && (j < min(i + w, n2) || (KIND != 0 && j == min(i + w, n2)));
  };
  if (threadIdx.x < NT) tile[threadIdx.x].s = -1;
  for (;;) {
    __syncthreads();
    if (wb == 0) {
      int need = 0;
      int cur = 0;
      while (ii > 0 && jj > 0) {
        if (!in_band(ii, jj)) {  // reads 255: a gap state holds, anything else moves left
          if (state >= 1 && state <= 4) {
          } else {
            state = 7;
          }
          if (state == 1 || state == 3) {
            push(2, 1);
            --ii;
          } else {
            push(1, 1);
            --jj;
          }
          continue;
        }
        const int s = (ii - 1) / kSgRows;
        int k = 0;
        for (; k < NT; ++k) {
          const SgTile &X = tile[(cur + k) % NT];
          if (X.s == s && jj >= X.ja && jj <= X.jb && ii <= X.tr) break;
        }
        if (k == NT) {
          need = 1;
          break;
        }
        cur = (cur + k) % NT;
        const SgTile X = tile[cur];
        const int rtop = kSgRows * s;  // rows above the tile end here
        // a tile's codes are bytes [column][row]
        const uint8_t *const code = reinterpret_cast<const uint8_t *>(codes_of(cur));
        auto in_tile = [&](int i, int j) { return i > rtop && j >= X.ja && (X.inside || in_band(i, j)); };
        do {
          // the next 32 cells in the direction of the state
          const int di = state == 2 || state >= 4 ? 0 : 1, dj = state == 1 || state == 3 ? 0 : 1;
          const int ci = ii - di * lane, cj = jj - dj * lane;
          const bool in = in_tile(ci, cj);
          const int c = in ? (int)code[(cj - X.ja) * kSgRows + (ci - 1 - rtop)] : 255;
          const bool hold = in && (state == 0 ? (c & 7) == 0 : ((c >> (state + 2)) & 1) != 0);
          const unsigned m = __ballot_sync(0xFFFFFFFFu, hold), mi = __ballot_sync(0xFFFFFFFFu, in);
          const int run = m == 0xFFFFFFFFu ? 32 : __ffs(~m) - 1;
          const int fresh = __shfl_sync(0xFFFFFFFFu, c & 7, run & 31);
          if (run > 0) {
            push(state == 0 ? 0u : (state == 1 || state == 3) ? 2u : 1u, run);
            ii -= di * run;
            jj -= dj * run;
          }
          if (run < 32 && ((mi >> run) & 1u)) {  // the cell the run ends at, if it lies in this tile, starts a new state
            state = fresh;
            if (state == 1 || state == 3) {
              push(2, 1);
              --ii;
            } else if (state != 0) {
              push(1, 1);
              --jj;
            }
          }
        } while (in_tile(ii, jj));
      }
      if (lane == 0) {
        more = need;
        if (need) {  // the next tiles in the direction of the state
          int i = ii, j = jj;
          const bool go_up = state != 2 && state != 4, go_left = state != 1 && state != 3;
          for (int k = 0; k < NT; ++k) {
            SgTile X{-1, 0, -1, 0, 0};
            if (i > 0 && j > 0) {
              X.s = (i - 1) / kSgRows;
              const int r0 = kSgRows * X.s + 1, jstart = max(r0 - w, 1);
              const int c0 = max((j - 1) / kSgTile * kSgTile + 1, jstart);
              X.ja = c0;
              X.jb = k == 0 ? j : min((j - 1) / kSgTile * kSgTile + kSgTile, min(min(r0 + kSgRows - 1, n1_eff) + w, n2));
              X.tr = k == 0 ? i : min(r0 + kSgRows - 1, rows);
              if (X.jb < X.ja) X.s = -1;
              const int r1 = r0 + kSgRows - 1;
              X.inside = r1 <= n1_eff && X.ja >= max(r1 - w, 1) && X.jb < min(r0 + w, n2);
              const int up = i - r0 + 1, lf = j - c0 + 1;  // moves until the diagonal leaves at the top, at the left
              const int d = !go_up ? lf : !go_left ? up : min(up, lf);
              if (go_up) i -= d;
              if (go_left) j -= d;
            }
            tile[k] = X;
          }
        }
      }
    }
    __syncthreads();
    if (!more) break;
    const SgTile X = tile[wb];
    if (X.s >= 0) {
      if (X.inside)
        sg_tile_codes<KIND, true>(T, ar, P, W, tb, X, codes_of(wb), feed, lane);
      else
        sg_tile_codes<KIND, false>(T, ar, P, W, tb, X, codes_of(wb), feed, lane);
    }
  }
  if (wb == 0) {
    if (ii > 0) push(2, ii);
    if (jj > 0) push(1, jj);
    push(0xFFFFFFFFu, 0);  // the last operation out
    if (lane == 0) {
      nops = nc;
      T.ncig = nc;
      if (full) T.status = 3;
    }
  }
  __syncthreads();
  nc = nops;
  for (int a = threadIdx.x; a < nc / 2; a += 32 * NT) {  // the reference reverses the walk (:915)
    const uint32_t tmp = out[a];
    out[a] = out[nc - 1 - a];
    out[nc - 1 - a] = tmp;
  }
}

void launch_sg_retrace(SgTask *tasks, const int *idx, int n, Arena ar, Params p, const SgWeights *wt, uint8_t *tb,
                       uint32_t *cig, int nsm, cudaStream_t st) {
  if (n <= 0) return;
  auto run = [&](auto kernel, int nt) {
    const int smem = nt * kSgTile * (32 * (int)sizeof(uint32_t) + (int)sizeof(SgFeed));
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    kernel<<<n, 32 * nt, smem, st>>>(tasks, idx, ar, p, wt ? *wt : SgWeights{}, tb, cig);
  };
  const bool few = n <= nsm;
  if (!wt)
    few ? run(sg_retrace_kernel<0, 8>, 8) : run(sg_retrace_kernel<0, 4>, 4);
  else if (wt->pieces == 1)
    few ? run(sg_retrace_kernel<1, 8>, 8) : run(sg_retrace_kernel<1, 4>, 4);
  else
    few ? run(sg_retrace_kernel<2, 8>, 8) : run(sg_retrace_kernel<2, 4>, 4);
}

// ------------------------------------------------------------------ traceback (:869-914)
// State machine of impl/sequenceAlignment3.cpp:869-914: start in the state that produced the cell; a gap state persists
// while the cell's continuation flag is set; unwritten cells (outside the band, and the unweighted DP's last band
// column) read 255; the remaining rows and columns pad the walk as D and I, and the CIGAR is reversed. 
// (The codes of sg_kernel, one CTA per DP; the flow's DPs are walked by sg_retrace_kernel above.)
//
// One warp per DP walks through shared-memory windows of the code store.  In the stripe / step / lane
// layout every move of the walk (diagonal, up, left) goes to a lower address, at most 2 x 32 x R + R bytes lower,
// so the warp stages the kSgTbWin bytes that end at the current cell with coalesced 16-byte loads and lane 0 walks
// them until the path leaves the window below; one memory round trip then serves about kSgTbWin / (32 R) moves
// instead of one.  The CIGAR is built and reversed as in sg_traceback_kernel.  tb_bytes: size of the code store
// (no load goes past it).
constexpr int kSgTbWin = 4096;

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__global__ void __launch_bounds__(128) sg_traceback_warp_kernel(SgTask *__restrict__ tasks, const int *__restrict__ idx,
                                                                int n, int w, const uint8_t *__restrict__ tb,
                                                                int64_t tb_bytes, uint32_t *__restrict__ cig) {
  constexpr int R = kSgR, kRows = 32 * R;
  // two windows per warp: lane 0 walks one while the warp's asynchronous copies fill the other with the window just
  // below it, where the walk goes next unless it crosses into the stripe above (a jump: then a synchronous fill)
  __shared__ __align__(16) uint8_t win2[4][2][kSgTbWin];
  const int lane = threadIdx.x & 31, wb = threadIdx.x >> 5;
  const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (gw >= n) return;  // whole warp
  SgTask &T = tasks[idx[gw]];
  const int n2 = T.n2;
  const int64_t span = 2 * (int64_t)w + kRows;
  const int64_t stride = (n2 < span ? (int64_t)n2 : span) + 32;
  int ii = T.end1, jj = T.end2, state = 0, nc = 0;
  uint32_t *out = cig + T.cig_off;
  uint32_t last = 0xFFFFFFFFu;
  int64_t wbase[2] = {-1, -1};  // window [wbase, wbase + kSgTbWin) of the code store in each buffer; -1: none
  int cur = 0;
  bool pending = false;  // the other buffer is being filled with the window below the current one
  int64_t base = -1;
  const uint8_t *win = win2[wb][0];
  bool full = false;
  auto push = [&](uint32_t op) {
    if (nc > 0 && (last & 0xFu) == op) {
      last += 1u << 4;
      out[nc - 1] = last;
    } else if (nc < T.cig_cap) {
      last = (1u << 4) | op;
      out[nc++] = last;
    } else {
      full = true;
    }
  };
  auto fill = [&](int b, int64_t from) {  // every lane: its share of [from, from + kSgTbWin), asynchronously
    for (int c = lane; c < kSgTbWin / 16; c += 32) {
      const int64_t a = from + 16 * (int64_t)c;
      if (a + 16 <= tb_bytes)
        cp_async16(&win2[wb][b][16 * c], tb + a);
      else
        *reinterpret_cast<uint4 *>(&win2[wb][b][16 * c]) = make_uint4(0, 0, 0, 0);
    }
    cp_async_commit();
  };
  for (;;) {
    // lane 0 walks while the next cell is outside the band (no read) or inside the window; the warp refills the
    // window when the walk needs a cell below it
    int64_t need = -1;
    if (lane == 0) {
      while (ii > 0 && jj > 0) {
        int code = 255;
        const int c0 = max(ii - w, 1), c1 = min(ii + w, n2);
        if (ii <= T.rows && jj >= c0 && jj < c1) {
          const int s = (ii - 1) / kRows, rr = (ii - 1) % kRows, l = rr / R, kk = rr % R;
          const int jstart = max(kRows * s + 1 - w, 1);
          const int64_t t = jj - jstart + l;
          const int64_t a = T.tb_off + (((int64_t)s * stride + t) * 32 + l) * R + kk;
          if (base < 0 || a < base || a >= base + kSgTbWin) {
            need = a;
            break;
          }
          code = win[a - base];
        }
        if (state == 0)
          state = code & 7;
        else if (!((code >> (state + 2)) & 1))
          state = 0;
        if (state == 0) state = code & 7;
        if (state == 0) {
          push(0);
          --ii;
          --jj;
        } else if (state == 1 || state == 3) {
          push(2);
          --ii;
        } else {
          push(1);
          --jj;
        }
      }
    }
    need = __shfl_sync(0xFFFFFFFFu, need, 0);
    if (need < 0) break;
    cp_async_wait_all();  // this lane's copies, for either buffer, have landed
    __syncwarp();
    if (pending && need >= wbase[1 - cur] && need < wbase[1 - cur] + kSgTbWin) {
      cur = 1 - cur;  // the prefetched window below
    } else {
      // the window that ends (16-byte aligned) just past the needed byte, clipped to the store
      wbase[cur] = (((need + 16) & ~(int64_t)15) - kSgTbWin);
      if (wbase[cur] < 0) wbase[cur] = 0;
      fill(cur, wbase[cur]);
      cp_async_wait_all();
      __syncwarp();
    }
    pending = false;
    base = wbase[cur];
    win = win2[wb][cur];
    if (base > 0) {  // prefetch the window below while lane 0 walks this one
      wbase[1 - cur] = base - kSgTbWin > 0 ? base - kSgTbWin : 0;
      fill(1 - cur, wbase[1 - cur]);
      pending = true;
    }
  }
  cp_async_wait_all();
  if (lane == 0) {
    while (ii > 0) push(2), --ii;
    while (jj > 0) push(1), --jj;
    for (int a = 0, b = nc - 1; a < b; ++a, --b) {  // the reference reverses the walk (:915)
      const uint32_t tmp = out[a];
      out[a] = out[b];
      out[b] = tmp;
    }
    T.ncig = nc;
    if (full) T.status = 3;
  }
}

void launch_sg_traceback(SgTask *tasks, const int *idx, int n, int bandwidth, const uint8_t *tb, int64_t tb_bytes,
                         uint32_t *cig, cudaStream_t st) {
  if (n <= 0) return;
  sg_traceback_warp_kernel<<<(n + 3) / 4, 128, 0, st>>>(tasks, idx, n, bandwidth, tb, tb_bytes, cig);
}

}  // namespace dcns
