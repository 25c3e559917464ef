// Seed-scan filter: which rows of the reference can give a window of the query a Smith-Waterman maximum of at least
// min_score.  The windows of the drivers overlap (38 columns every 8), so scanning each window by itself computes
// every (reference, query) cell 4.75 times, and nine windows in ten never reach min_score.  The filter computes every
// cell once, as an upper bound of the value any window's own DP can have there, and marks the places where the bound
// reaches the threshold; the exact window scan (seedscan.cu) then runs only there.  Windows that stay below
// min_score everywhere are never looked at again by the host, so what the filter leaves out cannot change a result.
//
// The bound.  a(i,j) = max(a(i-1,j-1) + s, q, 0), q = max(R(i-1,j), R(i,j-1)), R(i,j) = max(q + ext, a + open): a
// local alignment over the whole query in which a gap may turn between the two directions without opening anew.  By
// induction a is at least the H of any window's DP at (i,j), and R at least its E and F behind the cell.  A gap state
// in common costs one operation a cell less than E and F apart (three add-max operations per two cells where the
// exact scan takes four and a half), and lets through hardly more: a gap that turns once already costs open + ext.
//
// The check.  A cell with H >= T raises a(r,j) at every later row r by the vertical gap from it, so it is enough to
// look at every fourth row for a >= T + open + 2 ext: a third of a maximum per four cells instead of per cell.
//
// The tile.  One warp computes two column systems (the int16x2 halves) of 32 strips of 16 columns over a run of
// reference rows: lane l owns strip l of both systems and computes row t - l at step t, with the row's value to the
// left (a + open and R of lane l - 1's last column) by __shfl_up_sync.  A window's path spans 38 columns, so a system
// repeats the last three strips (48 columns) of the one before it and starts from zero there.  Reference rows before
// and after the tile's own are computed as they come (they only raise the bound), so no step is guarded.  State and
// scores take 48 registers and one 128-bit load from the warp's query profile per four columns; at 16 columns a lane
// the two shuffles of a step cost 2 of its 70 instructions.
//
// Measured on the 10,000-pair batch (534 G cells over all windows, 112 G over the pairs; serialised launch times):
// level 0 87 ms before, now 17.4 ms in the filter, 0.2 ms in its lists and 2.3 ms in the exact scan of the marked
// rows; the recursion rounds, which reuse the marks, 12 ms before and 1.8 ms now.  Bound: integer issue (ALU pipe at
// 78 %), as the exact scan.  The bound kept at match * window every 16 rows costs the filter 2 % and saves the exact
// scans 28 % (10.1 to 7.3 ms before the floor above min_score in those).  Widths of 8 to 24 columns a lane, chosen per
// pair to fit the query, would save 14 % of the columns but ran 1.5x slower mixed in one launch (instruction cache)
// and no faster sorted by width.
//
// References that are marked nearly everywhere: the filter stops where a pair's marks so far say that the exact scan
// would compute most rows anyway, a list of more rows than the whole scan's is not scanned, and one that is only too
// short is made again.  A pair of 200 kb that holds a 17-base word every 27, 60, 120 bases and no seed: 31.5, 32.5,
// 31.7 ms without the filter, 37.9, 38.0, 39.8 with the list's capacity as the only test, 32.1, 32.0, 11.9 now; of
// 40 and 2 kb 0.31 -> 0.71 -> 0.47, 0.47, 0.33.  The watch over the marks costs the filter 1.4 %.
#include <algorithm>
#include <type_traits>

#include "device_common.cuh"

namespace dcns {

namespace {

constexpr int kFC = kFiltCols;               // columns per lane and half
constexpr int kFNew = 32 - kFiltOverlap;     // strips of a system that no earlier system covers
constexpr int kFWarps = 4;

__device__ __forceinline__ uint32_t fpack2(int v) { return (uint32_t)(uint16_t)(int16_t)v * 0x00010001u; }

// The pair with task_begin <= t.
__device__ __forceinline__ int filt_pair_of(const FiltDesc &D, int t) {
  int lo = 0, hi = D.npairs - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (D.pairs[mid].task_begin <= t)
      lo = mid;
    else
      hi = mid - 1;
  }
  return lo;
}

// Blocks that the exact scan of a window pair around the lane's strip computes for a word of marks: those marked in
// this strip or the next three, and the warm-up before each run (some four blocks; runs closer than that are one).
__device__ __forceinline__ int filt_cost(uint32_t marks) {
  marks |= __shfl_down_sync(0xFFFFFFFFu, marks, 1);
  marks |= __shfl_down_sync(0xFFFFFFFFu, marks, 2);
  marks |= marks << 1;
  marks |= marks << 2;
  return __popc(marks | marks << 1);
}
// Whether a pair is marked nearly everywhere: most of its words of marks so far cost the exact scan five eighths of
// their rows or more (the filter is a fifth of the whole scan; words of few blocks count too little, since a run's
// warm-up may lie before them).  The rest of them are then set without the DP (marks only say where the exact scan
// looks), so that such a pair costs little more than the scan of every window that follows.
__device__ __forceinline__ bool filt_dense(unsigned long long seen) {
  const uint32_t words = (uint32_t)(seen >> 32), dense = (uint32_t)seen;
  return words >= 16 && dense > words / 2;
}

struct Stream {  // a lane's reference symbols, sixteen at a time
  const uint32_t *pk, *nm;
  int64_t k;  // arena index of the next sixteen
  __device__ __forceinline__ void load(uint32_t &w, uint32_t &n) {
    if (k < 0) {  // the arena's first sequence: A's in the places before its first base
      const int before = (int)-k;
      w = before < 16 ? __ldg(pk) << (2 * before) : 0u;
      n = before < 16 ? (__ldg(nm) << before) & 0xFFFFu : 0u;
    } else {
      const uint32_t a = __ldg(pk + (k >> 4)), b = __ldg(pk + (k >> 4) + 1);
      w = __funnelshift_r(a, b, 2u * (uint32_t)(k & 15));
      const uint32_t c = __ldg(nm + (k >> 5)), d = __ldg(nm + (k >> 5) + 1);
      n = __funnelshift_r(c, d, (uint32_t)(k & 31)) & 0xFFFFu;
    }
    k += 16;
  }
};

__global__ void __launch_bounds__(32 * kFWarps, 5)
    filter_kernel(FiltDesc D, Arena ar, int open, int ext, int match, int mismatch, int thr, int top) {
  __shared__ uint4 prof_all[kFWarps][4 * (kFC / 4) * 32];
  const int lane = threadIdx.x & 31, wb = threadIdx.x >> 5;
  const int t = blockIdx.x * kFWarps + wb;
  if (t >= D.ntasks) return;  // whole warp
  const int slot = filt_pair_of(D, t);
  const FiltPair P = D.pairs[slot];
  unsigned long long seen = __ldcg(D.seen + slot);
  const int rel = t - P.task_begin, ct = rel / P.nch, ch = rel % P.nch;
  uint4 *const prof = prof_all[wb];
  const uint32_t open2 = fpack2(open), ext2 = fpack2(ext), nopen2 = fpack2(-open);
  {
    // profile: score - open of both halves' columns against A, C, G, T; columns past the query hold -16384
    const int c0 = kFC * (2 * ct * kFNew + lane), c1 = c0 + kFC * kFNew;
    uint32_t *const w32 = reinterpret_cast<uint32_t *>(prof);
    for (int p = 0; p < kFC; ++p) {
      const int a = c0 + p < P.n2 ? base_code(ar, P.qry_base + c0 + p) : -1;
      const int b = c1 + p < P.n2 ? base_code(ar, P.qry_base + c1 + p) : -1;
#pragma unroll
      for (int sym = 0; sym < 4; ++sym) {
        const int c = sym + (sym >> 1);
        const int sa = a < 0 ? -16384 : score_of(c, a, match, mismatch) - open;
        const int sb = b < 0 ? -16384 : score_of(c, b, match, mismatch) - open;
        w32[((sym * (kFC / 4) + (p >> 2)) * 32 + lane) * 4 + (p & 3)] = (uint32_t)(uint16_t)sa | ((uint32_t)sb << 16);
      }
    }
    __syncwarp();
  }
  const int rows0 = ch * D.chunk, rows1 = min(P.n1, rows0 + D.chunk);
  const int rbeg = ch == 0 ? 0 : rows0 - D.warm;  // lane 0's row at step 0
  const int nblk = (rows1 - rbeg + 31 + 3 + 15) / 16;
  uint32_t *out = D.words + P.word_begin + (int64_t)rel * P.wpc * 64 + lane;
  const int strip = 2 * ct * kFNew + lane, strips = (P.n2 + kFC - 1) / kFC;  // strips of the query among the warp's
  const int used = __popc(__ballot_sync(0xFFFFFFFFu, strip < strips)) +
                   __popc(__ballot_sync(0xFFFFFFFFu, strip + kFNew < strips));
  if (filt_dense(seen)) {
    for (int k = 0; k < P.wpc; ++k, out += 64) out[0] = out[32] = ~0u;
    return;
  }
  Stream str{ar.pk, ar.nm, P.ref_base + rbeg - lane};
  uint32_t wcur, ncur, wnext, nnext;
  str.load(wcur, ncur);

  uint32_t Ga[kFC], Gb[kFC], R[kFC];  // a + open of the last row (two banks, as in the exact scan), R
#pragma unroll
  for (int p = 0; p < kFC; ++p) Ga[p] = open2, R[p] = open2;
  uint32_t lastT = open2, dg = open2, mrun;
  uint32_t acc0 = 0, acc1 = 0;
  const uint32_t thr2 = fpack2(thr + open - 1), top2 = fpack2(top + open);

  // One step: Gi holds the lane's previous row, Go receives this one.
  auto row = [&](uint32_t(&Gi)[kFC], uint32_t(&Go)[kFC], auto check, auto with_n) {
    uint32_t upT = __shfl_up_sync(0xFFFFFFFFu, lastT, 1);
    uint32_t left = __shfl_up_sync(0xFFFFFFFFu, R[kFC - 1], 1);
    upT = lane == 0 ? open2 : upT;
    left = lane == 0 ? open2 : left;
    const uint4 *pr = prof + (wcur & 3u) * (kFC / 4 * 32) + lane;
    const bool isn = decltype(with_n)::value && (ncur & 1u);
    wcur >>= 2;
    if (decltype(with_n)::value) ncur >>= 1;
    uint32_t gd = dg;
    uint4 q4 = make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int p = 0; p < kFC; ++p) {
      if ((p & 3) == 0) q4 = pr[(p >> 2) * 32];
      uint32_t s = (p & 3) == 0 ? q4.x : (p & 3) == 1 ? q4.y : (p & 3) == 2 ? q4.z : q4.w;
      if (decltype(with_n)::value) s = isn ? nopen2 : s;  // N scores 0 against everything
      const uint32_t q = __vmaxs2(R[p], left);
      const uint32_t a = __viaddmax_s16x2_relu(gd, s, q);
      gd = Gi[p];
      const uint32_t tv = __vadd2(a, open2);
      left = __viaddmax_s16x2(q, ext2, tv);
      R[p] = left;
      Go[p] = tv;
      if (decltype(check)::value && (p & 1)) mrun = __vimax3_s16x2(mrun, Go[p - 1], tv);
    }
    dg = upT;
    lastT = Go[kFC - 1];
  };
  using Yes = std::true_type;
  using No = std::false_type;
  for (int blk = 0; blk < nblk; ++blk) {
    str.load(wnext, nnext);
    mrun = 0x80008000u;
    if (!__any_sync(0xFFFFFFFFu, ncur != 0)) {
#pragma unroll 1
      for (int k = 0; k < 4; ++k) {
        row(Ga, Gb, No{}, No{});
        row(Gb, Ga, No{}, No{});
        row(Ga, Gb, No{}, No{});
        row(Gb, Ga, Yes{}, No{});
      }
    } else {
#pragma unroll 1
      for (int k = 0; k < 8; ++k) {
        row(Ga, Gb, No{}, Yes{});
        row(Gb, Ga, Yes{}, Yes{});
      }
    }
    // No window's own DP exceeds match * window, so the bound need not either: kept down every 16 rows, a long
    // alignment marks some 40 rows and columns around its path instead of half its score's worth.
#pragma unroll
    for (int p = 0; p < kFC; ++p) Ga[p] = __vmins2(Ga[p], top2), R[p] = __vmins2(R[p], top2);
    wcur = wnext, ncur = nnext;
    const uint32_t gt = __vcmpgts2(mrun, thr2);
    const uint32_t bit = 1u << (blk & 31);
    acc0 |= (gt & 0xFFFFu) ? bit : 0u;
    acc1 |= (gt >> 16) ? bit : 0u;
    if ((blk & 31) == 31 || blk == nblk - 1) {
      out[0] = acc0;
      out[32] = acc1;
      out += 64;
      bool dense = false;
      if (__any_sync(0xFFFFFFFFu, (acc0 | acc1) != 0))
        dense = 8 * (int)__reduce_add_sync(0xFFFFFFFFu, (unsigned)(filt_cost(acc0) + filt_cost(acc1))) >
                5 * used * ((blk & 31) + 1);
      acc0 = acc1 = 0;
      if (lane == 0) atomicAdd(D.seen + slot, (1ull << 32) | (dense ? 1u : 0u));
      if (blk == nblk - 1) break;
      if (filt_dense(seen)) {  // as it was a word ago: nothing waits for it
        for (int k = (blk >> 5) + 1; k < P.wpc; ++k, out += 64) out[0] = out[32] = ~0u;
        return;
      }
      seen = __ldcg(D.seen + slot);
    }
  }
}

// Calls emit(row_begin, row_end) for the runs of marked rows of columns [c_lo, c_hi) within rows [lo, hi), in row
// order; runs closer than the exact scan's warm-up are one (the rows between them would be computed twice).
template <class Emit>
__device__ __forceinline__ void filt_runs(const FiltDesc &D, const FiltPair &P, int c_lo, int c_hi, int lo, int hi,
                                          Emit &emit) {
  const int k0 = c_lo / kFC, k1 = (c_hi - 1) / kFC;
  int cs = -1, ce = -1;
  for (int ch = lo / D.chunk; ch <= (hi - 1) / D.chunk; ++ch) {
    const int rbeg = ch == 0 ? 0 : ch * D.chunk - D.warm;
    const int rlo = max(lo, ch * D.chunk), rhi = (int)min((int64_t)hi, (int64_t)(ch + 1) * D.chunk);
    const int w0 = (rlo - rbeg) >> 9, w1 = min(P.wpc - 1, (rhi - 1 - rbeg + 31) >> 9);
    for (int wi = w0; wi <= w1; ++wi) {
      uint32_t v = 0;
      int lmin = 31, lmax = 0;
      for (int k = k0; k <= k1; ++k) {
        const int sys = k >= kFiltOverlap ? (k - kFiltOverlap) / kFNew : 0, l = k - sys * kFNew;
        const int64_t task = (int64_t)(sys >> 1) * P.nch + ch;
        v |= __ldg(D.words + P.word_begin + (task * P.wpc + wi) * 64 + 32 * (sys & 1) + l);
        lmin = min(lmin, l), lmax = max(lmax, l);
      }
      while (v) {
        const int b = __ffs(v) - 1;
        const int len = __ffs(~(v >> b)) - 1;  // ones from bit b on (-1: all 32)
        const int nb = len < 0 ? 32 : len;
        v = nb + b >= 32 ? 0u : v & (0xFFFFFFFFu << (b + nb));
        const int a = max(rlo, rbeg + 512 * wi + 16 * b - lmax);
        const int e = min(rhi, rbeg + 512 * wi + 16 * (b + nb) - lmin);
        if (a >= e) continue;
        if (cs >= 0 && a - D.warm <= ce) {
          ce = max(ce, e);
        } else {
          if (cs >= 0) emit(cs, ce);
          cs = a, ce = e;
        }
      }
    }
  }
  if (cs >= 0) emit(cs, ce);
}

// A list's tiles from one thread's runs.  (Their rows are not counted: the plans of many items have longer tiles, whose
// warm-up matters little, and an addition per thread took a quarter of the plan.)
struct FiltEmit {
  const FiltTiles &T;
  int a, b;
  __device__ __forceinline__ void operator()(int rb, int re) {
    const int n = (re - rb + T.rows - 1) / T.rows, per = (re - rb + n - 1) / n;
    // one addition for the threads that are here together, whose tiles then lie next to each other: 4,000 pairs' plans
    // 161 and 159 us (an addition each, 32 bits; 172 and 198 in 64 bits) -> 65 and 58, their scans 1.04 -> 0.90 ms
    const unsigned here = __activemask();
    const int lead = __ffs(here) - 1;
    int before = 0, all = 0;
    for (unsigned m = here; m; m &= m - 1) {
      const int l = __ffs(m) - 1, v = __shfl_sync(here, n, l);
      before += l < (int)(threadIdx.x & 31) ? v : 0;
      all += v;
    }
    unsigned long long at = 0;
    if ((int)(threadIdx.x & 31) == lead) at = atomicAdd(T.count, (unsigned long long)all);
    at = __shfl_sync(here, at, lead) + (unsigned)before;
    for (int k = 0; k < n; ++k) {
      const int p = filt_place(at, k, T.cap);
      if (p < 0) break;
      T.list[p] = FiltTile{a, b, rb + k * per, min(re, rb + (k + 1) * per)};
    }
  }
};

// The same from a warp's runs: every lane holds one, and 32 of them go out at a time, each run's tiles written by all
// lanes.  What a warp holds at its end goes out with the other warps' of the block, by one addition to each counter:
// additions to one place are served one after the other, and two for each of some 25,000 warps took 50 us where the
// block's take 12.
constexpr int kPlanThreads = 256;
struct FiltEmitWarp {
  const FiltTiles &T;
  int a, b, warm, held = 0;
  int rb = 0, re = 0;  // the lane's run
  __device__ __forceinline__ void operator()(int from, int to) {
    if ((int)(threadIdx.x & 31) == held) rb = from, re = to;
    if (++held < 32) return;
    int n, per, end;
    const unsigned rows = tally(n, per, end);
    unsigned long long at = 0;
    if ((threadIdx.x & 31) == 31)
      at = atomicAdd(T.count, (unsigned long long)end), atomicAdd(T.count + 1, (unsigned long long)rows);
    write(__shfl_sync(0xFFFFFFFFu, at, 31), n, per, end);
    held = 0;
  }
  // Of the lane's run: its tiles and their rows; of the runs up to the lane's: their tiles.  The warp's rows.
  __device__ __forceinline__ unsigned tally(int &n, int &per, int &end) const {
    const int lane = threadIdx.x & 31;
    n = lane < held ? (re - rb + T.rows - 1) / T.rows : 0;
    per = n > 0 ? (re - rb + n - 1) / n : 0;
    end = n;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int v = __shfl_up_sync(0xFFFFFFFFu, end, d);
      if (lane >= d) end += v;
    }
    return __reduce_add_sync(0xFFFFFFFFu, n > 0 ? (unsigned)(re - rb + n * warm) : 0u);
  }
  __device__ __forceinline__ void write(unsigned long long at, int n, int per, int end) const {
    for (int r = 0; r < held; ++r) {
      const int rn = __shfl_sync(0xFFFFFFFFu, n, r), rper = __shfl_sync(0xFFFFFFFFu, per, r);
      const int from = __shfl_sync(0xFFFFFFFFu, rb, r), to = __shfl_sync(0xFFFFFFFFu, re, r);
      const int first = __shfl_sync(0xFFFFFFFFu, end, r) - rn;
      for (int k = threadIdx.x & 31; k < rn; k += 32) {
        const int p = filt_place(at, first + k, T.cap);
        if (p < 0) break;
        T.list[p] = FiltTile{a, b, from + k * rper, min(to, from + (k + 1) * rper)};
      }
    }
  }
  __device__ __forceinline__ void finish() const {  // every warp of the block
    constexpr int W = kPlanThreads / 32;
    __shared__ int tiles[W];
    __shared__ unsigned rows[W];
    __shared__ unsigned long long base;
    const int w = threadIdx.x >> 5;
    int n, per, end;
    const unsigned r = tally(n, per, end);
    if ((threadIdx.x & 31) == 31) tiles[w] = end, rows[w] = r;
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned long long t = 0, s = 0;
      for (int k = 0; k < W; ++k) t += (unsigned)tiles[k], s += rows[k];
      if (t) base = atomicAdd(T.count, t), atomicAdd(T.count + 1, s);
    }
    __syncthreads();
    if (held == 0) return;
    unsigned long long at = base;
    for (int k = 0; k < w; ++k) at += (unsigned)tiles[k];
    write(at, n, per, end);
  }
};

// The runs of part `part` of `parts` of the rows' words by a whole warp: the lanes load 32 words at a time, and the runs
// of the words that hold marks are followed in order by all lanes together.  A run that goes on in the next part is two.
__device__ __forceinline__ void filt_runs_warp(const FiltDesc &D, const FiltPair &P, int c_lo, int c_hi, int lo, int hi,
                                               int part, int parts, FiltEmitWarp &emit) {
  const int lane = threadIdx.x & 31;
  const int k0 = c_lo / kFC, k1 = (c_hi - 1) / kFC;
  int lmin = 31, lmax = 0;
  for (int k = k0; k <= k1; ++k) {
    const int l = k - (k >= kFiltOverlap ? (k - kFiltOverlap) / kFNew : 0) * kFNew;
    lmin = min(lmin, l), lmax = max(lmax, l);
  }
  const int ch0 = lo / D.chunk, items = ((hi - 1) / D.chunk - ch0 + 1) * P.wpc;
  const int per = ((items + parts - 1) / parts + 31) / 32 * 32;  // words of a part
  const int end = (int)min((int64_t)items, (int64_t)(part + 1) * per);
  int cs = -1, ce = -1;
  for (int64_t base = (int64_t)part * per; base < end; base += 32) {
    const int it = (int)base + lane;
    uint32_t v = 0;
    int row = 0, rlo = 0, rhi = 0;
    if (it < end) {
      const int ch = ch0 + it / P.wpc, wi = it % P.wpc;
      const int rbeg = ch == 0 ? 0 : ch * D.chunk - D.warm;
      rlo = max(lo, ch * D.chunk), rhi = (int)min((int64_t)hi, (int64_t)(ch + 1) * D.chunk);
      row = rbeg + 512 * wi;
      if (wi >= (rlo - rbeg) >> 9 && wi <= (rhi - 1 - rbeg + 31) >> 9) {
        for (int k = k0; k <= k1; ++k) {
          const int sys = k >= kFiltOverlap ? (k - kFiltOverlap) / kFNew : 0, l = k - sys * kFNew;
          const int64_t task = (int64_t)(sys >> 1) * P.nch + ch;
          v |= __ldg(D.words + P.word_begin + (task * P.wpc + wi) * 64 + 32 * (sys & 1) + l);
        }
      }
    }
    for (unsigned m = __ballot_sync(0xFFFFFFFFu, v != 0); m; m &= m - 1) {
      const int src = __ffs(m) - 1;
      uint32_t x = __shfl_sync(0xFFFFFFFFu, v, src);
      const int r = __shfl_sync(0xFFFFFFFFu, row, src);
      const int xlo = __shfl_sync(0xFFFFFFFFu, rlo, src), xhi = __shfl_sync(0xFFFFFFFFu, rhi, src);
      while (x) {
        const int b = __ffs(x) - 1;
        const int len = __ffs(~(x >> b)) - 1;
        const int nb = len < 0 ? 32 : len;
        x = nb + b >= 32 ? 0u : x & (0xFFFFFFFFu << (b + nb));
        const int a = max(xlo, r + 16 * b - lmax), e = min(xhi, r + 16 * (b + nb) - lmin);
        if (a >= e) continue;
        if (cs >= 0 && a - D.warm <= ce) {
          ce = max(ce, e);
        } else {
          if (cs >= 0) emit(cs, ce);
          cs = a, ce = e;
        }
      }
    }
  }
  if (cs >= 0) emit(cs, ce);
}

// Plans: one thread, or WARP one warp, per item.  A thread waits for each word before it looks at the next, so a plan
// of few items is as long as its longest reference has words; with a warp to each item, or to each part of it
// (blockIdx.y) where the items are so few that they leave multiprocessors idle, the words come 32 at a time.  Up to 256 items per multiprocessor: one pair of 5 kb (312 and 350 items)
// 66 -> 7 and 60 -> 7 us, two pairs of 200 kb 385 -> 140 and 472 -> 94 us.  The plans of 10,000 pairs have some 100,000
// items each, of a few words, and keep their threads.
constexpr int kPlanWarpItems = 256;

// Level-0 tiles: an item per two windows of a pair (slot of the level-0 table, duo).
template <bool WARP>
__global__ void __launch_bounds__(kPlanThreads, WARP ? 5 : 6)
    filter_plan_l0_kernel(FiltDesc D, L0Desc L, int64_t nduo, FiltTiles T) {
  const int64_t t = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / (WARP ? 32 : 1);
  int slot = 0, duo = 0, c_lo = 0, c_hi = 0;
  if (t < nduo) {
    int hi = D.npairs - 1;
    while (slot < hi) {  // the pair whose duos hold t
      const int mid = (slot + hi + 1) >> 1;
      if (D.pairs[mid].duo_begin <= t)
        slot = mid;
      else
        hi = mid - 1;
    }
    duo = (int)(t - D.pairs[slot].duo_begin);
    c_lo = 2 * duo * L.step;
    c_hi = min(D.pairs[slot].n2, min(2 * duo + 1, L.pairs[slot].nfast - 1) * L.step + L.window);
  }
  if constexpr (WARP) {
    FiltEmitWarp emit{T, slot, duo, D.warm};
    if (t < nduo) {
      const FiltPair P = D.pairs[slot];
      filt_runs_warp(D, P, c_lo, c_hi, 0, P.n1, (int)blockIdx.y, (int)gridDim.y, emit);
    }
    emit.finish();
  } else if (t < nduo) {
    FiltEmit emit{T, slot, duo};
    const FiltPair P = D.pairs[slot];
    filt_runs(D, P, c_lo, c_hi, 0, P.n1, emit);
  }
}

// Tiles of a round's tasks: an item per task.
template <bool WARP>
__global__ void __launch_bounds__(kPlanThreads, WARP ? 5 : 6)
    filter_plan_rec_kernel(FiltDesc D, const ScanTask *__restrict__ tasks, int first, int n, FiltTiles T) {
  const int64_t t = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / (WARP ? 32 : 1);
  ScanTask x{};
  if (t < n) x = tasks[first + (int)t];
  const bool on = x.tw > 0 && x.hi > x.lo;
  if constexpr (WARP) {
    FiltEmitWarp emit{T, first + (int)t, 0, D.warm};
    if (on)
      filt_runs_warp(D, D.pairs[D.slot[x.pair]], x.s2, x.s2 + x.tw, x.lo, x.hi, (int)blockIdx.y, (int)gridDim.y, emit);
    emit.finish();
  } else if (on) {
    FiltEmit emit{T, first + (int)t, 0};
    filt_runs(D, D.pairs[D.slot[x.pair]], x.s2, x.s2 + x.tw, x.lo, x.hi, emit);
  }
}

}  // namespace

void launch_filter(const FiltDesc &D, Arena ar, Params p, int thr, cudaStream_t st) {
  if (D.ntasks <= 0) return;
  filter_kernel<<<(D.ntasks + kFWarps - 1) / kFWarps, 32 * kFWarps, 0, st>>>(D, ar, p.open1, p.ext1, p.match,
                                                                            p.mismatch, thr, p.match * p.window);
}

// Parts of an item: of 128 words and more, while their warps all fit (32 to a multiprocessor).
unsigned plan_parts(const FiltDesc &D, int64_t items, int nsm) {
  return (unsigned)std::max<int64_t>(1, std::min<int64_t>((D.max_words + 127) / 128, 32 * nsm / items));
}

void launch_filter_plan_l0(const FiltDesc &D, L0Desc L, int64_t nduo, FiltTiles T, int nsm, cudaStream_t st) {
  if (nduo <= 0) return;
  if (nduo <= (int64_t)kPlanWarpItems * nsm)
    filter_plan_l0_kernel<true>
        <<<dim3((unsigned)((nduo + 7) / 8), plan_parts(D, nduo, nsm)), kPlanThreads, 0, st>>>(D, L, nduo, T);
  else
    filter_plan_l0_kernel<false><<<(unsigned)((nduo + 255) / 256), 256, 0, st>>>(D, L, nduo, T);
}

void launch_filter_plan_rec(const FiltDesc &D, const ScanTask *tasks, int first, int n, FiltTiles T, int nsm,
                            cudaStream_t st) {
  if (n <= 0) return;
  if (n <= kPlanWarpItems * nsm)
    filter_plan_rec_kernel<true>
        <<<dim3((unsigned)((n + 7) / 8), plan_parts(D, n, nsm)), kPlanThreads, 0, st>>>(D, tasks, first, n, T);
  else
    filter_plan_rec_kernel<false><<<(n + 255) / 256, 256, 0, st>>>(D, tasks, first, n, T);
}

}  // namespace dcns
