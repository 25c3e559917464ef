// Adaptive-band x-drop seed extension (SemiGlobal_xextend, impl/sequenceAlignment3.cpp:1234-1451, driven by
// x_extend_seed, impl/findSimilarFragmentsForPairedSequence4.cpp:205-285) and its traceback.
//
// Two forms of a pass, by band half-width w:
//   w <= 325   a group of lanes per pass, each lane a few neighbouring diagonals of the band in registers
//              (xdrop_band_kernel): one row per step, several passes per warp at narrow bands;
//   w > 325    one warp per pass across the band, the band rows in global scratch (xdrop_level_warp_kernel).
// The band is stored diagonal-relative: index k = j - i + w, so the diagonal predecessor of (i, j) sits at the same
// index in the previous row and the vertical predecessor at k + 1.
//
// A pass ends in one of three states: done, "restart" (the row maximum touched a band edge: the reference recomputes
// from scratch with 2w, and so does the next level), or "slot too small" (the direction codes outgrew the pass's
// traceback slot; the host relaunches it with a larger one).
//
// Direction codes (passes with a path) are 4-bit nibbles per band cell: bits 0-1 = winning state (0 diag, 1 vertical,
// 2 horizontal), bit 2 = vertical gap extended, bit 3 = horizontal gap extended.
#include <algorithm>
#include <type_traits>

#include "device_common.cuh"

namespace dcns {

__device__ __forceinline__ int xd_words_per_row(int w) { return (2 * w + 1 + 7) / 8; }

// How a band of half-width w is laid out over lanes, and its codes in memory.  Lane m of L owns the K band cells
// m K - pads .. m K - pads + K - 1 (the first `pads` of them lie left of the band) and stores a row's codes as `bytes`
// bytes.  Row i's bytes of lane m lie at ((i - 1 + m) L + m) * bytes (skew: lanes of one step write next to each
// other) or, for the warp form, at (i - 1) L bytes + m * bytes.
struct XBandLayout {
  int K, L, bytes, pads, skew;
};
__host__ __device__ inline XBandLayout xd_layout(int w) {
  const int nk = 2 * w + 1;
  XBandLayout b = nk <= 21    ? XBandLayout{3, 7, 2, 0, 1}
                  : nk <= 42  ? XBandLayout{6, 7, 4, 0, 1}
                  : nk <= 84  ? XBandLayout{6, 14, 4, 0, 1}
                  : nk <= 162 ? XBandLayout{6, 27, 4, 0, 1}
                  : nk <= 330 ? XBandLayout{11, 30, 8, 0, 1}
                  : nk <= 651 ? XBandLayout{21, 31, 12, 0, 1}
                              : XBandLayout{8, (nk + 7) / 8, 4, 0, 0};
  if (b.skew) b.pads = b.K * b.L - nk;
  return b;
}
// 32-bit words of a traceback slot of `rows` rows (a multiple of 4: slots start on 16-byte boundaries).
__host__ __device__ inline int64_t xd_slot(int w, int64_t rows) {
  const XBandLayout b = xd_layout(w);
  return ((rows + (b.skew ? b.L : 0)) * b.L * b.bytes + 15) / 16 * 4;
}
int64_t xd_slot_words(int w, int64_t rows) { return xd_slot(w, rows); }

struct XLevelArgs {
  XTask *tasks;
  XLevel L;
  int w;  // the level's band half-width (every pass of a level has it)
  int nsm;  // multiprocessors
};

// A traceback slot from the level's arena; passes of a host-driven round (no cursor) keep the one they were given.
__device__ __forceinline__ bool xd_take_slot(XTask &T, const XLevelArgs &A) {
  if (!A.L.tb_cursor) return true;
  const int64_t words = max((int64_t)4, xd_slot(T.w, min(T.n1, T.tb_rows)));
  if (words > INT32_MAX) return false;  // the capacity is an int: such a pass is retried with a whole-pass slot
  const unsigned long long off = atomicAdd(A.L.tb_cursor, (unsigned long long)words);
  if ((int64_t)off + words > A.L.tb_words) return false;
  T.tb_off = (int64_t)off;
  T.tb_cap = (int32_t)words;
  return true;
}

// Band-edge restarts go to the next level's list with the doubled band (as the reference does), passes whose slot did
// not fit to the retry list; a host-driven round reads the status itself.
__device__ __forceinline__ void xd_route(XTask &T, int id, const XLevelArgs &A) {
  if (!A.L.list_out) return;
  if (T.status == 1) {
    T.w *= 2;
    A.L.list_out[atomicAdd(A.L.count_out, 1)] = id;
  } else if (T.status == 2) {
    A.L.retry[atomicAdd(A.L.retry_count, 1)] = id;
  }
}

// ------------------------------------------------------------------ a group of lanes per pass
// One pass per group of L lanes (32 / L groups per warp), lane m owning K neighbouring diagonals.  In one step every
// lane of a group computes its K cells of one row, lane m one row behind lane m - 1: the horizontal gap state and the
// row's running maximum come from lane m - 1 as it left them a step ago, and the vertical gap state of the cell
// beyond the lane's last one from lane m + 1, which computes it as its first cell of this very step.  So a row costs
// one step of K cells and three shuffles whatever the band, every lane works on every step, and nothing but the
// sequences and the codes touches memory.  Scores come from a byte permutation: the row's profile (four
// scores by 2-bit code) under the column's selector, which moves one diagonal on per row.
//
// The last lane sees a row complete L - 1 steps after the first began it, and takes the row's decisions there (slot
// capacity, band-edge restart, score, x-drop, non-positive maximum); the steps the other lanes are ahead are
// discarded.  Groups take their next pass from the level's list as they finish.
//
// The row's first maximum travels as one word, value * 1024 + the cell counted from the band's end (1023 for its
// first cell, so that one test finds a maximum on either edge), and cells outside the DP hold -2^20: both hold while
// the higher score * the shorter sequence stays under 2^20 and the band at K L - P0 cells.  P0 >= 0: the band leaves
// exactly P0 cells of the first lane unused (the doubled bands of w = 10).  P0 = -1: any band, maximum and cell in two
// words.
//
// Passes with codes (P0 >= 0) hold 256 times the values and the codes below them: a vertical gap state ends in 1, a
// horizontal one in 2, a diagonal in 0, so the maxima settle ties as the reference's comparisons do (horizontal before
// vertical before diagonal) and leave the winner's code behind; 4 and 8 mark an extended gap, in copies that go to
// the codes only.  The gap's chain is one add-max a cell, as without codes.
//
// A row costs its instructions, 2-3 cycles each: 73 and 106 of them (119 and 192 with codes) at 3 and 6 cells a lane,
// where 95 and 130 (153 and 226) went with the profile's N test, the slot's and the last row's test and a branch to
// the decisions in every row.  Blocks that hold an N, begin a pass or may reach an end or the slot's run the full row
// (EDGES).  Level times per call, before -> after: two 200 kb pairs 8.01 -> 5.71 ms; 50,000 extension tasks
// 6.37 -> 5.11 ms; one 1 kb pair 190 -> 142 us.
//
// Measured on one GB300 against the forms this one replaces (one thread per pass, then 8-lane stripe wavefronts from
// row 96 or from band 40 on one warp; serialised level times per call): 10,000 pairs 41 -> 6.0 ms, of which 3x fewer
// reverse passes account for 9 ms; 50,000 extension tasks 28.8 -> 5.1 ms; 10,000-row passes of two 200 kb pairs
// 12.0 and 9.7 ms -> 1.2 and 1.05 ms at bands 10 and 20.  Bound: the latency of a row (0.12 us without codes, 0.15
// and 0.22 us with them: the shuffles, then the lane's cells) where passes are long or few, integer issue on short ones.
//
// Cells left of column 1 start from the same low value and never reach a cell inside (nothing is added to them but a
// few matches); cells right of column n2 feed only cells right of it, but the last column takes no vertical gap and
// the row's maximum must not see past it, so rows that reach it (i + w >= n2) test the column.
template <int K, int L, int P0, bool CODES>
__global__ void __launch_bounds__(128) xdrop_band_kernel(XLevelArgs A, Arena ar, Params P, uint8_t *__restrict__ tb) {
  constexpr bool WIDE = P0 < 0;
  constexpr int NG = 32 / L, KL = K * L, WN = (K + 7) / 8;
  constexpr int BYTES = K <= 4 ? 2 : 4 * WN;
  constexpr bool TAGS = CODES && !WIDE;  // codes below the values
  constexpr int S = TAGS ? 256 : 1;  // the scale of the cells' values
  constexpr int32_t NEG = WIDE ? kOut : -(1 << 20) * S, NEG_E = NEG | (TAGS ? 2 : 0), NEG_F = NEG | (TAGS ? 1 : 0);
  const int lane = threadIdx.x & 31, g = lane / L, m = lane - g * L;
  const bool in_group = g < NG, lead = m == 0, tail_lane = m == L - 1;
  const int first = in_group ? g * L : lane;
  const int w = A.w, nk = 2 * w + 1, pads = WIDE ? KL - nk : P0;
  const int m0 = pads / K, p0 = pads - m0 * K;  // the band's first cell
  const int n = *A.L.count_in;
  const int open = P.open1 * S, ext = P.ext1 * S, gext = max(P.ext1, P.open1) * S;
  // a horizontal gap extended: never where opening is dearer by the row (then e + ext < max(A, e) + open)
  const int ext_code = ext + (P.ext1 >= P.open1 ? 8 : 0);
  const uint32_t prof_rep = (uint32_t)(uint8_t)P.mismatch * 0x01010101u;
  const uint32_t prof_x = (uint32_t)(uint8_t)(P.match ^ P.mismatch);
  const int q0 = m * K - pads - w;  // query offset of the lane's cell p in row i: q0 + i - 1 + p

  int32_t M[K], F[K];
  uint32_t sel[K];
  int32_t e_out = NEG_E, best_out = 0, bk_out = 0;  // what the lane leaves to the next: gap state, row maximum (packed)
  Syms16 rs{0, 0}, qs{0, 0};
  SeqView s1{0, 0, 0}, s2{0, 0, 0};
  int id = -1, i = 0, n1 = 0, n2 = 0, last_step = 0;
  int score = 0, e1 = 0, e2 = 0, rows = 0, st = -1;  // the last lane's; st: the pass's status once it ended
  int row1 = 0;
  bool live = false;  // not WIDE: the last lane of a pass that goes on
  int32_t best = 0;  // not WIDE: the best row's packed maximum so far (of row e1)
  const int32_t xd = min(max(P.xdrop, -1), 1 << 20) * 1024;
  // the packed word's cell: KL - 1 - cell, and 1023 for the band's first
  const int32_t bc0 = m == 0 ? 1023 + P0 : KL - 1 - m * K;
  uint8_t *out = nullptr;
  bool more = in_group;
  // The first passes are dealt out, one to a warp over as many warps as the level needs (a warp per scheduler at
  // least), then a second to each, and so on; the rest go to whoever is free.  Fetched by all warps from the start,
  // the few passes of a wide level land on the schedulers whose blocks started first, two or three to each: 397
  // passes at band 80 of 50,000 extension tasks 0.75-1.25 -> 0.44 ms, one 1 kb pair's levels 142 -> 133 us.
  const int warp = blockIdx.x * 4 + (threadIdx.x >> 5);
  const int dealt_to = min((int)gridDim.x * 4, max((n + NG - 1) / NG, 4 * A.nsm)), dealt = NG * dealt_to;
  int next = warp < dealt_to && in_group ? g * dealt_to + warp : -1;
#pragma unroll
  for (int p = 0; p < K; ++p) M[p] = NEG, F[p] = NEG_F, sel[p] = 0x4444u;

  // Sixteen rows at a time: a pass that ends inside a block idles to its end (a few rows of some hundred), which
  // leaves the rows themselves free of votes.
  for (;;) {
    // groups without a pass take the level's next one
    while (__any_sync(0xFFFFFFFFu, id < 0 && more)) {
      const bool want = id < 0 && more;
      int q = n;
      if (want && lead) q = next >= 0 ? next : dealt + atomicAdd(A.L.fetch, 1);
      if (want) next = -1;
      q = __shfl_sync(0xFFFFFFFFu, q, first);
      if (want && q >= n) more = false;
      int ok = 1, cap = 0;
      long long off = 0;
      const bool take = want && more;
      if (take) {
        id = A.L.list_in[q];
        if (lead) {
          XTask &T = A.tasks[id];
          if (CODES) ok = xd_take_slot(T, A) ? 1 : 0;
          if (!ok) {
            T.status = 2;
            xd_route(T, id, A);
          } else if (T.n1 <= 0) {  // no row: done with nothing
            T.status = 0, T.rows = 0, T.score = 0, T.end1 = 0, T.end2 = 0;
            ok = 0;
          }
          off = T.tb_off;
          cap = T.tb_cap;
        }
      }
      ok = __shfl_sync(0xFFFFFFFFu, ok, first);
      off = __shfl_sync(0xFFFFFFFFu, off, first);
      cap = __shfl_sync(0xFFFFFFFFu, cap, first);
      if (take && !ok) id = -1;
      if (take && ok) {
        const XTask &T = A.tasks[id];
        n1 = T.n1, n2 = T.n2;
        s1 = SeqView{T.base1, T.a1, T.dir}, s2 = SeqView{T.base2, T.a2, T.dir};
        out = CODES ? tb + 4 * off + m * BYTES : nullptr;
        // steps whose bytes fit the slot (rows past it are never kept), at most 2^31 - 1 of them
        last_step = (int)min((int64_t)INT32_MAX, 4 * (int64_t)cap / (L * BYTES));
        i = 1 - m;
        score = e1 = e2 = rows = best = 0;
        st = -1;
        e_out = NEG_E, best_out = 0, bk_out = 0;
        // row 0: cell (0, 0) = 0, which is the diagonal of (1, 1), at band cell w; the rest is outside
#pragma unroll
        for (int p = 0; p < K; ++p) {
          M[p] = m * K + p - pads == w ? 0 : NEG;
          F[p] = NEG_F;
        }
        // selectors of row 1's first K - 1 cells, one place on (the row moves them back)
        sel[0] = 0x4444u;
#pragma unroll
        for (int p = 0; p < K - 1; ++p) {
          if (p % 16 == 0) qs = load16(ar, s2, n2, q0 + p);
          sel[p + 1] = TAGS ? sym_selector256(qs) : sym_selector(qs);
          next_sym(qs);
        }
      }
    }
    if (!__any_sync(0xFFFFFFFFu, id >= 0)) break;
    const bool have = id >= 0;
    if (have) {  // the next sixteen rows' symbols, from where the lane's pass is
      const int r = max(i, 1) - 1;
      qs = load16(ar, s2, n2, q0 + K - 1 + r);
      rs = load16(ar, s1, n1, r);
    }

    uint8_t *at = nullptr;
    if (CODES && have) at = out + (int64_t)(i + m - 1) * (L * BYTES);
    // ---- one row per lane.  `edges`: some lane has not begun its pass, may reach the last column or row or its slot's
    // end, or holds an N
    live = have && tail_lane;
    auto row = [&](auto edges) {
      constexpr bool EDGES = decltype(edges)::value;
      const bool on = !EDGES || (have && i >= 1);
      int32_t e = __shfl_up_sync(0xFFFFFFFFu, e_out, 1);
      int32_t b = __shfl_up_sync(0xFFFFFFFFu, best_out, 1);
      int32_t bk = WIDE ? __shfl_up_sync(0xFFFFFFFFu, bk_out, 1) : 0;
      const int lim = n2 - (q0 + i);  // cell p is in column q0 + i + p: p == lim is the last column
      uint32_t prof = 0, cw[WN];
#pragma unroll
      for (int c = 0; c < WN; ++c) cw[c] = 0;
      if (on) {
#pragma unroll
        for (int p = 0; p + 1 < K; ++p) sel[p] = sel[p + 1];
        if (EDGES) {
          sel[K - 1] = (TAGS ? sym_selector256(qs) : sym_selector(qs));
          prof = sym_profile(rs, P.match, P.mismatch);
          next_sym(qs);
          next_sym(rs);
        } else {  // no N
          sel[K - 1] = (qs.w & 3u) * (TAGS ? 0x1110u : 0x1111u) + (TAGS ? 0x8804u : 0x8880u);
          prof = prof_rep ^ __funnelshift_l(0u, prof_x, rs.w << 3);
          qs.w >>= 2, rs.w >>= 2;
        }
      }
      auto cell = [&](int p, int32_t fin) {
        if (WIDE ? (p == p0 && m == m0) : (p == P0 && m == 0)) e = NEG_E, b = 0, bk = 0;
        const int sc = perm_score(prof, 0u, sel[p]);
        if (EDGES) fin = p >= lim ? NEG_F : fin;
        int32_t v;
        if constexpr (TAGS) {
          const int32_t A_ = __viaddmax_s32(M[p], sc, fin);
          v = max(A_, e);
          const int32_t he = (A_ & ~255) + (open + 2);
          const int32_t he_code = __viaddmax_s32(e, ext_code, he);
          e = __viaddmax_s32(e, gext, he);
          if (EDGES) v = p > lim ? NEG : v;
          const int32_t c = v & ~255, h = c + (open + 1);
          const int32_t f_code = __viaddmax_s32(fin, ext + 4, h);
          F[p] = __viaddmax_s32(fin, ext, h);
          const uint32_t d = ((uint32_t)v & 3u) | ((uint32_t)f_code & ~3u);
          cw[p / 8] += (((d & 7u) | ((uint32_t)he_code & ~7u)) & 15u) * (1u << (4 * (p % 8)));
          v = c;
        } else if constexpr (CODES) {
          bool pv, ph, p1, p2;
          v = __vibmax_s32(fin, M[p] + sc, &pv);  // pv: the vertical gap wins ties with the diagonal
          v = __vibmax_s32(e, v, &ph);                 // ph: the horizontal gap wins ties
          if (EDGES) v = p > lim ? NEG : v;
          const int32_t h = v + open;
          F[p] = __vibmax_s32(fin + ext, h, &p1);
          e = __vibmax_s32(e + ext, h, &p2);
          const uint32_t d = (ph ? 2u : pv ? 1u : 0u) | (p1 ? 4u : 0u) | (p2 ? 8u : 0u);
          cw[p / 8] |= d << (4 * (p % 8));
        } else {
          // the gap's chain is one add-max a cell: max(e, A) + open and e + ext give max(e + max(ext, open), A + open)
          const int32_t A_ = __viaddmax_s32(M[p], sc, fin), ao = A_ + open;
          v = max(A_, e);
          if (EDGES) v = p > lim ? NEG : v;
          F[p] = EDGES ? __viaddmax_s32(fin, ext, v + open) : __viaddmax_s32(fin, ext, __viaddmax_s32(e, open, ao));
          e = __viaddmax_s32(e, gext, ao);
        }
        M[p] = v;
        if constexpr (WIDE) {
          if (v > b) b = v, bk = m * K + p;
        } else {
          b = __viaddmax_s32(v * (1024 / S) + (p == P0 ? bc0 : KL - 1 - m * K), -p, b);
        }
      };
      if (on) cell(0, F[1]);
      int32_t fr = __shfl_down_sync(0xFFFFFFFFu, F[0], 1);
      if (tail_lane) fr = NEG_F;
      if (on) {
#pragma unroll
        for (int p = 1; p < K; ++p) cell(p, p + 1 < K ? F[p + 1] : fr);
        e_out = e, best_out = b, bk_out = bk;
      }
      if constexpr (CODES) {  // the step's bytes of a group lie next to each other
        if (on && have && (!EDGES || i + m <= last_step)) {
          if constexpr (BYTES == 2) {
            *reinterpret_cast<uint16_t *>(at) = (uint16_t)cw[0];
          } else {
#pragma unroll
            for (int c = 0; c < WN; ++c) reinterpret_cast<uint32_t *>(at)[c] = cw[c];
          }
        }
        at += L * BYTES;
      }
      // the last lane's row is complete: take its decisions
      if constexpr (!WIDE) {
        if (!EDGES || on) {
          if (b > (best | 1023)) best = b, e1 = i;
          const int32_t low = __viaddmax_s32(best & ~1023, -xd, 1024);
          const bool last = EDGES && (i >= n1 || i + m > last_step);
          if (live && (b < low || ((uint32_t)(b + 1) & 1023u) <= 1u || last)) {
            const int c = b & 1023, k = c == 1023 ? 0 : KL - 1 - c - pads, j = i - w + k;
            if (CODES && EDGES && i + m > last_step)
              st = 2, rows = i - 1;
            else if (b >= 1024 && (k == 0 || k == 2 * w) && j != n2 && j != 1)
              st = 1, rows = i;
            else if (b < low || (EDGES && i >= n1))
              st = 0, rows = i;
            if (st >= 0) {
              live = false;
              score = best >> 10;
              row1 = e1;
              const int cb = best & 1023;
              e2 = score > 0 ? e1 - w + (cb == 1023 ? 0 : KL - 1 - cb - pads) : 0;
            }
          }
        }
      } else {
        if (on && have && tail_lane && st < 0) {
          if (CODES && i > last_step - (L - 1)) {
            st = 2;
          } else {
            rows = i;
            const int rb = b, k = bk - pads, j = rb > 0 ? i - w + k : -1;
            if (rb > 0 && j != n2 && j != 1 && (k == 0 || k == 2 * w)) {
              st = 1;
            } else {
              if (rb > score) score = rb, e1 = i, e2 = j;
              if (score - rb > P.xdrop || rb <= 0 || i >= n1) st = 0;
            }
          }
        }
      }
      ++i;
    };
    const bool ends = q0 + K - 1 + i + 15 >= n2 || (tail_lane && i + 15 >= n1) || (CODES && i + m + 15 > last_step);
    if (__any_sync(0xFFFFFFFFu, have && (i < 1 || ends || (qs.n | rs.n) != 0))) {
      for (int r = 0; r < 16; ++r) row(std::true_type{});
    } else {
      for (int r = 0; r < 16; ++r) row(std::false_type{});
    }
    const bool fin = have && tail_lane && st >= 0;
    if (fin) {
      XTask &T = A.tasks[id];
      T.status = st;
      T.rows = rows;
      if (st == 0) T.score = score, T.end1 = WIDE ? e1 : row1, T.end2 = e2;
      xd_route(T, id, A);
    }
    const unsigned done = __ballot_sync(0xFFFFFFFFu, fin);
    if (in_group && ((done >> (first + L - 1)) & 1u)) id = -1;
  }
}

// ------------------------------------------------------------------ wide bands: one warp per pass
// Lanes own consecutive band cells, 4 per lane in segments of 128.  The horizontal gap chain of a row,
//   e_{j+1} = max(e_j + g, A_j + open),  g = max(ext, open),  A_j = max(s + diag, F_above)
// (the value form of e += ext; e = max(e, M + open) with M = max(A, e)), is an affine map in max-plus algebra,
// f(e) = max(e + a, b); a lane's cells compose into one map, an exclusive warp scan of the maps gives every lane its
// incoming e, and the lane then replays its cells with the reference's exact comparisons.  Cells left of the row's
// first column reset e to OUT, as the reference starts each row with e = OUT.
constexpr int kXwSeg = 4;
constexpr int32_t kNegInf = -(1 << 30);

struct AffMax {
  int32_t a, b;  // e -> max(e + a, b); a <= kNegInf means "independent of e"
};

__device__ __forceinline__ int32_t aff_apply(AffMax f, int32_t e) {
  return f.a <= kNegInf ? f.b : max(e + f.a, f.b);
}
// g after f
__device__ __forceinline__ AffMax aff_then(AffMax f, AffMax g) {
  AffMax r;
  r.a = (f.a <= kNegInf || g.a <= kNegInf) ? kNegInf : f.a + g.a;
  r.b = (g.a <= kNegInf) ? g.b : max(f.b + g.a, g.b);
  return r;
}

// One pass of task T by the calling warp; M and F are the warp's scratch (2w + 2 ints each).  Lane 0 writes the
// pass's results into T.
__device__ void xdrop_warp_pass(XTask &T, const Arena &ar, const Params &P, uint32_t *__restrict__ tb,
                                int32_t *__restrict__ M, int32_t *__restrict__ F) {
  const int lane = threadIdx.x & 31;
  const int w = T.w, n1 = T.n1, n2 = T.n2, nk = 2 * w + 1;
  const int open = P.open1, ext = P.ext1, g = max(P.ext1, P.open1);
  const SeqView s1{T.base1, T.a1, T.dir}, s2{T.base2, T.a2, T.dir};
  for (int k = lane; k <= nk; k += 32) M[k] = kOut, F[k] = kOut;
  __syncwarp();
  const int wpr = xd_words_per_row(w);
  int score = 0, e1 = 0, e2 = 0, rows = 0, status = 0;
  for (int i = 1; i <= n1; ++i) {
    const int c0 = max(i - w, 1), c1 = min(i + w, n2);
    if (T.want_codes && (int64_t)i * wpr > T.tb_cap) {
      status = 2;
      break;
    }
    const int ci = s1.at(ar, i - 1);
    uint32_t *row_codes = tb + T.tb_off + (int64_t)(i - 1) * wpr;
    int32_t ecarry = kOut;  // e entering the segment's first cell
    int lbest = 0, lbestj = -1;
    for (int seg = 0; seg < nk; seg += 32 * kXwSeg) {
      const int k0 = seg + kXwSeg * lane;
      int32_t Mk[kXwSeg], Fk[kXwSeg];
#pragma unroll
      for (int q = 0; q < kXwSeg; ++q) {
        const int k = k0 + q;
        Mk[q] = k < nk ? M[k] : kOut;
        Fk[q] = k < nk ? F[k + 1] : kOut;
      }
      __syncwarp();  // every old value is read before any cell of this segment is rewritten
      // this lane's cells as one affine map of the incoming e
      AffMax f{0, kNegInf};
      int32_t A[kXwSeg], sv[kXwSeg], fin[kXwSeg];
      bool valid[kXwSeg], before[kXwSeg];
#pragma unroll
      for (int q = 0; q < kXwSeg; ++q) {
        const int k = k0 + q, j = i - w + k;
        valid[q] = k < nk && j >= c0 && j <= c1;
        before[q] = k < nk && j < c0;
        if (valid[q]) {
          const int32_t dg = (j == 1) ? (i == 1 ? 0 : kOut) : Mk[q];
          fin[q] = (j == c1) ? kOut : Fk[q];
          sv[q] = score_of(ci, s2.at(ar, j - 1), P.match, P.mismatch) + dg;
          A[q] = sv[q] > fin[q] ? sv[q] : fin[q];
          f = aff_then(f, AffMax{g, A[q] + open});
        } else if (before[q]) {
          f = AffMax{kNegInf, kOut};
        }
      }
      // exclusive scan of the lanes' maps
      AffMax incl = f;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        AffMax o;
        o.a = __shfl_up_sync(0xFFFFFFFFu, incl.a, d);
        o.b = __shfl_up_sync(0xFFFFFFFFu, incl.b, d);
        if (lane >= d) incl = aff_then(o, incl);
      }
      AffMax excl;
      excl.a = __shfl_up_sync(0xFFFFFFFFu, incl.a, 1);
      excl.b = __shfl_up_sync(0xFFFFFFFFu, incl.b, 1);
      if (lane == 0) excl = AffMax{0, kNegInf};
      int32_t e = aff_apply(excl, ecarry);
      const AffMax all{__shfl_sync(0xFFFFFFFFu, incl.a, 31), __shfl_sync(0xFFFFFFFFu, incl.b, 31)};
      const int32_t next_carry = aff_apply(all, ecarry);
      // replay the cells with the reference's comparisons
      uint32_t nib = 0;
#pragma unroll
      for (int q = 0; q < kXwSeg; ++q) {
        const int k = k0 + q, j = i - w + k;
        uint32_t cd = 0xFu;
        if (valid[q]) {
          uint32_t d = sv[q] > fin[q] ? 0u : 1u;
          int32_t v = A[q];
          if (!(v > e)) d = 2u, v = e;
          if (v > lbest) lbest = v, lbestj = j;
          const int32_t h = v + open, fx = fin[q] + ext;
          if (fx >= h) d |= 4u;
          e += ext;
          if (e >= h) d |= 8u;
          e = e >= h ? e : h;
          M[k] = v;
          F[k] = fx >= h ? fx : h;
          cd = d;
        } else if (before[q]) {
          e = kOut;
        }
        nib |= cd << (4 * q);
      }
      ecarry = next_carry;
      if (T.want_codes) {
        // 4 nibbles per lane = half a word: even lanes write the word shared with the next lane
        const uint32_t hi = __shfl_down_sync(0xFFFFFFFFu, nib, 1);
        const int word = k0 >> 3;
        if ((lane & 1) == 0 && word < wpr) row_codes[word] = nib | (hi << 16);
      }
      __syncwarp();
    }
    rows = i;
    // the row's first maximum: largest value, then smallest column
    const int best = __reduce_max_sync(0xFFFFFFFFu, lbest);
    int bestj = __reduce_min_sync(0xFFFFFFFFu, (lbest == best && lbestj >= 0) ? lbestj : 0x7FFFFFFF);
    if (best <= 0) bestj = -1;
    if (bestj != n2 && bestj != 1 && (bestj == c0 || bestj == c1)) {
      status = 1;
      break;
    }
    if (best > score) score = best, e1 = i, e2 = bestj;
    if (score - best > P.xdrop) break;
    if (best <= 0) break;
  }
  if (lane == 0) {
    T.status = status;
    T.rows = rows;
    if (status == 0) T.score = score, T.end1 = e1, T.end2 = e2;
  }
}


__global__ void __launch_bounds__(128) xdrop_level_warp_kernel(XLevelArgs A, Arena ar, Params P,
                                                               uint32_t *__restrict__ tb, int32_t *__restrict__ scratch,
                                                               int64_t per_warp) {
  const int n = *A.L.count_in;
  const int lane = threadIdx.x & 31;
  const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
  int32_t *M = scratch + per_warp * gw;
  for (int q = gw; q < n; q += nw) {
    const int id = A.L.list_in[q];
    XTask &T = A.tasks[id];
    int ok = 1;
    if (lane == 0 && T.want_codes) ok = xd_take_slot(T, A) ? 1 : 0;
    ok = __shfl_sync(0xFFFFFFFFu, ok, 0);
    __syncwarp();
    if (!ok) {
      if (lane == 0) {
        T.status = 2;
        xd_route(T, id, A);
      }
      continue;
    }
    xdrop_warp_pass(T, ar, P, tb, M, M + (2 * T.w + 2));
    __syncwarp();
    if (lane == 0) xd_route(T, id, A);
    __syncwarp();
  }
}

__global__ void xdrop_iota_kernel(int *list, int n, int *count) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) list[k] = k;
  if (k == 0) *count = n;
}

// The passes of the first level by falling bound on their rows, in kXdropOrderBins classes: counted, then placed.  A
// level's last passes run alone at a row's latency, so the long ones go first.
__device__ __forceinline__ int order_bin(const XTask &T, int max_rows) {
  const int64_t rows = min((int64_t)max(T.n1, 0), (int64_t)max(T.n2, 0) + T.w);
  return kXdropOrderBins - 1 - (int)min((int64_t)kXdropOrderBins - 1, rows * kXdropOrderBins / max(max_rows, 1));
}

__global__ void xdrop_order_count_kernel(const XTask *__restrict__ tasks, int n, int max_rows, int *bins) {
  __shared__ int h[kXdropOrderBins];
  if (threadIdx.x < kXdropOrderBins) h[threadIdx.x] = 0;
  __syncthreads();
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) atomicAdd(&h[order_bin(tasks[k], max_rows)], 1);
  __syncthreads();
  if (threadIdx.x < kXdropOrderBins && h[threadIdx.x]) atomicAdd(&bins[threadIdx.x], h[threadIdx.x]);
}

__global__ void xdrop_order_place_kernel(const XTask *__restrict__ tasks, int n, int max_rows,
                                         const int *__restrict__ bins, int *cursor, int *list, int *count) {
  __shared__ int h[kXdropOrderBins], at[kXdropOrderBins];
  if (threadIdx.x < kXdropOrderBins) h[threadIdx.x] = 0;
  __syncthreads();
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  int b = 0, r = 0;
  if (k < n) b = order_bin(tasks[k], max_rows), r = atomicAdd(&h[b], 1);
  __syncthreads();
  if (threadIdx.x < kXdropOrderBins) {
    int before = 0;
    for (int q = 0; q < (int)threadIdx.x; ++q) before += bins[q];
    at[threadIdx.x] = before + (h[threadIdx.x] ? atomicAdd(&cursor[threadIdx.x], h[threadIdx.x]) : 0);
  }
  __syncthreads();
  if (k < n) list[at[b] + r] = k;
  if (k == 0) *count = n;
}

// From 16 passes per multiprocessor on: fewer are all dealt out at once (four warps' worth), in any order.  50,000
// extension tasks: 11 us for 0.6 ms off the levels of 7.0 ms; a call of a few hundred passes would pay 8 us for nothing.
void launch_xdrop_list(const XTask *tasks, int *list, int n, int *count, int max_rows, int *bins, int nsm,
                       cudaStream_t st) {
  if (n <= nsm * 16) {
    xdrop_iota_kernel<<<(n + 255) / 256, 256, 0, st>>>(list, n, count);
    return;
  }
  xdrop_order_count_kernel<<<(n + 255) / 256, 256, 0, st>>>(tasks, n, max_rows, bins);
  xdrop_order_place_kernel<<<(n + 255) / 256, 256, 0, st>>>(tasks, n, max_rows, bins, bins + kXdropOrderBins, list,
                                                            count);
}

template <int K, int L, int P0, bool CODES>
void launch_band(const XLevelArgs &A, Arena ar, const Params &p, uint32_t *tb, int n_bound, int nsm, cudaStream_t st) {
  static const int per_sm = [] {
    int v = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, xdrop_band_kernel<K, L, P0, CODES>, 128, 0) != cudaSuccess) {
      (void)cudaGetLastError();
      v = 1;
    }
    return std::max(v, 1);
  }();
  const int passes = 4 * (32 / L);  // per block at a time
  const int blocks = (int)std::min<int64_t>((n_bound + passes - 1) / passes, (int64_t)nsm * per_sm);
  xdrop_band_kernel<K, L, P0, CODES><<<blocks, 128, 0, st>>>(A, ar, p, reinterpret_cast<uint8_t *>(tb));
}

// P0: the pads of the doubled bands 10, 20, 40, ... in this layout.
template <int K, int L, int P0>
void launch_band_form(const XLevelArgs &A, Arena ar, const Params &p, uint32_t *tb, int n_bound, int nsm, bool codes,
                      bool packed, cudaStream_t st) {
  const bool fixed = packed && K * L - (2 * A.w + 1) == P0;
  if (fixed && codes)
    launch_band<K, L, P0, true>(A, ar, p, tb, n_bound, nsm, st);
  else if (fixed)
    launch_band<K, L, P0, false>(A, ar, p, tb, n_bound, nsm, st);
  else if (codes)
    launch_band<K, L, -1, true>(A, ar, p, tb, n_bound, nsm, st);
  else
    launch_band<K, L, -1, false>(A, ar, p, tb, n_bound, nsm, st);
}

void launch_xdrop_level(XTask *tasks, const XLevel &lv, Arena ar, Params p, uint32_t *tb, int w, int n_bound, int nsm,
                        int32_t *scratch, int64_t per_warp, int warps, bool codes, bool packed, cudaStream_t st) {
  if (n_bound <= 0) return;
  const XLevelArgs A{tasks, lv, w, nsm};
  switch (xd_layout(w).skew ? xd_layout(w).K * xd_layout(w).L : 0) {
    case 21: return launch_band_form<3, 7, 0>(A, ar, p, tb, n_bound, nsm, codes, packed, st);
    case 42: return launch_band_form<6, 7, 1>(A, ar, p, tb, n_bound, nsm, codes, packed, st);
    case 84: return launch_band_form<6, 14, 3>(A, ar, p, tb, n_bound, nsm, codes, packed, st);
    case 162: return launch_band_form<6, 27, 1>(A, ar, p, tb, n_bound, nsm, codes, packed, st);
    case 330: return launch_band_form<11, 30, 9>(A, ar, p, tb, n_bound, nsm, codes, packed, st);
    case 651: return launch_band_form<21, 31, 10>(A, ar, p, tb, n_bound, nsm, codes, packed, st);
    default: xdrop_level_warp_kernel<<<(warps + 3) / 4, 128, 0, st>>>(A, ar, p, tb, scratch, per_warp);
  }
}

// ------------------------------------------------------------------ traceback of the passes with codes
// State machine of impl/sequenceAlignment3.cpp:1413-1438: start in the state that produced the cell; a gap state
// persists while the cell's continuation bit is set; ops are appended as the walk goes (no final reverse, because
// the walk over the reverse-complement pass already runs in forward order).  Cells outside the band or past the last
// row read 255.
//
// One warp per pass, a run at a time: the lanes load the next 32 cells in the direction of the state (a diagonal, a
// column or a row of the DP), and a ballot says how far the state holds.  Bound: one round trip to L2 per run or 32
// cells (a lane that walked cell by cell through a staged window took 3-4 times as long).
__device__ void xdrop_traceback_warp(XTask &T, const uint8_t *__restrict__ tb, uint32_t *__restrict__ cig, int lane) {
  const int w = T.w, rows = T.rows, cap = T.cig_cap;
  const XBandLayout B = xd_layout(w);
  const uint8_t *const base = tb + 4 * T.tb_off;
  int ii = T.end1, jj = T.end2, state = 0, nc = 0;
  uint32_t *const out = cig + T.cig_off;
  uint32_t last = 0xFFFFFFFFu;
  bool full = false;
  auto push = [&](uint32_t op, int n) {
    if (nc > 0 && (last & 0xFu) == op) {
      last += (uint32_t)n << 4;
    } else {
      if (nc >= cap) {
        full = true;
        return;
      }
      last = ((uint32_t)n << 4) | op;
      ++nc;
    }
    if (lane == 0) out[nc - 1] = last;
  };
  while (ii > 0 && jj > 0 && !full) {
    const int di = state == 2 || state > 3 ? 0 : 1, dj = state == 1 || state == 3 ? 0 : 1;
    const int ci = ii - di * lane, cj = jj - dj * lane, k = cj - ci + w;
    const bool in = ci > 0 && cj > 0 && ci <= rows && k >= 0 && k <= 2 * w;
    uint32_t nib = 0;
    if (in) {
      const int kk = k + B.pads, m = kk / B.K, p = kk - m * B.K;
      const int64_t at = B.skew ? ((int64_t)(ci - 1 + m) * B.L + m) * B.bytes : ((int64_t)(ci - 1) * B.L + m) * B.bytes;
      nib = (uint32_t)(__ldg(base + at + (p >> 1)) >> (4 * (p & 1))) & 0xFu;
    }
    if (!__shfl_sync(0xFFFFFFFFu, (int)in, 0)) {  // reads 255: a gap state holds, anything else moves left
      if (state != 1 && state != 2 && state != 3 && state != 4) state = 7;
      if (state == 1 || state == 3) {
        push(2, 1);
        --ii;
      } else {
        push(1, 1);
        --jj;
      }
      continue;
    }
    const bool hold = in && (state == 0 ? (nib & 3u) == 0 : state == 1 ? (nib & 4u) != 0 : state == 2 && (nib & 8u) != 0);
    const unsigned mk = __ballot_sync(0xFFFFFFFFu, hold);
    const int run = mk == 0xFFFFFFFFu ? 32 : __ffs(~mk) - 1;
    if (run > 0) {
      push(state == 0 ? 0u : state == 1 ? 2u : 1u, run);
      ii -= di * run;
      jj -= dj * run;
    }
    if (run < 32 && !full) {  // the cell the run ends at starts a new state
      const int there = __shfl_sync(0xFFFFFFFFu, (int)in, run), fresh = __shfl_sync(0xFFFFFFFFu, (int)(nib & 3u), run);
      if (there) {
        state = fresh;
        if (state == 1) {
          push(2, 1);
          --ii;
        } else if (state != 0) {
          push(1, 1);
          --jj;
        }
      }
    }
  }
  if (lane == 0) {
    if (full) T.status = 3;
    T.iii = ii;
    T.jjj = jj;
    T.ncig = nc;
  }
}

__global__ void __launch_bounds__(128) xdrop_traceback_kernel(XTask *__restrict__ tasks, const int *__restrict__ idx,
                                                              int n, const uint8_t *__restrict__ tb,
                                                              uint32_t *__restrict__ cig) {
  const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (gw >= n) return;  // whole warp
  xdrop_traceback_warp(tasks[idx[gw]], tb, cig, threadIdx.x & 31);
}

// Chained form: every task of the batch that finished with codes takes a CIGAR slot of end1 + end2 + 2 words from an
// arena sized for the bound n1 + n2 + 2 per task, then runs the walk above.
__global__ void __launch_bounds__(128) xdrop_traceback_all_kernel(XTask *__restrict__ tasks, int n,
                                                                  const uint8_t *__restrict__ tb,
                                                                  uint32_t *__restrict__ cig,
                                                                  unsigned long long *__restrict__ cig_cursor) {
  const int lane = threadIdx.x & 31;
  const int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (t >= n) return;  // whole warp
  XTask &T = tasks[t];
  if (T.status != 0 || !T.want_codes) return;
  if (lane == 0) {
    T.cig_cap = max(T.end1, 0) + max(T.end2, 0) + 2;
    T.cig_off = (int64_t)atomicAdd(cig_cursor, (unsigned long long)T.cig_cap);
  }
  __syncwarp();
  xdrop_traceback_warp(T, tb, cig, lane);
}

void launch_xdrop_traceback_all(XTask *tasks, int n, const uint32_t *tb, uint32_t *cig, unsigned long long *cig_cursor,
                                cudaStream_t st) {
  if (n <= 0) return;
  xdrop_traceback_all_kernel<<<(n + 3) / 4, 128, 0, st>>>(tasks, n, reinterpret_cast<const uint8_t *>(tb), cig,
                                                          cig_cursor);
}

// Dense offsets of the finished tasks' CIGARs in task order: one block; each thread sums a contiguous run of tasks,
// a block-wide exclusive scan of the run sums, then each thread assigns its run's offsets.
__global__ void __launch_bounds__(1024) xdrop_cigar_scan_kernel(XTask *__restrict__ tasks, int n,
                                                                unsigned long long *__restrict__ total) {
  __shared__ long long part[1024];
  const int t = threadIdx.x, per = (n + 1023) / 1024;
  const int lo = min(n, t * per), hi = min(n, lo + per);
  long long sum = 0;
  for (int k = lo; k < hi; ++k)
    if (tasks[k].status == 0 && tasks[k].want_codes) sum += tasks[k].ncig;
  part[t] = sum;
  __syncthreads();
  for (int d = 1; d < 1024; d <<= 1) {  // inclusive Hillis-Steele scan
    const long long v = t >= d ? part[t - d] : 0;
    __syncthreads();
    part[t] += v;
    __syncthreads();
  }
  long long off = part[t] - sum;
  for (int k = lo; k < hi; ++k)
    if (tasks[k].status == 0 && tasks[k].want_codes) {
      tasks[k].cig_dense = off;
      off += tasks[k].ncig;
    } else {
      tasks[k].cig_dense = -1;
    }
  if (t == 1023) *total = (unsigned long long)part[1023];
}

__global__ void xdrop_cigar_copy_kernel(const XTask *__restrict__ tasks, int n, const uint32_t *__restrict__ cig,
                                        uint32_t *__restrict__ dense) {
  const int k = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (k >= n) return;
  const XTask &T = tasks[k];
  if (T.cig_dense < 0) return;
  for (int q = lane; q < T.ncig; q += 32) dense[T.cig_dense + q] = cig[T.cig_off + q];
}

void launch_xdrop_cigar_pack(XTask *tasks, int n, const uint32_t *cig, uint32_t *dense, unsigned long long *total,
                             cudaStream_t st) {
  if (n <= 0) return;
  xdrop_cigar_scan_kernel<<<1, 1024, 0, st>>>(tasks, n, total);
  xdrop_cigar_copy_kernel<<<(n + 7) / 8, 256, 0, st>>>(tasks, n, cig, dense);
}

void launch_xdrop_traceback(XTask *tasks, const int *idx, int n, const uint32_t *tb, uint32_t *cig, cudaStream_t st) {
  if (n <= 0) return;
  xdrop_traceback_kernel<<<(n + 3) / 4, 128, 0, st>>>(tasks, idx, n, reinterpret_cast<const uint8_t *>(tb), cig);
}

}  // namespace dcns
