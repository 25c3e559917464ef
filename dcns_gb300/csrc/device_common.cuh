// Device helpers shared by the kernels: packed-sequence decode and score lookup.
#pragma once

#include "common.h"

namespace dcns {

// dCNS code (A0 C1 N2 G3 T4) of base k of the arena.
__device__ __forceinline__ int base_code(const Arena &ar, int64_t k) {
  const uint32_t w = __ldg(ar.pk + (k >> 4));
  const uint32_t two = (w >> ((uint32_t)(k & 15) * 2u)) & 3u;
  const uint32_t n = (__ldg(ar.nm + (k >> 5)) >> (uint32_t)(k & 31)) & 1u;
  return n ? 2 : (int)(two + (two >> 1));
}

// Scorei (model/Score.cpp:105-135): N (code 2) scores 0 against anything.
__device__ __forceinline__ int score_of(int a, int b, int match, int mismatch) {
  return (a == 2 || b == 2) ? 0 : (a == b ? match : mismatch);
}

// Sequence view for the DP kernels: forward (s[i] = seq[a + i]) or reverse-complement ending at a
// (s[i] = 4 - seq[a - i]).
struct SeqView {
  int64_t base;
  int32_t a, dir;
  __device__ __forceinline__ int at(const Arena &ar, int32_t i) const {
    return dir == 0 ? base_code(ar, base + a + i) : 4 - base_code(ar, base + a - i);
  }
};

// Sixteen symbols of a sequence view of n bases from offset o on: 2-bit codes and N bits, in reading order (an N
// carries code 0).  Offsets outside [0, n) give any symbols.
struct Syms16 {
  uint32_t w, n;
};
__device__ __forceinline__ Syms16 load16(const Arena &ar, const SeqView &s, int n, int o) {
  Syms16 r{0u, 0u};
  if (o <= -16 || o >= n) return r;
  const int64_t lo = s.base + s.a + (s.dir == 0 ? (int64_t)o : -(int64_t)o - 15);
  if (lo < 0) {
    const int sh = (int)-lo;  // at most 15
    r.w = __ldg(ar.pk) << (2 * sh);
    r.n = (__ldg(ar.nm) << sh) & 0xFFFFu;
  } else {
    r.w = __funnelshift_r(__ldg(ar.pk + (lo >> 4)), __ldg(ar.pk + (lo >> 4) + 1), 2u * (uint32_t)(lo & 15));
    r.n = __funnelshift_r(__ldg(ar.nm + (lo >> 5)), __ldg(ar.nm + (lo >> 5) + 1), (uint32_t)(lo & 31)) & 0xFFFFu;
  }
  if (s.dir != 0) {
    const uint32_t b = __brev(r.w);
    r.w = ~(((b >> 1) & 0x55555555u) | ((b << 1) & 0xAAAAAAAAu));
    r.n = __brev(r.n) >> 16;
  }
  for (uint32_t m = r.n; m; m &= m - 1) r.w &= ~(3u << (2 * (__ffs(m) - 1)));
  return r;
}
__device__ __forceinline__ void next_sym(Syms16 &s) { s.w >>= 2, s.n >>= 1; }

// Scores of a row's symbol against columns by byte permutation: the row's profile holds its score against the 2-bit
// codes 0..3 in bytes 0..3 (0 for a row N), and a column's selector picks its byte and repeats the sign (an N column
// picks the zeros behind the profile).
__device__ __forceinline__ uint32_t sym_selector(const Syms16 &s) {
  return ((s.w & 3u) | ((s.n & 1u) << 2)) * 0x1111u + 0x8880u;
}
// As sym_selector, for 256 times the score (byte 0 picks a zero behind the profile).
__device__ __forceinline__ uint32_t sym_selector256(const Syms16 &s) {
  return ((s.w & 3u) | ((s.n & 1u) << 2)) * 0x1110u + 0x8804u;
}
__device__ __forceinline__ uint32_t sym_profile(const Syms16 &s, int match, int mismatch) {
  const uint32_t rep = (uint32_t)(uint8_t)mismatch * 0x01010101u, x = (uint32_t)(uint8_t)(match ^ mismatch);
  return (s.n & 1u) ? 0u : rep ^ (x << (8u * (s.w & 3u)));
}
__device__ __forceinline__ int perm_score(uint32_t prof, uint32_t behind, uint32_t sel) {
  uint32_t d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(prof), "r"(behind), "r"(sel));
  return (int)d;
}

}  // namespace dcns
