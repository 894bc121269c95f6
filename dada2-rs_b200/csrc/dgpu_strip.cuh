// The banded ends-free aligner of the compare step, one warp per pair.
//
// The row-major recurrence (src/nwalign.rs:336-528) and, for end gap 0 and
// sequences of two or more bases, the vectorized one (src/nwalign.rs:665-1140)
// choose the same moves: the cells o_lo <= j - i <= o_hi, rows 0 and columns 0
// at zero, free gaps on the last row and column, ties up before left before
// diagonal. So one DP serves both, with homopolymer gaps or without.
#pragma once

#include "dgpu_common.h"

namespace dgpu {

// Shared memory of one warp's pair. s1 and s2 have kStripPad readable bytes
// past their ends (the DP loads one row ahead).
struct StripSmem {
  uint8_t* s1;      // center codes 1..4, bit 4 set inside a homopolymer run
  uint8_t* s2;      // raw codes
  uint8_t* qual;    // raw qualities
  uint8_t* tcode;   // per raw position: error-matrix row (see kUnaligned)
  uint2* stage;     // pointer words: all of them, or the traceback's window
  uint16_t* fidx;   // in stage, which is free after the traceback
};

__device__ __forceinline__ StripSmem carve_strip(unsigned char* base, const NwGeom& g) {
  StripSmem S;
  const size_t ls = align16(size_t(g.lmax) + kStripPad), lq = align16(size_t(g.lmax));
  S.s1 = base;
  S.s2 = base + ls;
  S.qual = base + 2 * ls;
  S.tcode = base + 2 * ls + lq;
  S.stage = reinterpret_cast<uint2*>(base + 2 * ls + 2 * lq);
  S.fidx = reinterpret_cast<uint16_t*>(S.stage);
  return S;
}

// Sets bit 4 of every position inside a run of three or more equal bases
// (src/nwalign.rs:211-227). In place: neighbours compare the low bits only.
__device__ __forceinline__ void flag_runs(int lane, uint8_t* s, int n) {
  for (int p = lane; p < n; p += 32) {
    const unsigned c = s[p] & 15u;
    const bool b1 = p >= 1 && (s[p - 1] & 15u) == c, b2 = b1 && p >= 2 && (s[p - 2] & 15u) == c;
    const bool a1 = p + 1 < n && (s[p + 1] & 15u) == c, a2 = a1 && p + 2 < n && (s[p + 2] & 15u) == c;
    if (b2 || a2 || (b1 && a1)) s[p] = uint8_t(c | 16u);
  }
}

// Offsets j - i of the band's first and last diagonal.
__device__ __forceinline__ void band_offsets(int band, int len1, int len2, int* o_lo, int* o_hi) {
  if (band >= 0) {
    *o_lo = max(-(band + max(len1 - len2, 0)), -len1);
    *o_hi = min(band + max(len2 - len1, 0), len2);
  } else {
    *o_lo = -len1;
    *o_hi = len2;
  }
}

// Walks the pointer words back from (len1, len2). Lane t tests whether the
// t-th step back is diagonal (the same diagonal, row i - t), so a run of
// diagonal steps and the gap that ends it are taken at once.
template <int C>
__device__ __forceinline__ bool strip_traceback(int lane, int len1, int len2, int o_lo, int W, const StripSmem& S,
                                                const uint2* planes, bool in_smem, uint32_t* ham_out,
                                                uint32_t* err_word, uint8_t* dbg0, uint8_t* dbg1, uint32_t* dbg_len) {
  constexpr int N = 2 * C, RPW = 32 / N, NB = RPW * N;
  for (int p = lane; p < len2; p += 32) S.tcode[p] = uint8_t(kUnaligned | (((S.s2[p] & 15u) - 1u) * 5u));
  __syncwarp();
  int i = len1, j = len2, slo = in_smem ? 0 : 0x7fffffff;
  uint32_t ham = 0, alen = 0;
  while (i > 0 && j > 0) {
    const int idx = j - i - o_lo;
    if (idx < 0 || idx >= W) {
      if (lane == 0) atomicOr(err_word, DERR_TRACEBACK);
      return false;
    }
    const int l = idx / N, k = idx - l * N;
    const int r = i + l - 1;
    if (!in_smem && (r / RPW < slo || (slo > 0 && r - slo * RPW < 31))) {  // stage the next words down
      const int hi = r / RPW, lo = max(0, hi - (kStripWindow - 1));
      __syncwarp();
      const uint4* src = reinterpret_cast<const uint4*>(planes + size_t(lo) * 32);
      uint4* dst = reinterpret_cast<uint4*>(S.stage);
      const int nv = (hi - lo + 1) * 16;
#pragma unroll 4
      for (int x = lane; x < nv; x += 32) dst[x] = __ldcg(src + x);
      __syncwarp();
      slo = lo;
    }
    const int rt = r - lane;  // the row this lane tests, as an insertion row
    const bool ok = lane < i && lane < j && rt >= slo * RPW;
    uint2 w = make_uint2(0u, 0u);
    int bit = 0;
    if (ok) {
      const int wt = rt / RPW;
      w = S.stage[(wt - slo) * 32 + l];
      bit = NB - 1 - ((rt - wt * RPW) * N + k);
    }
    const bool diag = ok && ((w.x >> bit) & 1u);
    const uint32_t nd = __ballot_sync(FULL, !diag);
    const int f = nd ? __ffs(nd) - 1 : 32;
    bool mm = false;
    if (lane < f) {
      const uint8_t a = S.s1[i - 1 - lane] & 15u, b = S.s2[j - 1 - lane] & 15u;
      S.tcode[j - 1 - lane] = uint8_t((unsigned(a) - 1u) * 4u + (unsigned(b) - 1u));
      mm = a != b;
      if (dbg0) {
        dbg0[alen + lane] = a;
        dbg1[alen + lane] = b;
      }
    }
    ham += __popc(__ballot_sync(FULL, mm));
    // the step after the run, where its lane holds it: 1 left, 0 up, -1 not known
    const int gap = __shfl_sync(FULL, ok ? int((w.y >> bit) & 1u) : -1, f & 31);
    i -= f;
    j -= f;
    alen += uint32_t(f);
    if (f < 32 && gap >= 0) {
      if (gap) {
        if (dbg0 && lane == 0) { dbg0[alen] = '-'; dbg1[alen] = S.s2[j - 1] & 15u; }
        --j;
      } else {
        if (dbg0 && lane == 0) { dbg0[alen] = S.s1[i - 1] & 15u; dbg1[alen] = '-'; }
        --i;
      }
      ++alen;
    }
  }
  if (dbg0) {  // row 0 moves left, column 0 moves up
    for (int t = lane; t < j; t += 32) { dbg0[alen + t] = '-'; dbg1[alen + t] = S.s2[j - 1 - t] & 15u; }
    for (int t = lane; t < i; t += 32) { dbg0[alen + t] = S.s1[i - 1 - t] & 15u; dbg1[alen + t] = '-'; }
  }
  alen += uint32_t(i + j);
  __syncwarp();
  if (dbg_len && lane == 0) *dbg_len = alen;
  *ham_out = ham;
  return true;
}

// The DP. Lane l owns the 2C neighbouring diagonals from o_lo + 2C l on, as
// two strips of C; row i of a lane's first strip is computed at step 2i + 2l
// and of its second one step later, so a step needs one value of a
// neighbouring lane and a row costs two shuffles, whatever C is. The bounds
// are the shuffle and add-max chain (few pairs) and integer issue (many). One
// cell per lane and anti-diagonal, as this replaces, cost a shuffle, the
// pointer's two ballots and the position's costs for every 32 cells: a call
// aligning 4,672 pairs of 1,400-1,550 nt (band 32, homopolymer gaps) went from
// 5.7 to 1.7 ms, one aligning 24,908 pairs of 250 nt (band 16) from 1.4 to
// 0.8 ms, and one of 4 such pairs from 51 to 30 us.
//
// Values are kept less the gap costs of their row and column (H = V - sum of
// gl over 1..j - sum of gu over 1..i): the two gap moves then cost nothing,
// a diagonal step adds w = score - gl(j) - gu(i), and a cell is one fused
// add-max on the chain from its left neighbour.
//
// A cell's two pointer bits (diagonal best; else left better than up) are the
// signs of differences, shifted into two words per lane: RPW = 32 / 2C rows
// per word, written as one 256-byte row of `planes` per RPW rows.
//
// The rows where some lane is before its first cell, or past the last row or
// column's start, take the SLOW form of the row; the rest need no tests.
//
// S.s1/S.s2 hold the codes, with the run flags when HOMO. Needs a band of
// W <= 62 C diagonals, so that the lane after the last
// one in use holds the mark outside the band (strip_cols).
template <int C, bool HOMO>
__device__ __noinline__ bool strip_align(int lane, int len1, int len2, int match, int mismatch, int gap, int hgap,
                                         int band, const StripSmem& S, uint2* planes, bool in_smem,
                                         uint32_t* ham_out, uint32_t* err_word, uint8_t* dbg0, uint8_t* dbg1,
                                         uint32_t* dbg_len) {
  constexpr int N = 2 * C, RPW = 32 / N;
  constexpr int BIG = 1 << 28;
  int o_lo, o_hi;
  band_offsets(band, len1, len2, &o_lo, &o_hi);
  const int W = o_hi - o_lo + 1;
  if (W > 62 * C) {
    if (lane == 0) atomicOr(err_word, DERR_UNSUPPORTED);
    return false;
  }
  const int nl = (W + N - 1) / N;
  const int lc = min(lane, nl - 1);  // idle lanes read what the last one does
  const int ol = o_lo + N * lc;
  int V[N], LB[N], Y[N];
  // before its first row a cell holds its value on row 0 (o >= 0) or column 0
  {
    int c1[N], c2[N];
#pragma unroll
    for (int k = 0; k < N; ++k) c1[k] = c2[k] = 0;
    if (HOMO) {
      const int top = max(-o_lo, o_hi);
      for (int b = 0; b < top; b += 32) {
        const int p = b + lane;
        const uint32_t m1 = __ballot_sync(FULL, p < len1 && (S.s1[p] & 16u));
        const uint32_t m2 = __ballot_sync(FULL, p < len2 && (S.s2[p] & 16u));
#pragma unroll
        for (int k = 0; k < N; ++k) {
          const int o = ol + k;
          const int n2 = min(max(o - b, 0), 32), n1 = min(max(-o - b, 0), 32);
          c2[k] += __popc(n2 == 32 ? m2 : m2 & ((1u << n2) - 1u));
          c1[k] += __popc(n1 == 32 ? m1 : m1 & ((1u << n1) - 1u));
        }
      }
    }
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const int idx = N * lane + k, o = ol + k;
      V[k] = idx >= W ? -BIG : -(gap * abs(o) + (HOMO ? (hgap - gap) * (o >= 0 ? c2[k] : c1[k]) : 0));
      LB[k] = (idx == 0 || idx == W) ? -BIG : 0;  // no left neighbour inside the band
    }
  }
  const int last = len1 + nl - 1;                                   // rows 1 .. len1 of every lane
  const int r_head = max(1 - o_lo, nl);                             // from here on every cell has started
  const int r_tail = min(len1, nl - 1 + len2 - (o_lo + N * nl - 1));  // from here on some cell may be on the last row or column
  uint32_t accD = 0, accL = 0;
  int cnt = 0;
  uint2* out = planes + lane;
  auto x_at = [&](int p, auto slow) -> int {
    constexpr bool SLOW = decltype(slow)::value;
    return S.s1[SLOW ? min(max(p, 0), len1 - 1) : p];
  };
  auto y_at = [&](int p, auto slow) -> int {
    constexpr bool SLOW = decltype(slow)::value;
    return S.s2[SLOW ? min(max(p, 0), len2 - 1) : p];
  };
  using Slow = std::integral_constant<bool, true>;
  using Fast = std::integral_constant<bool, false>;
  int x = x_at(-lc, Slow{});  // row r - lc = 1 - lc
#pragma unroll
  for (int k = 0; k < N; ++k) Y[k] = y_at(ol - lc + k, Slow{});
  // N rows from row count r on; cell k of row u reads column slot (k + u) % N
  auto rows = [&](int r, auto slow) {
    constexpr bool SLOW = decltype(slow)::value;
#pragma unroll
    for (int u = 0; u < N; ++u) {
      const int i = r + u - lc;
      const int xn = x_at(i, slow);
      const int yn = y_at(i + ol + N - 1, slow);
      const int xc = HOMO ? (x & 15) : x;
      const int cu = HOMO ? ((x & 16) ? -hgap : -gap) : -gap;
      // without runs both gap costs are the same constant
      const int wa = match + cu + (HOMO ? 0 : -gap), wb = mismatch + cu + (HOMO ? 0 : -gap);
      auto cell = [&](int k, int left, int up, bool up_late) -> int {
        const int y = Y[(k + u) % N];
        const int cl = HOMO ? ((y & 16) ? -hgap : -gap) : -gap;
        const int w = (HOMO ? (y & 15) : y) == xc ? wa : wb;
        const int dg = HOMO ? V[k] + w + cl : V[k] + w;
        if (SLOW) {
          if (i + ol + k == len2) up += cu;  // free on the last column
          if (i == len1) left += cl;         // and on the last row
        }
        const int sl = up - left - LB[k];
        const int sd = max(left + LB[k], up) - dg;
        accL = __funnelshift_l(uint32_t(sl), accL, 1);
        accD = __funnelshift_l(uint32_t(sd), accD, 1);
        // the value that arrives last joins last
        int v = up_late ? max(up, __viaddmax_s32(left, LB[k], dg)) : __viaddmax_s32(left, LB[k], max(up, dg));
        if (SLOW) v = (i >= 1 && i + ol + k >= 1) ? v : V[k];
        return v;
      };
      int left = __shfl_up_sync(FULL, V[N - 1], 1);
#pragma unroll
      for (int k = 0; k < C; ++k) left = V[k] = cell(k, left, V[k + 1], false);
      const int ub = __shfl_down_sync(FULL, V[0], 1);
#pragma unroll
      for (int k = C; k < N; ++k) left = V[k] = cell(k, left, k + 1 < N ? V[(k + 1) % N] : ub, k + 1 == N);
      Y[u] = yn;
      x = xn;
      if (++cnt == RPW) {
        *out = make_uint2(accD, accL);
        out += 32;
        cnt = 0;
      }
    }
  };
  int r = 1;
  for (; r <= last && r < r_head; r += N) rows(r, Slow{});
  for (; r + N - 1 < r_tail; r += N) rows(r, Fast{});
  for (; r <= last; r += N) rows(r, Slow{});
  if (cnt) {
    const int sh = (RPW - cnt) * N;
    *out = make_uint2(accD << sh, accL << sh);
  }
  __syncwarp();
  return strip_traceback<C>(lane, len1, len2, o_lo, W, S, planes, in_smem, ham_out, err_word, dbg0, dbg1, dbg_len);
}

// The narrowest strip that holds the pair's band. CMAX bounds it for the
// launch (the geometry's rule: strip_cols).
template <int CMAX, bool HOMO>
__device__ __forceinline__ bool strip_dispatch(int lane, int len1, int len2, const KParams& kp, bool homo,
                                               const StripSmem& S, uint2* planes, bool in_smem, uint32_t* ham,
                                               uint32_t* err_word, uint8_t* d0, uint8_t* d1, uint32_t* dl) {
  if (HOMO && homo) {
    flag_runs(lane, S.s1, len1);
    flag_runs(lane, S.s2, len2);
    __syncwarp();
  }
  const int hg = homo ? kp.homo_gap : kp.gap;
  int o_lo, o_hi;
  band_offsets(kp.band, len1, len2, &o_lo, &o_hi);
  const int need = strip_cols(o_hi - o_lo + 1);
#define STRIP_CASE(CC)                                                                                            \
  if (CC == CMAX || need <= CC)                                                                                   \
  return strip_align<CC, HOMO>(lane, len1, len2, kp.match, kp.mismatch, kp.gap, hg, kp.band, S, planes, in_smem, \
                               ham, err_word, d0, d1, dl)
  STRIP_CASE(1);
  if constexpr (CMAX >= 2) STRIP_CASE(2);
  if constexpr (CMAX >= 3) STRIP_CASE(3);
  if constexpr (CMAX >= 4) STRIP_CASE(4);
#undef STRIP_CASE
}

}  // namespace dgpu
