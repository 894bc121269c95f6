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
  uint2* stage;     // the pointer words, when they stay in shared memory
  uint16_t* fidx;   // in s1 and s2, which are free once the transition codes are there
};

__device__ __forceinline__ StripSmem carve_strip(unsigned char* base, const NwGeom& g) {
  StripSmem S;
  const size_t ls = align16(size_t(g.lmax) + kStripPad), lq = align16(size_t(g.lmax));
  S.s1 = base;
  S.s2 = base + ls;
  S.qual = base + 2 * ls;
  S.tcode = base + 2 * ls + lq;
  S.stage = reinterpret_cast<uint2*>(base + 2 * ls + 2 * lq);
  S.fidx = reinterpret_cast<uint16_t*>(base);
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

// Walks the pointer words back from (len1, len2). Lane t holds the words of
// row i - t of the lane's diagonals that the walk is on; two ballots turn the
// current diagonal's bits of the 32 rows into a run of diagonal steps and the
// gap that ends it, until the walk leaves the rows or the diagonals. The next
// 32 rows' words are on their way meanwhile. The bound is the chain of
// dependent instructions of one warp, about 200 cycles a run: a walk that also
// read its words anew for every run took 212,000 cycles for two unrelated
// 1,450-nt sequences (345 runs) and 34,000 for two copies of one.
template <int C, bool DBG>
__device__ __forceinline__ bool strip_traceback(int lane, int len1, int len2, int o_lo, int W, const StripSmem& S,
                                                const uint2* planes, uint32_t* ham_out, uint32_t* err_word,
                                                uint8_t* dbg0, uint8_t* dbg1, uint32_t* dbg_len) {
  constexpr int N = 2 * C;
  constexpr unsigned RPW = strip_rows_per_word(C), NB = RPW * N;
  const uint8_t* const s1 = S.s1;
  const uint8_t* const s2 = S.s2;
  uint8_t* const tcode = S.tcode;
  for (int p = lane; p < len2; p += 32) tcode[p] = uint8_t(kUnaligned | (((s2[p] & 15u) - 1u) * 5u));
  __syncwarp();
  int i = len1, j = len2;
  uint32_t mism = 0, alen = 0;
  // rows count as the DP inserted them: row i of lane l is its (i + l - 1)-th
  auto word_at = [&](int row, int l) -> uint2 {
    const unsigned r = unsigned(max(row, 1) + l - 1);
    return planes[(r / RPW) * 32 + l];
  };
  auto shift_of = [](int row, int l) -> unsigned { return NB - 1 - (unsigned(row + l - 1) % RPW) * N; };
  // The free gaps of the last row or column are the one place of long gap
  // runs: lane t tests the t-th next gap.
  const bool longer2 = len2 > len1;
  for (int g = 32; g == 32;) {
    const int it = longer2 ? i : i - lane, jt = longer2 ? j - lane : j, xt = jt - it - o_lo;
    bool same = it > 0 && jt > 0 && xt >= 0 && xt < W;
    if (same) {
      const int lt = xt / N;
      const uint2 v = word_at(it, lt);
      const unsigned b = shift_of(it, lt) - unsigned(xt - lt * N);
      same = !((v.x >> b) & 1u) && bool((v.y >> b) & 1u) == longer2;
    }
    g = __clz(__brev(~__ballot_sync(FULL, same)));
    if (DBG) {
      if (lane < g) {
        dbg0[alen + lane] = longer2 ? uint8_t('-') : uint8_t(s1[i - 1 - lane] & 15u);
        dbg1[alen + lane] = longer2 ? uint8_t(s2[j - 1 - lane] & 15u) : uint8_t('-');
      }
      alen += uint32_t(g);
    }
    i -= longer2 ? 0 : g;
    j -= longer2 ? g : 0;
  }
  uint2 wn = make_uint2(0u, 0u);
  int wn_l = -1, wn_i = 0;  // wn: the words of rows wn_i .. wn_i - 31 of lane wn_l
  bool bad = false;
  while (i > 0 && j > 0) {
    const int idx = j - i - o_lo;
    bad = unsigned(idx) >= unsigned(W);
    if (bad) break;
    const int l = idx / N, it = i - lane;
    const uint2 w = wn_l == l && wn_i == i ? wn : word_at(it, l);
    wn = word_at(it - 32, l);
    wn_l = l;
    wn_i = i - 32;
    const unsigned sh = shift_of(it, l);
    const unsigned a = s1[max(it - 1, 0)] & 15u;
    int k = idx - l * N, t0 = 0;
    do {
      const unsigned b = (sh - unsigned(k)) & 31u;
      const uint32_t d = __ballot_sync(FULL, (w.x >> b) & 1u), lf = __ballot_sync(FULL, (w.y >> b) & 1u);
      const int f = min(__clz(__brev(~(d >> t0))), min(i, j));
      const int u = lane - t0;
      if (unsigned(u) < unsigned(f)) {
        const unsigned c = s2[j - 1 - u] & 15u;
        tcode[j - 1 - u] = uint8_t((a - 1u) * 4u + (c - 1u));
        mism += a != c ? 1u : 0u;
        if (DBG) {
          dbg0[alen + u] = uint8_t(a);
          dbg1[alen + u] = uint8_t(c);
        }
      }
      if (DBG) alen += uint32_t(f);
      i -= f;
      j -= f;
      t0 += f;
      if (t0 >= 32 || min(i, j) == 0) break;
      const int left = int((lf >> t0) & 1u);
      if (DBG) {
        if (lane == 0) {
          dbg0[alen] = left ? uint8_t('-') : uint8_t(s1[i - 1] & 15u);
          dbg1[alen] = left ? uint8_t(s2[j - 1] & 15u) : uint8_t('-');
        }
        ++alen;
      }
      j -= left;
      i -= 1 - left;
      t0 += 1 - left;
      k += 1 - 2 * left;
    } while (t0 < 32 && unsigned(k) < unsigned(N) && min(i, j) > 0);
  }
  if (bad) {
    if (lane == 0) atomicOr(err_word, DERR_TRACEBACK);
    return false;
  }
  if (DBG) {  // row 0 moves left, column 0 moves up
    for (int t = lane; t < j; t += 32) { dbg0[alen + t] = '-'; dbg1[alen + t] = s2[j - 1 - t] & 15u; }
    for (int t = lane; t < i; t += 32) { dbg0[alen + t] = s1[i - 1 - t] & 15u; dbg1[alen + t] = '-'; }
    if (lane == 0) *dbg_len = alen + uint32_t(i + j);
  }
  __syncwarp();
  *ham_out = __reduce_add_sync(FULL, mism);
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
// 5.0 to 1.15 ms, one aligning 24,908 pairs of 250 nt (band 16) from 1.8 to
// 0.53 ms, and one of 4 such pairs from 51 to 30 us.
//
// Values are kept less the gap costs of their row and column (H = V - sum of
// gl over 1..j - sum of gu over 1..i): the two gap moves then cost nothing,
// a diagonal step adds w = score - gl(j) - gu(i), and a cell is one fused
// add-max on the chain from its left neighbour.
//
// A cell's two pointer bits (diagonal best; else left better than up) are the
// signs of differences, shifted into two words per lane: RPW = 16, 8, 4, 4 rows
// per word, written as one 256-byte row of `planes` per RPW rows.
//
// The rows where some lane is before its first cell, or past the last row or
// column's start, take the SLOW form of the row; the rest need no tests.
//
// S.s1/S.s2 hold the codes, with the run flags when HOMO. Needs a band of
// W <= 62 C diagonals, so that the lane after the last
// one in use holds the mark outside the band (strip_cols).
template <int C, bool HOMO, bool DBG>
__device__ __forceinline__ bool strip_align(int lane, int len1, int len2, int match, int mismatch, int gap, int hgap,
                                         int band, const StripSmem& S, uint2* planes,
                                         uint32_t* ham_out, uint32_t* err_word, uint8_t* dbg0, uint8_t* dbg1,
                                         uint32_t* dbg_len) {
  constexpr int N = 2 * C, RPW = strip_rows_per_word(C);
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
  int V[N], LB[N], Y[N], CL[HOMO ? N : 1];  // values; band-edge marks; column codes and gap costs
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
  for (int k = 0; k < N; ++k) {
    Y[k] = y_at(ol - lc + k, Slow{});
    if (HOMO) {
      CL[k] = (Y[k] & 16) ? -hgap : -gap;
      Y[k] &= 15;
    }
  }
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
        const int cl = HOMO ? CL[(k + u) % (HOMO ? N : 1)] : -gap;
        const int w = Y[(k + u) % N] == xc ? wa : wb;
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
      Y[u] = HOMO ? yn & 15 : yn;
      if (HOMO) CL[u % (HOMO ? N : 1)] = (yn & 16) ? -hgap : -gap;
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
  return strip_traceback<C, DBG>(lane, len1, len2, o_lo, W, S, planes, ham_out, err_word, dbg0, dbg1, dbg_len);
}

// The narrowest strip that holds the pair's band. CMAX bounds it for the
// launch (the geometry's rule: strip_cols).
template <int CMAX, bool HOMO, bool DBG = false>
__device__ __forceinline__ bool strip_dispatch(int lane, int len1, int len2, const KParams& kp, bool homo,
                                               const StripSmem& S, uint2* planes, uint32_t* ham,
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
  return strip_align<CC, HOMO, DBG>(lane, len1, len2, kp.match, kp.mismatch, kp.gap, hg, kp.band, S, planes, \
                               ham, err_word, d0, d1, dl)
  STRIP_CASE(1);
  if constexpr (CMAX >= 2) STRIP_CASE(2);
  if constexpr (CMAX >= 3) STRIP_CASE(3);
  if constexpr (CMAX >= 4) STRIP_CASE(4);
#undef STRIP_CASE
}

}  // namespace dgpu
