// tsu_packed.cuh -- the shared-ring align kernel: two diagonals per thread.
//
// The wavefront ring of the last max(x, o+e)+1 scores is 16-bit in shared
// memory, and one thread computes two neighbouring diagonals (one 32-bit
// word) at a time with per-halfword add-max / add-min instructions.  What
// bounds it is the integer ALU pipe (half an instruction per cycle and
// scheduler; ncu: 75 % busy in the one-diagonal form), so the layout is
// chosen to spend few ALU instructions per cell:
//   * an offset h is held as 2 h + kZero: an absent cell is any halfword below
//     kZero, and bit 0 is free.  A candidate enters a maximum with bit 0 set
//     when it wins ties, so one add-max both takes the maximum and records
//     which side won; I, D and M of two cells take nine such instructions with
//     all their source bits;
//   * absent cells stay below kZero: M rows store absent as 0, I climbs by 2
//     per diagonal it moves, at most 2 ring_w <= kZero (an I past the matrix
//     edge may wrap past 2^16 to absent, and climbs from there);
//   * every row has the same diagonal-to-position map (position = k - kbase)
//     and is all absent before its first write, so no read needs a range
//     test; a source row that does not exist at this score is a permanent
//     row of absent cells;
//   * the range of diagonals at score s follows from the penalties alone
//     (one more on each side per gap extension), clipped to [-m, n], so a step
//     has no reductions: its end test is one read of M on diagonal n - m;
//   * an M offset beyond the matrix edge is clamped to the edge instead of
//     dropped.  A clamped cell stands for a position that is reachable at no
//     higher cost, from which the alignment cannot end earlier than it does
//     through the cell that reached the edge, so neither the score nor the
//     cells on the backtrace's path change;
//   * with CIGARs a cell's history is its source bits alone (4 bits; 8 with
//     two gap pieces), not its offset: the backtrace follows the bits from the
//     end to score 0, and the matches between the edits are then found
//     again from the front, 512 bases per warp comparison.
// Measured on one B200 against the one-diagonal form (the same ring, limits
// per row kept by warp reductions, 4-byte history words; align pass, scores +
// CIGARs): 200,000 x 1 kbp at 5 % 31.9 -> 16.6 ms (scores only 24.0 -> 11.9),
// 1,000 x 10 kbp at 15 % on 16 warps 112 -> 50.5 ms, 20,000 x 1 kbp dual
// gap-affine on 8 warps 42.5 -> 15.4 ms.  A cell pair takes 75 warp
// instructions scored (90 with history) and a step 145, against 175 per 32
// cells before; issue slots are 86 % and the ALU pipe 68 % busy.
// Within a score bound (kBound): 1,000 x 10 kbp at 15 % 50.5 -> 27.1 ms with
// the probe, on 8 warps; two words per lane 32.0 -> 25.2 ms without it.
// Limits: sides of at most kPackedPlainLen bases (kPackedMaxLen with a bound),
// ACGT only, at most 128 score steps of ring depth; other pairs go to
// tsu_wide.cuh (with a bound), to the shared ring of one diagonal per thread
// (deeper rings with CIGARs, sides up to 32,000) or to the global ring
// (tsu_align.cuh).
#pragma once

#include <type_traits>

#include "tsu_common.cuh"
#include "tsu_extend.cuh"
#include "tsu_half2.cuh"

namespace tsu {

// Halfword of offset 0 (kZero): a multiple of 32 (the low 5 bits of a halfword
// are then twice the base's place in its 16-base word), at least 2 ring_w, and
// small enough for the longest side twice and 32 above it.  Launches without
// score bounds take 32768, where bit 15 says present (two instructions of 75
// less); bounded ones and the probe take 24576 for longer sides.
constexpr uint32_t kZeroPlain = 32768u, kZeroBound = 24576u;
static_assert(2 * kPackedMaxW <= kZeroBound && kZeroPlain + 2 * kPackedPlainLen + 32 <= 65535 &&
                  kZeroBound + 2 * kPackedMaxLen + 32 <= 65535,
              "16-bit offsets");

// ---- shared memory by byte address --------------------------------------------
// One address register per group, taken once: accesses are a register and a
// constant.  (Through pointers the base address of the block's shared memory
// was formed again at every step: 13 of its 200 instructions.)
#ifdef TSU_WARP_EMU
using smem_t = unsigned char*;
inline smem_t smem_addr(unsigned char* p) { return p; }
template <int kOff = 0>
inline uint32_t lds32(smem_t a) {
  uint32_t v;
  std::memcpy(&v, a + kOff, 4);
  return v;
}
inline uint32_t lds16(smem_t a) {
  uint16_t v;
  std::memcpy(&v, a, 2);
  return v;
}
inline void lds128(smem_t a, int& x, int& y, int& z, int& w) {
  int v[4];
  std::memcpy(v, a, 16);
  x = v[0], y = v[1], z = v[2], w = v[3];
}
inline void sts32(smem_t a, uint32_t v) { std::memcpy(a, &v, 4); }
inline void sts16(smem_t a, uint32_t v) {
  const uint16_t h = (uint16_t)v;
  std::memcpy(a, &h, 2);
}
inline void sts128(smem_t a, int x, int y, int z, int w) {
  const int v[4] = {x, y, z, w};
  std::memcpy(a, v, 16);
}
#else
using smem_t = uint32_t;
__device__ __forceinline__ smem_t smem_addr(unsigned char* p) {
  uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
  asm volatile("" : "+r"(a));  // opaque: kept in a register
  return a;
}
template <int kOff = 0>
__device__ __forceinline__ uint32_t lds32(smem_t a) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1+%2];" : "=r"(v) : "r"(a), "n"(kOff));
  return v;
}
__device__ __forceinline__ uint32_t lds16(smem_t a) {
  uint16_t v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ void lds128(smem_t a, int& x, int& y, int& z, int& w) {
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(x), "=r"(y), "=r"(z), "=r"(w) : "r"(a));
}
__device__ __forceinline__ void sts32(smem_t a, uint32_t v) {
  asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ void sts16(smem_t a, uint32_t v) {
  asm volatile("st.shared.u16 [%0], %1;" ::"r"(a), "h"((uint16_t)v) : "memory");
}
__device__ __forceinline__ void sts128(smem_t a, int x, int y, int z, int w) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
#endif

// 16 bases from position pos of the packed words at address w.
__device__ __forceinline__ uint32_t lds_win16(smem_t w, int pos) {
  const smem_t a = w + ((pos >> 4) << 2);
  return __funnelshift_r(lds32(a), lds32<4>(a), (uint32_t)pos << 1);
}
// lcp16 (tsu_extend.cuh) over words in shared memory.
__device__ __forceinline__ int lds_lcp(smem_t pw, int v, smem_t tw, int h, int rem) {
  int l = 0;
  while (l < rem) {
    const uint32_t d = lds_win16(pw, v + l) ^ lds_win16(tw, h + l);
    if (d) {
      l += h2_tz(d) >> 1;
      break;
    }
    l += 16;
  }
  return l < rem ? l : rem;
}

// 0xffff in each half that holds an offset.  (min() first: the sum that moves
// kZero to bit 15 then carries nothing.)
template <uint32_t kZero>
__device__ __forceinline__ uint32_t h2_present(uint32_t p) {
  if constexpr (kZero == 32768u) return h2_signmask(p);
  return h2_signmask(h2_min(p, (kZero + 16) * 0x10001u) + (32768u - kZero) * 0x10001u);
}

// ---- the cells of one word ---------------------------------------------------
// Byte offsets of the rows a step writes and reads.
struct PackedRows {
  int w_m, r_mx, r_mo, r_mo2, w_i, w_d, r_ie, r_de, w_i2, w_d2, r_ie2, r_de2;
};
// The pair's words and ends.
struct PackedPair {
  smem_t pws, tws;
  uint32_t m2, kend2;  // 2 m, 2 (n - m) + kZero in both halves
};

// Two cells of each of U words (at address at[u] = position word of row 0;
// k2[u]: 2 k + kZero of both): I, D and M of this score from the source rows
// into the score's rows.  om: M; valid: the halves that are present; bits
// (kBits): source bits, from bit 0 of each half: mismatch, deletion, I
// extended, D extended (two pieces: mismatch, D2, D1, I2, then I1, D1, I2, D2
// extended); ext: M minus its value before extension, per half.  U = 2 runs
// two independent chains of loads and maxima side by side: a cell is one chain
// from the ring's loads through the sequences' to the store, and wide rings
// leave an SM 16 warps to cover it.
template <int kModel, bool kBits, uint32_t kZero, int U>
__device__ __forceinline__ void packed_words_step(const PackedRows& r, const PackedPair& q, const smem_t (&at)[U],
                                                  const uint32_t (&k2)[U], uint32_t (&om)[U], uint32_t (&valid)[U],
                                                  uint32_t (&ext)[U], uint32_t (&bits)[U]) {
  constexpr bool kDual = kModel == kModelDual, kLin = kModel == kModelLinear;
  constexpr uint32_t kOne2 = 0x00010001u, kClean = 0xfffefffeu, kZero2 = kZero * 0x10001u;
  // I is kept as 2 (h - 1) + kZero, so that M[k-1] is its own insertion
  // candidate; bit 0 of ins, del: extension; of t: deletion over insertion;
  // of p: mismatch over both (ties go that way)
  uint32_t mo_l[U], mo_r[U], mx[U], ie[U], de[U], mo2_l[U], mo2_r[U], ie2[U], de2[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const uint32_t ob = lds32(at[u] + r.r_mo);
    mo_l[u] = h2_next(lds32<-4>(at[u] + r.r_mo), ob);  // M[s-o-e] on k-1
    mo_r[u] = h2_next(ob, lds32<4>(at[u] + r.r_mo));   // on k+1
    mx[u] = lds32(at[u] + r.r_mx);
    if constexpr (!kLin) {
      ie[u] = h2_next(lds32<-4>(at[u] + r.r_ie), lds32(at[u] + r.r_ie));
      de[u] = h2_next(lds32(at[u] + r.r_de), lds32<4>(at[u] + r.r_de));
    }
    if constexpr (kDual) {
      const uint32_t o2 = lds32(at[u] + r.r_mo2);
      mo2_l[u] = h2_next(lds32<-4>(at[u] + r.r_mo2), o2);
      mo2_r[u] = h2_next(o2, lds32<4>(at[u] + r.r_mo2));
      ie2[u] = h2_next(lds32<-4>(at[u] + r.r_ie2), lds32(at[u] + r.r_ie2));
      de2[u] = h2_next(lds32(at[u] + r.r_de2), lds32<4>(at[u] + r.r_de2));
    }
  }
  uint32_t p[U], c[U], vv[U], up[U], x0[U], x1[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    uint32_t t;
    if constexpr (!kLin) {
      const uint32_t ins = h2_addmax(ie[u], 3 * kOne2, mo_l[u]);
      const uint32_t del = h2_addmax(de[u], kOne2, mo_r[u]);
      const uint32_t insc = ins & kClean;
      sts32(at[u] + r.w_i, insc);
      sts32(at[u] + r.w_d, del & kClean);
      if constexpr (!kDual) {
        t = h2_addmax(insc, 2 * kOne2, del | kOne2);
        if constexpr (kBits) {
          const uint32_t f2 = (ins & kOne2) | ((del << 1) & (2 * kOne2));
          bits[u] = ((t << 1) & (2 * kOne2)) | (f2 << 2);
        }
      } else {
        const uint32_t ins2 = h2_addmax(ie2[u], 3 * kOne2, mo2_l[u]);
        const uint32_t del2 = h2_addmax(de2[u], kOne2, mo2_r[u]);
        sts32(at[u] + r.w_i2, ins2 & kClean);
        sts32(at[u] + r.w_d2, del2 & kClean);
        const uint32_t t1 = h2_max(insc, ins2 | kOne2);                      // I2 over I1
        const uint32_t t2 = h2_addmax(t1 & kClean, 2 * kOne2, del | kOne2);  // D1 over both
        t = h2_max(t2 & kClean, del2 | kOne2);                               // D2 over all
        if constexpr (kBits)
          bits[u] = ((t & kOne2) << 1) | ((t2 & kOne2) << 2) | ((t1 & kOne2) << 3) | ((ins & kOne2) << 4) |
                    ((del & kOne2) << 5) | ((ins2 & kOne2) << 6) | ((del2 & kOne2) << 7);
      }
    } else {
      t = h2_addmax(mo_l[u], 2 * kOne2, mo_r[u] | kOne2);
      if constexpr (kBits) bits[u] = (t & kOne2) << 1;
    }
    p[u] = h2_addmax(mx[u], 3 * kOne2, t & kClean);
    if constexpr (kBits) bits[u] |= p[u] & kOne2;
    // extend both M cells: clamp into [first, last] offset of the diagonal
    // (absent cells compare some window of it), compare 16 bases at the
    // halfword's place, add twice the matches
    up[u] = h2_min(k2[u], q.kend2) + q.m2;  // min(n, m + k)
    c[u] = h2_min(h2_max(p[u] & kClean, h2_max(k2[u], kZero2)), up[u]);
    vv[u] = c[u] - k2[u] + kZero2;
  }
  constexpr int kZeroByte = (int)(kZero >> 5) * 4;  // byte offset of halfword kZero's base word
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const smem_t h0 = q.tws + (((c[u] & 0xffffu) >> 5) << 2), h1 = q.tws + ((c[u] >> 21) << 2);
    const smem_t v0 = q.pws + (((vv[u] & 0xffffu) >> 5) << 2), v1 = q.pws + ((vv[u] >> 21) << 2);
    x0[u] = __funnelshift_r(lds32<-kZeroByte>(v0), lds32<4 - kZeroByte>(v0), vv[u]) ^
            __funnelshift_r(lds32<-kZeroByte>(h0), lds32<4 - kZeroByte>(h0), c[u]);
    x1[u] = __funnelshift_r(lds32<-kZeroByte>(v1), lds32<4 - kZeroByte>(v1), vv[u] >> 16) ^
            __funnelshift_r(lds32<-kZeroByte>(h1), lds32<4 - kZeroByte>(h1), c[u] >> 16);
  }
  uint32_t z[U], whole = 0;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    valid[u] = h2_present<kZero>(p[u]);
    z[u] = (uint32_t)(h2_tz(x0[u]) + (h2_tz(x1[u]) << 16)) & 0x003e003eu & valid[u];
    whole |= z[u];
  }
  if (whole & 0x00200020u) {  // a whole window matched: go on in that half
#pragma unroll
    for (int u = 0; u < U; ++u) {
#pragma unroll 1
      for (int half = 0; half < 32; half += 16) {
        if ((z[u] >> half) & 0x20u) {
          const uint32_t ch = (c[u] >> half) & 0xffffu, vh = (vv[u] >> half) & 0xffffu;
          const int rem = ((int)((up[u] >> half) & 0xffffu) - (int)ch) / 2 - 16;
          if (rem > 0)
            z[u] += (uint32_t)(2 * lds_lcp(q.pws, ((int)vh - (int)kZero) / 2 + 16, q.tws, ((int)ch - (int)kZero) / 2 + 16,
                                           rem))
                    << half;
        }
      }
    }
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    om[u] = h2_addmin(c[u], z[u], up[u]) & valid[u];
    ext[u] = om[u] - (c[u] & valid[u]);
    sts32(at[u] + r.w_m, om[u]);
  }
}

// The row tables of a group in shared memory (tab_m, tab_g, tab_g2: 16 bytes
// per M slot, I / D slot pair, I2 / D2 slot pair): byte offsets of the rows a
// score writes and reads, by its place in the ring: M {out, s-x, s-o-e,
// s-o2-e2}, I and D {out I, out D, I and D at s-e}, I2 and D2 likewise.
template <bool kDual>
__device__ __forceinline__ void packed_tables(const Pen& pen, int RB, smem_t tab_m, int gt, int GT) {
  const int rm = pen.rm, re = pen.re, re2 = pen.re2;
  const smem_t tab_g = tab_m + 16 * rm, tab_g2 = tab_g + 16 * re;
  auto back = [](int slot, int by, int depth) -> int { return slot < by ? slot - by + depth : slot - by; };
  for (int j = gt; j < rm; j += GT)
    sts128(tab_m + 16 * j, j * RB, back(j, pen.x, rm) * RB, back(j, pen.go, rm) * RB,
           kDual ? back(j, pen.go2, rm) * RB : 0);
  for (int j = gt; j < re; j += GT) {
    const int q = rm + back(j, pen.ge, re);
    sts128(tab_g + 16 * j, (rm + j) * RB, (rm + re + j) * RB, q * RB, (q + re) * RB);
  }
  for (int j = gt; j < re2; j += GT) {
    const int g0 = rm + 2 * re, q = g0 + back(j, pen.ge2, re2);
    sts128(tab_g2 + 16 * j, (g0 + j) * RB, (g0 + re2 + j) * RB, q * RB, (q + re2) * RB);
  }
}

// A pair's score by score bookkeeping, the same for every lane: the step's
// rows, the diagonals gained, which wavefronts exist (kDeep: rings deeper than
// 64 scores, of up to 128).
template <int kModel, bool kDeep>
struct PackedSteps {
  static constexpr bool kDual = kModel == kModelDual, kLin = kModel == kModelLinear;
  smem_t tab_m, tab_g, tab_g2, tab_end;
  smem_t tm, tg, tg2;
  int none_row;                // the row of absent cells
  int grow, grow_at;           // diagonals gained on each side, next score that gains one
  int grow2, grow2_at;         // the second gap piece
  // which of the last 64 scores (kDeep: had_m, the 64 before them) have an M
  // wavefront, which of the last 64 an I or D; once every score in reach has
  // all of them it stays so (full)
  unsigned long long has_m, had_m, has_g, has_g2;
  bool full;

  __device__ __forceinline__ void begin(const Pen& pen, smem_t tables, int none) {
    tab_m = tm = tables;
    tab_g = tg = tab_m + 16 * pen.rm;
    tab_g2 = tg2 = tab_g + 16 * pen.re;
    tab_end = tab_g2 + 16 * pen.re2;
    none_row = none;
    grow = grow2 = 0;
    grow_at = pen.go;
    grow2_at = kDual ? pen.go2 : INT_MAX;
    has_m = 1, had_m = 0, has_g = 0, has_g2 = 0;
    full = false;
  }
  __device__ __forceinline__ int gained() const { return kDual ? max(grow, grow2) : grow; }
  // To score s: its rows; true when a diagonal was gained.
  __device__ __forceinline__ bool next(const Pen& pen, int s, PackedRows* r) {
    tm = tm + 16 == tab_g ? tab_m : tm + 16;
    lds128(tm, r->w_m, r->r_mx, r->r_mo, r->r_mo2);
    if constexpr (!kLin) {
      tg = tg + 16 == tab_g2 ? tab_g : tg + 16;
      lds128(tg, r->w_i, r->w_d, r->r_ie, r->r_de);
    }
    if constexpr (kDual) {
      tg2 = tg2 + 16 == tab_end ? tab_g2 : tg2 + 16;
      lds128(tg2, r->w_i2, r->w_d2, r->r_ie2, r->r_de2);
    }
    bool wider = false;
    if (s >= grow_at) {
      ++grow;
      grow_at += pen.ge;
      wider = true;
    }
    if constexpr (kDual) {
      if (s >= grow2_at) {
        ++grow2;
        grow2_at += pen.ge2;
        wider = true;
      }
    }
    return wider;
  }
  // Whether the score has a wavefront (false: null step, wfa_gpu.cu:417-422;
  // no row of it is read); sources that do not exist become the row of absent
  // cells.
  __device__ __forceinline__ bool present(const Pen& pen, PackedRows* r) {
    if (full) return true;
    auto m_at = [&](int back) -> bool {
      return (((!kDeep || back <= 64) ? has_m >> (back - 1) : had_m >> (back - 65)) & 1) != 0;
    };
    const bool px = m_at(pen.x), po = m_at(pen.go);
    const bool pe = !kLin && ((has_g >> (pen.ge - 1)) & 1);
    const bool po2 = kDual && m_at(pen.go2);
    const bool pe2 = kDual && ((has_g2 >> (pen.ge2 - 1)) & 1);
    const bool pm = px | po | pe | po2 | pe2;
    if constexpr (kDeep) had_m = (had_m << 1) | (has_m >> 63);
    has_m = (has_m << 1) | (pm ? 1u : 0u);
    if constexpr (!kLin) has_g = (has_g << 1) | ((po | pe) ? 1u : 0u);
    if constexpr (kDual) has_g2 = (has_g2 << 1) | ((po2 | pe2) ? 1u : 0u);
    if (!pm) return false;
    const unsigned long long dm = kDeep && pen.rm > 64 ? ~0ull : (1ull << (pen.rm - 1)) - 1,
                             dh = kDeep ? (1ull << max(pen.rm - 65, 0)) - 1 : 0,
                             dg = kLin ? 0 : (1ull << pen.ge) - 1,
                             dg2 = kDual ? (1ull << pen.ge2) - 1 : 0;
    full = (has_m & dm) == dm && (!kDeep || (had_m & dh) == dh) && (kLin || (has_g & dg) == dg) && (!kDual || (has_g2 & dg2) == dg2);
    if (!px) r->r_mx = none_row;
    if (!po) r->r_mo = none_row;
    if constexpr (!kLin) {
      if (!pe) r->r_ie = r->r_de = none_row;
    }
    if constexpr (kDual) {
      if (!po2) r->r_mo2 = none_row;
      if (!pe2) r->r_ie2 = r->r_de2 = none_row;
    }
    return true;
  }
};

// Longest common prefix of pattern[v..] and text[h..], at most rem, by a
// whole warp: 512 bases per comparison.
__device__ __forceinline__ int warp_lcp(smem_t pw, int v, smem_t tw, int h, int rem, int lane) {
  int l = 0;
  while (l < rem) {
    const int at = l + 16 * lane;
    int lx = 0;  // lanes past the end stop the run at their start, which min() below cuts to rem
    if (at < rem) lx = h2_tz(lds_win16(pw, v + at) ^ lds_win16(tw, h + at)) >> 1;
    const unsigned stop = __ballot_sync(0xffffffffu, lx < 16);
    if (stop) {
      const int src = __ffs((int)stop) - 1;
      return min(l + 16 * src + __shfl_sync(0xffffffffu, lx, src), rem);
    }
    l += 512;
  }
  return rem;
}

template <class T>
__device__ __forceinline__ T ld_l2(const T* p) {
#ifdef TSU_WARP_EMU
  return *p;
#else
  return __ldcg(p);
#endif
}

// The CIGAR of a finished pair, by one warp.  First the walk: from the end
// (s_end, k_fin) along the source bits to score 0, 32 scores of history in
// registers at a time (lane l holds score top - l: 16 diagonals around the
// path; 8 with two gap pieces), each edit or gap written as one entry
// (length << 4 | op) downwards from out + cap.  Then the replay from the
// front: matches found again between the entries (lcp(v, h, at most)), runs written upwards from
// out.  Of e entries at most 2 e + 1 runs are written, 2 j + 1 of them before
// entry j is read, so with cap >= 2 e + 2 they share the space.  Returns the
// number of runs, or -1 on an inconsistency.
template <int kModel, class Lcp>
__device__ __forceinline__ int packed_cigar(const uint32_t* hist, int64_t hist_chunks,
                                            const int2* table, int s_end, int k_fin, int m, int n,
                                            const Pen& pen, int kbase, int lo0, int hi0, Lcp&& lcp,
                                            uint32_t* out, int cap, int lane) {
  constexpr unsigned FULL = 0xffffffffu;
  constexpr bool kDual = kModel == kModelDual, kLin = kModel == kModelLinear;
  constexpr int kCS = kDual ? 1 : 2;  // log2 of pairs of diagonals per 32-bit chunk
  int s = s_end, k = k_fin;
  int state = 0;  // 0: M; 1, 2: inside an I, D of the first gap piece; 3, 4: of the second
  int top = -1, c0 = 0;
  uint32_t d0 = 0, d1 = 0;
  int ne = 0;           // entries
  uint32_t gap = 0;     // the open gap's entry
  while (s > 0) {
    const int pos = k - kbase;
    const int ch = pos >> (kCS + 1);
    if (s > top || s <= top - 32 || ch < c0 || ch > c0 + 1) {
      top = s;
      c0 = (pos - (1 << kCS)) >> (kCS + 1);
      d0 = d1 = 0;
      if (s - lane > 0) {
        // (past L1: the blocks of a cluster write one history)
        const int2 te = ld_l2(table + s - lane);
        const int64_t i = (int64_t)te.y + c0 - te.x;
        if (i >= 0 && i < hist_chunks) d0 = ld_l2(hist + i);
        if (i + 1 >= 0 && i + 1 < hist_chunks) d1 = ld_l2(hist + i + 1);
      }
    }
    const uint32_t word = __shfl_sync(FULL, ch == c0 ? d0 : d1, top - s);
    uint32_t ins, ext;
    if constexpr (kDual) {
      const uint32_t b = word >> ((pos & 3) * 8);
      int comp = state;
      if (comp == 0) comp = (b & 1u) ? 0 : (b & 2u) ? 4 : (b & 4u) ? 2 : (b & 8u) ? 3 : 1;
      if (comp == 0) {
        if (lane == 0 && ne < cap) out[cap - 1 - ne] = (1u << 4) | kOpX;
        ++ne;
        s -= pen.x;
        continue;
      }
      ins = comp & 1;
      ext = (b >> (3 + comp)) & 1u;
      s -= ext ? (comp <= 2 ? pen.ge : pen.ge2) : (comp <= 2 ? pen.go : pen.go2);
      state = ext ? comp : 0;
    } else {
      const uint32_t b = word >> ((pos & 7) * 4);
      if (state == 0) {
        if (b & 1u) {
          if (lane == 0 && ne < cap) out[cap - 1 - ne] = (1u << 4) | kOpX;
          ++ne;
          s -= pen.x;
          continue;
        }
        state = (b & 2u) ? 2 : 1;
      }
      ins = state & 1;
      ext = kLin ? 0u : (b >> (1 + state)) & 1u;
      s -= ext ? pen.ge : pen.go;
      if (!ext) state = 0;
    }
    gap += 1u << 4;
    k += ins ? -1 : 1;
    if (!ext) {
      if (lane == 0 && ne < cap) out[cap - 1 - ne] = gap | (ins ? kOpI : kOpD);
      ++ne;
      gap = 0;
    }
  }
  if (s < 0 || gap || state || k < lo0 || k > hi0 || 2 * ne + 2 > cap) return -1;
  __syncwarp();
  // ---- replay
  int v = k < 0 ? -k : 0, h = k > 0 ? k : 0;  // the free leading gap
  int nr = 0;
  uint32_t cur = 0;  // the open run
  auto put = [&](uint32_t op, int len) {
    if (len <= 0) return;
    if (cur && (cur & 15u) == op) {
      cur += (uint32_t)len << 4;
      return;
    }
    if (cur) {
      if (lane == 0) out[nr] = cur;
      ++nr;
    }
    cur = ((uint32_t)len << 4) | op;
  };
  put(kOpD, v);
  put(kOpI, h);
  uint32_t ent = 0;
  for (int j = 0;; ++j) {
    const int rem = min(m - v, n - h);
    if (rem < 0) return -1;
    const int l = lcp(v, h, rem);
    put(kOpM, l);
    v += l;
    h += l;
    if (j == ne) break;
    if ((j & 31) == 0) {
      __syncwarp();
      ent = j + lane < ne ? out[cap - ne + j + lane] : 0u;
      __syncwarp();
    }
    const uint32_t e = __shfl_sync(FULL, ent, j & 31);
    const int len = (int)(e >> 4);
    const uint32_t op = e & 15u;
    put(op, len);
    if (op != kOpI) v += len;
    if (op != kOpD) h += len;
  }
  if (h - v != k_fin || h != min(n, m + k_fin)) return -1;
  put(kOpD, m - v);
  put(kOpI, n - h);
  if (cur) {
    if (lane == 0) out[nr] = cur;
    ++nr;
  }
  return nr;
}

// The body of align_kernel for the shared ring (see the head of this file).
// kBound: the pairs have score bounds (a.bound), end to end; kDeep: PackedSteps.
template <bool kCigar, int GW, int kModel, bool kBound, bool kDeep>
__device__ __forceinline__ void align_packed(const AlignArgs& a, unsigned char* smem_raw) {
  constexpr bool kDual = kModel == kModelDual;
  constexpr bool kLin = kModel == kModelLinear;
  constexpr unsigned FULL = 0xffffffffu;
  constexpr int GT = 32 * GW;
  constexpr uint32_t kZero = kBound ? kZeroBound : kZeroPlain;
  constexpr int kMaxLen = kBound ? kPackedMaxLen : kPackedPlainLen;
  constexpr int kCS = kDual ? 1 : 2;  // log2 of diagonal pairs per 32-bit history chunk
  const int tid = threadIdx.x;
  const int gid = tid / GT;
  const int gt = tid - gid * GT;
  const int lane = tid & 31;
  const int wig = gt >> 5;
  const int gpb = blockDim.x / GT;
  const int64_t ggroup = (int64_t)blockIdx.x * gpb + gid;
  const int rows = a.pen.slots() + 1;  // and the row of absent cells
  // 4 broadcast words, 2 GW partials of the free-end test, the row tables,
  // the ring, the sequences.  Bounded pairs share out the group's bytes each
  // by its own width and lengths.
  const int gbytes = kBound ? a.group_bytes : group_smem_bytes(a.pen, a.ring_w, kModeShared, a.seq_cap, GW, true);
  const smem_t bc = smem_addr(smem_raw) + (size_t)gid * gbytes;
  const smem_t part = bc + 16;
  const smem_t tab_m = bc + packed_head_bytes(Pen(), GW);
  const smem_t ring = bc + packed_head_bytes(a.pen, GW);
  const smem_t ring0 = ring + 8;  // position 0 of row 0
  int W = a.ring_w;
  int RB = packed_row_words(W) * 4;  // bytes per row
  if constexpr (!kBound) packed_tables<kDual>(a.pen, RB, tab_m, gt, GT);
  uint32_t* const hist = kCigar ? a.hist + ggroup * a.hist_cap : nullptr;
  const int hist_cap = (int)a.hist_cap;  // below 2^31 (tsu_plan.h)
  int2* const table = kCigar ? a.table + ggroup * (int64_t)a.table_cap : nullptr;

  for (;;) {
    unsigned qi;
    if constexpr (GW == 1) {
      unsigned q = 0;
      if (lane == 0) q = atomicAdd(a.queue, 1u);
      qi = __shfl_sync(FULL, q, 0);
    } else {
      if (gt == 0) sts32(bc, atomicAdd(a.queue, 1u));
      group_sync<GW>(gid);
      qi = lds32(bc);
    }
    if ((int64_t)qi >= a.n_order) break;
    const int64_t pair = a.order ? a.order[qi] : (int64_t)qi;
    const int m = a.seq.pat_len[pair];
    const int n = a.seq.txt_len[pair];
    const bool bytemode = a.pk.nonacgt[pair] | a.pk.nonacgt[a.seq.n + pair];
    const int pwn = 2 * (int)packed_words(m);  // uint32 words
    const int twn = 2 * (int)packed_words(n);
    const int k_end = n - m;
    int32_t st = kPairOk;
    if (bytemode || m > kMaxLen || n > kMaxLen || (!kBound && pwn + twn > a.seq_cap)) st = kPairScratch;
    int s_end = -1, k_fin = k_end;
    int s = 0;
    int hbase = 0;  // history chunks in use
    unsigned long long n_cells = 0;
    uint32_t n_steps = 0, n_ext2 = 0;  // n_ext2: twice the bases matched by this thread's extend steps
    const int ub = kBound ? a.bound[pair] : 0;  // an upper bound of the score
    // diagonals of score 0 (free beginnings), and the ring's window
    const int lo0 = kBound ? 0 : -min(a.ef_pb, m), hi0 = kBound ? 0 : min(a.ef_tb, n);
    int kbase = -m;
    if constexpr (kBound) {
      // the window: what a path within the bound can reach
      int lo_b = 0, hi_b = 0;
      if (ub != kNoBound) bound_reach(a.pen, m, n, ub, &lo_b, &hi_b);
      kbase = lo_b;
      W = packed_width(hi_b - lo_b + 1);
      RB = packed_row_words(W) * 4;
      if (packed_head_bytes(a.pen, GW) + rows * RB + 4 * (pwn + twn) > gbytes || W > kPackedMaxW) st = kPairScratch;
    } else if (m + n + 2 > W) {
      // its middle on the middle of the beginning, inside [-m, n]
      kbase = min(max((lo0 + hi0 - W) >> 1, -m), n + 1 - W);
    }
    if (lo0 < kbase || hi0 - kbase >= W || kbase < -(int)(kZero / 2) || k_end < -(int)(kZero / 2) ||
        (kBound && ub == kNoBound))
      st = kPairScratch;

    if (st == kPairOk) {
      const uint32_t* gpw = reinterpret_cast<const uint32_t*>(a.pk.words + a.pk.woff[pair]);
      const uint32_t* gtw = reinterpret_cast<const uint32_t*>(a.pk.words + a.pk.woff[a.seq.n + pair]);
      const smem_t pws = ring + rows * RB;
      const smem_t tws = pws + 4 * pwn;
      if constexpr (kBound) packed_tables<kDual>(a.pen, RB, tab_m, gt, GT);
      for (int i = gt; i < pwn; i += GT) sts32(pws + 4 * i, __ldg(gpw + i));
      for (int i = gt; i < twn; i += GT) sts32(tws + 4 * i, __ldg(gtw + i));
      // every row all absent, the words on both sides of it included
      for (int i = 16 * gt; i < rows * RB; i += 16 * GT) sts128(ring + i, 0, 0, 0, 0);
      group_sync<GW>(gid);
      const int k_hi = k_end + a.ef_pe;  // highest diagonal that may end with pattern characters left
      const bool free_te = !kBound && a.ef_te > 0;
      const int n_te = n - a.ef_te;
      const bool ends_free = !kBound && (a.ef_pe > 0 || free_te);
      // whether M at text offset om on diagonal k (om <= min(n, m + k)) ends the alignment
      auto ends_at = [&](int om, int k) -> bool {
        return (om >= n && k <= k_hi) || (free_te && om - k >= m && om >= n_te);
      };
      // ---- score 0
      int fk = INT_MAX;
      {
        for (int k = lo0 + gt; k <= hi0; k += GT) {
          const int p0 = k > 0 ? k : 0;
          const int om = p0 + lds_lcp(pws, p0 - k, tws, p0, min(m - (p0 - k), n - p0));
          sts16(ring0 + 2 * (k - kbase), 2 * (uint32_t)om + kZero);
          if (ends_free && fk == INT_MAX && ends_at(om, k)) fk = k;
        }
        n_cells = (unsigned)(hi0 - lo0 + 1);
      }
      // the cell on diagonal n - m (the row of absent cells' first one when
      // the window does not hold it)
      const int pend = k_end - kbase;
      const bool end_in = pend >= 0 && pend < W;
      const smem_t end_cell = ring0 + (end_in ? 2 * pend : 0);
      const uint32_t end_val = end_in ? 2 * (uint32_t)n + kZero : 0x10000u;
      // After a step: has the alignment ended?  (One barrier, which also
      // separates the step's writes from the next one's reads.)
      int flip = 0;  // the free-end partials are double-buffered by step computed
      auto ended = [&](int fkt, int row_m, bool free_ends) {
        if (free_ends) {
          fkt = __reduce_min_sync(FULL, fkt);
          if constexpr (GW > 1) {
            flip ^= 4 * GW;
            const smem_t pa = part + flip;
            if (lane == 0) sts32(pa + 4 * wig, (uint32_t)fkt);
            group_sync<GW>(gid);
            fkt = __reduce_min_sync(FULL, lane < GW ? (int)lds32(pa + 4 * lane) : INT_MAX);
          } else {
            __syncwarp();
          }
          if (fkt != INT_MAX) {
            s_end = s;
            k_fin = fkt;
          }
        } else {
          group_sync<GW>(gid);
          if (lds16(end_cell + row_m) >= end_val) s_end = s;
        }
      };
      ended(fk, 0, ends_free);

      const int64_t bound = score_bound(m, n, a.pen);
      // scores this launch can compute: past s_max the end would have been
      // found (an inconsistency), past the step table the pair is handed back
      const int s_max = (int)(bound < INT_MAX - 1 ? bound : INT_MAX - 1);
      const int s_lim = min(kBound ? ub : s_max, kCigar ? min(s_max, a.table_cap - 1) : s_max);
      const PackedPair pp{pws, tws, h2_dup(2 * (uint32_t)m), h2_dup((uint32_t)((int)kZero + 2 * k_end))};
      // 2 k + kZero of the diagonals at word w: kw0 + 4 w in each half, below
      // 2^16, so plain adds carry nothing
      const uint32_t kw0 = (uint32_t)((int)kZero + 2 * kbase) + ((uint32_t)((int)kZero + 2 * kbase + 2) << 16);
      PackedSteps<kModel, kDeep> steps;
      steps.begin(a.pen, tab_m, (rows - 1) * RB);
      PackedRows r{};
      // With a bound: a path on diagonal k at score s still pays at least one
      // gap extension per diagonal to n - m, so only diagonals within
      // (ub - s) / e of it can lie on a path that costs at most ub, and no
      // other cell can be a source of one that does.
      const int gem = a.pen.min_ge();
      int reach = kBound ? ub / gem : INT_MAX / 4;
      int reach_at = kBound ? ub - reach * gem + 1 : 0;  // next score that loses one
      // the score's diagonals, words, history chunks
      int lo = max(lo0, -m), hi = min(hi0, n);
      int wlo = (lo - kbase) >> 1, whi = (hi - kbase) >> 1;
      int hc0 = wlo >> kCS, chunks = (whi >> kCS) - hc0 + 1;
      auto run = [&](auto ends_tag) {
        constexpr bool kEnds = decltype(ends_tag)::value;
        while (s_end < 0) {
          ++s;
          bool moved = steps.next(a.pen, s, &r);
          if constexpr (kBound) {
            if (s >= reach_at) {
              --reach;
              reach_at += gem;
              moved = true;
            }
          }
          if (moved) {
            const int g = steps.gained();
            lo = max(lo0 - g, -m);
            hi = min(hi0 + g, n);
            if constexpr (kBound) {
              lo = max(lo, k_end - reach);
              hi = min(hi, k_end + reach);
            }
            if (lo < kbase || hi - kbase >= W) {
              st = kPairScratch;  // wider than the ring's window
              break;
            }
            wlo = (lo - kbase) >> 1;
            whi = (hi - kbase) >> 1;
            hc0 = wlo >> kCS;
            chunks = (whi >> kCS) - hc0 + 1;
          }
          if (s > s_lim) {
            st = s > s_max ? kPairInternal : kPairScratch;
            break;
          }
          // no wavefront, or (inside a gap opening near the bound) no diagonal
          // that a path can use
          if (!steps.present(a.pen, &r) || (kBound && lo > hi)) {
            --n_steps;
            continue;
          }
          uint8_t* hrow = nullptr;
          if constexpr (kCigar) {
            if (hbase + chunks > hist_cap) {
              st = kPairScratch;
              break;
            }
            if (gt == 0) table[s] = make_int2(hc0, hbase);
            hrow = reinterpret_cast<uint8_t*>(hist + (hbase - hc0));
            hbase += chunks;
          }
          fk = INT_MAX;
          // Every lane runs every iteration: lanes past the last word compute
          // it again and store the same values to the same places.
          auto words = [&](auto count, int w0) {
            constexpr int U = decltype(count)::value;
            int w[U];
            smem_t at[U];
            uint32_t k2[U], om[U], valid[U], ext[U], f[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
              w[u] = min(w0 + u * GT + lane, whi);
              at[u] = ring0 + 4 * w[u];
              k2[u] = kw0 + (uint32_t)w[u] * 0x00040004u;
            }
            packed_words_step<kModel, kCigar, kZero, U>(r, pp, at, k2, om, valid, ext, f);
#pragma unroll
            for (int u = 0; u < U; ++u) {
              if (w0 + u * GT + lane <= whi) n_ext2 = h2_sum(ext[u], n_ext2);
              if constexpr (kEnds) {
                const int k = kbase + 2 * w[u];
                if ((valid[u] & 1u) && k >= lo && ends_at((int)((om[u] & 0xffffu) - kZero) >> 1, k)) fk = min(fk, k);
                if ((valid[u] >> 31) && k < hi && ends_at((int)((om[u] >> 16) - kZero) >> 1, k + 1)) fk = min(fk, k + 1);
              }
              if constexpr (kCigar) {
                if constexpr (kDual)
                  reinterpret_cast<uint16_t*>(hrow)[w[u]] = (uint16_t)(f[u] | (f[u] >> 8));
                else
                  hrow[w[u]] = (uint8_t)(f[u] | (f[u] >> 12));
              }
            }
          };
          int w0 = wlo + 32 * wig;
          if constexpr (kBound) {
            for (; w0 + GT <= whi; w0 += 2 * GT) words(std::integral_constant<int, 2>{}, w0);
            if (w0 <= whi) words(std::integral_constant<int, 1>{}, w0);
          } else {
            for (; w0 <= whi; w0 += GT) words(std::integral_constant<int, 1>{}, w0);
          }
          n_cells += (unsigned)(hi - lo + 1);
          ended(fk, r.w_m, kEnds);
        }
      };
      if constexpr (kBound) {
        run(std::false_type{});
      } else {
        if (ends_free)
          run(std::true_type{});
        else
          run(std::false_type{});
      }
      n_steps += (uint32_t)s + (st == kPairOk ? 1u : 0u);

      if (st == kPairOk) {
        if (gt == 0) a.score[pair] = s_end * a.g;
        if constexpr (kCigar) {
          if (wig == 0) {
            // reserve the run bound 2*s/min_pen + 4 in the arena, then walk
            const int64_t bound = 2 * (int64_t)(s_end / a.pen.min_pen()) + 4;  // + a free gap at each end
            unsigned long long at = 0;
            if (lane == 0) at = atomicAdd(a.arena_cursor, (unsigned long long)bound);
            at = __shfl_sync(FULL, at, 0);
            int len = 0;
            if ((int64_t)at + bound > a.arena_cap) {
              st = kPairArena;
            } else {
              __syncwarp();
              len = packed_cigar<kModel>(
                  hist, hbase, table, s_end, k_fin, m, n, a.pen, kbase, lo0, hi0,
                  [&](int v, int h, int rem) { return warp_lcp(pws, v, tws, h, rem, lane); }, a.arena + at, (int)bound, lane);
              if (len < 0) {
                st = kPairInternal;
                len = 0;
              }
            }
            if (lane == 0) {
              a.cig_pos[pair] = (int64_t)at;
              a.cig_len[pair] = len;
            }
          }
        }
      }
    }
    if (a.work) {
      const unsigned we = __reduce_add_sync(FULL, n_ext2 >> 1);
      if (lane == 0 && we) atomicAdd(a.work + 2, (unsigned long long)we);
    }
    if (gt == 0) {
      a.status[pair] = st;
      if (st == kPairScratch || st == kPairArena) {
        const unsigned r = atomicAdd(a.retry_count, 1u);
        a.retry[r] = (int32_t)pair;
      }
      if (a.work) {
        atomicAdd(a.work, n_cells);
        atomicAdd(a.work + 1, (unsigned long long)n_steps);
      }
    }
    group_sync<GW>(gid);  // the group's shared memory is free for the next pair
  }
}

// Upper bounds of the scores of n_order pairs (order), end to end: the
// wavefronts of each pair inside a window of kProbeW diagonals that follows
// the furthest anti-diagonal, one warp per pair.  Whatever the window holds
// are cells of real alignments, so the score that reaches the end is the cost
// of one; it is the optimum unless the best path leaves the window.  bound:
// that score, or kNoBound (no end found within the score bound, bytes outside
// ACGT, sides beyond kPackedMaxLen or seq_cap).  Two words per lane and score
// whatever the pair: a latency chain of about 0.3 us per score, 1/20 of the
// work of the full wavefronts of a 10 kbp pair at 15 %, for which it halves
// the cells (see align_packed).
template <int kModel, bool kDeep>
__device__ __forceinline__ void probe_packed(const ProbeArgs& a, unsigned char* smem_raw) {
  constexpr unsigned FULL = 0xffffffffu;
  constexpr uint32_t kZero = kZeroBound;
  constexpr int W = kProbeW;
  constexpr int RB = packed_row_words(W) * 4;
  const int lane = threadIdx.x & 31;
  const int rows = a.pen.slots() + 1;
  const smem_t head = smem_addr(smem_raw) + (size_t)(threadIdx.x >> 5) * probe_smem_bytes(a.pen, a.seq_cap);
  const smem_t tables = head;
  const smem_t ring = head + 16 * (a.pen.rm + a.pen.re + a.pen.re2);
  const smem_t ring0 = ring + 8;
  const smem_t pws = ring + rows * RB;
  packed_tables<kModel == kModelDual>(a.pen, RB, tables, lane, 32);
  for (;;) {
    unsigned qi = 0;
    if (lane == 0) qi = atomicAdd(a.queue, 1u);
    qi = __shfl_sync(FULL, qi, 0);
    if ((int64_t)qi >= a.n_order) break;
    const int64_t pair = a.order[qi];
    const int m = a.seq.pat_len[pair], n = a.seq.txt_len[pair];
    const bool bytemode = a.pk.nonacgt[pair] | a.pk.nonacgt[a.seq.n + pair];
    const int pwn = 2 * (int)packed_words(m), twn = 2 * (int)packed_words(n);
    const int k_end = n - m;
    int found = kNoBound;
    if (!bytemode && m <= kPackedMaxLen && n <= kPackedMaxLen && pwn + twn <= a.seq_cap && k_end >= -(int)(kZero / 2)) {
      const uint32_t* gpw = reinterpret_cast<const uint32_t*>(a.pk.words + a.pk.woff[pair]);
      const uint32_t* gtw = reinterpret_cast<const uint32_t*>(a.pk.words + a.pk.woff[a.seq.n + pair]);
      const smem_t tws = pws + 4 * pwn;
      for (int i = lane; i < pwn; i += 32) sts32(pws + 4 * i, __ldg(gpw + i));
      for (int i = lane; i < twn; i += 32) sts32(tws + 4 * i, __ldg(gtw + i));
      for (int i = 16 * lane; i < rows * RB; i += 16 * 32) sts128(ring + i, 0, 0, 0, 0);
      __syncwarp();
      int kbase = -W / 2;
      {
        const int l = warp_lcp(pws, 0, tws, 0, min(m, n), lane);
        if (lane == 0) sts16(ring0 + 2 * -kbase, 2 * (uint32_t)l + kZero);
        if (l >= n && k_end == 0) found = 0;
        __syncwarp();
      }
      const int64_t sb = score_bound(m, n, a.pen);
      const int s_max = (int)(sb < INT_MAX - 1 ? sb : INT_MAX - 1);
      const PackedPair pp{pws, tws, h2_dup(2 * (uint32_t)m), h2_dup((uint32_t)((int)kZero + 2 * k_end))};
      const uint32_t end_val = 2 * (uint32_t)n + kZero;
      PackedSteps<kModel, kDeep> steps;
      steps.begin(a.pen, tables, (rows - 1) * RB);
      PackedRows r{};
      for (int s = 1; s <= s_max && found == kNoBound; ++s) {
        steps.next(a.pen, s, &r);
        if (!steps.present(a.pen, &r)) continue;
        const int g = steps.gained();
        const int lo = max(max(-g, -m), kbase), hi = min(min(g, n), kbase + W - 1);
        if (lo > hi) break;  // the window left the wavefronts
        const int wlo = (lo - kbase) >> 1, whi = (hi - kbase) >> 1;
        const uint32_t kw0 = (uint32_t)((int)kZero + 2 * kbase) + ((uint32_t)((int)kZero + 2 * kbase + 2) << 16);
        uint32_t far = 0;  // the furthest anti-diagonal of this lane's cells, and its position
        const bool look = (s & 15) == 0;
        for (int w0 = wlo; w0 <= whi; w0 += 64) {
          const int w[2] = {min(w0 + lane, whi), min(w0 + 32 + lane, whi)};
          const smem_t at[2] = {ring0 + 4 * w[0], ring0 + 4 * w[1]};
          const uint32_t k2[2] = {kw0 + (uint32_t)w[0] * 0x00040004u, kw0 + (uint32_t)w[1] * 0x00040004u};
          uint32_t om[2], valid[2], ext[2], f[2];
          packed_words_step<kModel, false, kZero, 2>(r, pp, at, k2, om, valid, ext, f);
          if (look) {
            // 2 h - k, positive from 1 << 16 on
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              const int k = kbase + 2 * w[u];
              const uint32_t f0 = (valid[u] & 1u) ? (uint32_t)((int)(om[u] & 0xffffu) - k + (1 << 16)) : 0u;
              const uint32_t f1 = (valid[u] >> 31) ? (uint32_t)((int)(om[u] >> 16) - k - 1 + (1 << 16)) : 0u;
              far = max(far, max(f0 * 128u + (uint32_t)(2 * w[u]), f1 * 128u + (uint32_t)(2 * w[u] + 1)));
            }
          }
        }
        __syncwarp();
        const int pend = k_end - kbase;
        if (pend >= 0 && pend < W && lds16(ring0 + 2 * pend + r.w_m) >= end_val) found = s;
        if (look) {
          far = (uint32_t)__reduce_max_sync(FULL, (int)far);
          const int off = (int)(far & 127u) - W / 2;
          // Off the middle by more than a quarter: move every row's cells, by
          // whole words, and the window with them.
          if (far >= 128u && (off > W / 4 || off < -W / 4)) {
            int words = off / 2;
            words = max(words, (-(int)(kZero / 2) - kbase + 1) / 2);
            for (int row = 0; row < rows - 1; ++row) {
              const smem_t at = ring0 + row * RB;
              uint32_t v[W / 64];
              for (int i = 0; i < W / 64; ++i) {
                const int from = lane + 32 * i + words;
                v[i] = from >= 0 && from < W / 2 ? lds32(at + 4 * from) : 0u;
              }
              __syncwarp();
              for (int i = 0; i < W / 64; ++i) sts32(at + 4 * (lane + 32 * i), v[i]);
            }
            __syncwarp();
            kbase += 2 * words;
          }
        }
      }
    }
    if (lane == 0) a.bound[pair] = found;
    __syncwarp();
  }
}

}  // namespace tsu
