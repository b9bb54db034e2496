// tsu_plan.h -- pass geometry of the align kernel (host only, no CUDA).
//
// Shared by the engine (tsu_engine.cu), the no-allocation entry point
// (tsu_noalloc.cu) and the CPU warp emulation used by the tests, so all run
// the kernel with the same group size, ring width, staging size and scratch
// capacities.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstdint>

#include "tsu_common.cuh"
#include "tsu_tuning.h"
#include "tsu_tuning_dual.h"

namespace tsu {

// A rung of the pass ladder: ring mode and warps per pair; single: on the
// shared ring, the kernel of one diagonal per thread whatever the pairs
// (shared_single).
struct PassChoice {
  int mode, gw;
  bool single = false;
};

struct PassGeom {
  int mode = kModeShared;
  int gw = 1;              // warps per pair
  int cta_threads = 128;   // threads per block
  int groups_per_cta = 4;  // pairs in flight per block
  int ring_w = 0;          // diagonals per ring slot
  int seq_cap = 0;         // staged sequence words per group (shared mode)
  int64_t hist_cap = 0;    // backtrace words per group
  int table_cap = 0;       // step-table entries per group
  int group_smem = 0;      // dynamic shared memory per group (bytes)
  int64_t ring_ints = 0;   // global ring int32 per group (global mode)
  int ckpt_k = 0;          // low-memory mode: checkpoint interval (0: off)
  int ckpt_cap = 0;        // checkpoints per group
  int64_t ckpt_bytes = 0;  // bytes per checkpoint
  bool single = false;     // shared ring, one diagonal per thread (shared_single)
  bool bounded = false;    // pairs with score bounds (plan_bounded, plan_wide)
  int wide_cell = 0;       // of these, the wide kernel's: bytes of a ring cell (2 or 4)
  int cluster = 1;         // blocks per pair (wide kernel)
};

constexpr int kSharedW1 = 384;         // shared-mode ring width for one warp per pair (diagonals)
constexpr int kSharedSeqWords1 = 544;  // staging area for one warp per pair (uint32 words)
constexpr int kSharedSeqWordsN = 4096; // staging area for a group of warps
constexpr int kSharedMaxLen = 32000;   // int16 ring limit
// A launch of the packed kernel takes pairs up to the end of their length
// band; the few beyond kPackedPlainLen are handed back one by one.
constexpr int kPackedBandLen = 16383;
// widest int16 ring of one diagonal per thread: a negative (invalid) I value
// grows by one per diagonal of the ring's width and must stay negative (the
// kernel's store clamp); the packed kernel's: kPackedMaxW
constexpr int kSharedMaxW = 16368;
constexpr int kSmemPerSM = 228 * 1024; // B200 shared memory per SM (bytes)

// Reduced-unit score expected at edit rate `hint` for a pair of length L.
inline int64_t hint_score(const Pen& pen, int64_t L, double hint) {
  return (int64_t)(hint * (double)L * (double)pen.max_pen()) + 16;
}

inline int cta_threads_for(int gw) { return gw <= 4 ? 128 : 32 * gw; }
inline int min_blocks_for(int mode, int gw) {
  return mode == kModeShared ? (gw <= 4 ? 6 : (gw == 8 ? 3 : 1)) : (gw <= 4 ? 4 : (gw == 8 ? 2 : 1));
}

// Whether a shared-ring launch over sides of up to maxlen runs the kernel of
// one diagonal per thread: rings deeper than the packed kernel's record of
// scores, and sides past its offsets.  (One warp stages at most 8,700 bases of
// both sides and hands longer pairs back either way: packed.)  Scores alone of
// the deepest rings go to the global ring instead, which holds more pairs (5,000
// pairs of 1 kbp at 1 and 5 %, penalties 5/200/4, shared against global: with
// CIGARs 50 and 234 ms, 97 and 922; scores 37 and 189, 12 and 93).  Depths of 65
// - 128 in the packed kernel, with bounds, against this one: 20,000 x 1 kbp,
// 5/60/4, 7.8 and 47 ms, 21 and 341; scores 7.1 and 38, 14 and 285.
inline bool shared_single(const Pen& pen, int64_t maxlen, int gw) {
  return !packed_fits(pen) || (gw > 1 && maxlen > kPackedBandLen);
}

// Ring width a shared-mode group of gw warps can hold with seq_cap staged
// words, at the block count the kernel is compiled for (packed: two diagonals
// per thread).
inline int shared_ring_width(const Pen& pen, int gw, int seq_cap, int smem_optin, bool packed) {
  const int ns = pen.slots();
  const int blocks = min_blocks_for(kModeShared, gw);
  const int per_cta = std::min(smem_optin, kSmemPerSM / blocks - 1024);
  const int gpc = cta_threads_for(gw) / (32 * gw);
  const int per_group = per_cta / gpc;
  const int fixed = group_smem_bytes(pen, 0, kModeShared, seq_cap, gw, packed) + 16;
  const int w = std::min((per_group - fixed) / (2 * (packed ? ns + 1 : ns)), packed ? kPackedMaxW : kSharedMaxW);
  return std::max(0, w & ~15);
}

// Shared ring width of a group of gw warps.  One warp per pair has a fixed
// width (kSharedW1), unless penalties with a very deep ring leave four such
// groups unable to fit one block; then the width one block can hold (below
// 64 diagonals the pass takes the global ring).
inline int shared_cap(const Pen& pen, int gw, int seq_cap, int smem_optin, bool packed) {
  if (gw != 1) return shared_ring_width(pen, gw, seq_cap, smem_optin, packed);
  const int gpc = cta_threads_for(1) / 32;
  if (gpc * group_smem_bytes(pen, kSharedW1, kModeShared, seq_cap, 1, packed) <= smem_optin) return kSharedW1;
  const int w = (smem_optin / gpc - group_smem_bytes(pen, 0, kModeShared, seq_cap, 1, packed) - 16) /
                (2 * (pen.slots() + (packed ? 1 : 0)));
  return std::max(0, w & ~15);
}

// mode/gw: the configuration of this pass.  Shared mode needs lengths within
// the int16 ring; otherwise the pass falls back to the global ring.
// low_mem (CIGAR passes): 0 off; > 0 checkpoint every low_mem scores; < 0
// an interval chosen here.  single: PassChoice::single.
inline PassGeom plan_geometry(const Pen& pen, int32_t max_m, int32_t max_n, int mode, int gw, double hint,
                              bool want_cigar, int smem_optin, int low_mem = 0, bool single = false) {
  PassGeom p;
  const bool lowmem = want_cigar && low_mem != 0;
  const int ns = pen.slots();
  const int ge = pen.min_ge();
  const int64_t maxlen = std::max(max_m, max_n);
  const int64_t s_hint = hint_score(pen, maxlen, hint);
  const int64_t full_w = (int64_t)max_m + max_n + 3;
  const int64_t width_hint = std::min<int64_t>(full_w, 2 * s_hint / ge + 3);
  p.gw = gw;
  p.cta_threads = cta_threads_for(gw);
  p.groups_per_cta = p.cta_threads / (32 * gw);
  const bool fits = maxlen <= kSharedMaxLen && (want_cigar || packed_fits(pen));
  p.mode = mode == kModeShared && fits ? kModeShared : kModeGlobal;
  p.single = p.mode == kModeShared && !lowmem && (single || shared_single(pen, maxlen, gw));
  const bool packed = p.mode == kModeShared && !lowmem && !p.single;
  if (p.mode == kModeShared) {
    const int64_t seqw = 2 * packed_words(max_m) + 2 * packed_words(max_n);
    p.seq_cap = (int)std::min<int64_t>(seqw, gw == 1 ? kSharedSeqWords1 : kSharedSeqWordsN);
    const int cap = shared_cap(pen, gw, p.seq_cap, smem_optin, packed);
    p.ring_w = (int)std::max<int64_t>(16, (std::min<int64_t>(full_w, cap) + 15) & ~15);
    if (cap < 64) p.mode = kModeGlobal, p.single = false;
  }
  if (p.mode == kModeGlobal) {
    p.ring_w = (int)full_w;
    // the pair's packed words staged in shared memory when
    // they fit beside the group's limits at the block count the kernel is
    // compiled for (0: read from global memory; always for 32-warp groups)
    const int64_t seqw = 2 * packed_words(max_m) + 2 * packed_words(max_n);
    const int per_cta = std::min(smem_optin, kSmemPerSM / min_blocks_for(kModeGlobal, gw) - 1024);
    const int gpc = cta_threads_for(gw) / (32 * gw);
    const int64_t room = per_cta / gpc - group_smem_bytes(pen, 0, kModeGlobal, 0, gw, false) - 48;
    p.seq_cap = (gw < 32 && seqw * 4 <= room) ? (int)seqw : 0;
  }
  p.group_smem = group_smem_bytes(pen, p.ring_w, p.mode, p.seq_cap, gw, packed);
  // Backtrace words up to score s: sum_j (2j/ge + 1) ~= s^2/ge + 2s.
  p.table_cap = want_cigar ? (int)std::min<int64_t>(s_hint + 1, INT32_MAX / 2) : 0;
  if (want_cigar) {
    const int64_t sq = s_hint * s_hint / ge + 2 * s_hint + 64;
    int64_t cells = std::min<int64_t>(sq, (s_hint + 1) * width_hint);
    // the packed kernel keeps 4 bits per cell (8 with two gap pieces), each
    // score's row rounded out to whole words at both ends
    if (packed && p.mode == kModeShared) cells = std::min<int64_t>(cells / (pen.dual() ? 4 : 8) + 3 * (s_hint + 1) + 64, INT32_MAX - 65536);
    p.hist_cap = std::min<int64_t>(cells, INT32_MAX - 64);
  }
  p.ring_ints = p.mode == kModeShared ? 0 : (int64_t)ns * p.ring_w;
  if (lowmem) {
    // The checkpoints of a pair (s_hint / K + 2 of ckpt_bytes) plus one
    // segment of history (K + 1 rows of at most width_hint words): K near
    // sqrt(s_hint * ckpt_bytes / (4 width_hint)) balances the two.  K is at
    // least the ring depth, so a backtrace step crosses one segment at most.
    p.ckpt_bytes = ckpt_bytes_for(pen, p.ring_w, p.mode);
    int64_t K = low_mem;
    if (K < 0) {
      const double k = std::sqrt((double)s_hint * (double)p.ckpt_bytes / (4.0 * (double)std::max<int64_t>(width_hint, 1)));
      K = (int64_t)k;
    }
    K = std::max<int64_t>(std::min<int64_t>(K, std::max<int64_t>(s_hint, 1)), pen.rm);
    p.ckpt_k = (int)K;
    p.ckpt_cap = (int)std::min<int64_t>(s_hint / K + 2, INT32_MAX / 2);
    p.hist_cap = std::min<int64_t>(p.hist_cap, (K + 1) * width_hint + 64);
  }
  return p;
}

// Retry ladder: the configuration of the pass after `prev` for n_pairs pairs
// of at most max_m x max_n that outgrew it.  The smallest group whose shared
// ring holds the widest possible wavefront (m + n + 3 diagonals, so it cannot
// overflow), else the largest shared group, then the global ring with
// global_gw (16) warps per pair (the pairs that reach it are the longest and
// most divergent ones; their count in flight is bounded by memory, not by
// warps).
// lowmem: low-memory passes, whose shared ring takes all sides up to
// kSharedMaxLen itself.
inline PassChoice next_pass(PassChoice prev, const Pen& pen, int32_t max_m, int32_t max_n, int smem_optin,
                            int global_gw = 16, bool lowmem = false) {
  const int64_t need_w = (int64_t)max_m + max_n + 3;
  const int64_t maxlen = std::max(max_m, max_n);
  if (prev.mode == kModeShared && maxlen <= kSharedMaxLen) {
    // sides past the packed kernel's offsets, handed back by it: the kernel of
    // one diagonal per thread, from the same warps on
    const bool single = !lowmem && (prev.single || maxlen > kPackedPlainLen);
    const bool again = single && !prev.single && !shared_single(pen, maxlen, prev.gw);
    const int least = again ? prev.gw : prev.gw + 1;
    const bool packed = !lowmem && !single && packed_fits(pen);
    const int64_t seqw =
        std::min<int64_t>(2 * packed_words(max_m) + 2 * packed_words(max_n), kSharedSeqWordsN);
    static const int kGW[] = {2, 4, 8, 16};
    for (int gw : kGW) {
      if (gw < least) continue;
      if (shared_ring_width(pen, gw, (int)seqw, smem_optin, packed) >= need_w) return {kModeShared, gw, single};
    }
    if (least <= 16) return {kModeShared, 16, single};
  }
  return {kModeGlobal, global_gw};
}

// The first rung at or above pc whose ring holds the wavefront width the
// hint predicts for pairs of at most max_m x max_n (2 s_hint / e + 3
// diagonals, at most m + n + 3): pc itself, a larger shared group, or the
// global ring with 8 or more warps.  Used when the hint is a per-pair
// estimate, so a pair that is bound to outgrow the shared ring does not
// start there; a wavefront wider than 16,384 diagonals gets 32 warps.
inline PassChoice fit_start(PassChoice pc, const Pen& pen, int32_t max_m, int32_t max_n, double hint,
                            int smem_optin) {
  const int64_t maxlen = std::max(max_m, max_n);
  const int64_t w =
      std::min<int64_t>((int64_t)max_m + max_n + 3, 2 * hint_score(pen, maxlen, hint) / pen.min_ge() + 3);
  if (pc.mode != kModeShared) return {kModeGlobal, w > 16384 ? 32 : pc.gw};
  if (maxlen > kSharedMaxLen) return {kModeGlobal, w > 16384 ? 32 : std::max(8, pc.gw)};
  const int64_t seqw = 2 * packed_words(max_m) + 2 * packed_words(max_n);
  static const int kGW[] = {1, 2, 4, 8, 16};
  for (int gw : kGW) {
    if (gw < pc.gw) continue;
    if (seqw > (gw == 1 ? kSharedSeqWords1 : kSharedSeqWordsN)) continue;
    const int cap = shared_cap(pen, gw, (int)seqw, smem_optin, !shared_single(pen, maxlen, gw));
    if (cap >= w && cap >= 64) return {kModeShared, gw};
  }
  // wavefronts wider than 16,384 diagonals: 32 warps (one 1024-thread block)
  return {kModeGlobal, w > 16384 ? 32 : std::max(8, pc.gw)};
}

// Length bands of the batched scheduler: max(m, n) < 1024, < 2048, < 4096,
// < 8192, < 16384, >= 16384.  Each band starts its ladder at the rung the
// autotuner measured fastest for it (tsu_tuning.h; the dual gap-affine
// kernels, with their deeper and wider rings: tsu_tuning_dual.h).
constexpr int kBands = 6;
inline int length_band(int32_t L) {
  if (L < 1024) return 0;
  if (L < 2048) return 1;
  if (L < 4096) return 2;
  if (L < 8192) return 3;
  if (L < 16384) return 4;
  return 5;
}
// The starting rung of each band in a table (a context's copy of the
// compiled one), adjusted for lengths beyond the int16 shared ring.
inline PassChoice band_start_in(const PassChoice* table, int band, int32_t maxlen) {
  PassChoice r = table[band < 0 ? 0 : (band >= kBands ? kBands - 1 : band)];
  if (r.mode == kModeShared && maxlen > kSharedMaxLen) r = {kModeGlobal, r.gw >= 8 ? r.gw : 8};
  return r;
}
inline const PassChoice* band_start_table(bool dual = false) {
  static const PassChoice kStart[kBands] = TSU_BAND_START;
  static const PassChoice kStartDual[kBands] = TSU_BAND_START_DUAL;
  return dual ? kStartDual : kStart;
}

// Edit-rate hint of the next retry pass.  Shared-ring passes keep the hint
// (they fail on ring width, staging or history); from the second global pass
// on it grows 4x up to kHintCeiling, at which the step table and the history
// cover the score bound of every pair (s_max <= max_pen * maxlen < s_hint,
// max_pen the dearest single-base edit), so a pass there can fail only on
// memory.
constexpr double kHintCeiling = 2.0;
inline double next_hint(double hint, bool grow) { return grow ? std::min(hint * 4.0, kHintCeiling) : hint; }

// CIGAR arena runs for a batch: 2*s/(cheapest edit) + 1 per pair at the hint.
inline int64_t arena_runs(const Pen& pen, int64_t n, int32_t max_m, int32_t max_n, double hint) {
  const int64_t maxlen = std::max(max_m, max_n);
  const int64_t per_pair = 2 * hint_score(pen, maxlen, hint) / pen.min_pen() + 1;
  return std::max<int64_t>(n * (std::min<int64_t>(per_pair, (int64_t)max_m + max_n + 1) + 3), 1024);
}

// ---- passes of pairs whose score bound is known ----------------------------

// Whether a pair of a large batch is worth a bound probe, by the width its full
// wavefronts are expected to reach at 4 % edits: 420 diagonals and 1,024 bases
// (gap-affine 4/6/2: from 1.2 kbp; edit distance: 4.9 kbp), 224 where the ring
// of one warp (kSharedW1 diagonals) takes over 14 KB, so that an SM holds few of
// them (two gap pieces 4/6/2/24/1: from 300 bp).  A probe computes 128
// diagonals and the bookkeeping of every score once more, so it saves nothing
// where the wavefronts are about that wide, and costs accurate pairs most.
// Probed / not, ms a scored call on one B200 at 0.5, 2, 5 and 15 %:
//   two pieces   20,000 x 100 bp  0.93 / 0.43  0.95 / 0.51  1.41 / 1.05  2.15 / 2.73
//                20,000 x 200 bp  0.96 / 0.45  1.33 / 0.96  1.87 / 2.23
//                20,000 x 300 bp  0.98 / 0.56  1.63 / 1.61  2.42 / 3.22
//                20,000 x 500 bp  1.24 / 0.92  2.01 / 2.52  3.34 / 5.16
//   affine 3/5/1  6,000 x 1 kbp   0.54 / 0.21  0.83 / 0.38  1.50 / 2.13
//   affine 4/6/2  2,000 x 1.5 kbp 0.31 / 0.17  0.47 / 0.26  0.68 / 0.53
//                   600 x 1.5 kbp 0.23 / 0.14  0.32 / 0.18  0.48 / 0.30  1.48 / 1.94
//                 6,000 x 2.5 kbp 0.68 / 0.54  1.20 / 1.17
//                 6,000 x 5 kbp   0.97 / 1.20  2.28 / 3.24
// Pairs below the line that outgrow their ring get a bound then.
constexpr int kBoundMinWidth = 420, kBoundMinWidthDeep = 224;
constexpr int kBoundMinRing = 14 << 10, kBoundMinLen = 1024;
struct BoundLimits {
  int32_t side = INT32_MAX;      // the longer side from which a pair of a large batch is probed
  int32_t few_side = INT32_MAX;  // the longer side from which few pairs get a bound (below)
  bool wants(int32_t m, int32_t n) const { return std::min(m, n) > 0 && std::max(m, n) >= side; }
};
// With no more such pairs than SMs each has an SM to itself, and a probe (0.35
// us per score on one warp) costs more than the narrower search saves until a
// pair outgrows the widest shared ring (148 x 8 kbp at 10 %: 3.1 ms either
// way; 100 of 12 kbp at 1 %: 0.53 ms without, 0.88 with): they start in that
// ring, and those that outgrow it get a bound when their full wavefronts at
// 16 % edits do not fit it anyway (few_side; gap-affine 4/6/2: from 8.2 kbp;
// 4/6/2/24/1, whose 37 rows leave 2,900 diagonals: from 1.1 kbp).  Only sides
// beyond that ring's offsets (kPackedBandLen) are probed at once.
inline BoundLimits bound_limits(const Pen& pen, int smem_optin) {
  BoundLimits b;
  // the shortest side whose expected width at `rate` edits reaches `width`
  auto from = [&](int64_t width, double rate) -> int32_t {
    int32_t lo = 0, hi = 1 << 27;
    while (lo < hi) {
      const int32_t L = lo + (hi - lo) / 2;
      if (2 * hint_score(pen, L, rate) / pen.min_ge() >= width)
        hi = L;
      else
        lo = L + 1;
    }
    return lo;
  };
  const bool deep = 2 * ((int64_t)pen.slots() + 1) * kSharedW1 > kBoundMinRing;
  b.side = deep ? from(kBoundMinWidthDeep, 0.04) : std::max(from(kBoundMinWidth, 0.04), kBoundMinLen);
  b.few_side = from(std::max(shared_ring_width(pen, 16, kSharedSeqWordsN, smem_optin, true), 64), 0.163);
  return b;
}

// What a pair of score bound ub needs: diagonals of the ring's window,
// 32-bit sequence words, and 32-bit history words (each side of the band grows
// to its crossing and shrinks again, one diagonal per gap extension; three
// words of rounding per score).
struct BoundNeed {
  int width = 0, words = 0;
  int64_t hist = 0;
};
inline BoundNeed bound_need(const Pen& pen, int32_t m, int32_t n, int32_t ub) {
  BoundNeed b;
  int lo, hi;
  bound_reach(pen, m, n, ub, &lo, &hi);
  b.width = hi - lo + 1;
  b.words = (int)(2 * packed_words(m) + 2 * packed_words(n));
  const int64_t h = hi, l = -(int64_t)lo, e = pen.min_ge();
  const int64_t cells = std::min<int64_t>(e * (h * h + l * l) + (int64_t)ub + 1, (int64_t)(b.width + 1) * ((int64_t)ub + 1));
  b.hist = cells / (pen.dual() ? 4 : 8) + 3 * ((int64_t)ub + 1) + 64;
  return b;
}

// Geometry of a launch of bounded pairs: bytes of shared memory per group
// (bounded_bytes of the pair that needs most at these warps), history and
// step table as their bounds say.
inline PassGeom plan_bounded(int bytes, int32_t max_ub, int64_t hist, int gw, bool want_cigar) {
  PassGeom p;
  p.mode = kModeShared;
  p.bounded = true;
  p.gw = gw;
  p.cta_threads = cta_threads_for(gw);
  p.groups_per_cta = p.cta_threads / (32 * gw);
  p.group_smem = bytes;
  if (want_cigar) {
    p.table_cap = max_ub + 2;
    p.hist_cap = std::min<int64_t>(hist, INT32_MAX - 65536);
  }
  return p;
}

// Classes of bounded pairs, one launch each: by how many of their kind an SM's
// shared memory holds (1, 2-3, 4-7, ... 64 and more: class 0 to 6).  Pairs of
// one class run at its widest member's ring, which costs none of them a place
// beyond the class; classes by width alone cut 10 kbp pairs at 4,096 diagonals
// and ran the last 13 of 309 as a wave of their own.
constexpr int kBoundClasses = 7;
inline int bound_class(int pairs_per_sm) {
  int c = 0;
  while (c < kBoundClasses - 1 && pairs_per_sm >= 2 << c) ++c;
  return c;
}

// Warps per pair of a bounded launch of n pairs whose shared memory is
// `bytes`: the fewest that keep 16 warps on an SM with the pairs it holds, and
// as many as fill 8 per SM when there are few pairs.  A step costs every warp
// of a group the same bookkeeping, so fewer warps do less work; below 16 they
// no longer cover the latency of a step (1,000 x 10 kbp at 15 % and 8,000
// uneven pairs, align ms, with at least 8: 31.5 and 42.1, 12: 27.0 and 38.3,
// 16: 27.1 and 38.5, 20: 38.1 and 47.1; 20,000 x 1 kbp dual gap-affine 8.7,
// 8.6, 8.5, 12.4).  0: the bytes do not fit a block.
inline int bounded_warps(int bytes, int64_t n, int sms, int smem_optin, int* pairs_per_sm = nullptr) {
  int best = 0;
  for (int gw = 1; gw <= 16; gw *= 2) {
    const int gpc = cta_threads_for(gw) / (32 * gw);
    const int64_t block = (int64_t)gpc * bytes;
    if (block > smem_optin) continue;
    const int64_t pairs = kSmemPerSM / (block + 1024) * gpc;
    best = gw;
    if (pairs_per_sm) *pairs_per_sm = (int)pairs;
    if (pairs * gw >= 16 && n * gw * 2 > (int64_t)sms * 8) break;
  }
  return best;
}

// Geometry of a launch of bounded pairs on the wide kernel: a ring of `width`
// diagonals in device memory, one block per pair.
inline PassGeom plan_wide(const Pen& pen, int32_t max_n, int width, int32_t max_ub, int64_t hist, bool want_cigar) {
  PassGeom p;
  p.mode = kModeGlobal;
  p.bounded = true;
  p.wide_cell = max_n <= kWide16MaxLen ? 2 : 4;
  p.gw = 16;
  p.cta_threads = 512;
  p.groups_per_cta = 1;
  p.group_smem = wide_smem_bytes(pen);
  p.ring_ints = (int64_t)(pen.slots() + 1) * wide_row_bytes(width, p.wide_cell) / 4;
  if (want_cigar) {
    p.table_cap = max_ub + 2;
    p.hist_cap = hist;
  }
  return p;
}
// Blocks per pair of a wide launch of n pairs (a cluster): as many as keep
// the clusters within 7 of every 8 SMs (a GPC's SMs rarely divide evenly).
inline int wide_cluster(int64_t n, int sms) {
  int c = 1;
  while (c < 8 && n * c * 2 <= (int64_t)sms * 7 / 8) c *= 2;
  return c;
}
// History a wide launch may keep (32-bit words below 2^31).  Scores alone are held
// to it too: it keeps the rows' byte offsets in the ring below 2^31.
constexpr int64_t kWideMaxHist = INT32_MAX - 65536;

// In low-memory mode (interval chosen here) every pair from this length on is
// probed: with its bound a pair's whole history, 4 bits per cell of a band
// that narrows again, takes less than the checkpoints and recomputed segment
// planned from the error hint, and is computed once.
constexpr int kBoundLowMemLen = 256;

// First launch of no more pairs than SMs whose length starts in the global
// ring: the widest shared ring instead, as far as its offsets reach; the ones
// that outgrow it get a bound.  Measured on one B200, 100 pairs each, global
// ring / probe at once / this: gap-affine 4/6/2 of 12 kbp at 1 % 0.97 / 0.88 /
// 0.53 ms, at 5 % 5.2 / 3.0 / 2.4, at 15 % 23 / 9.4 / 10.4; 4/6/2/24/1 of 1.2
// kbp at 4 % 0.83 / - / 0.39, of 2.5 kbp at 10 % 8.3 / 2.3 / 1.9, of 9 kbp at
// 1 % 8.0 / 1.2 / 0.74, at 4 % 40 / 4.1 / 5.8: noisy pairs of little more than
// the ring holds lose a part of the probe's gain, since the first ring's work is
// thrown away (100 of 16 kbp at 15 %: 181 / 13.7 / 24.6).  Bands whose rung the
// caller set keep it, here and in fill_warps, and are not probed.
inline PassChoice few_start(PassChoice pc, const Pen& pen, int32_t maxlen) {
  const PassChoice d = band_start_in(band_start_table(pen.dual()), length_band(maxlen), maxlen);
  if (pc.mode == kModeGlobal && pc.mode == d.mode && pc.gw == d.gw && maxlen <= kPackedBandLen) return {kModeShared, 16};
  return pc;
}

// Warps per pair of an unbounded shared-ring launch of n pairs: 16 when each
// pair can have an SM to itself (one pair of 1 kbp: 0.21 ms on 1 warp, 0.14 on
// 16; 148 of 8 kbp at 10 %: 3.1 ms, and 5.4 from 8 warps, whose ring they
// outgrow), else those of the rung, doubled while the launch leaves an SM
// fewer than 8 warps (600 pairs of 1 kbp: 0.22 ms on 1, 0.19 on 2, 0.26 on 4);
// at most one warp per 64 bases beyond the rung (20 pairs of 115 bp: 162 us a
// call on 1 warp, 168 on 16).  The kernel of one diagonal per thread keeps its
// rung, and so do low-memory passes, whose checkpoints are as wide as the ring.
inline PassChoice fill_warps(PassChoice pc, const Pen& pen, int64_t n, int32_t maxlen, int sms) {
  if (pc.mode != kModeShared || pc.single || shared_single(pen, maxlen, pc.gw)) return pc;
  while (pc.gw < 16 && (n <= sms || n * pc.gw * 2 <= (int64_t)sms * 8) && pc.gw * 128 <= maxlen) pc.gw *= 2;
  return pc;
}

}  // namespace tsu
