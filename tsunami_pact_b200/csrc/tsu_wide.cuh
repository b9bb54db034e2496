// tsu_wide.cuh -- bounded pairs beyond the 16-bit shared ring: sides of more
// than kPackedMaxLen bases, or a band wider than a block's shared memory.
//
// The same search as tsu_packed.cuh (score bound, ranges from the penalties and
// the bound, source bits as history, one end test per score), one diagonal per
// lane in 32-bit registers, the ring in device memory: one pair per block of
// 16 warps, rows of h + 1 (0: absent) in 16 bits for texts of up to 65,532
// bases and 32 bits for longer ones.  A block's scores are bound by issue and the
// ring's L2 traffic (five loads and three stores per cell), so 16-bit rows halve
// the time of the widest, and U = 4 cells per lane are in flight to cover its
// latency; few pairs are spread over clusters of up to 8 blocks, whose barrier
// between scores is then half of what a warp waits for (issue 35 %).
// The sequences are read through L1 (a few neighbouring words per warp).
#pragma once

#include "tsu_packed.cuh"

namespace tsu {

// Rows of one score in a ring of ST at byte offsets from base.
template <typename ST>
__device__ __forceinline__ ST* wide_row(unsigned char* base, int off) {
  return reinterpret_cast<ST*>(base + off);
}

struct WidePair {
  const uint32_t* pw;
  const uint32_t* tw;
  int m, n, kbase;
};

// I, D and M of U diagonals (positions w[u] of the window) from the source
// rows into the score's rows.  m1: M as h + 1 (0: absent); bits: source bits
// as packed_words_step's; ext: bases matched.
// kL2: read the ring past L1 (other blocks of the cluster write it).
template <bool kL2, typename ST>
__device__ __forceinline__ uint32_t wide_ld(const ST* p) {
#ifndef TSU_WARP_EMU
  if constexpr (kL2) return (uint32_t)__ldcg(p);
#endif
  return (uint32_t)*p;
}

template <int kModel, typename ST, int U, bool kL2>
__device__ __forceinline__ void wide_cells(unsigned char* base, const PackedRows& r, const WidePair& q, const int (&w)[U],
                                           uint32_t (&m1)[U], uint32_t (&bits)[U], uint32_t (&ext)[U]) {
  constexpr bool kDual = kModel == kModelDual, kLin = kModel == kModelLinear;
  const GlobalSeq P{q.pw}, T{q.tw};
  uint32_t mo_l[U], mo_r[U], mx[U], ie[U], de[U], mo2_l[U], mo2_r[U], ie2[U], de2[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    auto ld = [&](int row, int at) -> uint32_t { return wide_ld<kL2, ST>(wide_row<ST>(base, row) + at); };
    mo_l[u] = ld(r.r_mo, w[u] - 1);
    mo_r[u] = ld(r.r_mo, w[u] + 1);
    mx[u] = ld(r.r_mx, w[u]);
    if constexpr (!kLin) {
      ie[u] = ld(r.r_ie, w[u] - 1);
      de[u] = ld(r.r_de, w[u] + 1);
    }
    if constexpr (kDual) {
      mo2_l[u] = ld(r.r_mo2, w[u] - 1);
      mo2_r[u] = ld(r.r_mo2, w[u] + 1);
      ie2[u] = ld(r.r_ie2, w[u] - 1);
      de2[u] = ld(r.r_de2, w[u] + 1);
    }
  }
  // twice h + 1, bit 0 set by the side that wins ties; 0 and 1: absent
  const uint32_t cap = 2 * ((uint32_t)q.n + 2);
  auto ins_of = [&](uint32_t open, uint32_t extend, uint32_t* flag) -> uint32_t {
    const uint32_t v = max(2 * open, 2 * extend + 1);
    *flag = v & 1u;
    return v < 2 ? 0u : min((v & ~1u) + 2, cap);
  };
  uint32_t cx[U], ux[U];
  int v0[U], h0[U];
  bool valid[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    uint32_t t, fi = 0, fd = 0;
    if constexpr (!kLin) {
      const uint32_t ins = ins_of(mo_l[u], ie[u], &fi);
      const uint32_t dv = max(2 * mo_r[u], 2 * de[u] + 1);
      const uint32_t del = dv & ~1u;
      fd = dv & 1u;
      wide_row<ST>(base, r.w_i)[w[u]] = (ST)(ins >> 1);
      wide_row<ST>(base, r.w_d)[w[u]] = (ST)(del >> 1);
      if constexpr (!kDual) {
        t = max(ins, del | 1u);
        bits[u] = ((t & 1u) << 1) | (fi << 2) | (fd << 3);
      } else {
        uint32_t fi2;
        const uint32_t ins2 = ins_of(mo2_l[u], ie2[u], &fi2);
        const uint32_t dv2 = max(2 * mo2_r[u], 2 * de2[u] + 1);
        const uint32_t del2 = dv2 & ~1u;
        wide_row<ST>(base, r.w_i2)[w[u]] = (ST)(ins2 >> 1);
        wide_row<ST>(base, r.w_d2)[w[u]] = (ST)(del2 >> 1);
        const uint32_t t1 = max(ins, ins2 | 1u), t2 = max(t1 & ~1u, del | 1u);
        t = max(t2 & ~1u, del2 | 1u);
        bits[u] = ((t & 1u) << 1) | ((t2 & 1u) << 2) | ((t1 & 1u) << 3) | (fi << 4) | (fd << 5) | (fi2 << 6) |
                  ((dv2 & 1u) << 7);
      }
    } else {
      t = max(mo_l[u] ? 2 * mo_l[u] + 2 : 0u, 2 * mo_r[u] | 1u);
      bits[u] = (t & 1u) << 1;
    }
    const uint32_t p = max(t & ~1u, mx[u] ? 2 * mx[u] + 3 : 1u);
    bits[u] |= p & 1u;
    valid[u] = p >= 2;
    const int k = q.kbase + w[u];
    ux[u] = (uint32_t)max(min(q.n, q.m + k), -1) + 1u;  // last offset of the diagonal, and 1
    const uint32_t lx = (uint32_t)max(k, 0) + 1u;
    cx[u] = min(max(p >> 1, lx), ux[u]);
    h0[u] = max((int)cx[u] - 1, 0);
    v0[u] = max(h0[u] - k, 0);
  }
  uint32_t l[U];
#pragma unroll
  for (int u = 0; u < U; ++u) l[u] = (uint32_t)h2_tz(win16(P, v0[u]) ^ win16(T, h0[u])) >> 1;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const uint32_t most = ux[u] - cx[u];
    if (l[u] == 16 && most > 16 && valid[u]) l[u] = 16 + (uint32_t)lcp16(P, v0[u] + 16, T, h0[u] + 16, (int)most - 16);
    l[u] = min(l[u], most);
    ext[u] = valid[u] ? l[u] : 0u;
    m1[u] = valid[u] ? cx[u] + l[u] : 0u;
    wide_row<ST>(base, r.w_m)[w[u]] = (ST)m1[u];
  }
}

__device__ __forceinline__ int wide_warp_lcp(const WidePair& q, int v, int h, int rem, int lane) {
  const GlobalSeq P{q.pw}, T{q.tw};
  int l = 0;
  while (l < rem) {
    const int at = l + 16 * lane;
    int lx = 0;
    if (at < rem) lx = h2_tz(win16(P, v + at) ^ win16(T, h + at)) >> 1;
    const unsigned stop = __ballot_sync(0xffffffffu, lx < 16);
    if (stop) {
      const int src = __ffs((int)stop) - 1;
      return min(l + 16 * src + __shfl_sync(0xffffffffu, lx, src), rem);
    }
    l += 512;
  }
  return rem;
}

// The blocks of a cluster that share a pair.
#ifdef TSU_WARP_EMU
inline unsigned cluster_size() { return 1; }
inline unsigned cluster_rank() { return 0; }
inline void cluster_sync() {}
inline void cluster_sts32(smem_t a, unsigned, uint32_t v) { sts32(a, v); }
#else
__device__ __forceinline__ unsigned cluster_size() {
  unsigned v;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(v));
  return v;
}
__device__ __forceinline__ unsigned cluster_rank() {
  unsigned v;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(v));
  return v;
}
// Every thread of every block of the cluster; what they wrote before it
// (shared and global memory) is visible after it.
__device__ __forceinline__ void cluster_sync() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Store to the same shared memory address in block `rank` of the cluster.
__device__ __forceinline__ void cluster_sts32(smem_t a, unsigned rank, uint32_t v) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(r), "r"(v) : "memory");
}
#endif

// Scores (and CIGARs) of pairs with score bounds (a.bound), end to end, one
// block per pair, or one cluster of blocks (kCluster); a.ring_global,
// a.ring_stride (int32): the ring.  A step of a 50 kbp pair at 20 % (16,000
// cells) is 6 us of issue slots on one SM, and few pairs are that long: with a
// cluster each block computes every csize-th run of words of a score, reads
// the ring past L1, and a cluster barrier ends the score (11 pairs of 21 - 50
// kbp: 201 ms one block each, 78 ms on clusters of 8).
template <bool kCigar, int kModel, typename ST, bool kCluster, bool kDeep = true>
__device__ __forceinline__ void align_wide(const AlignArgs& a, unsigned char* smem_raw) {
  constexpr unsigned FULL = 0xffffffffu;
  constexpr int GW = 16, U = 4;
  const int csize = kCluster ? (int)cluster_size() : 1, crank = kCluster ? (int)cluster_rank() : 0;
  const int GT = 32 * GW * csize;  // threads per pair
  auto sync = [&]() {
    if constexpr (kCluster)
      cluster_sync();
    else
      group_sync<GW>(0);
  };
  // a word of every block's shared memory
  auto tell = [&](smem_t at, uint32_t v) {
    if constexpr (kCluster) {
      for (int c = 0; c < csize; ++c) cluster_sts32(at, (unsigned)c, v);
    } else {
      sts32(at, v);
    }
  };
  constexpr bool kDual = kModel == kModelDual;
  constexpr int kCS = kDual ? 1 : 2;  // log2 of pairs of diagonals per 32-bit history chunk
  const int gt = threadIdx.x + 32 * GW * crank, lane = gt & 31, wig = gt >> 5;  // in the pair's threads
  const int64_t grp = blockIdx.x / csize;
  const int rows = a.pen.slots() + 1;
  const smem_t bc = smem_addr(smem_raw);  // broadcast words: queue, end flag
  const smem_t tables = bc + packed_head_bytes(Pen(), GW);
  unsigned char* const ring = reinterpret_cast<unsigned char*>(a.ring_global + grp * a.ring_stride);
  uint32_t* const hist = kCigar ? a.hist + grp * a.hist_cap : nullptr;
  const int hist_cap = (int)a.hist_cap;
  int2* const table = kCigar ? a.table + grp * (int64_t)a.table_cap : nullptr;
  if constexpr (kCluster) cluster_sync();  // every block runs before another stores into it
  for (;;) {
    if (gt == 0) tell(bc, atomicAdd(a.queue, 1u));
    sync();
    const unsigned qi = lds32(bc);
    if ((int64_t)qi >= a.n_order) break;
    const int64_t pair = a.order[qi];
    const int m = a.seq.pat_len[pair], n = a.seq.txt_len[pair], k_end = n - m;
    const int ub = a.bound[pair];
    int st = kPairOk, s_end = -1, s = 0, hbase = 0;
    unsigned long long n_cells = 0;
    uint32_t n_steps = 0, n_ext = 0;
    int lo_b = 0, hi_b = 0;
    if (ub != kNoBound) bound_reach(a.pen, m, n, ub, &lo_b, &hi_b);
    const int kbase = lo_b;
    const int RB = wide_row_bytes(hi_b - lo_b + 1, (int)sizeof(ST));
    const bool bytemode = a.pk.nonacgt[pair] | a.pk.nonacgt[a.seq.n + pair];
    if (ub == kNoBound || bytemode || (int64_t)rows * RB > 4 * a.ring_stride ||
        (sizeof(ST) == 2 && n > kWide16MaxLen))
      st = kPairScratch;
    if (st == kPairOk) {
      const WidePair q{reinterpret_cast<const uint32_t*>(a.pk.words + a.pk.woff[pair]),
                       reinterpret_cast<const uint32_t*>(a.pk.words + a.pk.woff[a.seq.n + pair]), m, n, kbase};
      unsigned char* const ring0 = ring + 4 * sizeof(ST);  // position 0 of row 0
      packed_tables<kDual>(a.pen, RB, tables, (int)threadIdx.x, 32 * GW);
      {
        uint32_t* const z = reinterpret_cast<uint32_t*>(ring);
        const int words = rows * RB / 4;
        for (int i = gt; i < words; i += GT) z[i] = 0u;
      }
      sync();
      if (wig == 0) {
        const int l = wide_warp_lcp(q, 0, 0, min(m, n), lane);
        if (lane == 0) {
          wide_row<ST>(ring0, 0)[-kbase] = (ST)(l + 1);
          tell(bc + 4, l >= n && k_end == 0 ? 0u : 0xffffffffu);  // the score that ended, none yet
        }
      }
      sync();
      n_cells = 1;
      if (lds32(bc + 4) == 0) s_end = 0;
      const int64_t bound = score_bound(m, n, a.pen);
      const int s_max = (int)(bound < INT_MAX - 1 ? bound : INT_MAX - 1);
      const int s_lim = min(ub, kCigar ? min(s_max, a.table_cap - 1) : s_max);
      PackedSteps<kModel, kDeep> steps;
      steps.begin(a.pen, tables, (rows - 1) * RB);
      PackedRows r{};
      const int gem = a.pen.min_ge();
      int reach = ub / gem, reach_at = ub - reach * gem + 1;
      int lo = 0, hi = 0;
      const int pend = k_end - kbase;
      const uint32_t end_val = (uint32_t)n + 1u;
      while (s_end < 0) {
        ++s;
        bool moved = steps.next(a.pen, s, &r);
        if (s >= reach_at) {
          --reach;
          reach_at += gem;
          moved = true;
        }
        if (moved) {
          const int g = steps.gained();
          lo = max(max(-g, -m), k_end - reach);
          hi = min(min(g, n), k_end + reach);
          if (lo < lo_b || hi > hi_b) {
            st = kPairScratch;
            break;
          }
        }
        if (s > s_lim) {
          st = s > s_max ? kPairInternal : kPairScratch;
          break;
        }
        if (!steps.present(a.pen, &r) || lo > hi) {
          --n_steps;
          continue;
        }
        // whole pairs of diagonals, so that two lanes share a history byte
        const int wlo = (lo - kbase) & ~1, whi = (hi - kbase) | 1;
        uint8_t* hrow = nullptr;
        if constexpr (kCigar) {
          const int c0 = wlo >> (kCS + 1), chunks = (whi >> (kCS + 1)) - c0 + 1;
          if (hbase + chunks > hist_cap) {
            st = kPairScratch;
            break;
          }
          if (gt == 0) table[s] = make_int2(c0, hbase);
          hrow = reinterpret_cast<uint8_t*>(hist + (hbase - c0));
          hbase += chunks;
        }
        for (int w0 = wlo + 32 * wig; w0 <= whi; w0 += U * GT) {
          int w[U];
          uint32_t m1[U], f[U], ext[U];
#pragma unroll
          for (int u = 0; u < U; ++u) w[u] = min(w0 + u * GT + lane, whi);
          wide_cells<kModel, ST, U, kCluster>(ring0, r, q, w, m1, f, ext);
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const bool own = w0 + u * GT + lane <= whi;
            if (own) n_ext += ext[u];
            if (w[u] == pend && m1[u] >= end_val) tell(bc + 4, (uint32_t)s);
            if constexpr (kCigar) {
              if constexpr (kDual) {
                if (own) hrow[w[u]] = (uint8_t)f[u];
              } else {
                const uint32_t g = f[u] | (__shfl_xor_sync(FULL, f[u], 1) << 4);
                if (own && !(lane & 1)) hrow[w[u] >> 1] = (uint8_t)g;
              }
            }
          }
        }
        n_cells += (unsigned)(hi - lo + 1);
        sync();
        if (lds32(bc + 4) == (uint32_t)s) s_end = s;
      }
      n_steps += (uint32_t)s + (st == kPairOk ? 1u : 0u);
      if (st == kPairOk) {
        if (gt == 0) a.score[pair] = s_end * a.g;
        if constexpr (kCigar) {
          if (wig == 0) {
            const int64_t room = 2 * (int64_t)(s_end / a.pen.min_pen()) + 4;
            unsigned long long at = 0;
            if (lane == 0) at = atomicAdd(a.arena_cursor, (unsigned long long)room);
            at = __shfl_sync(FULL, at, 0);
            int len = 0;
            if ((int64_t)at + room > a.arena_cap) {
              st = kPairArena;
            } else {
              __syncwarp();
              len = packed_cigar<kModel>(
                  hist, hbase, table, s_end, k_end, m, n, a.pen, kbase, 0, 0,
                  [&](int v, int h, int rem) { return wide_warp_lcp(q, v, h, rem, lane); }, a.arena + at, (int)room, lane);
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
      const unsigned we = __reduce_add_sync(FULL, n_ext);
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
    sync();  // the block's ring and flags are free for the next pair
  }
}

// probe_packed (tsu_packed.cuh) for pairs of any length: the same window of
// kProbeW diagonals, 32-bit cells in shared memory, sequences through L1.
template <int kModel, bool kDeep = true>
__device__ __forceinline__ void probe_wide(const ProbeArgs& a, unsigned char* smem_raw) {
  constexpr unsigned FULL = 0xffffffffu;
  constexpr int W = kProbeW, U = W / 32;
  constexpr int RB = wide_row_bytes(W, 4);
  const int lane = threadIdx.x & 31;
  const int rows = a.pen.slots() + 1;
  unsigned char* const mine = smem_raw + (size_t)(threadIdx.x >> 5) * wide_probe_smem_bytes(a.pen);
  const smem_t tables = smem_addr(mine);
  unsigned char* const ring = mine + 16 * (a.pen.rm + a.pen.re + a.pen.re2);
  unsigned char* const ring0 = ring + 16;
  packed_tables<kModel == kModelDual>(a.pen, RB, tables, lane, 32);
  for (;;) {
    unsigned qi = 0;
    if (lane == 0) qi = atomicAdd(a.queue, 1u);
    qi = __shfl_sync(FULL, qi, 0);
    if ((int64_t)qi >= a.n_order) break;
    const int64_t pair = a.order[qi];
    const int m = a.seq.pat_len[pair], n = a.seq.txt_len[pair], k_end = n - m;
    const bool bytemode = a.pk.nonacgt[pair] | a.pk.nonacgt[a.seq.n + pair];
    int found = kNoBound;
    if (!bytemode) {
      WidePair q{reinterpret_cast<const uint32_t*>(a.pk.words + a.pk.woff[pair]),
                 reinterpret_cast<const uint32_t*>(a.pk.words + a.pk.woff[a.seq.n + pair]), m, n, -W / 2};
      for (int i = lane; i < rows * RB / 4; i += 32) reinterpret_cast<uint32_t*>(ring)[i] = 0u;
      __syncwarp();
      {
        const int l = wide_warp_lcp(q, 0, 0, min(m, n), lane);
        if (lane == 0) wide_row<uint32_t>(ring0, 0)[-q.kbase] = (uint32_t)l + 1u;
        if (l >= n && k_end == 0) found = 0;
        __syncwarp();
      }
      const int64_t sb = score_bound(m, n, a.pen);
      const int s_max = (int)(sb < INT_MAX - 1 ? sb : INT_MAX - 1);
      PackedSteps<kModel, kDeep> steps;
      steps.begin(a.pen, tables, (rows - 1) * RB);
      PackedRows r{};
      for (int s = 1; s <= s_max && found == kNoBound; ++s) {
        steps.next(a.pen, s, &r);
        if (!steps.present(a.pen, &r)) continue;
        const int g = steps.gained();
        const int lo = max(max(-g, -m), q.kbase), hi = min(min(g, n), q.kbase + W - 1);
        if (lo > hi) break;  // the window left the wavefronts
        const int wlo = lo - q.kbase, whi = hi - q.kbase;
        int w[U];
        uint32_t m1[U], f[U], ext[U];
#pragma unroll
        for (int u = 0; u < U; ++u) w[u] = min(wlo + 32 * u + lane, whi);
        wide_cells<kModel, uint32_t, U, false>(ring0, r, q, w, m1, f, ext);
        __syncwarp();
        const int pend = k_end - q.kbase;
        if (pend >= wlo && pend <= whi && wide_row<uint32_t>(ring0, r.w_m)[pend] >= (uint32_t)n + 1u) found = s;
        if ((s & 15) == 0) {
          // the furthest anti-diagonal 2 h - k, and then its position
          int far = INT_MIN;
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (m1[u]) far = max(far, 2 * ((int)m1[u] - 1) - (q.kbase + w[u]));
          const int best = __reduce_max_sync(FULL, far);
          int at = -1;
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (m1[u] && 2 * ((int)m1[u] - 1) - (q.kbase + w[u]) == best) at = max(at, w[u]);
          at = __reduce_max_sync(FULL, at);
          const int off = at - W / 2;
          if (at >= 0 && (off > W / 4 || off < -W / 4)) {
            for (int row = 0; row < rows - 1; ++row) {
              uint32_t* const c = wide_row<uint32_t>(ring0, row * RB);
              uint32_t v[U];
#pragma unroll
              for (int u = 0; u < U; ++u) {
                const int from = lane + 32 * u + off;
                v[u] = from >= 0 && from < W ? c[from] : 0u;
              }
              __syncwarp();
#pragma unroll
              for (int u = 0; u < U; ++u) c[lane + 32 * u] = v[u];
            }
            __syncwarp();
            q.kbase += off;
          }
        }
      }
    }
    if (lane == 0) a.bound[pair] = found;
    __syncwarp();
  }
}

}  // namespace tsu
