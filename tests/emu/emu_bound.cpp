// emu_bound.cpp -- the bound probe, then the shared-ring align kernel planned
// from its bounds, through the CPU warp emulator (test infrastructure;
// compiled by tests/test_bound_probe.py with AddressSanitizer).
//
// Input (stdin):  x o e o2 e2 cigar gw loose wide N, then N records "m n\n<pattern>\n<text>\n"
//   (o2 < 0: one gap piece; o < 0: gap-linear); loose: added to each bound;
//   wide: 0, or the wide probe and kernel with ring cells of 2 or 4 bytes
// Output: per pair "bound<TAB>score<TAB>ops" (score -1: no bound, not aligned).
#include "warp_emu.h"
// clang-format off
#include "../../tsunami_pact_b200/csrc/tsu_kernels.cuh"
#include "../../tsunami_pact_b200/csrc/tsu_plan.h"
// clang-format on

#include <cstdio>
#include <iostream>
#include <string>

template <class T>
static T* block(size_t n) {  // exact-size zeroed heap block
  T* p = static_cast<T*>(std::malloc(sizeof(T) * (n ? n : 1)));
  std::memset((void*)p, 0, sizeof(T) * (n ? n : 1));
  return p;
}

template <int kM, bool kCigar>
static void align(int gw, int threads, size_t smem, const tsu::AlignArgs& a) {
  switch (gw) {
    case 1: emu::launch(1, threads, smem, [&] { tsu::align_kernel<kCigar, tsu::kModeShared, 1, kM | tsu::kBoundFlag>(a); }); break;
    default: emu::launch(1, threads, smem, [&] { tsu::align_kernel<kCigar, tsu::kModeShared, 4, kM | tsu::kBoundFlag>(a); }); break;
  }
}

template <int kM>
static void align_wide(bool cigar, int cell, size_t smem, const tsu::AlignArgs& a) {
  if (cell == 2)
    emu::launch(1, 512, smem, [&] { cigar ? tsu::wide_kernel<true, kM, uint16_t>(a) : tsu::wide_kernel<false, kM, uint16_t>(a); });
  else
    emu::launch(1, 512, smem, [&] { cigar ? tsu::wide_kernel<true, kM, uint32_t>(a) : tsu::wide_kernel<false, kM, uint32_t>(a); });
}

int main() {
  int X, O, E, O2, E2, cigar, gw, loose, wide;
  int64_t N;
  if (!(std::cin >> X >> O >> E >> O2 >> E2 >> cigar >> gw >> loose >> wide >> N)) return 2;
  std::vector<std::string> pats(N), txts(N);
  for (int64_t i = 0; i < N; ++i) {
    int m, n;
    std::cin >> m >> n;
    std::cin.get();
    pats[i].resize(m);
    std::cin.read(&pats[i][0], m);
    std::cin.get();
    txts[i].resize(n);
    std::cin.read(&txts[i][0], n);
    std::cin.get();
  }
  int g = 1;
  const tsu::Pen rp = O < 0 ? tsu::reduce_linear(X, E, &g) : tsu::reduce_penalties(X, O, E, O2, E2, &g);
  int64_t ptot = 0, ttot = 0, words = 0;
  for (int64_t i = 0; i < N; ++i) {
    ptot += pats[i].size(), ttot += txts[i].size();
    words += tsu::packed_words(pats[i].size()) + tsu::packed_words(txts[i].size());
  }
  uint8_t *pb = block<uint8_t>(ptot), *tb = block<uint8_t>(ttot);
  int64_t *po = block<int64_t>(N), *to = block<int64_t>(N), *woff = block<int64_t>(2 * N);
  int32_t *pl = block<int32_t>(N), *tl = block<int32_t>(N), *order = block<int32_t>(N);
  int64_t pa = 0, ta = 0, w = 0;
  int seq_cap = 0;
  for (int64_t i = 0; i < N; ++i) {
    po[i] = pa, to[i] = ta, pl[i] = pats[i].size(), tl[i] = txts[i].size(), order[i] = (int32_t)(N - 1 - i);
    std::memcpy(pb + pa, pats[i].data(), pl[i]);
    std::memcpy(tb + ta, txts[i].data(), tl[i]);
    pa += pl[i], ta += tl[i];
  }
  for (int64_t j = 0; j < 2 * N; ++j) {
    woff[j] = w;
    w += tsu::packed_words(j < N ? pl[j] : tl[j - N]);
  }
  for (int64_t i = 0; i < N; ++i)
    seq_cap = std::max<int>(seq_cap, 2 * tsu::packed_words(pl[i]) + 2 * tsu::packed_words(tl[i]));
  tsu::SeqView sv{N, pb, po, pl, tb, to, tl};
  tsu::PackView pk{block<uint64_t>(words), woff, block<uint8_t>(2 * N)};
  emu::launch(1, 64, 0, [&] { tsu::pack_kernel(sv, pk); });

  unsigned* queue = block<unsigned>(2);
  int32_t* bound = block<int32_t>(N);
  for (int64_t i = 0; i < N; ++i) bound[i] = tsu::kNoBound;
  tsu::ProbeArgs b{sv, pk, order, N, rp, seq_cap, bound, queue};
  const int threads = 64;
  const size_t psmem = 2 * (size_t)(wide ? tsu::wide_probe_smem_bytes(rp) : tsu::probe_smem_bytes(rp, seq_cap));
  emu::launch(1, threads, psmem, [&] {
    if (wide && rp.linear())
      tsu::wide_probe_kernel<tsu::kModelLinear>(b);
    else if (wide && rp.dual())
      tsu::wide_probe_kernel<tsu::kModelDual>(b);
    else if (wide)
      tsu::wide_probe_kernel<tsu::kModelAffine>(b);
    else if (rp.linear())
      tsu::probe_kernel<tsu::kModelLinear>(b);
    else if (rp.dual())
      tsu::probe_kernel<tsu::kModelDual>(b);
    else
      tsu::probe_kernel<tsu::kModelAffine>(b);
  });
  std::vector<int32_t> found(bound, bound + N), todo;
  int bytes = 0, width = 0;
  int32_t ub = 0;
  int64_t hist = 0, runs = 0;
  for (int64_t i = 0; i < N; ++i) {
    if (bound[i] == tsu::kNoBound) continue;
    bound[i] += loose;
    const tsu::BoundNeed need = tsu::bound_need(rp, pl[i], tl[i], bound[i]);
    width = std::max(width, need.width);
    bytes = std::max(bytes, tsu::bounded_bytes(rp, need.width, need.words, gw)), ub = std::max(ub, bound[i]), hist = std::max(hist, need.hist);
    runs += 2 * (int64_t)bound[i] / rp.min_pen() + 4;
    todo.push_back((int32_t)i);
  }
  tsu::PassGeom geo = wide ? tsu::plan_wide(rp, wide == 2 ? 0 : tsu::kWide16MaxLen + 1, width, ub, hist, cigar != 0)
                           : tsu::plan_bounded(bytes, ub, hist, gw, cigar != 0);
  const int groups = geo.groups_per_cta;
  int32_t *score = block<int32_t>(N), *status = block<int32_t>(N), *clen = block<int32_t>(N), *retry = block<int32_t>(N);
  int64_t* cpos = block<int64_t>(N);
  unsigned long long* cnt = block<unsigned long long>(4);
  std::memcpy(order, todo.data(), 4 * todo.size());
  queue[0] = queue[1] = 0;
  tsu::AlignArgs a{};
  a.seq = sv, a.pk = pk, a.order = order, a.n_order = (int64_t)todo.size(), a.pen = rp, a.g = g;
  a.group_bytes = geo.group_smem;
  a.hist = block<uint32_t>(cigar ? groups * geo.hist_cap : 0), a.hist_cap = geo.hist_cap;
  a.table = block<int2>(cigar ? groups * geo.table_cap : 0), a.table_cap = geo.table_cap;
  a.score = score, a.status = status;
  a.arena = block<uint32_t>(runs), a.arena_cursor = cnt, a.arena_cap = runs;
  a.cig_pos = cpos, a.cig_len = clen, a.queue = queue, a.retry = retry, a.retry_count = queue + 1, a.work = cnt + 1;
  a.bound = bound;
  a.wide_cell = geo.wide_cell, a.ring_global = block<int32_t>(geo.ring_ints), a.ring_stride = geo.ring_ints;
  const size_t smem = (size_t)groups * geo.group_smem;
  if (wide && rp.linear())
    align_wide<tsu::kModelLinear>(cigar, wide, smem, a);
  else if (wide && rp.dual())
    align_wide<tsu::kModelDual>(cigar, wide, smem, a);
  else if (wide)
    align_wide<tsu::kModelAffine>(cigar, wide, smem, a);
  else if (rp.linear())
    cigar ? align<tsu::kModelLinear, true>(gw, geo.cta_threads, smem, a) : align<tsu::kModelLinear, false>(gw, geo.cta_threads, smem, a);
  else if (rp.dual())
    cigar ? align<tsu::kModelDual, true>(gw, geo.cta_threads, smem, a) : align<tsu::kModelDual, false>(gw, geo.cta_threads, smem, a);
  else
    cigar ? align<tsu::kModelAffine, true>(gw, geo.cta_threads, smem, a) : align<tsu::kModelAffine, false>(gw, geo.cta_threads, smem, a);
  static const char code2c[16] = {'M', 'I', 'D', '?', '?', '?', '?', '?', 'X', '?', '?', '?', '?', '?', '?', '?'};
  for (int64_t i = 0; i < N; ++i) {
    if (found[i] == tsu::kNoBound) {
      std::printf("none\t-1\t\n");
      continue;
    }
    if (status[i] != tsu::kPairOk) {
      std::fprintf(stderr, "pair %lld status %d\n", (long long)i, status[i]);
      return 4;
    }
    std::string line = std::to_string(found[i] * g) + "\t" + std::to_string(score[i]) + "\t";
    if (cigar)
      for (int r = 0; r < clen[i]; ++r) line.append(a.arena[cpos[i] + r] >> 4, code2c[a.arena[cpos[i] + r] & 15]);
    std::printf("%s\n", line.c_str());
  }
  return 0;
}
