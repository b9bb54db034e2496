"""The pack kernel with 4 to 32 lanes per sequence: every length and alignment
around a word, forward and reversed, on the CPU's warp emulation (exact-size
buffers under AddressSanitizer); large batches of short reads on the GPU."""
import subprocess

import numpy as np
import pytest

from test_kernel_emu import EMU_DIR

SRC = r"""
#include "@EMU@/warp_emu.h"
#include "@EMU@/../../tsunami_pact_b200/csrc/tsu_kernels.cuh"
#include <cstdio>
#include <string>
#include <vector>
using namespace tsu;
template <bool kRev, int kLanes>
static int check(int n, int gap) {
  std::vector<int64_t> po(n), to(n), woff(2 * n);
  std::vector<int32_t> pl(n), tl(n);
  int64_t a = 0, b = 0, words = 0;
  for (int i = 0; i < n; ++i) {
    pl[i] = i % 83, tl[i] = (i * 7) % 131;
    po[i] = a, to[i] = b;
    a += pl[i] + i % gap, b += tl[i];
  }
  for (int j = 0; j < 2 * n; ++j) woff[j] = words, words += packed_words(j < n ? pl[j] : tl[j - n]);
  std::vector<uint8_t> pat(a ? a : 1), txt(b ? b : 1), bad(2 * n);
  unsigned s = 5;
  auto base = [&] { s = s * 1664525u + 1013904223u; return "ACGT"[(s >> 20) & 3]; };
  for (auto& c : pat) c = base();
  for (auto& c : txt) c = base();
  for (int i = 0; i < n; i += 5) if (tl[i]) txt[to[i] + (i * 3) % tl[i]] = "N@[a\xc1"[i % 5];
  std::vector<uint64_t> w(words, ~0ull);
  const SeqView sv{n, pat.data(), po.data(), pl.data(), txt.data(), to.data(), tl.data()};
  const PackView pk{w.data(), woff.data(), bad.data()};
  emu::launch(1, 64, 0, [&] { pack_kernel<kRev, kLanes>(sv, pk); });
  for (int j = 0; j < 2 * n; ++j) {
    const int i = j < n ? j : j - n, len = j < n ? pl[i] : tl[i];
    const uint8_t* q = j < n ? pat.data() + po[i] : txt.data() + to[i];
    bool out = false;
    std::vector<uint64_t> want(packed_words(len), 0);
    for (int p = 0; p < len; ++p) {
      const uint8_t c = q[kRev ? len - 1 - p : p];
      out |= std::string("ACGT").find((char)c) == std::string::npos;
      want[p / 32] |= (uint64_t)((c >> 1) & 3) << (2 * (p % 32));
    }
    if (out != (bad[j] != 0)) return std::printf("flag of %d\n", j), 1;
    for (size_t k = 0; k < want.size(); ++k)
      if (w[woff[j] + k] != want[k]) return std::printf("word %zu of %d (%d bases)\n", k, j, len), 1;
  }
  return 0;
}
int main() {
  int r = 0;
  for (int n : {1, 3, 97}) {
    r |= check<false, 4>(n, 5) | check<false, 8>(n, 4) | check<false, 16>(n, 3) | check<false, 32>(n, 2);
    r |= check<true, 4>(n, 2) | check<true, 8>(n, 3) | check<true, 16>(n, 4) | check<true, 32>(n, 5);
  }
  // the rule: 148 SMs, 303,104 threads
  const int want[][3] = {{2, 100, 32}, {20000, 150, 16}, {75776, 60, 4}, {75775, 60, 8}, {200000, 2048, 4},
                         {200000, 2049, 8}, {200000, 8193, 32}};
  for (auto& q : want)
    if (pack_lanes(q[0], q[1], 148) != q[2]) r |= std::printf("lanes of %d x %d: %d\n", q[0], q[1], pack_lanes(q[0], q[1], 148));
  return r != 0;
}
"""


def test_every_group_size(tmp_path):
    src = tmp_path / "pack.cpp"
    src.write_text(SRC.replace("@EMU@", EMU_DIR))
    exe = str(tmp_path / "pack")
    subprocess.run(["g++", "-std=c++20", "-O1", "-g", "-w", "-fsanitize=address,undefined", "-fno-sanitize-recover=undefined",
                    "-o", exe, str(src), "-lpthread"], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, (r.stdout + r.stderr)[-2000:]


@pytest.mark.gpu
@pytest.mark.parametrize("pairs, longest", [(40000, 60), (20000, 300), (10000, 90), (200, 40)])
@pytest.mark.parametrize("bidirectional", [False, True])
def test_short_reads_gpu(oracle, pairs, longest, bidirectional):
    """Batches on either side of the rule's lines, a few pairs with an N."""
    import tsunami_pact_b200 as T

    rng = np.random.default_rng(pairs)
    lens = rng.integers(0, longest + 1, pairs).astype(np.int32)
    pbuf, poff, plen, tbuf, toff, tlen = T.gen_batch(pairs, lens, rng.uniform(0, 0.1, pairs))
    pbuf = pbuf.copy()
    for i in range(0, pairs, 500):
        if plen[i]:
            pbuf[poff[i] + plen[i] // 2] = ord("N")
    osc = oracle.align_batch_arrays(pbuf, poff, plen, tbuf, toff, tlen, 4, 6, 2, cigar=False)[0]
    with T.Aligner(4, 6, 2) as al:
        scores = al.align_arrays(pbuf, poff, plen, tbuf, toff, tlen, cigar=False, bidirectional=bidirectional)[0]
        assert np.array_equal(scores, osc)
