"""Deep rings and long sides on the shared ring: penalties whose ring holds 65 -
128 scores (the two-diagonal kernel's second word of its record) and more (the
kernel of one diagonal per thread), and sides past the two-diagonal kernel's
offsets.  Where such pairs start (tsu_plan.h), on the CPU; their results on the
CPU's warp emulation and on the GPU."""
import ctypes
import os
import random
import subprocess

import numpy as np
import pytest

from test_kernel_emu import EMU_DIR, _edited, check, check_dual, emu  # noqa: F401

PLAN = r"""
#include "warp_emu.h"
#include "../../tsunami_pact_b200/csrc/tsu_plan.h"
#include <cstdio>
#include <cstdlib>
using namespace tsu;
// x o e o2 e2 mode gw m n cigar -> mode gw ring_w single (the pass), then the next rung's mode gw single
int main(int, char** v) {
  auto a = [&](int i) { return std::atoi(v[i]); };
  int g = 1;
  const Pen p = reduce_penalties(a(1), a(2), a(3), a(4), a(5), &g);
  const int side = a(8) > a(9) ? a(8) : a(9);
  const PassChoice table[kBands] = {{a(6), a(7)}, {a(6), a(7)}, {a(6), a(7)}, {a(6), a(7)}, {a(6), a(7)}, {a(6), a(7)}};
  const PassChoice c = band_start_in(table, length_band(side), side);
  const PassGeom q = plan_geometry(p, a(8), a(9), c.mode, c.gw, 0.1, a(10) != 0, 232448);
  const PassChoice n = next_pass(c, p, a(8), a(9), 232448);
  std::printf("%d %d %d %d %d %d %d\n", q.mode, q.gw, q.ring_w, q.single ? 1 : 0, n.mode, n.gw, n.single ? 1 : 0);
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    src = d / "plan.cpp"
    src.write_text(PLAN.replace('"warp_emu.h"', f'"{EMU_DIR}/warp_emu.h"').replace('"../..', f'"{EMU_DIR}/../..'))
    exe = str(d / "plan")
    subprocess.run(["g++", "-std=c++20", "-O1", "-o", exe, str(src), "-lpthread"], check=True)

    def run(pen, mode, gw, m, n, cigar=1):
        o2, e2 = (pen[3], pen[4]) if len(pen) == 5 else (-1, 0)
        r = subprocess.run([exe] + [str(x) for x in (*pen[:3], o2, e2, mode, gw, m, n, cigar)], capture_output=True, check=True)
        return [int(x) for x in r.stdout.split()]

    return run


def test_where_they_start(plan):
    """mode 0 is the shared ring.  Ring widths: 384 diagonals on one warp where
    four such rings fit a block (232,448 bytes), else what one block holds; on
    more warps the SM's 228 KB over the blocks the kernel is compiled for."""
    # rm 65, re 5 (5/60/4) and rm 72, re 2 (4/70/1): one warp
    for pen in ((5, 60, 4), (4, 70, 1)):
        for cigar in (0, 1):
            mode, gw, width, single = plan(pen, 0, 1, 1000, 1000, cigar)[:4]
            assert (mode, gw, single) == (0, 1, 0) and 336 <= width <= 384, (pen, width)
    # rm 83: 8 warps; rm 129 (4/119/9): the last two-diagonal one is 128 deep
    for pen, gw, want in (((19, 39, 3, 81, 1), 8, [0, 8, 0]), ((31, 32, 31), 1, [0, 1, 0]), ((4, 118, 9), 1, [0, 1, 0]),
                          ((4, 119, 9), 1, [0, 1, 1])):
        q = plan(pen, 0, gw, 1000, 1000)
        assert q[:2] + q[3:4] == want, (pen, q)
    # deeper: the shared ring with CIGARs, the global one for scores; a gap
    # extension past 63 scores likewise
    for pen in ((5, 200, 4), (4, 1, 64)):
        q = plan(pen, 0, 1, 1000, 1000)
        assert q[:2] + q[3:4] == [0, 1, 1] and plan(pen, 0, 1, 1000, 1000, 0)[0] == 1, (pen, q)
    # 4/6/2: the caller's rung for sides up to 32,000, the global ring beyond
    for side, want in ((16351, [0, 16, 0]), (16383, [0, 16, 0]), (16384, [0, 16, 1]), (32000, [0, 16, 1]),
                       (32001, [1, 16, 0])):
        q = plan((4, 6, 2), 0, 16, side, side)
        assert q[:2] + q[3:4] == want, (side, q)
    # pairs that the two-diagonal kernel hands back for their length run again
    # on the same warps; the others go on to the global ring
    assert plan((4, 6, 2), 0, 16, 16352, 16352)[4:] == [0, 16, 1]
    assert plan((4, 6, 2), 0, 16, 16351, 16351)[4:] == [1, 16, 0]
    assert plan((4, 6, 2), 0, 16, 20000, 20000)[4:] == [1, 16, 0]
    # one warp hands long pairs back whatever they are; the others of its
    # launch keep the shared ring
    assert plan((4, 6, 2), 0, 1, 20000, 20000)[:4] == [0, 1, 384, 0]


@pytest.mark.parametrize("gw", [1, 2])
def test_deep_rings_emulated(emu, oracle, gw):  # noqa: F811
    rng = random.Random(65)
    pairs = [_edited(rng, rng.randint(30, 90), 0.15) for _ in range(6)] + [("", "ACGTA"), ("ACGTN", "ACGTA")]
    for pen in ((5, 60, 4), (4, 70, 1), (4, 118, 9), (5, 200, 4), (3, 1, 70), (127, 60, 63)):
        rungs = check(emu, oracle, pairs, pen, gw=gw)[2]
        # (two warps of a block leave the widest of these rings under 64 diagonals)
        assert rungs.startswith(f"s{gw}") or (gw == 2 and pen not in ((5, 60, 4), (4, 70, 1))), (pen, rungs)
    check_dual(emu, oracle, pairs, (19, 39, 3, 81, 1), gw=gw)


@pytest.mark.gpu
@pytest.mark.parametrize("pen", [(5, 60, 4), (4, 70, 1), (4, 118, 9), (127, 60, 63), (5, 200, 4), (19, 39, 3, 81, 1),
                                 (70, -1, 1)])
def test_deep_rings_gpu(oracle, pen):
    """Defaults and every number of warps; with CIGARs the first pass is on the
    shared ring."""
    import tsunami_pact_b200 as T

    rng = np.random.default_rng(4)
    lens = rng.integers(100, 1020, 300).astype(np.int32)
    pbuf, poff, plen, tbuf, toff, tlen = T.gen_batch(4, lens, rng.uniform(0.005, 0.06, 300))
    pats = [bytes(pbuf[poff[i]:poff[i] + plen[i]]) for i in range(300)]
    txts = [bytes(tbuf[toff[i]:toff[i] + tlen[i]]) for i in range(300)]
    dual = len(pen) == 5
    linear = pen[1] < 0
    osc, oops = (oracle.align_batch_linear(pats, txts, pen[0], pen[2]) if linear
                 else (oracle.align_batch2 if dual else oracle.align_batch)(pats, txts, *pen))
    kw = {"metric": "gap_linear"} if linear else {"gap_opening2": pen[3], "gap_extension2": pen[4]} if dual else {}
    L = T.lib()
    L.tsu_set_band_start.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_int]
    with T.Aligner(pen[0], max(pen[1], 0), pen[2], **kw) as al:
        for gw in (0, 1, 2, 4, 8, 16, 32):
            if gw:
                assert L.tsu_set_band_start(al._h, 0, 0, gw) == 0
            scores, ops = al.align(pats, txts)
            assert list(scores) == list(osc) and ops == oops, gw
            assert "s" in al.pass_log(), al.pass_log()
            assert list(al.align(pats, txts, cigar=False)[0]) == list(osc), gw


@pytest.mark.gpu
def test_long_sides_gpu(oracle):
    """Accurate pairs of 16,351 - 32,001 bases with free ends: from the
    caller's 16 warps, and after being handed back by the default rung."""
    import tsunami_pact_b200 as T

    lens = np.array([16351, 16352, 16383, 16384, 24000, 32000, 32001], np.int32)
    pbuf, poff, plen, tbuf, toff, tlen = T.gen_batch(6, lens, np.full(len(lens), 0.004))
    pats = [bytes(pbuf[poff[i]:poff[i] + plen[i]])[: lens[i]] for i in range(len(lens))]
    txts = [bytes(tbuf[toff[i]:toff[i] + tlen[i]])[: lens[i]] for i in range(len(lens))]
    free = (20, 20, 20, 20)
    want = [oracle.align_ends_free(p, t, free, 4, 6, 2) for p, t in zip(pats, txts)]
    L = T.lib()
    L.tsu_set_band_start.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_int]
    with T.Aligner(4, 6, 2) as al:
        al.set_ends_free(*free)
        for i in range(len(lens)):  # the default: band 4 on the shared ring, band 5 on the global one
            scores, ops = al.align(pats[i:i + 1], txts[i:i + 1])
            assert (int(scores[0]), ops[0]) == want[i], i
            log = [p.split("x")[0] for p in al.pass_log().split()]
            assert log == [["s16"], ["s16", "s16"], ["s16", "s16"]][i] if i < 3 else log[0][0] == "g", (i, log)
        for band in (4, 5):
            assert L.tsu_set_band_start(al._h, band, 0, 16) == 0
        for i in range(len(lens)):
            scores, ops = al.align(pats[i:i + 1], txts[i:i + 1])
            assert (int(scores[0]), ops[0]) == want[i], i
            assert al.pass_log().split()[0][0] == ("s" if lens[i] <= 32000 else "g")
        scores, ops = al.align(pats, txts)
        assert [(int(s), o) for s, o in zip(scores, ops)] == want


@pytest.mark.gpu
def test_one_warp_entries_gpu(oracle):
    """Score-only entries that keep one warp per pair: short pairs beside one of
    20 kbp, and a deep ring."""
    import torch

    import tsunami_pact_b200 as T
    from test_zz_no_alloc import _call_noalloc, _device_batch, _noalloc_fn

    t = _device_batch(torch, 7, [500, 900, 20000, 700, 64, 0], [0.05, 0.02, 0.003, 0.01, 0.1, 0])
    h = [x.cpu().numpy() for x in t]
    for pen in ((4, 6, 2), (5, 60, 4)):
        osc = oracle.align_batch_arrays(*h, *pen, cigar=False)[0]
        rc, out = _call_noalloc(*_noalloc_fn(), t, pen)
        assert rc == 0 and np.array_equal(out.cpu().numpy(), osc)
        with T.Aligner(*pen) as al:
            out = torch.zeros(len(osc), dtype=torch.int32, device="cuda:0")
            al.align_device(*t, out, one_warp=True)
            assert np.array_equal(out.cpu().numpy(), osc)
            assert "s1x" in al.pass_log(), al.pass_log()
