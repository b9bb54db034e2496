"""That score bounds are found and used: the probe finds one for every pair it
can (on the CPU's warp emulation), batches of many long pairs run their bounded
launches, and the wide kernel runs on clusters of every size."""
import ctypes
import random

import numpy as np
import pytest

from test_bound_probe import _align, _pairs, _run, emu_bound  # noqa: F401


@pytest.mark.parametrize("pen", [(4, 6, 2), (5, 11, 3), (4, 6, 2, 24, 1), (1, -1, 1), (3, -1, 1), (5, 60, 4), (70, -1, 1)])
@pytest.mark.parametrize("wide", [0, 2])
def test_probe_finds_every_bound(emu_bound, oracle, pen, wide):  # noqa: F811
    """Every pair of ACGT gets a bound, the drifting one included; it is the
    optimum where 128 diagonals hold the whole search (at most 60 edits)."""
    pairs = _pairs(random.Random(sum(pen)))
    if wide:
        pairs = pairs[:2] + pairs[5:]
    for (p, t), (ub, _, _) in zip(pairs, _run(emu_bound, pairs, pen, False, 16 if wide else 1, 0, wide)):
        if b"N" in p:
            assert ub == "none"
            continue
        assert ub != "none", (p, t, pen)
        best = _align(oracle, p, t, pen)[0]
        edits = oracle.align_linear(p, t, 1, 1)[0]
        assert int(ub) >= best and (edits > 60 or int(ub) == best), (p, t, pen, ub, best)


def _batch(seed, lens, rates):
    import tsunami_pact_b200 as T

    b = T.gen_batch(seed, np.asarray(lens, np.int32), np.asarray(rates))
    return ([bytes(b[0][b[1][i]:b[1][i] + b[2][i]]) for i in range(len(lens))],
            [bytes(b[3][b[4][i]:b[4][i] + b[5][i]]) for i in range(len(lens))])


@pytest.mark.gpu
@pytest.mark.parametrize("kw, lo, hi", [({}, 1300, 3000), ({"gap_opening2": 24, "gap_extension2": 1}, 1000, 2500),
                                        ({"metric": "edit"}, 4900, 6000)])
def test_many_bounded_pairs_gpu(oracle, kw, lo, hi):
    """300 ordinary pairs past the line from which pairs get a bound, ten of
    8 - 16 kbp, drifting, unrelated and unequal ones: the oracle's results, from
    several launches, with fewer cells than the same pairs computed without
    bounds (bands set to the shared ring)."""
    import tsunami_pact_b200 as T

    rng = np.random.default_rng(17)
    lens = np.concatenate([rng.integers(lo, hi, 300), rng.integers(8000, 16300, 10)])
    pats, txts = _batch(6, lens, np.concatenate([rng.uniform(0.02, 0.12, 300), rng.uniform(0.02, 0.06, 10)]))
    txts[3], txts[4], pats[5] = txts[7], txts[4][: len(txts[4]) // 2], pats[5][300:]
    txts[6] = b"".join(pats[6][i:i + 40] + txts[8][i:i + 9] for i in range(0, len(pats[6]), 40))
    run = {"metric": oracle.align_batch_linear, "gap_opening2": oracle.align_batch2}.get(next(iter(kw), ""), oracle.align_batch)
    osc, oops = run(pats, txts, *((1, 1) if "metric" in kw else ()))
    L = T.lib()
    L.tsu_set_band_start.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_int]
    with T.Aligner(4, 6, 2, **kw) if "metric" not in kw else T.Aligner(**kw) as al:
        scores, ops = al.align(pats, txts)
        assert list(scores) == list(osc) and ops == oops
        log, cells = [p.split("x")[0] for p in al.pass_log().split()], al.timing()["cells"]
        assert list(al.align(pats, txts, cigar=False)[0]) == list(osc)
        for band in range(6):
            assert L.tsu_set_band_start(al._h, band, 0, 16) == 0
        scores, ops = al.align(pats, txts)
        assert list(scores) == list(osc) and ops == oops
        assert len(set(log)) >= 2 and cells < 0.9 * al.timing()["cells"], (log, cells, al.timing()["cells"])


@pytest.mark.gpu
@pytest.mark.parametrize("length, rate", [(20464, 0.01), (65533, 0.002)])
@pytest.mark.parametrize("pairs", [16, 17, 33, 65])
def test_cluster_sizes_gpu(oracle, pairs, length, rate):
    """8, 4 and 2 blocks per pair and one, with ring cells of 16 bits and (texts
    of more than 65,532 bases) 32."""
    import tsunami_pact_b200 as T

    pats, txts = _batch(9, [length] * pairs, [rate] * pairs)
    txts = [t + b"ACGT" * 20 if length > 65532 else t for t in txts]
    osc, oops = oracle.align_batch(pats, txts, 4, 6, 2)
    with T.Aligner(4, 6, 2) as al:
        scores, ops = al.align(pats, txts)
        assert list(scores) == list(osc) and ops == oops
        assert al.pass_log().startswith(f"g16x{pairs}:{pairs}@"), al.pass_log()
        assert list(al.align(pats, txts, cigar=False)[0]) == list(osc)
