"""The shared-ring kernel that computes two diagonals per thread
(tsunami_pact_b200/csrc/tsu_packed.cuh) where its layout can go wrong: every
parity of n + m and of the end diagonal, wavefronts around a warp's 64
diagonals, scores without a wavefront (null steps), ring depths up to and past
its 64, sides up to and past its longest, ring windows off the matrix edge.
Scores and CIGARs equal the oracles'; on the CPU through the warp emulator, on
the GPU at sizes the emulator cannot run."""
import random

import numpy as np
import pytest

from test_kernel_emu import _b, _edited, check, check_dual, check_ends_free, check_linear, emu  # noqa: F401


def _rand(rng, n):
    return "".join(rng.choice("ACGT") for _ in range(n))


@pytest.mark.parametrize("gw", [1, 2])
def test_parities_and_word_edges(emu, oracle, gw):  # noqa: F811
    """Lengths 0-3 in every combination, then n + m and n - m of both
    parities with wavefronts of 60-70 and 124-132 diagonals."""
    rng = random.Random(5)
    pairs = [(_rand(rng, m), _rand(rng, n)) for m in range(4) for n in range(4)]
    for m in (61, 62, 63, 64):
        for n in (63, 64, 65):
            pairs.append((_rand(rng, m), _rand(rng, n)))
    check(emu, oracle, pairs, gw=gw)
    check_linear(emu, oracle, pairs, 1, 1, gw=gw)
    check_dual(emu, oracle, pairs[:20], (4, 6, 2, 24, 1), gw=gw)


@pytest.mark.parametrize("pen", [(7, 13, 5), (31, 32, 31), (60, 3, 1), (64, 1, 1), (2, 0, 1), (63, 62, 1)])
def test_null_steps_and_deep_rings(emu, oracle, pen):  # noqa: F811
    """Penalties whose low scores are mostly unreachable, and rings of up to
    64 scores and just past it (the latter run on the global ring)."""
    rng = random.Random(sum(pen))
    pairs = [_edited(rng, rng.randint(0, 40), 0.1) for _ in range(6)] + [("", "ACGTA"), ("ACGTA", ""), ("A", "T")]
    check(emu, oracle, pairs, pen)


def test_longest_sides(emu, oracle):  # noqa: F811
    """Sides of 16,351 (the longest) and 16,352 bases (handed back), with runs of matches over many 512-base comparisons."""
    rng = random.Random(8)
    pairs = []
    for n in (16351, 16352):
        p = _rand(rng, n)
        t = list(p)
        t[5] = "ACGT"[("ACGT".index(t[5]) + 1) % 4]
        t[n - 1] = "ACGT"[("ACGT".index(t[n - 1]) + 1) % 4]
        pairs += [(p, "".join(t)), (p[1:], p)]
    check(emu, oracle, pairs)


@pytest.mark.parametrize("free", [(0, 0, 150, 150), (150, 150, 0, 0), (1, 2, 3, 4), (90, 0, 0, 90)])
def test_free_ends_and_windows(emu, oracle, free):  # noqa: F811
    """Beginnings of many diagonals in a ring narrower than the matrix: its
    window off the middle, and at either edge of the matrix."""
    rng = random.Random(sum(free))
    pairs = []
    for _ in range(4):
        core = _rand(rng, rng.randint(250, 330))
        pairs.append((_rand(rng, 40) + core, _rand(rng, 60) + core + _rand(rng, 30)))
        pairs.append((_rand(rng, 20), _rand(rng, 380)))
        pairs.append((_rand(rng, 380), _rand(rng, 21)))
    check_ends_free(emu, oracle, pairs, free)


@pytest.mark.gpu
def test_long_wide_pairs_gpu(oracle):
    """Long divergent pairs on one wide shared ring: diagonals k with m + k
    past 16,384, both signs of n - m, single sides at the limit."""
    import tsunami_pact_b200 as T

    rng = np.random.default_rng(12)
    lens = [16352, 16351, 15000, 12001, 12000, 9000, 16353, 16383]
    pbuf, poff, plen, tbuf, toff, tlen = T.gen_batch(7, np.array(lens, np.int32), rng.uniform(0.06, 0.12, len(lens)))
    pats = [bytes(pbuf[poff[i]:poff[i] + plen[i]]) for i in range(len(lens))]
    txts = [bytes(tbuf[toff[i]:toff[i] + tlen[i]]) for i in range(len(lens))]
    txts[2], pats[3], txts[4] = txts[2][1500:], pats[3][1201:], txts[4][:11000]
    with T.Aligner(4, 6, 2) as al:
        scores, ops = al.align(pats, txts)
        only, _ = al.align(pats, txts, cigar=False)
    osc, oops = oracle.align_batch(pats, txts, 4, 6, 2)
    assert list(scores) == list(osc) and ops == oops
    assert list(only) == list(osc)
