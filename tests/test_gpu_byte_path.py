"""Pairs with bytes outside ACGT: the byte path of the global ring on every
number of warps and in every penalty model, and the default path of a batch of
two-piece pairs, call after call."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
DUAL = (4, 6, 2, 24, 1)


def _with_ns(seed, n, lo, hi, every=1):
    """n pairs of lo..hi bp at 1 - 12 %; every `every`-th has one to three Ns."""
    import tsunami_pact_b200 as T

    rng = np.random.default_rng(seed)
    lens = rng.integers(lo, hi + 1, n).astype(np.int32)
    pbuf, poff, plen, tbuf, toff, tlen = T.gen_batch(seed, lens, rng.uniform(0.01, 0.12, n))
    pats = [bytes(pbuf[poff[i]:poff[i] + plen[i]]) for i in range(n)]
    txts = [bytes(tbuf[toff[i]:toff[i] + tlen[i]]) for i in range(n)]
    for i in range(0, n, every):
        for where in rng.integers(0, len(pats[i]) - 1, 1 + i % 3):
            pats[i] = pats[i][:where] + b"N" + pats[i][where + 1:]
    return pats, txts


def _tails(seed):
    """Pairs whose last edit lies 0 - 24 bases before their ends, with an N in
    front of it, behind it, or at both sequences' last base."""
    rng = np.random.default_rng(seed)
    pats, txts = [], []
    for back in range(25):
        for kind in range(3):
            for n_at in ("front", "tail", "end"):
                p = bytes(b"ACGT"[c] for c in rng.integers(0, 4, 40 + 7 * kind + back))
                at = len(p) - back - 1
                other = b"ACGT"[(b"ACGT".index(p[at]) + 1) % 4:][:1]
                t = [p[:at] + other + p[at + 1:], p[:at] + p[at + 1:], p[:at] + other + p[at:]][kind]
                if n_at == "end":
                    p, t = p[:-1] + b"N", t[:-1] + b"N"
                else:
                    q = 3 if n_at == "front" else at + back // 2
                    p = p[:q] + b"N" + p[q + 1:]
                pats.append(p)
                txts.append(t)
    return pats, txts


@pytest.mark.parametrize("gw", [1, 2, 4, 8, 16, 32])
@pytest.mark.parametrize("model", ["affine", "dual", "linear", "affine low memory", "dual low memory"])
def test_windows_at_the_ends(oracle, model, gw):
    """Every length of the last window of a match run."""
    import tsunami_pact_b200 as T

    pats, txts = _tails(3)
    kw = {"gap_opening2": 24, "gap_extension2": 1} if "dual" in model else {"metric": "edit"} if model == "linear" else {}
    osc, oops = (oracle.align_batch2(pats, txts, *DUAL) if "dual" in model
                 else oracle.align_batch_linear(pats, txts, 1, 1) if model == "linear"
                 else oracle.align_batch(pats, txts, 4, 6, 2))
    L = T.lib()
    L.tsu_set_band_start.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_int]
    with T.Aligner(**kw) if model == "linear" else T.Aligner(4, 6, 2, **kw) as al:
        if "low" in model:
            al.set_low_memory(20)
        assert L.tsu_set_band_start(al._h, 0, 1, gw) == 0
        for call in range(3):
            scores, ops = al.align(pats, txts)
            assert list(scores) == list(osc) and ops == oops, call
        assert f"g{gw}x" in al.pass_log()
        assert list(al.align(pats, txts, cigar=False)[0]) == list(osc)


@pytest.mark.parametrize("gw", [1, 2, 4, 8, 16, 32])
def test_global_rung(oracle, gw):
    """Pairs that start on the global ring with gw warps: the same, right
    results each time (the pass log names the rung)."""
    import tsunami_pact_b200 as T

    pats, txts = _with_ns(11, 40, 1500, 2500)
    osc, oops = oracle.align_batch2(pats, txts, *DUAL)
    L = T.lib()
    L.tsu_set_band_start.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_int]
    with T.Aligner(4, 6, 2, gap_opening2=24, gap_extension2=1) as al:
        for band in range(6):
            assert L.tsu_set_band_start(al._h, band, 1, gw) == 0
        for call in range(25):
            scores, ops = al.align(pats, txts)
            assert list(scores) == list(osc) and ops == oops, call
            assert f"g{gw}x" in al.pass_log()


def test_default_path(oracle):
    """Many reads of 1 - 4 kbp, every other one with Ns, as a caller without
    settings has them aligned; with their CIGARs and scored only."""
    import tsunami_pact_b200 as T

    pats, txts = _with_ns(12, 400, 1000, 4000, every=2)
    osc, oops = oracle.align_batch2(pats, txts, *DUAL)
    with T.Aligner(4, 6, 2, gap_opening2=24, gap_extension2=1) as al:
        for call in range(12):
            scores, ops = al.align(pats, txts)
            assert list(scores) == list(osc) and ops == oops, call
        assert list(al.align(pats, txts, cigar=False)[0]) == list(osc)
        one = [al.align(pats[:1], txts[:1]) for _ in range(60)]
        assert all(int(s[0]) == osc[0] and o == oops[:1] for s, o in one)
