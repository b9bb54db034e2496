"""Score bounds (the probe of tsunami_pact_b200/csrc/tsu_packed.cuh) and the
alignments they narrow: the probe's bound is never below the optimum, and with
it, or with any larger one, scores and CIGARs are the oracle's."""
import os
import random
import shutil
import subprocess

import numpy as np
import pytest

from test_kernel_emu import EMU_DIR, SRCS, _b, _edited

EXE = os.path.join(EMU_DIR, "_build", "emu_bound")


@pytest.fixture(scope="module")
def emu_bound():
    srcs = SRCS + [os.path.join(EMU_DIR, "emu_bound.cpp")]
    os.makedirs(os.path.dirname(EXE), exist_ok=True)
    if not os.path.exists(EXE) or os.path.getmtime(EXE) < max(os.path.getmtime(s) for s in srcs):
        tmp = f"{EXE}.{os.getpid()}"
        subprocess.run(["g++", "-std=c++20", "-O1", "-g", "-fsanitize=address,undefined", "-fno-omit-frame-pointer",
                        "-fno-sanitize-recover=undefined", "-o", tmp, os.path.join(EMU_DIR, "emu_bound.cpp"), "-lpthread"],
                       check=True)
        shutil.move(tmp, EXE)
    return EXE


def _run(exe, pairs, pen, cigar=True, gw=1, loose=0, wide=0):
    o2, e2 = (pen[3], pen[4]) if len(pen) == 5 else (-1, 0)
    hdr = f"{pen[0]} {pen[1]} {pen[2]} {o2} {e2} {int(cigar)} {gw} {loose} {wide} {len(pairs)}\n"
    body = b"".join(f"{len(p)} {len(t)}\n".encode() + p + b"\n" + t + b"\n" for p, t in pairs)
    env = dict(os.environ, ASAN_OPTIONS="detect_leaks=0:abort_on_error=1", UBSAN_OPTIONS="halt_on_error=1")
    r = subprocess.run([exe], input=hdr.encode() + body, capture_output=True, env=env, timeout=600)
    assert r.returncode == 0, r.stderr.decode()[-3000:]
    return [ln.split("\t") for ln in r.stdout.decode().split("\n")[: len(pairs)]]


def _align(oracle, p, t, pen):
    if pen[1] < 0:
        return oracle.align_linear(p, t, pen[0], pen[2])
    return oracle.align2(p, t, *pen) if len(pen) == 5 else oracle.align(p, t, *pen)


def _pairs(rng):
    pairs = [_edited(rng, rng.randint(100, 400), rng.choice([0.02, 0.1, 0.2])) for _ in range(5)]
    p, t = _edited(rng, 250, 0.05)
    pairs += [(p, p), ("", ""), ("A", ""), ("ACGTN", "ACGT"), (p[:200], p[:90] + p[140:]), (p[:60], p + t[:100])]
    # the path drifts past the probe's 128 diagonals, one gap after another
    q = "".join(rng.choice("ACGT") for _ in range(500))
    pairs.append((q, "".join(q[i:i + 35] + "".join(rng.choice("ACGT") for _ in range(12)) for i in range(0, 500, 35))))
    return [(_b(a), _b(b)) for a, b in pairs]


@pytest.mark.parametrize("pen", [(4, 6, 2), (5, 11, 3), (4, 6, 2, 24, 1), (1, -1, 1), (3, -1, 1)])
@pytest.mark.parametrize("gw,loose,cigar,wide", [(1, 0, True, 0), (1, 7, True, 0), (4, 0, True, 0), (1, 0, False, 0),
                                                 (16, 0, True, 2), (16, 3, True, 4)])
def test_bounded_equals_oracle(emu_bound, oracle, pen, gw, loose, cigar, wide):
    """wide: the kernels of sides beyond the 16-bit ring (tsu_wide.cuh)."""
    pairs = _pairs(random.Random(sum(pen) + gw + loose))
    if wide:
        pairs = pairs[:2] + pairs[5:]
    for (p, t), (ub, s, ops) in zip(pairs, _run(emu_bound, pairs, pen, cigar, gw, loose, wide)):
        if b"N" in p:
            assert ub == "none"
            continue
        es, eops = _align(oracle, p, t, pen)
        assert ub == "none" or (int(ub) >= es and int(s) == es and ops == (eops if cigar else "")), (p, t, pen, ub, s, es)


@pytest.mark.gpu
@pytest.mark.parametrize("low_memory", [False, True])
def test_long_pairs_gpu(oracle, low_memory):
    """Pairs past the 16-bit shared ring: 20-34 kbp, a text of more than
    65,532 bases, a band wider than a block's ring, a pair with bytes outside
    ACGT; with and without low-memory mode (whose short pairs get bounds too)."""
    import tsunami_pact_b200 as T

    rng = np.random.default_rng(8)
    lens = np.array([20464, 30000, 34000, 66000, 66000, 20400, 21000, 300, 255], np.int32)
    rates = np.array([0.02, 0.1, 0.15, 0.01, 0.004, 0.3, 0.02, 0.1, 0.1])
    pbuf, poff, plen, tbuf, toff, tlen = T.gen_batch(9, lens, rates)
    pats = [bytes(pbuf[poff[i]:poff[i] + plen[i]]) for i in range(len(lens))]
    txts = [bytes(tbuf[toff[i]:toff[i] + tlen[i]]) for i in range(len(lens))]
    pats[1], txts[4] = pats[1][700:], txts[4][: 66000 - 300]
    pats[6] = pats[6][:5000] + b"N" + pats[6][5001:]
    osc, oops = oracle.align_batch(pats, txts, 4, 6, 2)
    with T.Aligner(4, 6, 2) as al:
        if low_memory:
            al.set_low_memory(-1)
        scores, ops = al.align(pats, txts)
        assert list(scores) == list(osc) and ops == oops
        assert list(al.align(pats, txts, cigar=False)[0]) == list(osc)


@pytest.mark.gpu
@pytest.mark.parametrize("kw", [{}, {"gap_opening2": 24, "gap_extension2": 1}, {"metric": "edit"}])
def test_bounded_batches_gpu(oracle, kw):
    """Batches whose long pairs get bounds: ordinary ones, drifting and
    unrelated ones, unequal lengths, sides at the packed kernel's limit, bytes
    outside ACGT, short pairs beside them; few pairs (many warps each) and
    many."""
    import tsunami_pact_b200 as T

    rng = np.random.default_rng(31)
    lens = np.array([1300, 1400, 3000, 5000, 9000, 16500, 20463, 20464, 150, 700] + [2000] * 60, np.int32)
    rates = np.concatenate([[0.15, 0.3, 0.1, 0.08, 0.05, 0.01, 0.01, 0.01, 0.1, 0.02], rng.uniform(0.01, 0.15, 60)])
    pbuf, poff, plen, tbuf, toff, tlen = T.gen_batch(5, lens, rates)
    pats = [bytes(pbuf[poff[i]:poff[i] + plen[i]]) for i in range(len(lens))]
    txts = [bytes(tbuf[toff[i]:toff[i] + tlen[i]]) for i in range(len(lens))]
    txts[10], pats[11], txts[12] = txts[10][:1500], pats[11][400:], txts[30]
    if "gap_opening2" not in kw:
        pats[13] = pats[13][:900] + b"N" + pats[13][901:]
    txts[14] = b"".join(pats[14][i:i + 40] + txts[15][i:i + 9] for i in range(0, 2000, 40))
    run = {"metric": oracle.align_batch_linear, "gap_opening2": oracle.align_batch2}.get(next(iter(kw), ""), oracle.align_batch)
    args = (1, 1) if "metric" in kw else ()
    osc, oops = run(pats, txts, *args)
    with T.Aligner(4, 6, 2, **kw) if "metric" not in kw else T.Aligner(**kw) as al:
        for sl in (slice(0, None), slice(2, 4)):
            scores, ops = al.align(pats[sl], txts[sl])
            assert list(scores) == list(osc[sl]) and ops == oops[sl]
            assert list(al.align(pats[sl], txts[sl], cigar=False)[0]) == list(osc[sl])
