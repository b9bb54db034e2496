"""Batches of reads with bytes outside ACGT, more of them than SMs: no probe and
no second start on a ring that hands them back, beside pairs that do need one;
scores and CIGARs are the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pairs(seed, lens, rates, n_every):
    import tsunami_pact_b200 as T

    b = T.gen_batch(seed, np.asarray(lens, np.int32), np.asarray(rates))
    pats = [bytes(b[0][b[1][i]:b[1][i] + b[2][i]]) for i in range(len(lens))]
    txts = [bytes(b[3][b[4][i]:b[4][i] + b[5][i]]) for i in range(len(lens))]
    for i in range(0, len(lens), n_every):
        q = len(pats[i]) // 3
        pats[i] = pats[i][:q] + b"N" + pats[i][q + 1:]
    return pats, txts


def _run(oracle, pats, txts):
    import tsunami_pact_b200 as T

    osc, oops = oracle.align_batch(pats, txts, 4, 6, 2)
    with T.Aligner(4, 6, 2) as al:
        scores, ops = al.align(pats, txts)
        assert list(scores) == list(osc) and ops == oops
        log, timing = al.pass_log(), al.timing()
        assert list(al.align(pats, txts, cigar=False)[0]) == list(osc)
    return [p.split("@")[0] for p in log.split()], timing


def test_short_reads_with_ns(oracle):
    """400 reads of 150 bp, all with an N: their first pass, and the global
    ring."""
    log, timing = _run(oracle, *_pairs(21, [150] * 400, [0.02] * 400, 1))
    assert len(log) == 2 and log[0].startswith("s") and log[1].startswith("g16x") and log[1].endswith(":400"), log
    assert timing["retried_pairs"] == 400


def test_beside_pairs_that_outgrow_their_ring(oracle):
    """1 kbp at 1 % and at 15 % (which outgrow one warp's ring and run again
    with bounds), a third of all with an N."""
    rates = np.where(np.arange(900) % 2 == 0, 0.01, 0.15)
    log, timing = _run(oracle, *_pairs(22, [1000] * 900, rates, 3))
    assert log[-1].startswith("g16x") and log[-1].endswith(":300"), log
    # the first pass, the bounded ones, the global one; every retried pair once
    assert sum(int(p.split(":")[1]) for p in log) - 900 == timing["retried_pairs"], (log, timing["retried_pairs"])


def test_probed_reads_with_ns(oracle):
    """200 of 500 pairs of 2 kbp, probed at once, with an N: one plain pass,
    then the ladder, and no bound for them in between."""
    log, timing = _run(oracle, *_pairs(23, [2000] * 500, [0.03] * 500, 2))
    assert sum(p.endswith(":250") for p in log) >= 2, log
    assert log.count(log[0]) == 1 and timing["retried_pairs"] == sum(
        int(p.split(":")[1]) for p in log) - 500, (log, timing["retried_pairs"])
