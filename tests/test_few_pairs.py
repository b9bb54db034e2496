"""No more pairs than SMs: the first launch takes the widest shared ring, and
the pairs that outgrow it run again with a bound (few_start, bound_limits in
tsu_plan.h)."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("kw, lens, rates", [
    ({"gap_opening2": 24, "gap_extension2": 1}, (900, 1092, 1093, 1500, 2900, 5000), (0.01, 0.2, 0.12, 0.25, 0.1, 0.06)),
    ({}, (8000, 8208, 8209, 9000, 12000, 16351, 16352, 16383, 16384), (0.02, 0.2, 0.2, 0.25, 0.01, 0.02, 0.02, 0.03, 0.02)),
    ({"metric": "edit"}, (8192, 16383, 16384), (0.05, 0.05, 0.05)),
])
def test_few_long_pairs(oracle, kw, lens, rates):
    """Sides around the lines of the rule: the ones from which outgrown pairs
    get a bound, the reach of the plain packed offsets and of the shared ring;
    pairs that fit the ring and pairs that outgrow it; a pair of unequal
    sides.  Whole numbers: equal to the oracle."""
    import tsunami_pact_b200 as T

    pbuf, poff, plen, tbuf, toff, tlen = T.gen_batch(3, np.array(lens, np.int32), np.array(rates))
    pats = [bytes(pbuf[poff[i]:poff[i] + plen[i]]) for i in range(len(lens))]
    txts = [bytes(tbuf[toff[i]:toff[i] + tlen[i]]) for i in range(len(lens))]
    txts[0] = txts[0][: lens[0] // 2]
    run = {"metric": oracle.align_batch_linear, "gap_opening2": oracle.align_batch2}.get(next(iter(kw), ""), oracle.align_batch)
    osc, oops = run(pats, txts, *((1, 1) if "metric" in kw else ()))
    with T.Aligner(4, 6, 2, **kw) if "metric" not in kw else T.Aligner(**kw) as al:
        for sl in [slice(0, None)] + [slice(i, i + 1) for i in range(len(lens))]:
            scores, ops = al.align(pats[sl], txts[sl])
            assert list(scores) == list(osc[sl]) and ops == oops[sl]
        assert list(al.align(pats, txts, cigar=False)[0]) == list(osc)
