"""Base cases of a few bidirectional pairs: all at once where 32 MB hold them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw, length, rate, pairs, at_once", [({"metric": "edit"}, 3000, 0.15, 30, True), ({}, 3000, 0.05, 30, True),
                                                              ({}, 50000, 0.2, 1, False)])
def test_leaves_in_one_wave(oracle, kw, length, rate, pairs, at_once):
    import tsunami_pact_b200 as T

    b = T.gen_batch(7, np.full(pairs, length, np.int32), np.full(pairs, rate))
    with T.Aligner(**kw) as al:
        scores, off, runs = al.align_arrays(*b, bidirectional=True)
        groups, leaves = map(int, al.pass_log().split()[-1].split("@")[0].split("x")[1].split(":"))
        held = al.timing()["device_bytes"]
    p, t = bytes(b[0][b[1][0]:b[1][0] + b[2][0]]), bytes(b[3][b[4][0]:b[4][0] + b[5][0]])
    ops = T.runs_to_ops(runs[off[0]:off[1]])
    if "metric" in kw:
        assert scores[0] == oracle.align_linear(p, t, 1, 1)[0] == sum(c != "M" for c in ops)
    else:
        assert oracle.cigar_cost(ops, p, t, 4, 6, 2) == scores[0]
    assert (groups == leaves) == at_once, (groups, leaves)
    assert at_once or held < 40 << 20
