"""Low-memory mode and the device memory a mixed batch holds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_mixed_batch_holds_no_more_than_its_largest_part(oracle):
    """Lengths that fall into several launches: each alone, and all in one
    call.  Run one after the other the launches share one scratch buffer, so
    the call holds its largest launch's, and the inputs and runs of all (a few
    percent here)."""
    import tsunami_pact_b200 as T

    parts = [(4000, 148), (8000, 60), (12000, 30), (2000, 300)]

    def held(groups):
        lens = np.concatenate([np.full(n, length, np.int32) for length, n in groups])
        b = T.gen_batch(3, lens, np.full(len(lens), 0.2))
        with T.Aligner(4, 6, 2, mem_budget=44 << 30) as al:
            al.set_low_memory(-1)
            scores, off, runs = al.align_arrays(*b)
            return al.timing()["device_bytes"], b, scores.copy()

    alone = [held([g])[0] for g in parts]
    mixed, b, scores = held(parts)
    assert mixed <= 1.25 * max(alone), (mixed, alone)
    few = np.concatenate([np.arange(3), 148 + np.arange(2), 238 + np.arange(3)])
    pats = [bytes(b[0][b[1][i]:b[1][i] + b[2][i]]) for i in few]
    txts = [bytes(b[3][b[4][i]:b[4][i] + b[5][i]]) for i in few]
    assert list(scores[few]) == list(oracle.align_batch(pats, txts, 4, 6, 2, cigar=False)[0])
