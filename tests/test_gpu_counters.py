"""The counters that tsu_timing reports, where a kernel could get them wrong."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("length", [16000, 16390, 20463, 20464, 40000])
def test_ext_bases_of_a_long_match(length):
    """One mismatch at base 5 and matches to the end: score 0 is extended
    before the counted steps, so the second M cell alone counts, with the
    length - 6 bases behind the mismatch (a run of 16,384 and more fills bit 15
    of a 16-bit half)."""
    import tsunami_pact_b200 as T

    p = b"ACGTTGCA" * (length // 8) + b"A" * (length % 8)
    t = p[:5] + b"A" + p[6:]
    assert p[5:6] != b"A"
    with T.Aligner(4, 6, 2) as al:
        scores, ops = al.align([p], [t])
        assert int(scores[0]) == 4 and ops[0].count("X") == 1
        assert al.timing()["ext_bases"] == length - 6
        al.align([p] * 200, [t] * 200)  # more pairs than SMs: bounds from the first pass on
        assert al.timing()["ext_bases"] == 200 * (length - 6)
