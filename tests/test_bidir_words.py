"""The breakpoint kernel's two-cells-per-lane form (tsunami_pact_b200/csrc/
tsu_bidir.cuh: interior words of wide wavefronts on 16-bit rings) against the
oracle: wavefronts of several warps' words, both parities of the ring's rows
(odd ones go cell by cell) and of the pattern's length."""
import random

import pytest

from test_bidir_kernel import _check, _edited, emu_bidir  # noqa: F401


def _rand(rng, n):
    return "".join(rng.choice("ACGT") for _ in range(n)).encode()


@pytest.mark.parametrize("gw", [1, 4])
@pytest.mark.parametrize("odd", [0, 1])
def test_wide_wavefronts(emu_bidir, oracle, gw, odd):  # noqa: F811
    rng = random.Random(17 + 2 * gw + odd)
    recs = [(*_edited(rng, 400, 0.3), "M", "M", None), (*_edited(rng, 333, 0.25), "I", "D", None)]
    recs.append((_rand(rng, 260), _rand(rng, 241), "M", "M", None))
    recs.append((_rand(rng, 240), _rand(rng, 261), "D", "I", None))
    big = max(len(p) + len(t) for p, t, *_ in recs)
    # the longest pair sets the ring's row length, m + n + 3 diagonals
    recs.append((b"A", b"C" * (big + 1 - (big + odd) % 2), "M", "M", None))
    _check(emu_bidir, oracle, recs, (4, 6, 2), gw)
