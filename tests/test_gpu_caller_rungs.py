"""tsu_set_band_start: a band whose rung the caller set starts there, for few
pairs and for pairs that would otherwise get a bound first."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SHARED = [(0, g) for g in (1, 2, 4, 8, 16, 32)]
GLOBAL = [(1, g) for g in (1, 8, 32)]


@pytest.mark.parametrize("kw", [{}, {"gap_opening2": 24, "gap_extension2": 1}, {"metric": "edit"}])
@pytest.mark.parametrize("pairs, length, rungs", [(1, 900, SHARED + GLOBAL), (30, 2500, [(0, 4), (1, 8)]),
                                                  (200, 3000, [(0, 8), (0, 16), (1, 4)]), (2, 17000, [(0, 16), (1, 16)])])
def test_first_pass_is_the_callers(oracle, kw, pairs, length, rungs):
    import tsunami_pact_b200 as T

    b = T.gen_batch(5, np.full(pairs, length, np.int32), np.full(pairs, 0.01))
    pats = [bytes(b[0][b[1][i]:b[1][i] + b[2][i]]) for i in range(pairs)]
    txts = [bytes(b[3][b[4][i]:b[4][i] + b[5][i]]) for i in range(pairs)]
    run = {"metric": oracle.align_batch_linear, "gap_opening2": oracle.align_batch2}.get(next(iter(kw), ""), oracle.align_batch)
    osc, oops = run(pats, txts, *((1, 1) if "metric" in kw else ()))
    L = T.lib()
    L.tsu_set_band_start.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_int]
    with T.Aligner(4, 6, 2, **kw) if "metric" not in kw else T.Aligner(**kw) as al:
        for mode, gw in rungs:
            for band in range(6):
                assert L.tsu_set_band_start(al._h, band, mode, gw) == 0
            scores, ops = al.align(pats, txts)
            assert list(scores) == list(osc) and ops == oops, (mode, gw)
            assert al.pass_log().startswith(f"{'sg'[mode]}{gw}x"), (mode, gw, al.pass_log())
