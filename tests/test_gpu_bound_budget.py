"""Bounds and the device budget: a call that runs without them is not refused
for the buffers that they need."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pairs, length, rate", [(60000, 100, 0.02), (3000, 1000, 0.12), (2000, 1500, 0.05)])
def test_least_budget(oracle, pairs, length, rate):
    """The least budget, to 1 %, of batches whose pairs all fit their first ring, all
    outgrow it (and run again with bounds), or are probed at once: no more than
    what one warp per pair without any of it needs at the same history, and
    results are the oracle's there."""
    import ctypes

    import tsunami_pact_b200 as T

    b = T.gen_batch(5, np.full(pairs, length, np.int32), np.full(pairs, rate))
    osc = oracle.align_batch_arrays(*b, 4, 6, 2, cigar=False)[0]
    L = T.lib()
    L.tsu_set_band_start.argtypes = [ctypes.c_void_p] + [ctypes.c_int] * 3
    L.tsu_get_band_start.argtypes = [ctypes.c_void_p, ctypes.c_int] + [ctypes.POINTER(ctypes.c_int)] * 2

    def run(mb, as_compiled):
        try:
            with T.Aligner(4, 6, 2, mem_budget=int(mb * 1e6)) as al:
                for band in range(6):
                    m, w = ctypes.c_int(), ctypes.c_int()
                    L.tsu_get_band_start(al._h, band, ctypes.byref(m), ctypes.byref(w))
                    if as_compiled:
                        assert L.tsu_set_band_start(al._h, band, m.value, w.value) == 0
                return al.align_arrays(*b)[0].copy()
        except T.AlignError:
            return None

    def least(as_compiled):
        lo, hi = 0.0, 1.0
        while run(hi, as_compiled) is None:
            lo, hi = hi, 2 * hi
        while hi - lo > 0.005 * hi:
            mid = (lo + hi) / 2
            lo, hi = (mid, hi) if run(mid, as_compiled) is None else (lo, mid)
        return hi

    own, plain = least(False), least(True)
    assert own <= 1.02 * plain, (own, plain)
    for mb in (own, 1.05 * own, 1.3 * own, 3 * own):
        assert np.array_equal(run(mb, False), osc), mb
